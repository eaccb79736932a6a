// deltaSPH right-hand side on sm_103a: one thread (or 2 / 4 lanes) per fluid particle in
// cell-sorted order, gathering over its pairs (a CSR row, or its segment list of accepted
// candidates from the cell rows) and over the wall particles of the neighboring cells.
// Every sum is a gather into registers — no atomics, deterministic order: fluid neighbors in
// cell order, then walls, added to the fluid sum the way the reference adds its wall
// module's result (`x += simulation.boundaryModule...`).
//
// Each kernel body takes its scene's grid, parameters and cell-table offset explicitly, so
// the same code serves one scene (sph_* entry points) and a batch of independent scenes
// concatenated in one particle array (sph_batch_* entry points, scene table + per-particle
// scene index).
//
// Reference formulas (relative density rho~, absolute rho = rho~ rho0, V = A / rho~):
//   continuity     src/modules/momentum.py:13-19 (+ wall solidBoundary.py:746-770)
//   MOG diffusion  src/modules/densityDiffusion.py:56-63
//   deltaSPH diff. src/modules/densityDiffusion.py:12-52 (+ wall L / grad parts,
//                  solidBoundary.py:676-717), pinv2x2 src/util.py:386-433
//   Tait EOS       src/modules/pressure.py:82-83 (wall: solidBoundary.py:802-804)
//   pressure acc.  src/modules/pressure.py:13-19 (+ wall solidBoundary.py:846-890)
//   art. viscosity src/modules/diffusion.py:12-25 (+ wall solidBoundary.py:820-844)
//   laminar visc.  src/modules/laminar.py:12-27 (index choices kept: r = x_j - x_i, mu_j = rho_i nu)
//   gravity        src/modules/gravity.py:46-57
//   mDBC density   src/modules/solidBoundary.py:561-617
#include <cstring>

#include "sph_math.cuh"

namespace sph {

// ---------------------------------------------------------------------------- mDBC
// Shepard and first-order MLS sums over the fluid particles within h of wall b's ghost, then the
// 3x3 pseudo-inverse solve, wall density, volume and Tait pressure.  One scene has few walls,
// so its launch is one wall's chain: a cell row's candidates are tested 32 at a time (all loads
// in flight), the accepted ones summed with four records in flight, and kLanes = 4 lanes take a
// row each.  Every row is summed by itself and the rows are added in order, so a wall's sums
// are the same with 1 lane, which a batch's hundreds of thousands of walls fill the GPU with.
// 1,380 walls 20 -> 10.2 us a launch, 5,976 walls 35 -> 9.3 us, the 210,000 walls of 50 served
// tanks 78 -> 34 us, most of it by the shorter solve (pinv3_solve).
struct MdbcRec {
  float2 x;
  float area, rho;
};

constexpr int kMdbcSums = 12;
constexpr int kMdbcSplitWalls = 32768;   // walls up to which a launch takes 4 lanes per wall

// s += the sums of the candidates [j0, j1) of one cell row; float sums (GB300's FP64 rate is
// low), the 3x3 solve runs in double.
__device__ __forceinline__ int mdbc_row(float2 xg, int j0, int j1, const FluidView& F, const SphParams& P,
                                        float (&s)[kMdbcSums]) {
  int cnt = 0;
  const auto use = [&](const MdbcRec& f) {
    // e = (x_g - x_j) / r from one rsqrt (zero below r = 1e-7, as the reference's e_ij)
    const float dx = xg.x - f.x.x, dy = xg.y - f.x.y;
    const float r2 = dx * dx + dy * dy;
    const float ir = r2 >= 1e-14f ? rsqrt_normal(r2) : 0.f;
    const float q = r2 * ir * P.inv_h;
    const float k = kW(q, P.c_w);
    const float gwr = kGW(q, P.c_g) * ir;
    const float ggx = gwr * dx, ggy = gwr * dy;
    const float mass = f.area * P.rho0;
    const float Vj = f.area * rcp_normal(f.rho);
    const float xx = f.x.x - xg.x, xy = f.x.y - xg.y;
    s[0] += mass * k;        // Shepard numerator and denominator
    s[1] += Vj * k;
    s[2] += mass * ggx;      // first-order MLS: gradient sums and moments
    s[3] += mass * ggy;
    s[4] += Vj * ggx;
    s[5] += Vj * ggy;
    s[6] += Vj * k * xx;
    s[7] += Vj * k * xy;
    s[8] += Vj * xx * ggx;
    s[9] += Vj * xx * ggy;
    s[10] += Vj * xy * ggx;
    s[11] += Vj * xy * ggy;
  };
  const auto load = [&](int j) { return MdbcRec{__ldg(F.x + j), __ldg(F.area + j), __ldg(F.rho + j)}; };
  for (int c = j0; c < j1; c += 32) {
    uint32_t w = c + 32 <= F.n ? segment_mask_full(F.x, c, j1, xg.x, xg.y, P.thr)
                               : segment_mask(F.x, c, j1, xg.x, xg.y, P.thr);
    cnt += __popc(w);
    while (w) {
      int j[4];
      bool ok[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        ok[t] = w != 0;
        j[t] = ok[t] ? c - 1 + __ffs(w) : c;
        w &= w - 1;   // 0 stays 0
      }
      const MdbcRec f0 = load(j[0]), f1 = load(j[1]), f2 = load(j[2]), f3 = load(j[3]);
      use(f0);
      if (ok[1]) use(f1);
      if (ok[2]) use(f2);
      if (ok[3]) use(f3);
    }
  }
  return cnt;
}

// Lane `sub` of wall b's kLanes; `live` false: a lane that only takes part in the sums.
template <int kLanes>
__device__ __forceinline__ void mdbc_body(int b, bool live, int sub, const FluidView& F, const WallView& W,
                                          const sph_grid& g, const SphParams& P, int coff) {
  const float2 xg = W.xg[b];
  float s[kMdbcSums] = {};
  int cnt = 0;
  const int32_t* cs = F.cell_start + coff;
  int x0 = 0, x1 = -1, y0 = 0, rows = 0;
  if (live && grid_ok(g, P.cell_capacity)) {
    const float fcx = ceilf(__fdiv_rn(__fsub_rn(xg.x, g.qmin[0]), g.hmax));
    const float fcy = ceilf(__fdiv_rn(__fsub_rn(xg.y, g.qmin[1]), g.hmax));
    if (fcx > -1e9f && fcx < 1e9f && fcy > -1e9f && fcy < 1e9f) {
      const int cx = (int)fcx, cy = (int)fcy, r = P.search_radius;
      x0 = max(cx - r, 0);
      x1 = min(cx + r, g.cells_x - 1);
      y0 = max(cy - r, 0);
      rows = x0 <= x1 ? max(min(cy + r, g.cells_y - 1) - y0 + 1, 0) : 0;
    }
  }
  const auto row_sums = [&](int q, float (&t)[kMdbcSums]) {
    const int32_t* row = cs + (y0 + q) * g.cells_x;
    return mdbc_row(xg, __ldg(row + x0), __ldg(row + x1 + 1), F, P, t);
  };
  if constexpr (kLanes == 1) {
    for (int q = 0; q < rows; ++q) {
      float t[kMdbcSums] = {};
      cnt += row_sums(q, t);
#pragma unroll
      for (int k = 0; k < kMdbcSums; ++k) s[k] += t[k];
    }
  } else {
    for (int q = 0; __any_sync(0xffffffffu, q < rows); q += kLanes) {
      float t[kMdbcSums] = {};
      int c = q + sub < rows ? row_sums(q + sub, t) : 0;
#pragma unroll
      for (int k = 0; k < kMdbcSums; ++k) {
        s[k] += t[k];   // lane 0: the first row; the others' come in order
#pragma unroll
        for (int l = 1; l < kLanes; ++l) {
          const float v = __shfl_sync(0xffffffffu, t[k], l, kLanes);
          if (sub == 0) s[k] += v;
        }
      }
#pragma unroll
      for (int o = 1; o < kLanes; o <<= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
      cnt += c;
    }
  }
  if (!live || sub != 0) return;
  double rho_b = 1.0;
  if (cnt > 10) {
    const float A[3][3] = {{s[1], s[6], s[7]}, {s[4], s[8], s[9]}, {s[5], s[10], s[11]}};
    const float bb[3] = {s[0], s[2], s[3]};
    double res[3];
    pinv3_solve(A, bb, res);
    const float2 xb = W.x[b];
    rho_b = (res[0] + ((double)xb.x - xg.x) * res[1] + ((double)xb.y - xg.y) * res[2]) / P.rho0;
  } else if (cnt > 0) {
    rho_b = ((double)s[0] / (double)s[1]) / P.rho0;
  }
  const float rb = (float)fmax(rho_b, 1.0);
  W.rho[b] = rb;
  W.vol[b] = W.area[b] / rb;
  W.p[b] = tait(rb, P);
}

// ---------------------------------------------------------------------------- neighbor records
// What neighbor j brings to every pair term, computed once per particle instead of once
// per pair: xv = (x, y, vx, vy) and q = (rho_j, V_j = A_j / rho~_j, p_j V_j with p_j =
// Tait(rho~_j), m_j = rho_j V_j).  Two 16-byte loads per pair replace four scalar loads, a
// division and the Tait power.
// The two float4 lie in arrays of their own, n apart (xv_of, q_of): the lanes' loads of one of
// them spread over all of the L1's 16-byte columns, where one 32-byte record per particle
// left every other column to the other half (pass 1 of a serving step of 3.1 M particles
// 322 us instead of 328, its records 111 instead of 114).
struct Rec {
  float4 xv, q;
};

__device__ __forceinline__ float4* xv_of(Rec* r) { return reinterpret_cast<float4*>(r); }
__device__ __forceinline__ const float4* xv_of(const Rec* r) { return reinterpret_cast<const float4*>(r); }
__device__ __forceinline__ float4* q_of(Rec* r, int n) { return reinterpret_cast<float4*>(r) + n; }
__device__ __forceinline__ const float4* q_of(const Rec* r, int n) { return reinterpret_cast<const float4*>(r) + n; }

__device__ __forceinline__ void prep_body(int i, const FluidView& F, const SphParams& P, Rec* __restrict__ rec) {
  const float2 x = F.x[i], v = F.v[i];
  const float rt = F.rho[i];
  const float V = F.area[i] / rt, rho = rt * P.rho0;
  xv_of(rec)[i] = make_float4(x.x, x.y, v.x, v.y);
  q_of(rec, F.n)[i] = make_float4(rho, V, tait(rt, P) * V, rho * V);
}

// Pair geometry in the form the sums need: d = x_i - x_j, r2 = |d|^2 and the Wendland
// gradient as gradW_ij = gd * d, gd = kGW(q) / r = -20 c_g (1 - q)^3 / h (zero when
// r < 1e-7, where the reference's e_ij is zero).  Every dot product with gradW then folds
// into gd: (x_j - x_i) . gradW = -gd r2, u . gradW = gd (u . d).
struct PairG {
  float dx, dy, r2, gd;
};

// kScaled = false: gd without its constant factor gk (a sum that is linear in gd takes gk
// once at the end).
template <bool kScaled = true>
__device__ __forceinline__ PairG pair_g(float xi, float yi, float xj, float yj, const SphParams& P) {
  PairG g;
  g.dx = xi - xj;
  g.dy = yi - yj;
  g.r2 = g.dx * g.dx + g.dy * g.dy;
  const bool apart = g.r2 >= 1e-14f;
  const float r = g.r2 * rsqrt_normal(g.r2);   // NaN at r2 = 0, dropped by the select
  const float a = apart ? 1.0f - r * P.inv_h : 0.f;
  g.gd = kScaled ? P.gk * (a * a * a) : a * a * a;
  return g;
}

// ---------------------------------------------------------------------------- pass 1
// dpdt (continuity + MOG), acceleration (gravity, pressure, artificial and laminar
// viscosity) and, for the deltaSPH scheme, the renormalization matrix L_i and the density
// gradient <grad rho>_i = -L_i^+ sum_j 2 (rho_j - rho_i) V_j gradW_ij (+ walls), all in one
// sweep over the row: L_i^+ is applied to the summed vector once instead of to every term.
// For the deltaSPH scheme the diffusion D_i = sum_j psi_ij . gradW_ij V_j, psi_ij =
// 2 (rho_j - rho_i) x_ji / (|x_ji|^2 + eps) - (<grad rho>_i + <grad rho>_j), is split: pass 1
// sums the parts it can, ddiff = 2 sum_j (rho_j - rho_i) (x_ji . gradW) V_j / (|x_ji|^2 + eps)
// - <grad rho>_i . sum_j V_j gradW_ij, and the diffusion pass subtracts
// sum_j (<grad rho>_j V_j) . gradW_ij, the only part that needs the neighbors' gradients.
struct WallRec {
  float2 x;
  float vol, rho, p;
};

struct Pass1 {
  float dpdt, ax, ay;
  float4 L;        // renormalization matrix, fluid + walls
  float2 grad_rho;
  float ddiff;     // deltaSPH: the pass-1 part of D_i
};

// kTpp lanes per particle (kCells only): lane `sub` sums its share of the pairs and walls, the
// lanes add their sums, and lane 0 finishes (gravity, L^+); the other lanes return a zero
// record.  `live` false: a lane past the last particle, which only takes part in the sums.
// kScheme: the density diffusion (0 none, 1 MOG, 2 deltaSPH) fixed at compile time, or -1:
// read from P.diffusion.  kByFour (kCells, one lane): four pairs' records in flight at a time,
// and the walls' bounds together; the same sums in the same order, for small launches.
template <bool kCells, int kTpp = 1, int kScheme = -1, bool kByFour = false>
__device__ __forceinline__ Pass1 pass1_body(int i, const FluidView& F, const Rec* __restrict__ rec,
                                            const WallView& W, const sph_grid& g,
                                            const SphParams& P, int coff, const Segments& S, int sub = 0,
                                            bool live = true) {
  const float4 si = xv_of(rec)[i];
  const float rhoi = q_of(rec, F.n)[i].x, pi = tait(F.rho[i], P);
  const int scheme = kScheme >= 0 ? kScheme : P.diffusion;
  const bool renorm = scheme == 2;
  const float mu8 = 4.0f * (2.0f * rhoi * P.kinematic);   // 4 (mu_i + mu_j), both rho_i nu
  float dp_f = 0.f, mog = 0.f, bx = 0.f, by = 0.f;   // b = sum_j V_j gradW_ij (deltaSPH)
  float pax = 0.f, pay = 0.f, vax = 0.f, vay = 0.f, lax = 0.f, lay = 0.f;
  float l00 = 0.f, l01 = 0.f, l11 = 0.f, gfx = 0.f, gfy = 0.f;
  const auto load = [&](int j) { return Rec{__ldg(xv_of(rec) + j), __ldg(q_of(rec, F.n) + j)}; };
  const auto fluid_pair = [&](const Rec& other) {
    const float4 sj = other.xv, qj = other.q;
    const float rhoj = qj.x, Vj = qj.y, pVj = qj.z, mj = qj.w;
    const PairG e = pair_g(si.x, si.y, sj.x, sj.y, P);   // gradW = e.gd * d
    const float ux = sj.z - si.z, uy = sj.w - si.w;       // u_j - u_i
    const float ud = ux * e.dx + uy * e.dy;               // (u_j - u_i) . d
    const float ir2 = rcp_normal(e.r2 + P.eps);
    const float rg = -e.gd * e.r2;                        // (x_j - x_i) . gradW
    const float mg = mj * e.gd;
    dp_f -= mg * ud;
    // MOG diffusion (for deltaSPH the first part of its diffusion, formed below from the
    // renormalization product): (rho_j - rho_i) V_j (x_j - x_i) . gradW / (r^2 + eps), x 2 after the sum
    if (scheme == 1) mog += (rhoj - rhoi) * ir2 * rg * Vj;
    const float pf = fmaf(pi, Vj, pVj) * e.gd;            // (p_i + p_j) V_j gd
    pax += pf * e.dx;
    pay += pf * e.dy;
    const float irs = rcp_normal(rhoi + rhoj);
    const float wg = mg * (irs * ir2);
    const float vf = fminf(-ud, 0.f) * wg;                // pi_ij, (u_j - u_i) . (x_j - x_i) = -ud
    vax += vf * e.dx;
    vay += vf * e.dy;
    const float term = e.r2 * irs * wg;                   // laminar: mu8 term (u_j - u_i), mu8 after the sum
    lax += term * ux;
    lay += term * uy;
    if (renorm) {
      // V_j (x_j - x_i) (x) gradW = -t d (x) d: symmetric, one off-diagonal sum
      const float t = Vj * e.gd;
      const float tx = t * e.dx, ty = t * e.dy;
      l00 -= tx * e.dx;
      l01 -= tx * e.dy;
      l11 -= ty * e.dy;
      bx += tx;
      by += ty;
      const float s = (rhoj - rhoi) * t;                  // x 2 after the sum
      gfx += s * e.dx;
      gfy += s * e.dy;
      mog -= s * (e.r2 * ir2);                            // (rho_j - rho_i) V_j (-gd r^2) / (r^2 + eps)
    }
  };
  if constexpr (kCells) {
    if constexpr (kByFour) {
      stored_pairs_by_four(i, F, g, coff, P.search_radius, S.nseg, S.start, S.mask, si.x, si.y, P.thr, load,
                           fluid_pair);
    } else {
      if (live) stored_pairs<kTpp>(i, F, g, coff, P.search_radius, S.nseg, S.start, S.mask, si.x, si.y, P.thr,
                                   [&](int j) { fluid_pair(load(j)); }, sub);
    }
  } else {
    static_assert(kTpp == 1, "CSR rows run one lane per particle");
    const int k0 = F.offsets[i], k1 = row_end(F, i, k0);
    for (int k = k0; k < k1; ++k) fluid_pair(load(__ldg(F.cols + k)));
  }
  if constexpr (kTpp > 1) {
    dp_f = lane_sum<kTpp>(dp_f);
    mog = lane_sum<kTpp>(mog);
    pax = lane_sum<kTpp>(pax);
    pay = lane_sum<kTpp>(pay);
    vax = lane_sum<kTpp>(vax);
    vay = lane_sum<kTpp>(vay);
    lax = lane_sum<kTpp>(lax);
    lay = lane_sum<kTpp>(lay);
    l00 = lane_sum<kTpp>(l00);
    l01 = lane_sum<kTpp>(l01);
    l11 = lane_sum<kTpp>(l11);
    gfx = lane_sum<kTpp>(gfx);
    gfy = lane_sum<kTpp>(gfy);
    bx = lane_sum<kTpp>(bx);
    by = lane_sum<kTpp>(by);
  }
  float dp_w = 0.f, pwx = 0.f, pwy = 0.f, vwx = 0.f, vwy = 0.f;
  float w00 = 0.f, w01 = 0.f, w10 = 0.f, w11 = 0.f, gwx = 0.f, gwy = 0.f;
  if (W.n > 0) {
    const float thr = P.thr;
    bool any = false;   // a wall of this lane's (kTpp > 1)
    const auto load_wall = [&](int b) { return WallRec{__ldg(W.x + b), W.vol[b], W.rho[b], W.p[b]}; };
    const auto wall_pair = [&](const WallRec& wall) {
      any = true;
      const PairG e = pair_g(si.x, si.y, wall.x.x, wall.x.y, P);   // fluid side: d = x_f - x_b
      const float Vb = wall.vol, rhob = wall.rho * P.rho0, pb = wall.p;
      const float ud = -(si.z * e.dx + si.w * e.dy);       // (u_b - u_f) . d, walls at rest
      dp_w -= e.gd * ud * Vb * rhob;
      const float pf = (pi + pb) * Vb * e.gd;
      pwx += pf * e.dx;
      pwy += pf * e.dy;
      if (P.boundary_diffusion) {
        const float vf = fminf(-ud, 0.f) * rcp_normal(e.r2 + P.eps) * Vb * rhob *
                         rcp_normal(rhoi + rhob) * e.gd;
        vwx += vf * e.dx;
        vwy += vf * e.dy;
      }
      if (renorm) {
        const float t = Vb * e.gd;
        const float tx = t * e.dx, ty = t * e.dy;
        w00 -= tx * e.dx;
        w01 -= tx * e.dy;
        w10 -= ty * e.dx;
        w11 -= ty * e.dy;
        const float s = (rhob - rhoi) * 2.0f * t;
        gwx += s * e.dx;
        gwy += s * e.dy;
      }
    };
    if (kTpp == 1 || live) {
      int cx, cy;
      cell_of(F.keys[i] - (uint32_t)coff, g, &cx, &cy);
      if constexpr (kByFour) {
        for_each_wall_by_four(W, g, P.search_radius, cx, cy, si.x, si.y, thr, load_wall, wall_pair, coff);
      } else if constexpr (kTpp == 1) {
        for_each_wall(W, g, P.search_radius, cx, cy, si.x, si.y, thr,
                      [&](int b, float2 xb) { wall_pair(WallRec{xb, W.vol[b], W.rho[b], W.p[b]}); }, coff);
      } else {
        for_each_wall_lanes<kTpp>(W, g, P.search_radius, cx, cy, si.x, si.y, thr, sub,
                                  [&](int b, float2 xb) { wall_pair(WallRec{xb, W.vol[b], W.rho[b], W.p[b]}); },
                                  coff);
      }
    }
    if constexpr (kTpp > 1) {
      if (__any_sync(0xffffffffu, any)) {
        dp_w = lane_sum<kTpp>(dp_w);
        pwx = lane_sum<kTpp>(pwx);
        pwy = lane_sum<kTpp>(pwy);
        vwx = lane_sum<kTpp>(vwx);
        vwy = lane_sum<kTpp>(vwy);
        w00 = lane_sum<kTpp>(w00);
        w01 = lane_sum<kTpp>(w01);
        w10 = lane_sum<kTpp>(w10);
        w11 = lane_sum<kTpp>(w11);
        gwx = lane_sum<kTpp>(gwx);
        gwy = lane_sum<kTpp>(gwy);
      }
    }
  }
  if (kTpp > 1 && (sub != 0 || !live)) return Pass1{};
  Pass1 o;
  o.dpdt = dp_f + dp_w;
  if (scheme == 1) o.dpdt += P.diff_k * (2.0f * mog);
  float ax, ay;
  if (P.point_source) {
    float dx = si.x - P.point_cx, dy = si.y - P.point_cy;
    float dist = sqrtf(dx * dx + dy * dy);
    if (dist > 1e-7f) {
      dx /= dist;
      dy /= dist;
    }
    ax = -P.point_mag * dx * dist;
    ay = -P.point_mag * dy * dist;
  } else {
    ax = P.gx;
    ay = P.gy;
  }
  const float ir = -1.0f / rhoi;
  ax += ir * pax + ir * pwx;
  ay += ir * pay + ir * pwy;
  ax += P.visc_k * vax + P.visc_k * vwx;
  ay += P.visc_k * vay + P.visc_k * vwy;
  o.ax = ax - mu8 * lax;
  o.ay = ay - mu8 * lay;
  o.L = make_float4(l00 + w00, l01 + w01, l01 + w10, l11 + w11);
  gfx *= 2.0f;
  gfy *= 2.0f;
  o.grad_rho = make_float2(0.f, 0.f);
  o.ddiff = 0.f;
  if (renorm) {
    const float4 Li = pinv2x2_fast(o.L.x, o.L.y, o.L.z, o.L.w);
    const float fx = Li.x * gfx + Li.y * gfy, fy = Li.z * gfx + Li.w * gfy;
    const float wx = Li.x * gwx + Li.y * gwy, wy = Li.z * gwx + Li.w * gwy;
    o.grad_rho = make_float2(-fx - wx, -fy - wy);
    o.ddiff = 2.0f * mog - (o.grad_rho.x * bx + o.grad_rho.y * by);
  }
  return o;
}

// D_i = sum_j [2 (rho_j - rho_i)/(|x_ji|^2 + eps) x_ji - (<grad rho>_i + <grad rho>_j)] . gradW_ij V_j
// (the deltaSPH density diffusion before its h delta c0 factor).
// sum_j (<grad rho>_j V_j) . gradW_ij, the part of the deltaSPH diffusion that needs the
// neighbors' gradients.  kHoldsGV: gbuf holds <grad rho> V (the batch's pass 1 stores it
// so); otherwise it holds <grad rho> and V_j comes from the neighbor record (the same
// product, so both give the same bits).  kCells: pairs from the segment lists instead of the
// CSR row.
struct DiffRec {
  float2 x, g;
  float V;
};

template <bool kCells, int kTpp = 1, bool kHoldsGV = true, bool kByFour = false>
__device__ __forceinline__ float diffusion_sum(int i, const FluidView& F, const Rec* __restrict__ rec,
                                               const SphParams& P, const float2* __restrict__ gbuf,
                                               const sph_grid& g, int coff, const Segments& S, int sub = 0,
                                               bool live = true) {
  const float2 xi = F.x[i];
  float acc = 0.f;
  const auto load = [&](int j) { return DiffRec{__ldg(F.x + j), __ldg(gbuf + j), kHoldsGV ? 0.f : __ldg(&q_of(rec, F.n)[j].y)}; };
  const auto pair = [&](const DiffRec& other) {
    const float2 xj = other.x;
    float2 gv = other.g;
    if constexpr (!kHoldsGV) gv = make_float2(gv.x * other.V, gv.y * other.V);
    const PairG e = pair_g<false>(xi.x, xi.y, xj.x, xj.y, P);   // gk after the sum
    acc += (gv.x * e.dx + gv.y * e.dy) * e.gd;
  };
  if constexpr (kCells) {
    if constexpr (kByFour) {
      stored_pairs_by_four(i, F, g, coff, P.search_radius, S.nseg, S.start, S.mask, xi.x, xi.y, P.thr, load, pair);
    } else {
      if (live) stored_pairs<kTpp, true>(i, F, g, coff, P.search_radius, S.nseg, S.start, S.mask, xi.x, xi.y, P.thr,
                                         [&](int j) { pair(load(j)); }, sub);
    }
  } else {
    static_assert(kTpp == 1, "CSR rows run one lane per particle");
    const int k0 = F.offsets[i], k1 = row_end(F, i, k0);
    for (int k = k0; k < k1; ++k) pair(load(__ldg(F.cols + k)));
  }
  return lane_sum<kTpp>(acc) * P.gk;
}

// semiImplicitEuler, src/simulationBase.py:647-652 with integrateValues :564-569, for one
// particle with its own values.
__device__ __forceinline__ void sie_apply(int i, float2 xi, float2 vi, float rti, float2 ai, float dpi, float dt,
                                          float rho0, int continuum, float2* __restrict__ xo,
                                          float2* __restrict__ vo, float* __restrict__ ro, int32_t* status) {
  const float2 vn = make_float2(vi.x + dt * ai.x, vi.y + dt * ai.y);
  const float2 xn = make_float2(xi.x + dt * (vi.x + dt * ai.x), xi.y + dt * (vi.y + dt * ai.y));
  xo[i] = xn;
  vo[i] = vn;
  const float rn = continuum ? rti + dt * dpi / rho0 : rti;
  ro[i] = rn;
  if (!isfinite(xn.x) || !isfinite(xn.y) || !isfinite(vn.x) || !isfinite(vn.y) || !isfinite(rn))
    flag(status, SPH_FLAG_NONFINITE);
}

// ---------------------------------------------------------------------------- one scene
template <int kLanes>
__global__ void __launch_bounds__(128) k_mdbc(FluidView F, WallView W, const sph_grid* __restrict__ gp, SphParams P) {
  const int b = (blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
  if (kLanes == 1 && b >= W.n) return;
  mdbc_body<kLanes>(min(b, W.n - 1), b < W.n, threadIdx.x % kLanes, F, W, *gp, P, 0);
}

__global__ void __launch_bounds__(256) k_prep(FluidView F, SphParams P, Rec* __restrict__ rec) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= F.n) return;
  prep_body(i, F, P, rec);
}

// Neighbor record and segment list of particle i by kRowLanes lanes, for launches too small to
// hide one thread's chain of candidate tests: a lane tests a cell row each, then places its row's
// non-empty segments behind those of the rows before it, the list that segments_body makes.  It
// keeps the masks of two segments (rows of up to 64 candidates) and forms later ones again.
// `live` false: a lane that only takes part.  Records and segments of 8,192 particles
// 6.1 -> 4.9 us, 16,384: 6.9 -> 5.4, 32,400: 7.0 -> 5.9; 65,536 take 7.3 with one lane, 9.6 with four.
constexpr int kRowLanes = 4;
constexpr int kRowLanesMax = 32768;   // particles up to which it is faster

__device__ __noinline__ uint32_t segment_mask_again(const float2* __restrict__ x, int c, int e, float xi, float yi,
                                                    float thr) {
  return segment_mask(x, c, e, xi, yi, thr);
}

__device__ __forceinline__ void prep_rows(int i, bool live, int sub, const FluidView& F, const sph_grid& g, int coff,
                                          const SphParams& P, Rec* __restrict__ rec, int32_t* __restrict__ nseg,
                                          int32_t* __restrict__ seg_start, uint32_t* __restrict__ seg_mask) {
  const size_t n = (size_t)F.n;
  int cx = 0, cy = -(1 << 20);
  float2 xi = make_float2(0.f, 0.f);
  if (live) {
    cell_of(F.keys[i] - (uint32_t)coff, g, &cx, &cy);
    xi = F.x[i];
    if (sub == kRowLanes - 1) prep_body(i, F, P, rec);
  }
  const int r = P.search_radius;
  const int x0 = max(cx - r, 0), x1 = min(cx + r, g.cells_x - 1), y0 = max(cy - r, 0);
  const int rows = live && x0 <= x1 ? min(cy + r, g.cells_y - 1) - y0 + 1 : 0;
  int first = 0;   // segments of the rows already placed
  for (int q = 0; __any_sync(0xffffffffu, q < rows); q += kRowLanes) {
    int b = 0, e = 0;
    if (q + sub < rows) {
      const int32_t* row = F.cell_start + coff + (y0 + q + sub) * g.cells_x;
      b = __ldg(row + x0);
      e = __ldg(row + x1 + 1);
    }
    uint32_t w0 = 0, w1 = 0;   // the row's first two segments
    int mine = 0;
    for (int c = b; c < e; c += 32) {
      const uint32_t w = c + 32 <= F.n ? segment_mask_full(F.x, c, e, xi.x, xi.y, P.thr)
                                       : segment_mask(F.x, c, e, xi.x, xi.y, P.thr);
      if (c == b) w0 = w;
      if (c == b + 32) w1 = w;
      mine += w != 0;
    }
    int k = mine, all = mine;
#pragma unroll
    for (int o = 1; o < kRowLanes; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, k, o, kRowLanes);
      if (sub >= o) k += v;
      all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    k += first - mine;
    first += all;
    const auto place = [&](int c, uint32_t w) {
      if (w == 0 || k >= kMaxSegments) return;
      seg_start[k * n + i] = c;
      seg_mask[k * n + i] = w;
      ++k;
    };
    place(b, w0);
    place(b + 32, w1);
    for (int c = b + 64; c < e && k < kMaxSegments; c += 32) place(c, segment_mask_again(F.x, c, e, xi.x, xi.y, P.thr));
  }
  if (live && sub == 0) nseg[i] = first <= kMaxSegments ? first : -1;
}

// Neighbor records and segment lists of one scene, kLanes (1 or kRowLanes) per particle.
template <int kLanes>
__global__ void __launch_bounds__(256) k_prep_cells(FluidView F, SphParams P, const sph_grid* __restrict__ gp,
                                                    Rec* __restrict__ rec, int32_t* __restrict__ nseg,
                                                    int32_t* __restrict__ seg_start,
                                                    uint32_t* __restrict__ seg_mask) {
  const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes);
  if constexpr (kLanes == 1) {
    if (i >= F.n) return;
    prep_body(i, F, P, rec);
    segments_body(i, F, *gp, 0, P.search_radius, P.thr, nseg, seg_start, seg_mask);
  } else {
    prep_rows(i, i < F.n, threadIdx.x % kLanes, F, *gp, 0, P, rec, nseg, seg_start, seg_mask);
  }
}

// The walls' densities and the records of one scene in one launch: the first wall_blocks blocks
// take four lanes per wall, the others the records.  Both only read the sorted state; the
// walls are a chain of latencies (a cell row, its candidates, a solve in double) in a few blocks.
// 8,192 particles with 1,380 walls: 9.4 us (9.4 + 4.4 one after the other).
template <int kLanes>
__global__ void __launch_bounds__(128) k_walls_and_prep(FluidView F, WallView W, SphParams P,
                                                        const sph_grid* __restrict__ gp, Rec* __restrict__ rec,
                                                        int32_t* __restrict__ nseg, int32_t* __restrict__ seg_start,
                                                        uint32_t* __restrict__ seg_mask, int wall_blocks) {
  if ((int)blockIdx.x < wall_blocks) {
    const int b = (blockIdx.x * blockDim.x + threadIdx.x) / 4;
    mdbc_body<4>(min(b, W.n - 1), b < W.n, threadIdx.x % 4, F, W, *gp, P, 0);
    return;
  }
  const int i = (int)(((int64_t)(blockIdx.x - wall_blocks) * blockDim.x + threadIdx.x) / kLanes);
  if constexpr (kLanes == 1) {
    if (i >= F.n) return;
    prep_body(i, F, P, rec);
    segments_body(i, F, *gp, 0, P.search_radius, P.thr, nseg, seg_start, seg_mask);
  } else {
    prep_rows(i, i < F.n, threadIdx.x % kLanes, F, *gp, 0, P, rec, nseg, seg_start, seg_mask);
  }
}

// One scene's right-hand side.
template <bool kCells, int kScheme, bool kByFour>
__global__ void __launch_bounds__(128) k_dsph_pass1(FluidView F, const Rec* __restrict__ rec, WallView W,
                                                    const sph_grid* __restrict__ gp, SphParams P, Segments S,
                                                    float* __restrict__ dpdt, float2* __restrict__ acc,
                                                    float4* __restrict__ Lout, float2* __restrict__ grad_rho) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= F.n) return;
  const Pass1 o = pass1_body<kCells, 1, kScheme, kByFour>(i, F, rec, W, *gp, P, 0, S);
  dpdt[i] = (kScheme >= 0 ? kScheme : P.diffusion) == 2 ? o.dpdt + P.diff_k * o.ddiff : o.dpdt;
  acc[i] = make_float2(o.ax, o.ay);
  if (Lout) Lout[i] = o.L;
  if (grad_rho) grad_rho[i] = o.grad_rho;
}

template <bool kCells, bool kByFour>
__global__ void __launch_bounds__(128) k_dsph_diffusion(FluidView F, const Rec* __restrict__ rec,
                                                        const sph_grid* __restrict__ gp, SphParams P, Segments S,
                                                        const float2* __restrict__ grad_rho,
                                                        float* __restrict__ dpdt) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= F.n) return;
  dpdt[i] -= P.diff_k * diffusion_sum<kCells, 1, false, kByFour>(i, F, rec, P, grad_rho, *gp, 0, S);
}

__global__ void k_sie(int n, const float2* __restrict__ x, const float2* __restrict__ v,
                      const float* __restrict__ rho, const float2* __restrict__ a, const float* __restrict__ dpdt,
                      const float* __restrict__ dt_ptr, float rho0, int continuum, float2* __restrict__ xo,
                      float2* __restrict__ vo, float* __restrict__ ro, int32_t* status, double* time) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (time && i == 0) *time += (double)*dt_ptr;
  sie_apply(i, x[i], v[i], rho[i], a[i], continuum ? dpdt[i] : 0.f, *dt_ptr, rho0, continuum, xo, vo, ro, status);
}

// ---------------------------------------------------------------------------- batch of scenes
// scenes[sid[i]] gives particle i's grid, parameters, cell-table offset and time step.
template <int kLanes>
__global__ void __launch_bounds__(128, 8) k_batch_mdbc(FluidView F, WallView W, const SceneDev* __restrict__ scenes,
                                                       const int32_t* __restrict__ wsid) {
  const int b = (blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
  const int sid = b < W.n ? wsid[b] : -1;   // -1: wall of no scene (free slot of a pooled batch)
  if (kLanes == 1 && sid < 0) return;
  const SceneDev& S = scenes[max(sid, 0)];
  mdbc_body<kLanes>(min(b, W.n - 1), sid >= 0, threadIdx.x % kLanes, F, W, S.g, S.P, S.coff);
}

// Neighbor records and segment lists of a small batch.
__global__ void __launch_bounds__(256) k_batch_prep_rows(FluidView F, const SceneDev* __restrict__ scenes,
                                                         const int32_t* __restrict__ sid, Rec* __restrict__ rec,
                                                         int32_t* __restrict__ nseg, int32_t* __restrict__ seg_start,
                                                         uint32_t* __restrict__ seg_mask) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) / kRowLanes;
  const int s = i < F.n ? sid[i] : -1;   // -1: particle of no scene
  const SceneDev& S = scenes[max(s, 0)];
  prep_rows(i, s >= 0, threadIdx.x % kRowLanes, F, S.g, S.coff, S.P, rec, nseg, seg_start, seg_mask);
}

// Neighbor records and, with pairs from the cell rows (nseg != NULL), the segment lists.
__global__ void __launch_bounds__(256) k_batch_prep(FluidView F, const SceneDev* __restrict__ scenes,
                                                    const int32_t* __restrict__ sid, Rec* __restrict__ rec,
                                                    int32_t* __restrict__ nseg,
                                                    int32_t* __restrict__ seg_start, uint32_t* __restrict__ seg_mask) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= F.n || sid[i] < 0) return;   // particle of no scene: never anyone's neighbor
  const SceneDev& S = scenes[sid[i]];
  prep_body(i, F, S.P, rec);
  if (nseg) segments_body(i, F, S.g, S.coff, S.P.search_radius, S.P.thr, nseg, seg_start, seg_mask);
}

// The update of one particle of a batch with its scene's dt.  If the neighbor list
// overflowed (the fill set SPH_FLAG_PAIR_CAPACITY) the step is not applied: the sorted
// inputs are copied unchanged.
__device__ __forceinline__ void batch_update(int i, const FluidView& F, float ax, float ay, float dpdt,
                                             const SceneDev& S, float2* __restrict__ xo, float2* __restrict__ vo,
                                             float* __restrict__ ro, int32_t* status) {
  if (*status & SPH_FLAG_PAIR_CAPACITY) {
    xo[i] = F.x[i];
    vo[i] = F.v[i];
    ro[i] = F.rho[i];
    return;
  }
  sie_apply(i, F.x[i], F.v[i], F.rho[i], make_float2(ax, ay), dpdt, S.dt, S.P.rho0, 1, xo, vo, ro, status);
}

// Pass 1 of the particles [p_lo, p_hi).  Particles of scenes without the deltaSPH density
// diffusion are complete after it and are updated here; the others hand dpdt, acc and
// <grad rho> to k_batch_diffusion, which finishes and updates them.  kCells: pairs from the
// segment lists; kTpp lanes per particle (kCells only).  With kTpp > 1 no lane leaves
// before the lane sums: lanes past p_hi take part with nothing to add.
// Large batches (one lane, pairs from the cell rows) take 48 registers, ten blocks per SM: a serving step
// of 3.1 M particles 318 us, with nine 322, with eight 326, with eleven (spilled sums) 522.
template <bool kCells, int kTpp, int kScheme, bool kByFour = false>
__global__ void __launch_bounds__(128, kByFour ? 6 : kCells && kTpp == 1 ? 10 : 9) k_batch_pass1(FluidView F, const Rec* __restrict__ rec, WallView W,
                                                     const SceneDev* __restrict__ scenes,
                                                     const int32_t* __restrict__ sid, float* __restrict__ dpdt,
                                                     float2* __restrict__ acc, float2* __restrict__ grad_rho,
                                                     const Segments seg, float2* __restrict__ xo,
                                                     float2* __restrict__ vo, float* __restrict__ ro,
                                                     int32_t* status, int p_lo, int p_hi) {
  int i, sub = 0;
  bool live = true;
  if constexpr (kTpp == 1) {
    i = p_lo + (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= p_hi || sid[i] < 0) return;
  } else {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t ii = p_lo + g / kTpp;
    sub = (int)(g % kTpp);
    live = ii < p_hi;
    i = live ? (int)ii : p_lo;
    live = live && sid[i] >= 0;   // a particle of no scene takes part in the lane sums only
  }
  const SceneDev& S = scenes[sid[i] < 0 ? 0 : sid[i]];
  const SphParams P = S.P;   // the fields the loop reads, in registers
  const Pass1 o = pass1_body<kCells, kTpp, kScheme, kByFour>(i, F, rec, W, S.g, P, S.coff, seg, sub,
                                                             kTpp == 1 || live);
  if (kTpp > 1 && (!live || sub != 0)) return;
  if ((kScheme >= 0 ? kScheme : P.diffusion) == 2) {
    dpdt[i] = o.dpdt + P.diff_k * o.ddiff;
    acc[i] = make_float2(o.ax, o.ay);
    const float Vi = q_of(rec, F.n)[i].y;
    grad_rho[i] = make_float2(o.grad_rho.x * Vi, o.grad_rho.y * Vi);   // <grad rho> V for the diffusion pass
    return;
  }
  batch_update(i, F, o.ax, o.ay, o.dpdt, S, xo, vo, ro, status);
}

template <bool kCells, int kTpp, bool kByFour = false>
__global__ void __launch_bounds__(128) k_batch_diffusion(FluidView F, const Rec* __restrict__ rec,
                                                         const SceneDev* __restrict__ scenes,
                                                         const int32_t* __restrict__ sid,
                                                         const float2* __restrict__ grad_rho, const Segments seg,
                                                         const float* __restrict__ dpdt,
                                                         const float2* __restrict__ acc, float2* __restrict__ xo,
                                                         float2* __restrict__ vo, float* __restrict__ ro,
                                                         int32_t* status, int p_lo, int p_hi) {
  int i, sub = 0;
  bool live = true;
  if constexpr (kTpp == 1) {
    i = p_lo + (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= p_hi || sid[i] < 0) return;
  } else {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t ii = p_lo + g / kTpp;
    sub = (int)(g % kTpp);
    live = ii < p_hi;
    i = live ? (int)ii : p_lo;
    live = live && sid[i] >= 0;
  }
  const SceneDev& S = scenes[sid[i] < 0 ? 0 : sid[i]];
  const bool act = live && S.P.diffusion == 2;   // the same on all lanes of a particle
  if (kTpp == 1 && !act) return;
  const SphParams P = S.P;   // the fields the loop reads, in registers
  const float sum = diffusion_sum<kCells, kTpp, true, kByFour>(i, F, rec, P, grad_rho, S.g, S.coff, seg, sub,
                                                               kTpp == 1 || act);
  if (kTpp > 1 && (!act || sub != 0)) return;
  const float d = dpdt[i] - P.diff_k * sum;
  const float2 a = acc[i];
  batch_update(i, F, a.x, a.y, d, S, xo, vo, ro, status);
}

// ---------------------------------------------------------------------------- RK4 helpers
// RK4 stage / combination, src/simulationBase.py:679-705: out = base + c * (k_u, k_a, k_d / rho0).
__global__ void k_rk_axpy(int n, const float2* __restrict__ x0, const float2* __restrict__ v0,
                          const float* __restrict__ r0, const float2* __restrict__ ku, const float2* __restrict__ ka,
                          const float* __restrict__ kd, const float* __restrict__ dt_ptr, float c, float rho0,
                          float2* __restrict__ xo, float2* __restrict__ vo, float* __restrict__ ro, int32_t* status) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float h = c * *dt_ptr;
  const float2 u = ku[i], a = ka[i], x = x0[i], v = v0[i];
  const float2 xn = make_float2(x.x + h * u.x, x.y + h * u.y);
  const float2 vn = make_float2(v.x + h * a.x, v.y + h * a.y);
  const float rn = r0[i] + h * kd[i] / rho0;
  xo[i] = xn;
  vo[i] = vn;
  ro[i] = rn;
  if (!isfinite(xn.x) || !isfinite(xn.y) || !isfinite(vn.x) || !isfinite(vn.y) || !isfinite(rn))
    flag(status, SPH_FLAG_NONFINITE);
}

// A whole RK4 stage: s (+)= w k, then out = base + c dt k, or the step's end from the sums (last).
// One launch where a sum and an update were two of about 1.3 us.
__global__ void k_rk_stage(int n, const float2* __restrict__ x0, const float2* __restrict__ v0,
                           const float* __restrict__ r0, const float2* __restrict__ ku, const float2* __restrict__ ka,
                           const float* __restrict__ kd, float w, int init, int last, float2* __restrict__ su,
                           float2* __restrict__ sa, float* __restrict__ sd, const float* __restrict__ dt_ptr, float c,
                           float rho0, float2* __restrict__ xo, float2* __restrict__ vo, float* __restrict__ ro,
                           int32_t* status, double* time) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float dt = *dt_ptr;
  if (time && i == 0) *time += (double)dt;
  float2 u = ku[i], a = ka[i];
  float d = kd[i];
  float2 pu = make_float2(w * u.x, w * u.y), pa = make_float2(w * a.x, w * a.y);
  float pd = w * d;
  if (!init) {
    const float2 cu = su[i], ca = sa[i];
    pu = make_float2(cu.x + w * u.x, cu.y + w * u.y);
    pa = make_float2(ca.x + w * a.x, ca.y + w * a.y);
    pd = sd[i] + w * d;
  }
  su[i] = pu;
  sa[i] = pa;
  sd[i] = pd;
  if (last) {
    u = pu;
    a = pa;
    d = pd;
  }
  const float h = c * dt;
  const float2 x = x0[i], v = v0[i];
  const float2 xn = make_float2(x.x + h * u.x, x.y + h * u.y);
  const float2 vn = make_float2(v.x + h * a.x, v.y + h * a.y);
  const float rn = r0[i] + h * d / rho0;
  xo[i] = xn;
  vo[i] = vn;
  ro[i] = rn;
  if (!isfinite(xn.x) || !isfinite(xn.y) || !isfinite(vn.x) || !isfinite(vn.y) || !isfinite(rn))
    flag(status, SPH_FLAG_NONFINITE);
}

// s (+)= w * k for the RK4 sums; init = 1 overwrites.
__global__ void k_rk_accum(int n, const float2* __restrict__ ku, const float2* __restrict__ ka,
                           const float* __restrict__ kd, float w, int init, float2* __restrict__ su,
                           float2* __restrict__ sa, float* __restrict__ sd) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float2 u = ku[i], a = ka[i];
  float d = kd[i];
  if (init) {
    su[i] = make_float2(w * u.x, w * u.y);
    sa[i] = make_float2(w * a.x, w * a.y);
    sd[i] = w * d;
  } else {
    float2 s = su[i], t = sa[i];
    su[i] = make_float2(s.x + w * u.x, s.y + w * u.y);
    sa[i] = make_float2(t.x + w * a.x, t.y + w * a.y);
    sd[i] += w * d;
  }
}

// Permute per-particle arrays into a new order: out[s] = in[order[s]] (4-, 8- and 16-byte elements).
template <typename T>
__global__ void k_permute(const uint32_t* __restrict__ order, int n, const T* __restrict__ in, T* __restrict__ out) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < n) out[s] = in[order[s]];
}

// Up to kMaxArrays per-particle arrays gathered in one pass: out_k[s] = in_k[order[s]], or
// a plain copy when order is null.  One launch reads order once instead of once per array.
__global__ void __launch_bounds__(256) k_permute_arrays(const uint32_t* __restrict__ order, int n, ArraySet a) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  copy_rows(a, s, order ? (int)order[s] : s);
}

}  // namespace sph

using namespace sph;

extern "C" {

sph_status_t sph_mdbc_wall_density(const sph_fluid_view* fluid, const sph_wall_view* walls, const sph_grid* grid,
                                   const sph_params* params, void* stream) {
  SPH_VIEW_CHECK(fluid);
  SPH_VIEW_CHECK(walls);
  SPH_REQUIRE(grid && params && params->support > 0.f, "mdbc: bad arguments");
  if (walls->n == 0) return SPH_OK;
  const FluidView F = to_fluid(fluid);
  const WallView W = to_walls(walls);
  const SphParams P = to_params(params);
  if (W.n <= kMdbcSplitWalls)
    k_mdbc<4><<<grid_for(4 * walls->n, 128), 128, 0, as_stream(stream)>>>(F, W, grid, P);
  else
    k_mdbc<1><<<grid_for(walls->n, 128), 128, 0, as_stream(stream)>>>(F, W, grid, P);
  SPH_CHECK_LAUNCH("mdbc_wall_density");
  return SPH_OK;
}

// Neighbor records (two float4 per particle), then, for pairs from the cell rows, the
// segment lists: kMaxSegments masks and starts and a count per particle.
constexpr size_t kRecordBytes = 2 * sizeof(float4),
                 kMaskBytes = kMaxSegments * (sizeof(uint32_t) + sizeof(int32_t)) + sizeof(int32_t);
size_t sph_deltasph_scratch_bytes(int64_t n) { return (size_t)(n > 0 ? n : 0) * (kRecordBytes + kMaskBytes) + 256; }
static_assert(sizeof(Rec) == kRecordBytes, "a neighbor record is two float4");

sph_status_t sph_deltasph_segment_lists(int64_t n, size_t* masks_offset, size_t* starts_offset,
                                        size_t* counts_offset, int32_t* max_segments) {
  SPH_REQUIRE(n >= 0 && masks_offset && starts_offset && counts_offset && max_segments,
              "deltasph_segment_lists: bad arguments");
  *masks_offset = (size_t)n * kRecordBytes;
  *starts_offset = *masks_offset + (size_t)n * kMaxSegments * sizeof(uint32_t);
  *counts_offset = *starts_offset + (size_t)n * kMaxSegments * sizeof(int32_t);
  *max_segments = kMaxSegments;
  return SPH_OK;
}

}  // extern "C"

// Particles of a launch up to which the force passes keep four pairs' records in flight per thread
// (same sums, 78 instead of 56 registers): pass 1 and diffusion of one scene, us, without / with:
// 8,100 particles 16.6 + 9.5 / 14.6 + 7.7, 36,864: 15.6 + 9.8 / 15.3 + 8.3, 65,536: 17.3 + 10.3 /
// 18.1 + 9.7, 131,044: 21.9 + 12.3 / 27.8 + 13.2.
constexpr int kByFourMax = 49152;

// Particles up to which the walls' densities run beside the records (k_walls_and_prep; its
// registers cost the records some of their warps), us, beside / one after the other, the walls of a
// tank twice as wide and high: 49,152: 9.1 / 15.8, 153,863: 12.0 / 20.0, 262,144: 14.6 / 24.2,
// 1,024,000: 43.0 / 50.1.
constexpr int kWallsBesideMax = 1 << 20;

// The neighbor records in caller scratch, 32-byte aligned.
static bool records_from_scratch(void* scratch, size_t bytes, int64_t n, Rec** rec, Segments* seg = nullptr) {
  if (!scratch) return false;
  const uintptr_t base = reinterpret_cast<uintptr_t>(scratch);
  const uintptr_t p = (base + 31) & ~(uintptr_t)31;
  if ((p - base) + (size_t)n * (kRecordBytes + (seg ? kMaskBytes : 0)) > bytes) return false;
  *rec = reinterpret_cast<Rec*>(p);
  if (seg) {
    uint32_t* m = reinterpret_cast<uint32_t*>(*rec + n);
    int32_t* st = reinterpret_cast<int32_t*>(m + kMaxSegments * n);
    seg->mask = m;
    seg->start = st;
    seg->nseg = st + kMaxSegments * n;
  }
  return true;
}

extern "C" {

static sph_status_t forces(const sph_fluid_view* fluid, const sph_wall_view* walls, const sph_grid* grid,
                           const sph_params* params, float* dpdt, float* acc, float* L, float* grad_rho, void* scratch,
                           size_t scratch_bytes, bool with_walls, void* stream) {
  SPH_VIEW_CHECK(fluid);
  SPH_VIEW_CHECK(walls);
  SPH_REQUIRE(grid && params && dpdt && acc && params->support > 0.f, "deltasph_forces: bad arguments");
  SPH_REQUIRE(params->density_diffusion != 2 || grad_rho, "deltasph_forces: deltaSPH diffusion needs grad_rho");
  if (fluid->n == 0) return with_walls ? sph_mdbc_wall_density(fluid, walls, grid, params, stream) : SPH_OK;
  // no CSR list (offsets and cols NULL): the pairs come from the cell rows
  const bool cells = !fluid->offsets && !fluid->cols;
  SPH_REQUIRE(cells ? fluid->cell_start && fluid->keys : fluid->offsets && fluid->cols,
              "deltasph_forces: give offsets and cols, or neither with keys and the cell table");
  Rec* rec;
  Segments seg{};
  SPH_REQUIRE(records_from_scratch(scratch, scratch_bytes, fluid->n, &rec, cells ? &seg : nullptr),
              "deltasph_forces: scratch smaller than sph_deltasph_scratch_bytes(n)");
  cudaStream_t st = as_stream(stream);
  const FluidView F = to_fluid(fluid);
  const WallView W = to_walls(walls);
  const SphParams P = to_params(params);
  const int n = F.n;
  float2* ac = reinterpret_cast<float2*>(acc);
  float4* Lo = reinterpret_cast<float4*>(L);
  float2* gr = reinterpret_cast<float2*>(grad_rho);
  const int nb = grid_for(n, 128);
#define SPH_PASS1(C, K, B4) k_dsph_pass1<C, K, B4><<<nb, 128, 0, st>>>(F, rec, W, grid, P, seg, dpdt, ac, Lo, gr)
#define SPH_DIFFUSION(C, B4) k_dsph_diffusion<C, B4><<<nb, 128, 0, st>>>(F, rec, grid, P, seg, gr, dpdt)
  const bool beside = cells && with_walls && W.n > 0 && W.n <= kMdbcSplitWalls && n <= kWallsBesideMax;
  if (with_walls && !beside) {
    const sph_status_t r = sph_mdbc_wall_density(fluid, walls, grid, params, stream);
    if (r != SPH_OK) return r;
  }
  if (!cells) {
    k_prep<<<grid_for(n, 256), 256, 0, st>>>(F, P, rec);
    SPH_PASS1(false, -1, false);
    if (P.diffusion == 2) SPH_DIFFUSION(false, false);
  } else {
    int32_t* ns = const_cast<int32_t*>(seg.nseg);
    int32_t* ss = const_cast<int32_t*>(seg.start);
    uint32_t* sm = const_cast<uint32_t*>(seg.mask);
    const int wb = beside ? grid_for(4 * (int64_t)W.n, 128) : 0;
    if (beside && n <= kRowLanesMax)
      k_walls_and_prep<kRowLanes><<<wb + grid_for(kRowLanes * (int64_t)n, 128), 128, 0, st>>>(F, W, P, grid, rec, ns, ss,
                                                                                           sm, wb);
    else if (beside)
      k_walls_and_prep<1><<<wb + grid_for(n, 128), 128, 0, st>>>(F, W, P, grid, rec, ns, ss, sm, wb);
    else if (n <= kRowLanesMax)
      k_prep_cells<kRowLanes><<<grid_for(kRowLanes * (int64_t)n, 256), 256, 0, st>>>(F, P, grid, rec, ns, ss, sm);
    else
      k_prep_cells<1><<<grid_for(n, 256), 256, 0, st>>>(F, P, grid, rec, ns, ss, sm);
    const bool by_four = n <= kByFourMax;
    if (P.diffusion == 2) {
      if (by_four) {
        SPH_PASS1(true, 2, true);
        SPH_DIFFUSION(true, true);
      } else {
        SPH_PASS1(true, 2, false);
        SPH_DIFFUSION(true, false);
      }
    } else if (by_four) {
      SPH_PASS1(true, -1, true);
    } else if (P.diffusion == 1) {
      SPH_PASS1(true, 1, false);
    } else {
      SPH_PASS1(true, -1, false);
    }
  }
#undef SPH_PASS1
#undef SPH_DIFFUSION
  SPH_CHECK_LAUNCH("deltasph_forces");
  return SPH_OK;
}

sph_status_t sph_deltasph_forces(const sph_fluid_view* fluid, const sph_wall_view* walls, const sph_grid* grid,
                                 const sph_params* params, float* dpdt, float* acc, float* L, float* grad_rho,
                                 void* scratch, size_t scratch_bytes, void* stream) {
  return forces(fluid, walls, grid, params, dpdt, acc, L, grad_rho, scratch, scratch_bytes, false, stream);
}

sph_status_t sph_deltasph_wall_forces(const sph_fluid_view* fluid, const sph_wall_view* walls, const sph_grid* grid,
                                      const sph_params* params, float* dpdt, float* acc, float* L, float* grad_rho,
                                      void* scratch, size_t scratch_bytes, void* stream) {
  return forces(fluid, walls, grid, params, dpdt, acc, L, grad_rho, scratch, scratch_bytes, true, stream);
}

sph_status_t sph_integrate_step(int64_t n, const float* x, const float* v, const float* rho, const float* acc,
                                const float* dpdt, const float* dt, float rest_density, int32_t continuum_density,
                                float* x_out, float* v_out, float* rho_out, int32_t* status, double* time,
                                void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && x && v && rho && acc && dt && x_out && v_out && rho_out,
              "integrate_semi_implicit_euler: bad arguments");
  SPH_REQUIRE(!continuum_density || dpdt, "integrate_semi_implicit_euler: continuum density needs dpdt");
  if (n == 0) return SPH_OK;
  k_sie<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(
      (int)n, reinterpret_cast<const float2*>(x), reinterpret_cast<const float2*>(v), rho,
      reinterpret_cast<const float2*>(acc), dpdt, dt, rest_density, continuum_density, reinterpret_cast<float2*>(x_out),
      reinterpret_cast<float2*>(v_out), rho_out, status, time);
  SPH_CHECK_LAUNCH("integrate_semi_implicit_euler");
  return SPH_OK;
}

sph_status_t sph_integrate_semi_implicit_euler(int64_t n, const float* x, const float* v, const float* rho,
                                               const float* acc, const float* dpdt, const float* dt,
                                               float rest_density, int32_t continuum_density, float* x_out,
                                               float* v_out, float* rho_out, int32_t* status, void* stream) {
  return sph_integrate_step(n, x, v, rho, acc, dpdt, dt, rest_density, continuum_density, x_out, v_out, rho_out, status,
                            nullptr, stream);
}

sph_status_t sph_batch_deltasph_step(const sph_fluid_view* fluid, const sph_wall_view* walls, const void* scenes,
                                     const int32_t* sid, const int32_t* wall_sid, float* dpdt, float* acc,
                                     float* grad_rho, int32_t any_renormalized, float* x_out, float* v_out,
                                     float* rho_out, int32_t* status, int32_t phases, int32_t ngroups,
                                     const sph_force_group* groups, void* scratch, size_t scratch_bytes,
                                     void* stream) {
  SPH_VIEW_CHECK(fluid);
  SPH_VIEW_CHECK(walls);
  SPH_REQUIRE(scenes && sid && x_out && v_out && rho_out && status, "batch_deltasph_step: bad arguments");
  SPH_REQUIRE(walls->n == 0 || wall_sid, "batch_deltasph_step: walls need wall_sid");
  SPH_REQUIRE(!any_renormalized || (dpdt && acc && grad_rho),
              "batch_deltasph_step: deltaSPH diffusion needs dpdt, acc, grad_rho");
  // no CSR list (offsets and cols NULL): the pairs come from the cell rows
  const bool cells = !fluid->offsets && !fluid->cols;
  SPH_REQUIRE(cells || (fluid->offsets && fluid->cols), "batch_deltasph_step: give both offsets and cols, or neither");
  SPH_REQUIRE(fluid->cell_start && fluid->keys, "batch_deltasph_step: bad arguments");
  const int n = (int)fluid->n;
  // force groups: by default one group, one lane per particle, any schemes
  const sph_force_group all{0, n, 1, -1};
  SPH_REQUIRE(ngroups >= 0 && (ngroups == 0 || groups), "batch_deltasph_step: bad groups");
  const int ng = ngroups ? ngroups : 1;
  const sph_force_group* G = ngroups ? groups : &all;
  SPH_REQUIRE(G[0].begin == 0 && G[ng - 1].end == n, "batch_deltasph_step: the groups must tile [0, n)");
  for (int k = 0; k < ng; ++k) {
    SPH_REQUIRE(G[k].begin <= G[k].end && (k == 0 || G[k].begin == G[k - 1].end),
                "batch_deltasph_step: the groups must tile [0, n) in order");
    SPH_REQUIRE(G[k].tpp == 1 || (cells && (G[k].tpp == 2 || G[k].tpp == 4)),
                "batch_deltasph_step: lanes per particle must be 1 (2 or 4 with pairs from the cell rows)");
    SPH_REQUIRE(G[k].scheme >= -1 && G[k].scheme <= 2, "batch_deltasph_step: bad diffusion scheme");
  }
  if (n == 0) return SPH_OK;
  Rec* rec;
  Segments seg{};
  SPH_REQUIRE(records_from_scratch(scratch, scratch_bytes, n, &rec, cells ? &seg : nullptr),
              "batch_deltasph_step: scratch smaller than sph_deltasph_scratch_bytes(n)");
  cudaStream_t st = as_stream(stream);
  const FluidView F = to_fluid(fluid);
  const WallView W = to_walls(walls);
  const SceneDev* S = static_cast<const SceneDev*>(scenes);
  if (W.n > 0 && (phases & SPH_PHASE_WALLS)) {
    if (W.n <= kMdbcSplitWalls)
      k_batch_mdbc<4><<<grid_for(4 * (int64_t)W.n, 128), 128, 0, st>>>(F, W, S, wall_sid);
    else
      k_batch_mdbc<1><<<grid_for(W.n, 128), 128, 0, st>>>(F, W, S, wall_sid);
  }
  if (phases & SPH_PHASE_RECORDS) {
    int32_t* ns = const_cast<int32_t*>(seg.nseg);
    int32_t* ss = const_cast<int32_t*>(seg.start);
    uint32_t* sm = const_cast<uint32_t*>(seg.mask);
    if (cells && n <= kRowLanesMax)
      k_batch_prep_rows<<<grid_for(kRowLanes * (int64_t)n, 256), 256, 0, st>>>(F, S, sid, rec, ns, ss, sm);
    else
      k_batch_prep<<<grid_for(n, 256), 256, 0, st>>>(F, S, sid, rec, ns, ss, sm);
  }
  float2* xo = reinterpret_cast<float2*>(x_out);
  float2* vo = reinterpret_cast<float2*>(v_out);
  float2* gr = reinterpret_cast<float2*>(grad_rho);
  float2* ac = reinterpret_cast<float2*>(acc);
  // kernel variants: CSR rows run one lane and read the scheme per scene; cell rows have 1, 2
  // or 4 lanes and a scheme of MOG, deltaSPH or read per scene
  auto pass1 = [&](int lo, int hi, int t, int scheme) {
    const int nb = grid_for((int64_t)(hi - lo) * t, 128);
#define SPH_PASS1(C, T, K, ...)                                                                                \
  k_batch_pass1<C, T, K, ##__VA_ARGS__><<<nb, 128, 0, st>>>(F, rec, W, S, sid, dpdt, ac, gr,                   \
                                                            C ? seg : Segments{}, xo, vo, rho_out, status, lo, \
                                                            hi)
    if (!cells) {
      SPH_PASS1(false, 1, -1);
      return;
    }
    const int k = scheme == 1 || scheme == 2 ? scheme : -1;
    if (t == 1 && hi - lo <= kByFourMax) {
      if (k == 2) SPH_PASS1(true, 1, 2, true);
      else SPH_PASS1(true, 1, -1, true);
    } else if (t == 1) {
      if (k == 2) SPH_PASS1(true, 1, 2);
      else if (k == 1) SPH_PASS1(true, 1, 1);
      else SPH_PASS1(true, 1, -1);
    } else if (t == 2) {
      if (k == 2) SPH_PASS1(true, 2, 2);
      else if (k == 1) SPH_PASS1(true, 2, 1);
      else SPH_PASS1(true, 2, -1);
    } else {
      if (k == 2) SPH_PASS1(true, 4, 2);
      else if (k == 1) SPH_PASS1(true, 4, 1);
      else SPH_PASS1(true, 4, -1);
    }
#undef SPH_PASS1
  };
  for (int k = 0; k < ng && (phases & SPH_PHASE_PASS1); ++k)
    if (G[k].end > G[k].begin) pass1((int)G[k].begin, (int)G[k].end, G[k].tpp, G[k].scheme);
  for (int k = 0; k < ng && any_renormalized && (phases & SPH_PHASE_DIFFUSION); ++k) {
    const int lo = (int)G[k].begin, hi = (int)G[k].end, t = G[k].tpp;
    if (hi <= lo || G[k].scheme == 0 || G[k].scheme == 1) continue;   // no deltaSPH scene in the group
    const int nb = grid_for((int64_t)(hi - lo) * t, 128);
    if (!cells)
      k_batch_diffusion<false, 1><<<nb, 128, 0, st>>>(F, rec, S, sid, gr, Segments{}, dpdt, ac, xo, vo, rho_out,
                                                      status, lo, hi);
    else if (t == 1 && hi - lo <= kByFourMax)
      k_batch_diffusion<true, 1, true><<<nb, 128, 0, st>>>(F, rec, S, sid, gr, seg, dpdt, ac, xo, vo, rho_out,
                                                           status, lo, hi);
    else if (t == 1)
      k_batch_diffusion<true, 1><<<nb, 128, 0, st>>>(F, rec, S, sid, gr, seg, dpdt, ac, xo, vo, rho_out, status, lo,
                                                     hi);
    else if (t == 2)
      k_batch_diffusion<true, 2><<<nb, 128, 0, st>>>(F, rec, S, sid, gr, seg, dpdt, ac, xo, vo, rho_out, status, lo,
                                                     hi);
    else
      k_batch_diffusion<true, 4><<<nb, 128, 0, st>>>(F, rec, S, sid, gr, seg, dpdt, ac, xo, vo, rho_out, status, lo,
                                                     hi);
  }
  SPH_CHECK_LAUNCH("batch_deltasph_step");
  return SPH_OK;
}

size_t sph_scene_bytes(void) { return sizeof(SceneDev); }

sph_status_t sph_scene_encode(const sph_params* params, const sph_grid* grid_host, int32_t cell_offset, float dt,
                              void* out_host) {
  SPH_REQUIRE(params && grid_host && out_host && params->support > 0.f, "scene_encode: bad arguments");
  SceneDev s;
  s.P = to_params(params);
  s.g = *grid_host;
  s.coff = cell_offset;
  s.dt = dt;
  memcpy(out_host, &s, sizeof(s));
  return SPH_OK;
}

sph_status_t sph_rk_axpy(int64_t n, const float* x0, const float* v0, const float* rho0_field, const float* ku,
                         const float* ka, const float* kd, const float* dt, float c, float rest_density, float* x_out,
                         float* v_out, float* rho_out, int32_t* status, void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && x0 && v0 && rho0_field && ku && ka && kd && dt && x_out && v_out && rho_out,
              "rk_axpy: bad arguments");
  if (n == 0) return SPH_OK;
  k_rk_axpy<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(
      (int)n, reinterpret_cast<const float2*>(x0), reinterpret_cast<const float2*>(v0), rho0_field,
      reinterpret_cast<const float2*>(ku), reinterpret_cast<const float2*>(ka), kd, dt, c, rest_density,
      reinterpret_cast<float2*>(x_out), reinterpret_cast<float2*>(v_out), rho_out, status);
  SPH_CHECK_LAUNCH("rk_axpy");
  return SPH_OK;
}

sph_status_t sph_rk_stage(int64_t n, const float* x0, const float* v0, const float* rho0_field, const float* ku,
                          const float* ka, const float* kd, float w, int32_t init, int32_t last, float* su, float* sa,
                          float* sd, const float* dt, float c, float rest_density, float* x_out, float* v_out,
                          float* rho_out, int32_t* status, double* time, void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && x0 && v0 && rho0_field && ku && ka && kd && su && sa && sd && dt && x_out &&
                  v_out && rho_out,
              "rk_stage: bad arguments");
  if (n == 0) return SPH_OK;
  k_rk_stage<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(
      (int)n, reinterpret_cast<const float2*>(x0), reinterpret_cast<const float2*>(v0), rho0_field,
      reinterpret_cast<const float2*>(ku), reinterpret_cast<const float2*>(ka), kd, w, init, last,
      reinterpret_cast<float2*>(su), reinterpret_cast<float2*>(sa), sd, dt, c, rest_density,
      reinterpret_cast<float2*>(x_out), reinterpret_cast<float2*>(v_out), rho_out, status, time);
  SPH_CHECK_LAUNCH("rk_stage");
  return SPH_OK;
}

sph_status_t sph_rk_accumulate(int64_t n, const float* ku, const float* ka, const float* kd, float w, int32_t init,
                               float* su, float* sa, float* sd, void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && ku && ka && kd && su && sa && sd, "rk_accumulate: bad arguments");
  if (n == 0) return SPH_OK;
  k_rk_accum<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(
      (int)n, reinterpret_cast<const float2*>(ku), reinterpret_cast<const float2*>(ka), kd, w, init,
      reinterpret_cast<float2*>(su), reinterpret_cast<float2*>(sa), sd);
  SPH_CHECK_LAUNCH("rk_accumulate");
  return SPH_OK;
}

sph_status_t sph_permute_arrays(const uint32_t* order, int64_t n, int32_t count, const int32_t* elem_bytes,
                                const void* const* in, void* const* out, void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && count >= 0 && count <= kMaxArrays && (count == 0 || (elem_bytes && in && out)),
              "permute_arrays: bad arguments");
  if (n == 0 || count == 0) return SPH_OK;
  ArraySet a;
  SPH_REQUIRE(array_set_from(count, elem_bytes, in, out, &a),
              "permute_arrays: each array needs distinct in/out and 4, 8 or 16-byte elements");
  k_permute_arrays<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(order, (int)n, a);
  SPH_CHECK_LAUNCH("permute_arrays");
  return SPH_OK;
}

sph_status_t sph_permute(const uint32_t* order, int64_t n, int32_t elem_bytes, const void* in, void* out, void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && order && in && out, "permute: bad arguments");
  if (n == 0) return SPH_OK;
  cudaStream_t st = as_stream(stream);
  const int nb = grid_for(n, 256);
  switch (elem_bytes) {
    case 4:
      k_permute<uint32_t><<<nb, 256, 0, st>>>(order, (int)n, static_cast<const uint32_t*>(in), static_cast<uint32_t*>(out));
      break;
    case 8:
      k_permute<uint2><<<nb, 256, 0, st>>>(order, (int)n, static_cast<const uint2*>(in), static_cast<uint2*>(out));
      break;
    case 16:
      k_permute<uint4><<<nb, 256, 0, st>>>(order, (int)n, static_cast<const uint4*>(in), static_cast<uint4*>(out));
      break;
    default:
      set_error_text("permute: elem_bytes must be 4, 8 or 16");
      return SPH_ERR_INVALID_ARGUMENT;
  }
  SPH_CHECK_LAUNCH("permute");
  return SPH_OK;
}

}  // extern "C"
