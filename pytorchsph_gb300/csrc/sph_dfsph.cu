// DFSPH on sm_103a (src/modules/dfsph.py with the solid-wall PBSPH terms of
// src/modules/solidBoundary.py:294-520).
//
// The pressure solve (densitySolve / divergenceSolve, dfsph.py:195-260) runs as ONE
// cooperative kernel: every iteration is  accel from p (all particles)  -> grid barrier ->
// pressure-sum, residual, relaxed-Jacobi update and the block partials of the error ->
// grid barrier -> every block sums the partials in the same order (identical double result
// everywhere, so every block takes the same loop decision).  The loop is bounded by
// max_iters, so every thread meets every barrier the same number of times.
#include <cooperative_groups.h>

#include <mutex>

#include "sph_math.cuh"

namespace cg = cooperative_groups;

namespace sph {

struct DfsphBufs {
  // fluid, sorted order
  float* rho;         // relative density incl. the wall contribution
  float* vol;         // A / rho_fluid_only (fluidVolume)
  float* aact;        // A / rho (fluidActualArea)
  float2* vstar;      // predicted velocity
  float* alpha;
  float* source;
  float* p;           // pressure (fluidPressure2)
  float2* pa;         // predicted pressure acceleration
  float* res;
  // walls
  float* wrho;        // wall relative density (summation, clamped <= 1)
  float* waact;       // A_b / rho_b
  float* walpha;
  float* wsource;
  float* wp;
  float* wres;
  const float* wterm; // static wall-wall density term
  // solver output
  double* partials;   // [gridDim.x] block partial errors
  float* errors;      // [max_iters + 1] error history
  int32_t* iters;     // iteration count
  // pair records of the Jacobi sweeps, one 16-byte gather per neighbor and phase:
  float4* rec_p;      // (x, y, m = A rho0, p / (rho rho0)^2), its pressure part updated every sweep
  float4* rec_a;      // (x, y, predicted pressure acceleration)
  float* fdt;         // dt^2 A_act
  // pairs from the cell rows (kCells kernels): neighbor lists made by the density pass
  int4* list;         // [list_slots(n)] four neighbors each, see fluid_pairs
  int32_t* chunks;    // of particle i: fluid chunks + 256 x wall chunks, or -1: more than list_chunks in all
  int4* wlist;        // [wall_chunks nb] the walls' fluid neighbors, four each
  int32_t* wchunks;   // chunks of wall b, or -1: more than wall_chunks
  int list_chunks, wall_chunks;   // a particle's and a wall's places for chunks
};

// Neighbor list chunks (of four) per particle: the caller's list_capacity, which it takes from support and
// area with headroom.  A particle whose list does not fit tests its cell rows again in every sweep:
// one right-hand side of 262,144 particles at support 3 / 4 / 5 dx takes 648 / 566 / 796 us with
// lists that fit and 662 / 1,165 / 1,609 with room for 48 (over CSR rows 960 / 900 / 1,308).
constexpr int kListChunks = 12;      // list_capacity 0: a lattice at support 3 dx (29) 1.6 times as dense
constexpr int kMaxListChunks = 255;  // `chunks` holds the fluid's in 8 bits

// A wall's fluid neighbors are less than half a particle's (the first layer sees about 14 at 3 dx).
static int wall_chunks(int list_chunks) { return (2 * list_chunks + 2) / 3; }

// The fluid pairs of particle i for lane `sub` of its kTpp lanes: use(load(j)) for its share of
// the neighbor list (kCells) or of the CSR row.  A list is kept in chunks of four neighbors,
// filled up with i itself (whose gradient is zero in every sum here), chunk c of particle i at
// list[((c / kTpp) n + i) kTpp + c % kTpp]: a warp's loads are contiguous, one 16-byte load
// gives four neighbors whose records are in flight together, and the next chunk is loaded
// ahead.  The sweeps read every list many times over; a CSR row per thread costs them a cache
// line per lane and load (58 % of the SM's load wavefronts), segment masks 53 instructions a
// pair.  Both pressure solves of 262,144 settling particles (16 sweeps of pairs and walls): 1292 ->
// 702 us, of which the walls' lists gave 320.
template <bool kCells, int kTpp, typename Load, typename Use>
__device__ __forceinline__ void fluid_pairs(int i, const FluidView& F, const sph_grid& g, const SphParams& P,
                                            const DfsphBufs& B, float xi, float yi, int sub, Load&& load, Use&& use) {
  if constexpr (kCells) {
    int chunks = __ldg(B.chunks + i);
    if (chunks < 0) {
      int cx, cy;
      cell_of(F.keys[i], g, &cx, &cy);
      cell_pairs<kTpp>(F, g, P.search_radius, 0, cx, cy, xi, yi, P.thr, [&](int j) { use(load(j)); }, sub);
      return;
    }
    chunks &= 255;
    const int4* p = B.list + (size_t)i * kTpp + sub;
    const size_t step = (size_t)F.n * kTpp;
    int4 next = make_int4(i, i, i, i);
    if (sub < chunks) next = __ldg(p);
    for (int c = sub; c < chunks; c += kTpp) {
      const int4 j = next;
      p += step;
      if (c + kTpp < chunks) next = __ldg(p);
      const auto r0 = load(j.x), r1 = load(j.y), r2 = load(j.z), r3 = load(j.w);
      use(r0);
      use(r1);
      use(r2);
      use(r3);
    }
  } else {
    const int k0 = F.offsets[i], kn = row_end(F, i, k0);
    for (int k = k0 + sub; k < kn; k += kTpp) use(load(__ldg(F.cols + k)));
  }
}

// The walls of particle i the same way: use(b) for its share of the wall chunks behind its
// fluid chunks (kCells; a chunk is filled up with -1), or of the walls in its cells.  Walls
// tested candidate by candidate were the longest chain of every sweep.
template <bool kCells, int kTpp, typename Use>
__device__ __forceinline__ void wall_pairs(int i, const FluidView& F, const WallView& W, const sph_grid& g,
                                           const SphParams& P, const DfsphBufs& B, float xi, float yi, int sub,
                                           Use&& use) {
  const int chunks = kCells ? __ldg(B.chunks + i) : -1;
  if (chunks < 0) {
    int cx, cy;
    cell_of(F.keys[i], g, &cx, &cy);
    for_each_wall_lanes<kTpp>(W, g, P.search_radius, cx, cy, xi, yi, P.thr, sub, [&](int b, float2) { use(b); });
    return;
  }
  const int c0 = chunks & 255, c1 = c0 + (chunks >> 8);
  for (int c = c0 + (sub + kTpp - c0 % kTpp) % kTpp; c < c1; c += kTpp) {   // chunk c belongs to lane c % kTpp
    const int4 b = __ldg(B.list + ((size_t)(c / kTpp) * F.n + i) * kTpp + c % kTpp);
    if (b.x >= 0) use(b.x);
    if (b.y >= 0) use(b.y);
    if (b.z >= 0) use(b.z);
    if (b.w >= 0) use(b.w);
  }
}

// The solver's block: 4 x 256 threads per SM at 64 registers.  Both solves of 262,144 particles:
// 702 us, with 5 blocks (48 registers) 845, with 2 x 512 threads 684 but 16,384 particles 14 %
// slower (fewer SMs have a block).
constexpr int kSolveThreads = 256, kSolveBlocks = 4;

// What a pair needs of its neighbor: a float4 record with two more floats, or with one.
struct PairRec {
  float4 a;
  float2 q;
};
struct SweepRec {
  float4 a;
  float f;
};

// Lanes that share one wall's candidates: walls are few, so a wall per thread left its chain
// of ~81 candidate loads on the critical path of every sweep.
constexpr int kWallLanes = 8;

// The fluid neighbors of wall b at xb, shared by kWallLanes lanes: use(j) for every fluid
// particle that passes the wall-side pair test, from the wall's list (kCells; a chunk is
// filled up with -1) or from the cells around it.
template <typename Use>
__device__ __forceinline__ void wall_candidates(const FluidView& F, const sph_grid& g, const SphParams& P, float2 xb,
                                                int sub, Use&& use) {
  const float fcx = ceilf(__fdiv_rn(__fsub_rn(xb.x, g.qmin[0]), g.hmax));
  const float fcy = ceilf(__fdiv_rn(__fsub_rn(xb.y, g.qmin[1]), g.hmax));
  if (!(grid_ok(g, P.cell_capacity) && fcx > -1e9f && fcx < 1e9f && fcy > -1e9f && fcy < 1e9f)) return;
  for_each_member<kWallLanes>(F.cell_start, g, P.search_radius, (int)fcx, (int)fcy, sub, [&](int j) {
    const float2 xj = __ldg(F.x + j);
    if (dist2_ref(xb.x, xb.y, xj.x, xj.y) <= P.thr) use(j);
  });
}

template <bool kCells, typename Use>
__device__ __forceinline__ void wall_fluid_pairs(int b, const FluidView& F, const sph_grid& g, const SphParams& P,
                                                 const DfsphBufs& B, float2 xb, int sub, Use&& use) {
  const int chunks = kCells ? __ldg(B.wchunks + b) : -1;
  if (chunks < 0) {
    wall_candidates(F, g, P, xb, sub, use);
    return;
  }
  for (int c = sub; c < chunks; c += kWallLanes) {
    const int4 j = __ldg(B.wlist + (size_t)b * B.wall_chunks + c);
    if (j.x >= 0) use(j.x);
    if (j.y >= 0) use(j.y);
    if (j.z >= 0) use(j.z);
    if (j.w >= 0) use(j.w);
  }
}

// ---------------------------------------------------------------- densities
// The neighbor list of particle i while it is made: neighbors enter at the end of `four`, which
// is stored whenever it holds four new ones.
struct ListWriter {
  const DfsphBufs& B;
  int i, n, shift, k;   // 1 << shift lanes per particle
  int4 four;
  __device__ __forceinline__ void store(int c) {
    if (c < B.list_chunks) B.list[(((size_t)(c >> shift) * n + i) << shift) + (c & ((1 << shift) - 1))] = four;
  }
  __device__ __forceinline__ void add(int j) {
    four = make_int4(four.y, four.z, four.w, j);
    if ((++k & 3) == 0) store(k / 4 - 1);
  }
  __device__ __forceinline__ void fill_up(int j) {   // ends the list of one kind on a whole chunk
    while (k & 3) add(j);
  }
};

// The density sum rho_fluid of particle i and its neighbors' list, one test per candidate; the
// sum has k_nl_count's terms in its order (the solver's source 1 - rho would turn another
// order's rounding into relative errors of 1e-5 in the pressure).
__device__ __forceinline__ float search_body(int i, const FluidView& F, const sph_grid& g, const SphParams& P,
                                             float c_w, ListWriter& out) {
  int cx, cy;
  cell_of(F.keys[i], g, &cx, &cy);
  const float2 xi = F.x[i];
  const int r = P.search_radius;
  const int x0 = max(cx - r, 0), x1 = min(cx + r, g.cells_x - 1);
  const int y0 = max(cy - r, 0), y1 = min(cy + r, g.cells_y - 1);
  float acc = 0.f;
  for (int yy = y0; yy <= y1 && x0 <= x1; ++yy) {
    const int row = yy * g.cells_x;
    const int b = __ldg(F.cell_start + row + x0), e = __ldg(F.cell_start + row + x1 + 1);
    for (int c = b; c < e; c += 32) {
      uint32_t w = segment_mask_density(F.x, F.area, c, e, xi.x, xi.y, P.thr, P.inv_h, acc);
      while (w) {
        out.add(c - 1 + __ffs(w));
        w &= w - 1;
      }
    }
  }
  return acc * c_w;
}

// fluid: rho = rho_fluid (kCells: summed here while the neighbor lists are made; else from the
// count pass) + sum_b W A_b  (solidBoundary.py:522-549)
template <bool kCells>
__global__ void __launch_bounds__(128) k_dfsph_fluid_density(FluidView F, WallView W, const sph_grid* __restrict__ gp,
                                                             SphParams P, float c_w, int lanes,
                                                             const float* __restrict__ rho_fluid, DfsphBufs B) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= F.n) return;
  const sph_grid g = *gp;
  ListWriter out{B, i, F.n, 31 - __clz(lanes), 0, make_int4(i, i, i, i)};
  float rf;
  int fluid_chunks = 0;
  if constexpr (kCells) {
    rf = search_body(i, F, g, P, c_w, out);
    if (rho_fluid) rf = rho_fluid[i];
    out.fill_up(i);
    fluid_chunks = out.k / 4;
  } else {
    rf = rho_fluid[i];
  }
  float rw = 0.f;
  if (W.n > 0) {
    int cx, cy;
    cell_of(F.keys[i], g, &cx, &cy);
    const float2 xi = F.x[i];
    const float thr = P.thr;
    const auto wall = [&](int b, float2 xb, float area) {
      const Geo e = geo(xb.x, xb.y, xi.x, xi.y, P.inv_h);
      rw += kW(e.q, P.c_w) * area;
      if (kCells) out.add(b);
    };
    if constexpr (kCells) {   // the walls of a row tested together: the particles beside walls end last
      struct At {
        int b;
        float2 x;
        float area;
      };
      for_each_wall_by_four(
          W, g, P.search_radius, cx, cy, xi.x, xi.y, thr, [&](int b) { return At{b, __ldg(W.x + b), __ldg(W.area + b)}; },
          [&](const At& a) { wall(a.b, a.x, a.area); });
    } else {
      for_each_wall(W, g, P.search_radius, cx, cy, xi.x, xi.y, thr, [&](int b, float2 xb) { wall(b, xb, W.area[b]); });
    }
  }
  if constexpr (kCells) {
    out.fill_up(-1);
    const int all = out.k / 4;
    B.chunks[i] = all <= B.list_chunks ? fluid_chunks + 256 * (all - fluid_chunks) : -1;
  }
  const float A = F.area[i];
  const float r = rf + rw;
  B.rho[i] = r;
  B.vol[i] = A / rf;
  B.aact[i] = A / r;
}

// walls: rho_b = min(term_b + sum_f W A_f, 1), A_b^act = A_b / rho_b (kCells: and the wall's list
// of fluid neighbors, each lane's where its group's lanes before it have placed theirs)
template <bool kCells>
__global__ void __launch_bounds__(128) k_dfsph_wall_density(FluidView F, WallView W, const sph_grid* __restrict__ gp,
                                                            SphParams P, DfsphBufs B) {
  const int b = (blockIdx.x * blockDim.x + threadIdx.x) / kWallLanes, sub = threadIdx.x % kWallLanes;
  const sph_grid g = *gp;
  float s = 0.f;
  int found = 0;
  const float2 xb = b < W.n ? W.x[b] : make_float2(0.f, 0.f);
  if (b < W.n)
    wall_candidates(F, g, P, xb, sub, [&](int j) {
      const float2 xj = __ldg(F.x + j);
      const Geo e = geo(xb.x, xb.y, xj.x, xj.y, P.inv_h);
      s += kW(e.q, P.c_w) * F.area[j];
      ++found;
    });
  s = lane_sum<kWallLanes>(s);
  if constexpr (kCells) {
    int at = found, all = found;   // neighbors of the lanes up to this one, and of the group
#pragma unroll
    for (int o = 1; o < kWallLanes; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, at, o, kWallLanes);
      if (sub >= o) at += v;
      all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    at -= found;
    if (b < W.n) {
      int32_t* list = reinterpret_cast<int32_t*>(B.wlist + (size_t)b * B.wall_chunks);
      if (all <= 4 * B.wall_chunks) {
        wall_candidates(F, g, P, xb, sub, [&](int j) { list[at++] = j; });
        for (int k = all + sub; k < (all + 3) / 4 * 4; k += kWallLanes) list[k] = -1;
      }
      if (sub == 0) B.wchunks[b] = all <= 4 * B.wall_chunks ? (all + 3) / 4 : -1;
    }
  }
  if (b >= W.n || sub != 0) return;
  const float rb = fminf(B.wterm[b] + s, 1.0f);
  B.wrho[b] = rb;
  B.waact[b] = W.area[b] / rb;
}

// static wall-wall density term: sum over wall neighbors of W * A_b' (solidBoundary.py:180-200)
__global__ void __launch_bounds__(128) k_wall_wall_term(WallView W, const sph_grid* __restrict__ gp, SphParams P,
                                                        float* __restrict__ term) {
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= W.n) return;
  const sph_grid g = *gp;
  const float2 xb = W.x[b];
  float fcx = ceilf(__fdiv_rn(__fsub_rn(xb.x, g.qmin[0]), g.hmax));
  float fcy = ceilf(__fdiv_rn(__fsub_rn(xb.y, g.qmin[1]), g.hmax));
  float s = 0.f;
  if (grid_ok(g, P.cell_capacity) && fcx > -1e9f && fcx < 1e9f && fcy > -1e9f && fcy < 1e9f) {
    const float thr = P.thr;
    for_each_wall(W, g, P.search_radius, (int)fcx, (int)fcy, xb.x, xb.y, thr, [&](int c, float2 xc) {
      const Geo e = geo(xb.x, xb.y, xc.x, xc.y, P.inv_h);
      s += kW(e.q, P.c_w) * W.area[c];
    });
  }
  term[b] = s;
}

// ---------------------------------------------------------------- solver set-up
// The spiky gradient of pair (i, j) as gs * d with d = x_i - x_j: spikyGrad = e kGS(q), e =
// d / r, so gs = kGS(q) / r, from one reciprocal square root (0 when r < 1e-7, where the
// reference's e is zero).
__device__ __forceinline__ float spiky_gd(float r2, const SphParams& P) {
  if (!(r2 >= 1e-14f)) return 0.f;
  const float rs = rsqrt_normal(r2);
  return kGS(r2 * rs * P.inv_h, P.c_s) * rs;
}

// The Wendland gradient the same way: gradW = e kGW(q) = gw * d.
__device__ __forceinline__ float wendland_gd(float r2, const SphParams& P) {
  if (!(r2 >= 1e-14f)) return 0.f;
  const float rs = rsqrt_normal(r2);
  return kGW(r2 * rs * P.inv_h, P.c_g) * rs;
}

// v* = v + dt a, and the pair records of the preparation pass: rec_a = (x, y, v*),
// rec_p = (A_act, A_act^2 / (A rho0)) (both rewritten by the solve before it reads them).
__global__ void k_dfsph_vstar(FluidView F, SphParams P, DfsphBufs B, const float2* __restrict__ acc,
                              const float* __restrict__ dt_ptr) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= F.n) return;
  const float dt = *dt_ptr;
  const float2 a = acc[i], u = F.v[i], x = F.x[i];
  const float2 vs = make_float2(u.x + dt * a.x, u.y + dt * a.y);
  B.vstar[i] = vs;
  B.rec_a[i] = make_float4(x.x, x.y, vs.x, vs.y);
  const float aa = B.aact[i];
  B.rec_p[i] = make_float4(aa, aa * aa / (F.area[i] * P.rho0), 0.f, 0.f);
}

// The pair records of the viscosity pass: rec_a = (x, y, v), rec_p = (V, rho rho0).
__global__ void k_dfsph_visc_records(FluidView F, SphParams P, DfsphBufs B) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= F.n) return;
  const float2 x = F.x[i], u = F.v[i];
  B.rec_a[i] = make_float4(x.x, x.y, u.x, u.y);
  B.rec_p[i] = make_float4(B.vol[i], B.rho[i] * P.rho0, 0.f, 0.f);
}

// alpha (dfsph.py:58-83 + solidBoundary.py:443-479) and source (dfsph.py:85-100, 154-161 +
// solidBoundary.py:481-520) per fluid particle.  Wall terms only in the density solve.
template <bool kCells, int kTpp>
__global__ void __launch_bounds__(128) k_dfsph_prepare(FluidView F, WallView W, const sph_grid* __restrict__ gp,
                                                       SphParams P, DfsphBufs B, const float* __restrict__ dt_ptr,
                                                       int density) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) / kTpp, sub = threadIdx.x % kTpp;
  const bool live = row < F.n;
  const int i = live ? row : F.n - 1;   // lanes past the last particle only take part in the sums
  const float dt = *dt_ptr;
  const float4 me = B.rec_a[i];
  const float2 xi = make_float2(me.x, me.y);
  const float2 vi = make_float2(me.z, me.w);
  float k1x = 0.f, k1y = 0.f, k2 = 0.f, src = 0.f;
  const sph_grid g = *gp;
  const auto load = [&](int j) {   // (x, y, v*) and (A_act, A_act^2 / m)
    return PairRec{__ldg(B.rec_a + j), __ldg(reinterpret_cast<const float2*>(B.rec_p + j))};
  };
  if (live) fluid_pairs<kCells, kTpp>(i, F, g, P, B, xi.x, xi.y, sub, load, [&](const PairRec& rec) {
    const float4 rj = rec.a;
    const float2 qj = rec.q;
    const float dx = xi.x - rj.x, dy = xi.y - rj.y;
    const float gd = spiky_gd(dx * dx + dy * dy, P);
    const float gx = gd * dx, gy = gd * dy;
    const float aj = qj.x;
    k1x += aj * gx;
    k1y += aj * gy;
    k2 += qj.y * (gx * gx + gy * gy);
    src += -dt * aj * ((vi.x - rj.z) * gx + (vi.y - rj.w) * gy);
  });
  float w1x = 0.f, w1y = 0.f, w2 = 0.f, wsrc = 0.f;
  if (density && W.n > 0) {
    if (live) wall_pairs<kCells, kTpp>(i, F, W, g, P, B, xi.x, xi.y, sub, [&](int b) {
      const float2 xb = __ldg(W.x + b);
      const Geo e = geo(xb.x, xb.y, xi.x, xi.y, P.inv_h);   // e = (x_b - x_f)/r
      const float gs = kGS(e.q, P.c_s);
      const float gx = gs * e.ex, gy = gs * e.ey;
      const float ab = B.waact[b], Ab = W.area[b];
      w1x += ab * gx;
      w1y += ab * gy;
      w2 += (ab * ab / (Ab * P.rho0)) * (gx * gx + gy * gy);
      wsrc += ab * ((0.f - vi.x) * gx + (0.f - vi.y) * gy);
    });
  }
  k1x = lane_sum<kTpp>(k1x) + lane_sum<kTpp>(w1x);
  k1y = lane_sum<kTpp>(k1y) + lane_sum<kTpp>(w1y);
  k2 = lane_sum<kTpp>(k2) + lane_sum<kTpp>(w2);
  src = lane_sum<kTpp>(src);
  wsrc = lane_sum<kTpp>(wsrc);
  if (!live || sub != 0) return;
  const float aa = B.aact[i], Ai = F.area[i];
  const float fac = -dt * dt * aa;
  float alpha = fac / (Ai * P.rho0) * (k1x * k1x + k1y * k1y) + fac * k2;
  alpha = fminf(fmaxf(alpha, -1.0f), -1e-7f);
  B.alpha[i] = alpha;
  float s = src + (-dt) * wsrc;
  B.source[i] = density ? 1.0f - B.rho[i] + s : s;
  B.p[i] = 0.f;
}

// wall alpha and source (PBSPH branch, solidBoundary.py:463-466, 499-503)
template <bool kCells>
__global__ void __launch_bounds__(128) k_dfsph_wall_prepare(FluidView F, WallView W, const sph_grid* __restrict__ gp,
                                                            SphParams P, DfsphBufs B, const float* __restrict__ dt_ptr) {
  const int b = (blockIdx.x * blockDim.x + threadIdx.x) / kWallLanes, sub = threadIdx.x % kWallLanes;
  const float dt = *dt_ptr;
  float t = 0.f, s = 0.f;
  if (b < W.n) {
    const float2 xb = W.x[b];
    wall_fluid_pairs<kCells>(b, F, *gp, P, B, xb, sub, [&](int j) {
      const float2 xj = __ldg(F.x + j);
      const Geo e = geo(xb.x, xb.y, xj.x, xj.y, P.inv_h);   // e = (x_b - x_f)/r
      const float gs = kGS(e.q, P.c_s);
      const float gx = gs * e.ex, gy = gs * e.ey;
      const float af = B.aact[j];
      t += (af * af / (F.area[j] * P.rho0)) * (gx * gx + gy * gy);
      const float2 vj = B.vstar[j];
      s += af * ((0.f - vj.x) * gx + (0.f - vj.y) * gy);
    });
  }
  t = lane_sum<kWallLanes>(t);
  s = lane_sum<kWallLanes>(s);
  if (b >= W.n || sub != 0) return;
  const float ab = B.waact[b];
  B.walpha[b] = fminf(-dt * dt * ab * t, -0.0001f * P.h * P.h);
  B.wsource[b] = 1.0f - B.wrho[b] + (-dt) * s;
  B.wp[b] = 0.f;
}

// ---------------------------------------------------------------- solver phases

// predicted pressure acceleration of fluid particle i (dfsph.py:25-42 + solidBoundary.py:310-403),
// the fluid pairs from the records rec_p = (x, y, m, p / rho^2); lane `sub` of kTpp sums
// its share of the row and (wall) of the walls, and every lane returns the whole.
template <bool kCells, int kTpp>
__device__ __forceinline__ float2 pressure_accel(const FluidView& F, const WallView& W, const sph_grid& g,
                                                 const SphParams& P, const DfsphBufs& B, int i, int sub, bool live,
                                                 bool walls) {
  float ax = 0.f, ay = 0.f, wx = 0.f, wy = 0.f;
  if (live) {
    const float4 me = B.rec_p[i];
    const float ppi = me.w;
    fluid_pairs<kCells, kTpp>(i, F, g, P, B, me.x, me.y, sub, [&](int j) { return B.rec_p[j]; },
                              [&](const float4& rj) {
      const float dx = me.x - rj.x, dy = me.y - rj.y;
      const float f = -rj.z * (ppi + rj.w) * spiky_gd(dx * dx + dy * dy, P);
      ax += f * dx;
      ay += f * dy;
    });
    if (walls) {
      wall_pairs<kCells, kTpp>(i, F, W, g, P, B, me.x, me.y, sub, [&](int b) {
        const float2 xb = __ldg(W.x + b);
        // spiky(e_bf) = gd (x_b - x_f), used negated
        const float dx = xb.x - me.x, dy = xb.y - me.y;
        const float gd = spiky_gd(dx * dx + dy * dy, P);
        const float rb = B.wrho[b] * P.rho0;
        const float pb = B.wp[b] / (rb * rb);
        const float f = (W.area[b] * P.rho0) * (ppi + pb) * gd;
        wx += f * dx;
        wy += f * dy;
      });
    }
  }
  ax = lane_sum<kTpp>(ax);
  ay = lane_sum<kTpp>(ay);
  if (walls) {
    ax += lane_sum<kTpp>(wx);
    ay += lane_sum<kTpp>(wy);
  }
  return make_float2(ax, ay);
}

// The particles of the grid's groups of kTpp lanes: group q of the grid takes particles q,
// q + groups, ...; every lane of a warp stays in the loop while one of its groups has a
// particle (`live`), so that the sums' shuffles meet.
template <int kTpp, typename Fn>
__device__ __forceinline__ void for_each_row(int n, int groups, Fn&& fn) {
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int in_warp = (threadIdx.x & 31) / kTpp;
  for (int q = (tid / 32) * (32 / kTpp); q < n; q += groups) fn(q + in_warp, q + in_warp < n);
}

template <bool kCells, int kTpp>
__global__ void __launch_bounds__(kSolveThreads, kSolveBlocks) k_dfsph_solve(FluidView F, WallView W, const sph_grid* __restrict__ gp,
                                                     SphParams P, DfsphBufs B, const float* __restrict__ dt_ptr,
                                                     int density, int min_iters, int max_iters, float thr_err,
                                                     float omega_f, float omega_b, int32_t* status) {
  cg::grid_group grid = cg::this_grid();
  const sph_grid g = *gp;
  const float dt = *dt_ptr;
  const bool walls = density && W.n > 0;
  const int tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int nthreads = gridDim.x * blockDim.x;
  const int groups = nthreads / kTpp, sub = threadIdx.x % kTpp;
  const double count = (double)F.n + (walls ? (double)W.n : 0.0);
  __shared__ double s_part[kSolveThreads], s_err;
  // the pair records: positions, masses and dt^2 A_act are fixed during the solve
  for (int i = tid; i < F.n; i += nthreads) {
    const float2 xi = F.x[i];
    const float ri = B.rho[i] * P.rho0;
    B.rec_p[i] = make_float4(xi.x, xi.y, F.area[i] * P.rho0, B.p[i] / (ri * ri));
    B.fdt[i] = dt * dt * B.aact[i];
  }
  grid.sync();
  double err = 0.0;
  int it = 0;
  while ((it < min_iters || err > (double)thr_err) && it <= max_iters) {
    // phase A: predicted acceleration from the current pressures
    for_each_row<kTpp>(F.n, groups, [&](int i, bool live) {
      const float2 a = pressure_accel<kCells, kTpp>(F, W, g, P, B, i, sub, live, walls);
      if (live && sub == 0) {
        B.pa[i] = a;
        const float4 me = B.rec_p[i];
        B.rec_a[i] = make_float4(me.x, me.y, a.x, a.y);
      }
    });
    grid.sync();
    // phase B: pressure sums, residuals, relaxed Jacobi updates, error partials
    double local = 0.0;
    for_each_row<kTpp>(F.n, groups, [&](int i, bool live) {
      float ks = 0.f, wks = 0.f;
      if (live) {
        const float4 me = B.rec_a[i];
        const auto load = [&](int j) { return SweepRec{B.rec_a[j], B.fdt[j]}; };
        fluid_pairs<kCells, kTpp>(i, F, g, P, B, me.x, me.y, sub, load, [&](const SweepRec& rec) {
          const float4 rj = rec.a;
          const float dx = me.x - rj.x, dy = me.y - rj.y;
          ks += rec.f * ((me.z - rj.z) * dx + (me.w - rj.w) * dy) * spiky_gd(dx * dx + dy * dy, P);
        });
        if (walls) {
          wall_pairs<kCells, kTpp>(i, F, W, g, P, B, me.x, me.y, sub, [&](int b) {
            const float2 xb = __ldg(W.x + b);
            const float dx = xb.x - me.x, dy = xb.y - me.y;
            const float gd = spiky_gd(dx * dx + dy * dy, P);
            wks -= dt * dt * B.waact[b] * gd * (me.z * dx + me.w * dy);
          });
        }
      }
      ks = lane_sum<kTpp>(ks);
      if (walls) ks += lane_sum<kTpp>(wks);
      if (live && sub == 0) {
        const float r = ks - B.source[i];
        B.res[i] = r;
        float pn = B.p[i] - omega_f * r / B.alpha[i];
        if (density) pn = fmaxf(pn, 0.f);
        if (!isfinite(pn)) flag(status, SPH_FLAG_NONFINITE);
        B.p[i] = pn;
        const float ri = B.rho[i] * P.rho0;
        B.rec_p[i].w = pn / (ri * ri);
        local += (double)fmaxf(r, -thr_err);
      }
    });
    if (walls) {
      // the last groups take the walls: the first ones may have had a particle more
      const int wsub = threadIdx.x % kWallLanes;
      for (int q = (nthreads - 1 - tid) / 32 * (32 / kWallLanes); q < W.n; q += nthreads / kWallLanes) {
        const int b = q + (threadIdx.x & 31) / kWallLanes;
        float bks = 0.f;
        if (b < W.n) {
          const float2 xb = W.x[b];
          wall_fluid_pairs<kCells>(b, F, g, P, B, xb, wsub, [&](int j) {
            const float4 rj = B.rec_a[j];
            const float dx = xb.x - rj.x, dy = xb.y - rj.y;
            bks -= B.fdt[j] * spiky_gd(dx * dx + dy * dy, P) * (rj.z * dx + rj.w * dy);
          });
        }
        bks = lane_sum<kWallLanes>(bks);
        if (b < W.n && wsub == 0) {
          const float rb = bks - B.wsource[b];
          B.wres[b] = rb;
          B.wp[b] = fmaxf(B.wp[b] - omega_b * rb / B.walpha[b], 0.f);
          local += (double)fmaxf(rb, -thr_err);
        }
      }
    }
    // block partial of the error, then the mean over all blocks' partials: one warp of the block
    // sums each (every SM's FP64 pipe is shared by its warps, and a sum repeated in each of
    // them took 5 us of an iteration), always in the same order, so that every block forms the
    // same double and takes the same loop decision
    s_part[threadIdx.x] = local;
    __syncthreads();
    if (threadIdx.x < 32) {
      double t = 0.0;
#pragma unroll
      for (int w = 0; w < kSolveThreads; w += 32) t += s_part[w + threadIdx.x];
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (threadIdx.x == 0) B.partials[blockIdx.x] = t;
    }
    grid.sync();
    if (threadIdx.x < 32) {
      double t = 0.0;
      for (int k = threadIdx.x; k < (int)gridDim.x; k += 32) t += B.partials[k];
      for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
      if (threadIdx.x == 0) s_err = t / count;
    }
    __syncthreads();
    err = s_err;
    if (tid == 0) B.errors[it] = (float)err;
    ++it;
  }
  // final acceleration with the converged pressures (dfsph.py:303-309)
  for_each_row<kTpp>(F.n, groups, [&](int i, bool live) {
    const float2 a = pressure_accel<kCells, kTpp>(F, W, g, P, B, i, sub, live, walls);
    if (live && sub == 0) B.pa[i] = a;
  });
  if (tid == 0) *B.iters = it;
}

// ---------------------------------------------------------------- viscosity (DFSPH steps 11-12)
// artificial viscosity with walls and laminar viscosity; V = A / rho_fluid_only (the volume
// set before the wall density is added, src/dfsph.py:151-163), rho = rho~ rho0 incl. walls.
template <bool kCells, int kTpp>
__global__ void __launch_bounds__(128) k_dfsph_viscosity(FluidView F, WallView W, const sph_grid* __restrict__ gp,
                                                         SphParams P, DfsphBufs B, float2* __restrict__ acc) {
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) / kTpp, sub = threadIdx.x % kTpp;
  const bool live = row < F.n;
  const int i = live ? row : F.n - 1;   // lanes past the last particle only take part in the sums
  const float4 me = B.rec_a[i];
  const float2 xi = make_float2(me.x, me.y), vi = make_float2(me.z, me.w);
  const float rhoi = B.rho[i] * P.rho0;
  float vax = 0.f, vay = 0.f, lax = 0.f, lay = 0.f;
  const sph_grid g = *gp;
  const auto load = [&](int j) {   // (x, y, v) and (V, rho rho0)
    return PairRec{__ldg(B.rec_a + j), __ldg(reinterpret_cast<const float2*>(B.rec_p + j))};
  };
  if (live) fluid_pairs<kCells, kTpp>(i, F, g, P, B, xi.x, xi.y, sub, load, [&](const PairRec& rec) {
    const float4 rj = rec.a;
    const float2 qj = rec.q;
    const float2 vj = make_float2(rj.z, rj.w);
    const float Vj = qj.x, rhoj = qj.y;
    const float dx = xi.x - rj.x, dy = xi.y - rj.y;
    const float d2 = dx * dx + dy * dy;
    const float gd = wendland_gd(d2, P);
    const float gx = gd * dx, gy = gd * dy;
    const float ux = vj.x - vi.x, uy = vj.y - vi.y;
    const float rx = -dx, ry = -dy;
    const float r2 = rx * rx + ry * ry + P.eps;
    // one correctly rounded reciprocal each for r^2 + eps and rho_i + rho_j, shared by both terms
    const float ir2 = __frcp_rn(r2), irs = __frcp_rn(rhoi + rhoj);
    const float mj = rhoj * Vj, mr = mj * irs * ir2;
    const float vf = fminf(ux * rx + uy * ry, 0.f) * mr;
    vax += vf * gx;
    vay += vf * gy;
    const float term = 8.0f * rhoi * P.kinematic * (rx * gx + ry * gy) * irs * mr;
    lax -= term * (vi.x - vj.x);
    lay -= term * (vi.y - vj.y);
  });
  float vwx = 0.f, vwy = 0.f;
  if (W.n > 0 && P.boundary_diffusion) {
    if (live) wall_pairs<kCells, kTpp>(i, F, W, g, P, B, xi.x, xi.y, sub, [&](int b) {
      const float2 xb = __ldg(W.x + b);
      const Geo e = geo(xi.x, xi.y, xb.x, xb.y, P.inv_h);
      const float gw = kGW(e.q, P.c_g);
      const float gx = gw * e.ex, gy = gw * e.ey;
      const float rb = B.wrho[b];
      const float Vb = W.area[b] / rb, rhob = rb * P.rho0;
      const float rx = -e.dx, ry = -e.dy;
      const float r2 = rx * rx + ry * ry + P.eps;
      const float pij = fminf(-vi.x * rx - vi.y * ry, 0.f) / r2;
      const float vf = pij * Vb * rhob / (rhoi + rhob);
      vwx += vf * gx;
      vwy += vf * gy;
    });
  }
  vax = lane_sum<kTpp>(vax);
  vay = lane_sum<kTpp>(vay);
  lax = lane_sum<kTpp>(lax);
  lay = lane_sum<kTpp>(lay);
  vwx = lane_sum<kTpp>(vwx);
  vwy = lane_sum<kTpp>(vwy);
  if (!live || sub != 0) return;
  float2 a = acc[i];
  a.x += P.visc_k * vax + P.visc_k * vwx + lax;
  a.y += P.visc_k * vay + P.visc_k * vwy + lay;
  acc[i] = a;
}

// a += pa (fluidAcceleration += fluidPredAccel, src/dfsph.py:179, 185)
__global__ void k_add2(int n, const float2* __restrict__ b, float2* __restrict__ a) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float2 x = a[i], y = b[i];
  a[i] = make_float2(x.x + y.x, x.y + y.y);
}

__global__ void k_fill2(int n, float gx, float gy, float2* __restrict__ a) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = make_float2(gx, gy);
}

// ---------------------------------------------------------------- adaptive dt (adaptiveDT.py:59-95)
__global__ void __launch_bounds__(256) k_dt_partials(int n, const float2* __restrict__ v, const float2* __restrict__ a,
                                                     float h, float* __restrict__ part) {
  float vmax = 0.f, amin = INFINITY;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float2 u = v[i], b = a[i];
    vmax = fmaxf(vmax, sqrtf(u.x * u.x + u.y * u.y));
    amin = fminf(amin, sqrtf(h / sqrtf(b.x * b.x + b.y * b.y)));
  }
  for (int o = 16; o > 0; o >>= 1) {
    vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    amin = fminf(amin, __shfl_xor_sync(0xffffffffu, amin, o));
  }
  __shared__ float sv[8], sa[8];
  if ((threadIdx.x & 31) == 0) {
    sv[threadIdx.x >> 5] = vmax;
    sa[threadIdx.x >> 5] = amin;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
      vmax = fmaxf(vmax, sv[w]);
      amin = fminf(amin, sa[w]);
    }
    part[2 * blockIdx.x] = vmax;
    part[2 * blockIdx.x + 1] = amin;
  }
}

__global__ void k_dt_final(int nparts, const float* __restrict__ part, float h, float kinematic, float cfl, float c0,
                           int acoustic_from_c0, float dt_min, float dt_max, float* __restrict__ dt) {
  // one warp over the parts (one thread took 14 us of every step for the 304 of a large scene)
  float vmax = 0.f, amin = INFINITY;
  for (int k = threadIdx.x; k < nparts; k += 32) {
    vmax = fmaxf(vmax, part[2 * k]);
    amin = fminf(amin, part[2 * k + 1]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    vmax = fmaxf(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    amin = fminf(amin, __shfl_xor_sync(0xffffffffu, amin, o));
  }
  if (threadIdx.x != 0) return;
  const double visc = 0.125 * (double)h * h / kinematic;
  const double accdt = 0.25 * (double)amin;
  const double vdt = acoustic_from_c0 ? (double)cfl * h / c0 : 0.4 * (double)h / vmax;
  double m = dt_max;
  if (dt_min != 0.f) {
    m = fmin(m, visc);
    m = fmin(m, accdt);
    if (!isnan(vdt)) m = fmin(m, vdt);
  }
  const double target = m > dt_min ? m : dt_min;
  const double cur = *dt;
  *dt = (float)fmin(fmax(target, cur * 0.5), cur * 1.05);
}

}  // namespace sph

using namespace sph;

// Lanes per particle: as many as keep the GPU's ~155 k resident solver threads busy without a
// lane's chunk of the list costing more than it hides.  Both pressure solves of a settling block
// (16 sweeps), us with 8 / 4 / 2 / 1 lanes: 4,096 particles 221 / 241 / 271 / 350; 16,384:
// 270 / 246 / 257 / 324; 65,536: - / - / 365 / 406; 131,044: 747 / 605 / 529 / 553 (before
// the error's sum was cut to one warp); 262,144: - / - / 724 / 702.
static int dfsph_lanes(int64_t n) { return n <= 8192 ? 8 : n <= 32768 ? 4 : n <= 196608 ? 2 : 1; }

// Chunks for a list_capacity (0: kListChunks).
static int list_chunks(int32_t capacity) {
  return capacity <= 0 ? kListChunks : std::min((capacity + 3) / 4, kMaxListChunks);
}

// List slots (int4) of n particles with c chunks: a particle's chunks are dealt to its lanes, so their
// number is rounded up to the lanes (chunk k < c lies below (k / lanes + 1) lanes n).
static size_t list_slots(int64_t n, int c) {
  const int lanes = dfsph_lanes(n);
  return (size_t)n * ((c + lanes - 1) / lanes * lanes);
}

// n: the fluid count, which places the pair records (and, with pairs from the cell rows, the
// neighbor lists behind them) inside b->records.
static DfsphBufs to_bufs(const sph_dfsph_buffers* b, int64_t n, int64_t nb, bool cells) {
  DfsphBufs B;
  B.rho = b->rho;
  B.vol = b->volume;
  B.aact = b->actual_area;
  B.vstar = reinterpret_cast<float2*>(b->vstar);
  B.alpha = b->alpha;
  B.source = b->source;
  B.p = b->pressure;
  B.pa = reinterpret_cast<float2*>(b->pred_accel);
  B.res = b->residual;
  B.wrho = b->wall_rho;
  B.waact = b->wall_actual_area;
  B.walpha = b->wall_alpha;
  B.wsource = b->wall_source;
  B.wp = b->wall_pressure;
  B.wres = b->wall_residual;
  B.wterm = b->wall_density_term;
  B.partials = b->partials;
  B.errors = b->errors;
  B.iters = b->iters;
  B.rec_p = b->records ? reinterpret_cast<float4*>(b->records) : nullptr;
  B.rec_a = B.rec_p ? B.rec_p + n : nullptr;
  B.fdt = B.rec_p ? b->records + 8 * n : nullptr;
  // the lists start 16-byte aligned: 9 n floats rounded up to a multiple of four
  B.list = cells && B.rec_p ? reinterpret_cast<int4*>(b->records + (9 * n + 3) / 4 * 4) : nullptr;
  B.list_chunks = cells ? list_chunks(b->list_capacity) : 0;
  B.wall_chunks = wall_chunks(B.list_chunks);
  B.wlist = B.list ? B.list + list_slots(n, B.list_chunks) : nullptr;
  B.chunks = B.list ? reinterpret_cast<int32_t*>(B.wlist + B.wall_chunks * nb) : nullptr;
  B.wchunks = B.list ? B.chunks + n : nullptr;
  return B;
}

// Pairs from the cell rows: the view has no CSR list.
static bool cell_rows(const sph_fluid_view* f) { return !f->offsets && !f->cols; }

// Runs the kernel variant of the view: kCells and, with pairs from the cell rows, its lanes.
#define SPH_DFSPH_VARIANT(cells, lanes, CALL)   \
  do {                                          \
    if (!(cells)) {                             \
      CALL(false, 1);                           \
    } else if ((lanes) == 1) {                  \
      CALL(true, 1);                            \
    } else if ((lanes) == 2) {                  \
      CALL(true, 2);                            \
    } else if ((lanes) == 4) {                  \
      CALL(true, 4);                            \
    } else {                                    \
      CALL(true, 8);                            \
    }                                           \
  } while (0)

// Cooperative grid size of k_dfsph_solve per GPU (resident blocks x SMs), computed on the
// first solve on that GPU; GPUs of one process may differ in SM count.
constexpr int kCoopMaxDevices = 64;
static int g_coop_blocks[kCoopMaxDevices][9] = {{0}};   // by lanes (0: CSR rows)
static std::mutex g_coop_mu;

extern "C" {

size_t sph_dfsph_records_count(int64_t n, int64_t nb, int32_t cell_rows) {
  if (n < 0 || nb < 0) return 0;
  if (!cell_rows) return (size_t)n * 9;
  const int c = list_chunks(cell_rows == 1 ? 0 : cell_rows);
  return (size_t)(9 * n + 3) / 4 * 4 + 4 * list_slots(n, c) + (size_t)n + (size_t)nb * (4 * wall_chunks(c) + 1);
}

size_t sph_dfsph_partials_count(void) { return (size_t)kNumSMs * 8; }

sph_status_t sph_dfsph_wall_wall_term(const sph_wall_view* walls, const sph_grid* grid, const sph_params* params,
                                      float* term, void* stream) {
  SPH_VIEW_CHECK(walls);
  SPH_REQUIRE(grid && params && term, "dfsph_wall_wall_term: bad arguments");
  if (walls->n == 0) return SPH_OK;
  k_wall_wall_term<<<grid_for(walls->n, 128), 128, 0, as_stream(stream)>>>(to_walls(walls), grid, to_params(params),
                                                                           term);
  SPH_CHECK_LAUNCH("dfsph_wall_wall_term");
  return SPH_OK;
}

sph_status_t sph_dfsph_densities(const sph_fluid_view* fluid, const sph_wall_view* walls, const sph_grid* grid,
                                 const sph_params* params, const float* rho_fluid, const sph_dfsph_buffers* bufs,
                                 void* stream) {
  SPH_VIEW_CHECK(fluid);
  SPH_VIEW_CHECK(walls);
  const bool cells = cell_rows(fluid);
  SPH_REQUIRE(grid && params && bufs && (cells || rho_fluid), "dfsph_densities: bad arguments");
  SPH_REQUIRE(!cells || (bufs->records && fluid->cell_start && fluid->keys &&
                         (reinterpret_cast<uintptr_t>(bufs->records) & 15) == 0),
              "dfsph_densities: pairs from the cell rows need keys, the cell table and 16-byte aligned records");
  cudaStream_t st = as_stream(stream);
  const FluidView F = to_fluid(fluid);
  const WallView W = to_walls(walls);
  const SphParams P = to_params(params);
  const DfsphBufs B = to_bufs(bufs, fluid->n, walls->n, cells);
  // as sph_nl_count scales its density sum
  const float c_w = (float)(7.0 / 3.14159265358979323846) / (params->support * params->support);
  if (fluid->n > 0) {
    if (cells)
      k_dfsph_fluid_density<true>
          <<<grid_for(fluid->n, 128), 128, 0, st>>>(F, W, grid, P, c_w, dfsph_lanes(fluid->n), rho_fluid, B);
    else
      k_dfsph_fluid_density<false><<<grid_for(fluid->n, 128), 128, 0, st>>>(F, W, grid, P, c_w, 1, rho_fluid, B);
  }
  if (walls->n > 0) {
    const int nb = grid_for(walls->n, 128 / kWallLanes);
    if (cells)
      k_dfsph_wall_density<true><<<nb, 128, 0, st>>>(F, W, grid, P, B);
    else
      k_dfsph_wall_density<false><<<nb, 128, 0, st>>>(F, W, grid, P, B);
  }
  SPH_CHECK_LAUNCH("dfsph_densities");
  return SPH_OK;
}

sph_status_t sph_dfsph_solve(const sph_fluid_view* fluid, const sph_wall_view* walls, const sph_grid* grid,
                             const sph_params* params, const sph_dfsph_buffers* bufs, const float* acc_in,
                             const float* dt, int32_t density, int32_t* status, void* stream) {
  SPH_VIEW_CHECK(fluid);
  SPH_VIEW_CHECK(walls);
  SPH_REQUIRE(grid && params && bufs && acc_in && dt, "dfsph_solve: bad arguments");
  const int n = (int)fluid->n;
  if (n == 0) return SPH_OK;
  cudaStream_t st = as_stream(stream);
  SPH_REQUIRE(bufs->records && (reinterpret_cast<uintptr_t>(bufs->records) & 15) == 0,
              "dfsph_solve: records must be a 16-byte aligned array of 9 n floats");
  FluidView F = to_fluid(fluid);
  WallView W = to_walls(walls);
  SphParams P = to_params(params);
  const bool cells = cell_rows(fluid);
  const int lanes = cells ? dfsph_lanes(n) : 1;
  DfsphBufs B = to_bufs(bufs, n, walls->n, cells);
  k_dfsph_vstar<<<grid_for(n, 256), 256, 0, st>>>(F, P, B, reinterpret_cast<const float2*>(acc_in), dt);
#define SPH_PREPARE(C, T) k_dfsph_prepare<C, T><<<grid_for(n, 128 / T), 128, 0, st>>>(F, W, grid, P, B, dt, density)
  SPH_DFSPH_VARIANT(cells, lanes, SPH_PREPARE);
#undef SPH_PREPARE
  if (density && W.n > 0) {
    const int nb = grid_for(W.n, 128 / kWallLanes);
    if (cells)
      k_dfsph_wall_prepare<true><<<nb, 128, 0, st>>>(F, W, grid, P, B, dt);
    else
      k_dfsph_wall_prepare<false><<<nb, 128, 0, st>>>(F, W, grid, P, B, dt);
  }
  const void* kernel = nullptr;
#define SPH_SOLVE(C, T) kernel = (const void*)k_dfsph_solve<C, T>
  SPH_DFSPH_VARIANT(cells, lanes, SPH_SOLVE);
#undef SPH_SOLVE
  SPH_CHECK_LAUNCH("dfsph_solve(prepare)");
  int dev = 0;
  cudaError_t de = cudaGetDevice(&dev);
  if (de != cudaSuccess || dev < 0 || dev >= kCoopMaxDevices) {
    set_error("dfsph_solve(device)", de);
    return SPH_ERR_CUDA;
  }
  int coop_blocks = 0;
  {
    std::lock_guard<std::mutex> lock(g_coop_mu);
    const int v = cells ? lanes : 0;
    if (g_coop_blocks[dev][v] == 0) {
      int per_sm = 0, sms = 0;
      cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kSolveThreads, 0);
      if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      if (e != cudaSuccess || per_sm < 1 || sms < 1) {
        set_error("dfsph_solve(occupancy)", e);
        return SPH_ERR_CUDA;
      }
      g_coop_blocks[dev][v] = std::min(per_sm, 8) * sms;
    }
    coop_blocks = g_coop_blocks[dev][v];
  }
  int blocks = std::min(coop_blocks, (int)sph_dfsph_partials_count());
  blocks = std::min(blocks, std::max(1, grid_for(n, kSolveThreads / lanes)));
  int density_i = density;
  int min_it = density ? params->min_density_iters : params->min_divergence_iters;
  int max_it = density ? params->max_density_iters : params->max_divergence_iters;
  float thr = density ? params->density_threshold : params->divergence_threshold;
  float omega_f = params->omega_fluid;
  float omega_b = params->omega_boundary;
  void* args[] = {&F, &W, (void*)&grid, &P, &B, (void*)&dt, &density_i, &min_it, &max_it, &thr, &omega_f, &omega_b,
                  (void*)&status};
  cudaError_t e = cudaLaunchCooperativeKernel(kernel, blocks, kSolveThreads, args, 0, st);
  if (e != cudaSuccess) {
    set_error("dfsph_solve(cooperative launch)", e);
    return SPH_ERR_CUDA;
  }
  return SPH_OK;
}

sph_status_t sph_dfsph_viscosity(const sph_fluid_view* fluid, const sph_wall_view* walls, const sph_grid* grid,
                                 const sph_params* params, const sph_dfsph_buffers* bufs, float* acc, void* stream) {
  SPH_VIEW_CHECK(fluid);
  SPH_VIEW_CHECK(walls);
  SPH_REQUIRE(grid && params && bufs && acc, "dfsph_viscosity: bad arguments");
  if (fluid->n == 0) return SPH_OK;
  SPH_REQUIRE(bufs->records && (reinterpret_cast<uintptr_t>(bufs->records) & 15) == 0,
              "dfsph_viscosity: records must be a 16-byte aligned array of 9 n floats");
  const FluidView F = to_fluid(fluid);
  const SphParams P = to_params(params);
  const bool cells = cell_rows(fluid);
  const DfsphBufs B = to_bufs(bufs, fluid->n, walls->n, cells);
  const WallView W = to_walls(walls);
  const int lanes = cells ? dfsph_lanes(fluid->n) : 1;
  cudaStream_t st = as_stream(stream);
  k_dfsph_visc_records<<<grid_for(fluid->n, 256), 256, 0, st>>>(F, P, B);
#define SPH_VISCOSITY(C, T)                                                                  \
  k_dfsph_viscosity<C, T><<<grid_for(fluid->n, 128 / T), 128, 0, st>>>(F, W, grid, P, B,     \
                                                                       reinterpret_cast<float2*>(acc))
  SPH_DFSPH_VARIANT(cells, lanes, SPH_VISCOSITY);
#undef SPH_VISCOSITY
  SPH_CHECK_LAUNCH("dfsph_viscosity");
  return SPH_OK;
}

sph_status_t sph_add_float2(int64_t n, const float* b, float* a, void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && a && b, "add_float2: bad arguments");
  if (n == 0) return SPH_OK;
  k_add2<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>((int)n, reinterpret_cast<const float2*>(b),
                                                           reinterpret_cast<float2*>(a));
  SPH_CHECK_LAUNCH("add_float2");
  return SPH_OK;
}

sph_status_t sph_fill_float2(int64_t n, float x, float y, float* a, void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && a, "fill_float2: bad arguments");
  if (n == 0) return SPH_OK;
  k_fill2<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>((int)n, x, y, reinterpret_cast<float2*>(a));
  SPH_CHECK_LAUNCH("fill_float2");
  return SPH_OK;
}

size_t sph_dt_scratch_bytes(void) { return (size_t)2 * kNumSMs * 2 * sizeof(float); }

sph_status_t sph_update_dt(int64_t n, const float* v, const float* acc, float support, float kinematic, float cfl,
                           float c0, int32_t acoustic_from_c0, float dt_min, float dt_max, float* dt, void* scratch,
                           size_t scratch_bytes, void* stream) {
  SPH_REQUIRE(n > 0 && n < (1LL << 31) && v && acc && dt && kinematic > 0.f, "update_dt: bad arguments");
  if (!scratch || scratch_bytes < sph_dt_scratch_bytes()) {
    set_error_text("update_dt: scratch too small");
    return SPH_ERR_SCRATCH_TOO_SMALL;
  }
  cudaStream_t st = as_stream(stream);
  int parts = (int)std::min<int64_t>(2 * kNumSMs, (n + 255) / 256);
  float* part = static_cast<float*>(scratch);
  k_dt_partials<<<parts, 256, 0, st>>>((int)n, reinterpret_cast<const float2*>(v), reinterpret_cast<const float2*>(acc),
                                       support, part);
  k_dt_final<<<1, 32, 0, st>>>(parts, part, support, kinematic, cfl, c0, acoustic_from_c0, dt_min, dt_max, dt);
  SPH_CHECK_LAUNCH("update_dt");
  return SPH_OK;
}

}  // extern "C"
