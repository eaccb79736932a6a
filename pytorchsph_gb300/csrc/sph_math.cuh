// Device math of the SPH summations: Wendland C2 / spiky kernels (src/kernels.py:20-33),
// pair geometry (src/modules/neighborSearch.py:218-223), the reference's closed-form 2x2
// pseudo-inverse (src/util.py:386-433) and a 3x3 pseudo-inverse for mDBC.
#pragma once

#include "sph_common.cuh"

namespace sph {

// Parameters shared by every summation kernel (by value in the launch).
struct SphParams {
  float h, inv_h;
  float thr;        // sq_threshold(h): the pair test v <= thr for support h
  float c_w;        // 7 / (pi h^2)           Wendland W
  float c_g;        // 7 / (pi h^3)           Wendland gradient (times 20 q (1-q)^3)
  float c_s;        // 30 / (pi h^3)          spiky gradient
  float gk;         // -20 c_g / h: gradW = gk (1 - q)^3 (x_i - x_j)
  float eps;        // 0.1 h^2
  float rho0, c0, gamma;
  float tait_k;     // rho0 c0^2 / gamma
  float visc_k;     // h alpha c0
  float diff_k;     // h delta c0
  float kinematic;
  float gx, gy;     // constant gravity
  int point_source; // gravity = -g (x - c)  (potential field)
  float point_mag, point_cx, point_cy;
  int diffusion;    // 0 none, 1 MOG, 2 deltaSPH
  int boundary_diffusion;
  int search_radius;
  int cell_capacity;
};

// Wall particles, sorted by their cell in the fluid grid; quantities per sorted wall.
struct WallView {
  const float2* x;         // wall positions
  const float2* xg;        // ghost positions
  const float* area;       // boundaryVolume (pi r^2)
  const int32_t* cell_start;  // wall cell table in the fluid grid (cells+2)
  int n;
  float* rho;              // relative wall density
  float* vol;              // A_b / rho_b
  float* p;                // wall pressure
};

__device__ __forceinline__ float kW(float q, float c_w) {
  float a = 1.0f - q;
  float a2 = a * a;
  return a2 * a2 * (1.0f + 4.0f * q) * c_w;
}

// gradW = e * kGW(q): Wendland gradient magnitude factor -C/h^3 * 20 q (1-q)^3.
__device__ __forceinline__ float kGW(float q, float c_g) {
  float a = 1.0f - q;
  return -c_g * 20.0f * q * a * a * a;
}

// spikyGrad = e * kGS(q): -30/(pi h^3) (1-q)^2.
__device__ __forceinline__ float kGS(float q, float c_s) {
  float a = 1.0f - q;
  return -c_s * a * a;
}

// Approximate reciprocal square root and reciprocal of a positive NORMAL float (every caller
// passes a value >= 1e-30): the same hardware approximation as rsqrtf(x) and
// __fdividef(1, x), in their .ftz forms, which skip the scaling that the default forms wrap
// around it for subnormal inputs.  For normal inputs the results are the same.
__device__ __forceinline__ float rsqrt_normal(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

__device__ __forceinline__ float rcp_normal(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

struct Geo {
  float dx, dy;   // x_row - x_col
  float r, q;
  float ex, ey;   // unit vector, 0 when r < 1e-7
};

__device__ __forceinline__ Geo geo(float xi, float yi, float xj, float yj, float inv_h) {
  Geo g;
  g.dx = xi - xj;
  g.dy = yi - yj;
  g.r = sqrtf(g.dx * g.dx + g.dy * g.dy);
  if (g.r >= 1e-7f) {
    float ir = 1.0f / g.r;
    g.ex = g.dx * ir;
    g.ey = g.dy * ir;
  } else {
    g.ex = 0.f;
    g.ey = 0.f;
  }
  g.q = g.r * inv_h;
  return g;
}

__device__ __forceinline__ float tait(float rho_rel, const SphParams& P) {
  float r7;
  if (P.gamma == 7.0f) {
    float r2 = rho_rel * rho_rel;
    float r4 = r2 * r2;
    r7 = r4 * r2 * rho_rel;
  } else {
    r7 = powf(rho_rel, P.gamma);
  }
  return P.tait_k * (r7 - 1.0f);
}

// pinv2x2, src/util.py:386-433: closed-form SVD pseudo-inverse, singular values <= 1e-5
// dropped.  M = [[a, b], [c, d]]; returns [[o00, o01], [o10, o11]] in a float4 (row major).
__device__ __forceinline__ float4 pinv2x2(float a, float b, float c, float d) {
  float theta = 0.5f * atan2f(2 * a * c + 2 * b * d, a * a + b * b - c * c - d * d);
  float ct = cosf(theta), st = sinf(theta);
  float S1 = a * a + b * b + c * c + d * d;
  float t = a * a + b * b - c * c - d * d;
  float u = a * c + b * d;
  float S2 = sqrtf(t * t + 4 * u * u);
  float o1 = sqrtf((S1 + S2) * 0.5f);
  float o2 = sqrtf((S1 - S2) * 0.5f);
  float phi = 0.5f * atan2f(2 * a * b + 2 * c * d, a * a - b * b + c * c - d * d);
  float cp = cosf(phi), sp = sinf(phi);
  float v1 = (a * ct + c * st) * cp + (b * ct + d * st) * sp;
  float v2 = (a * st - c * ct) * sp + (-b * st + d * ct) * cp;
  float s11 = (v1 > 0.f) ? 1.f : ((v1 < 0.f) ? -1.f : 0.f);
  float s22 = (v2 > 0.f) ? 1.f : ((v2 < 0.f) ? -1.f : 0.f);
  // V = [[cp s11, -sp s22], [sp s11, cp s22]]; U = [[ct, -st], [st, ct]]
  float i1 = fabsf(o1) > 1e-5f ? 1.0f / o1 : 0.f;
  float i2 = fabsf(o2) > 1e-5f ? 1.0f / o2 : 0.f;
  // V S^-1 = [[cp s11 i1, -sp s22 i2], [sp s11 i1, cp s22 i2]]; times U^T = [[ct, st], [-st, ct]]
  float m00 = cp * s11 * i1, m01 = -sp * s22 * i2, m10 = sp * s11 * i1, m11 = cp * s22 * i2;
  return make_float4(m00 * ct - m01 * st, m00 * st + m01 * ct, m10 * ct - m11 * st, m10 * st + m11 * ct);
}

// pinv2x2 of a well-conditioned M: there the pseudo-inverse is the inverse adj(M) / det, a
// few operations instead of the closed form's atan2 / cos / sin.  With S1 = |M|_F^2 and
// sigma_max^2 = (S1 + sqrt(S1^2 - 4 det^2)) / 2 (no cancellation), sigma_min^2 = det^2 /
// sigma_max^2.  Taken when sigma_min > 0.1 sigma_max and sigma_min > 2e-5 (twice the 1e-5
// cutoff): there the closed form in float32 is itself within ~1e-5 of the inverse (its small
// singular value carries a relative error of ~FLT_EPSILON (sigma_max / sigma_min)^2).  Any
// other M (free-surface particles, non-finite input) goes through pinv2x2.
__device__ __forceinline__ float4 pinv2x2_fast(float a, float b, float c, float d) {
  const float det = a * d - b * c;
  const float S1 = a * a + b * b + c * c + d * d;
  const float s1sq = 0.5f * (S1 + sqrtf(fmaxf(S1 * S1 - 4.0f * det * det, 0.0f)));
  const float d2 = det * det;
  if (d2 > 0.01f * s1sq * s1sq && d2 > 4e-10f * s1sq && isfinite(d2)) {
    const float id = 1.0f / det;
    return make_float4(d * id, -b * id, -c * id, a * id);
  }
  return pinv2x2(a, b, c, d);
}

// x = pinv(A) b for a 3x3 A in double (torch.linalg.pinv semantics: singular values below
// 3 * FLT_EPSILON * sigma_max are dropped).  Eigen-decomposition of A^T A by cyclic Jacobi
// rotations (at most 16 sweeps), then pinv(A) b = sum_k v_k ((A v_k) . b) / sigma_k^2.
// Kept out of line: its arrays would otherwise set the register count of every caller's
// common path (pinv3_solve below).
static __device__ __noinline__ void pinv3_solve_jacobi(const double A[3][3], const double b[3], double x[3]) {
  double S[3][3];
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) S[r][c] = A[0][r] * A[0][c] + A[1][r] * A[1][c] + A[2][r] * A[2][c];
  double V[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
  for (int sweep = 0; sweep < 16; ++sweep) {
    double off = fabs(S[0][1]) + fabs(S[0][2]) + fabs(S[1][2]);
    double diag = fabs(S[0][0]) + fabs(S[1][1]) + fabs(S[2][2]);
    if (off <= 1e-300 || off <= 1e-17 * diag) break;
    for (int p = 0; p < 2; ++p)
      for (int q = p + 1; q < 3; ++q) {
        double apq = S[p][q];
        if (fabs(apq) <= 1e-300) continue;
        double tau = (S[q][q] - S[p][p]) / (2.0 * apq);
        double t = (tau >= 0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
        double c = 1.0 / sqrt(1.0 + t * t), s = t * c;
        for (int k = 0; k < 3; ++k) {  // S = J^T S J
          double skp = S[k][p], skq = S[k][q];
          S[k][p] = c * skp - s * skq;
          S[k][q] = s * skp + c * skq;
        }
        for (int k = 0; k < 3; ++k) {
          double spk = S[p][k], sqk = S[q][k];
          S[p][k] = c * spk - s * sqk;
          S[q][k] = s * spk + c * sqk;
        }
        for (int k = 0; k < 3; ++k) {
          double vkp = V[k][p], vkq = V[k][q];
          V[k][p] = c * vkp - s * vkq;
          V[k][q] = s * vkp + c * vkq;
        }
        S[p][q] = S[q][p] = 0.0;   // what the rotation is for; its rounding would keep the sweeps going
      }
  }
  double lmax = fmax(fmax(S[0][0], S[1][1]), S[2][2]);
  double smax = sqrt(fmax(lmax, 0.0));
  double tol = 3.0 * 1.1920928955078125e-07 * smax;
  x[0] = x[1] = x[2] = 0.0;
  for (int k = 0; k < 3; ++k) {
    double sig = sqrt(fmax(S[k][k], 0.0));
    if (!(sig > tol)) continue;
    double av[3];
    for (int r = 0; r < 3; ++r) av[r] = A[r][0] * V[0][k] + A[r][1] * V[1][k] + A[r][2] * V[2][k];
    double coef = (av[0] * b[0] + av[1] * b[1] + av[2] * b[2]) / (sig * sig);
    for (int r = 0; r < 3; ++r) x[r] += V[r][k] * coef;
  }
}

// x = pinv(A) b of float32 sums, solved in double.  While the Frobenius condition bound
// ||A|| ||A^-1|| stays below 2.5e6, under the 1/(3 FLT_EPSILON) = 2.8e6 at which a singular value
// would be dropped, pinv(A) = A^-1, applied through the adjugate; |det| > 1e-10 ||A||^3 keeps the
// determinant's rounding below 1e-5, far under what the float32 sums contribute at such
// conditions (the Jacobi sweeps work on A^T A and lose more).  GB300 does two double
// operations a clock and SM, and a launch waits for its slowest wall: so A is scaled by a power
// of two (exact) and the bounds run in float, about 60 double operations in all, and only
// systems that may lose a singular value go to the sweeps (some 5,000 operations; with a bound
// of 1e5 the corner walls of a tank did).
__device__ inline void pinv3_solve(const float A[3][3], const float b[3], double x[3]) {
  float amax = 0.f;
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 3; ++c) amax = fmaxf(amax, fabsf(A[r][c]));
  const int ex = (__float_as_int(amax) >> 23) & 255;
  if (ex >= 2 && ex <= 252) {
    const float sc = __int_as_float((254 - ex) << 23);   // amax * sc in [1, 2)
    float f[3][3], na = 0.f;
    double d[3][3];
    for (int r = 0; r < 3; ++r)
      for (int c = 0; c < 3; ++c) {
        f[r][c] = A[r][c] * sc;
        na = fmaf(f[r][c], f[r][c], na);
        d[r][c] = f[r][c];
      }
    // cofactor (r, c) = a b - c d as fma(a, b, -(c d)); in float only for the norm
    const auto cof = [](double p, double q, double u, double v) { return fma(p, q, -(u * v)); };
    const auto sqr = [](float p, float q, float u, float v) {
      const float c = fmaf(p, q, -(u * v));
      return c * c;
    };
    const double c00 = cof(d[1][1], d[2][2], d[1][2], d[2][1]), c01 = cof(d[1][2], d[2][0], d[1][0], d[2][2]),
                 c02 = cof(d[1][0], d[2][1], d[1][1], d[2][0]);
    const double det = fma(d[0][0], c00, fma(d[0][1], c01, d[0][2] * c02));
    const float nc = sqr(f[1][1], f[2][2], f[1][2], f[2][1]) + sqr(f[1][2], f[2][0], f[1][0], f[2][2]) +
                     sqr(f[1][0], f[2][1], f[1][1], f[2][0]) + sqr(f[0][2], f[2][1], f[0][1], f[2][2]) +
                     sqr(f[0][0], f[2][2], f[0][2], f[2][0]) + sqr(f[0][1], f[2][0], f[0][0], f[2][1]) +
                     sqr(f[0][1], f[1][2], f[0][2], f[1][1]) + sqr(f[0][2], f[1][0], f[0][0], f[1][2]) +
                     sqr(f[0][0], f[1][1], f[0][1], f[1][0]);
    const float ds = (float)det, ds2 = ds * ds;
    // ||A^-1||_F = ||adj A||_F / |det|
    if (na * nc < 6.25e12f * ds2 && ds2 > 1e-20f * (na * na * na)) {
      const double c10 = cof(d[0][2], d[2][1], d[0][1], d[2][2]), c11 = cof(d[0][0], d[2][2], d[0][2], d[2][0]),
                   c12 = cof(d[0][1], d[2][0], d[0][0], d[2][1]);
      const double c20 = cof(d[0][1], d[1][2], d[0][2], d[1][1]), c21 = cof(d[0][2], d[1][0], d[0][0], d[1][2]),
                   c22 = cof(d[0][0], d[1][1], d[0][1], d[1][0]);
      const double id = (double)sc / det;  // A^-1 = sc adj(sc A) / det(sc A), adj(A)[r][c] = cofactor c_cr
      const double b0 = b[0], b1 = b[1], b2 = b[2];
      x[0] = fma(c00, b0, fma(c10, b1, c20 * b2)) * id;
      x[1] = fma(c01, b0, fma(c11, b1, c21 * b2)) * id;
      x[2] = fma(c02, b0, fma(c12, b1, c22 * b2)) * id;
      return;
    }
  }
  const double Ad[3][3] = {{A[0][0], A[0][1], A[0][2]}, {A[1][0], A[1][1], A[1][2]}, {A[2][0], A[2][1], A[2][2]}};
  const double bd[3] = {b[0], b[1], b[2]};
  pinv3_solve_jacobi(Ad, bd, x);
}

// Iterate the wall particles whose cell is within +-r of fluid cell (cx, cy) and that pass
// the wall-side predicate sqrtf(fmaf(dx,dx,dy*dy)) < h_b with dx = x_b - x_f: exactly the
// wall->fluid pairs of searchExisting (src/modules/neighborSearch.py:231-252).
// `coff` is the scene's first slot in the (batched) cell tables; 0 for a single scene.
template <typename F>
__device__ __forceinline__ void for_each_wall(const WallView& W, const sph_grid& g, int r, int cx, int cy, float xf,
                                              float yf, float thr_b, F&& f, int coff = 0) {
  const int x0 = max(cx - r, 0), x1 = min(cx + r, g.cells_x - 1);
  if (x0 > x1) return;
  const int y0 = max(cy - r, 0), y1 = min(cy + r, g.cells_y - 1);
  const int32_t* cs = W.cell_start + coff;
  for (int yy = y0; yy <= y1; ++yy) {
    const int row = yy * g.cells_x;
    const int b0 = __ldg(cs + row + x0), b1 = __ldg(cs + row + x1 + 1);
    for (int b = b0; b < b1; ++b) {
      const float2 xb = __ldg(W.x + b);
      if (dist2_ref(xb.x, xb.y, xf, yf) <= thr_b) f(b, xb);
    }
  }
}

// The members of the cells within r of (cx, cy) that a cell table lists, dealt to kLanes
// consecutive lanes: f(j) for every kLanes-th member j.  Three rows of cells at a time: their six
// bounds are loaded together and the rows are walked as one range, so that a lane's chain is
// the bounds and then members that do not wait for each other.
template <int kLanes, typename Fn>
__device__ __forceinline__ void for_each_member(const int32_t* __restrict__ cs, const sph_grid& g, int r, int cx,
                                                int cy, int sub, Fn&& f) {
  const int x0 = max(cx - r, 0), x1 = min(cx + r, g.cells_x - 1);
  if (x0 > x1) return;
  const int y1 = min(cy + r, g.cells_y - 1);
  for (int yy = max(cy - r, 0); yy <= y1; yy += 3) {
    const int32_t* row = cs + (int64_t)yy * g.cells_x;
    const int two = yy + 1 <= y1 ? g.cells_x : 0, three = yy + 2 <= y1 ? 2 * g.cells_x : 0;
    const int b0 = __ldg(row + x0), b1 = __ldg(row + two + x0), b2 = __ldg(row + three + x0);
    const int n0 = __ldg(row + x1 + 1) - b0;
    const int e1 = __ldg(row + two + x1 + 1), e2 = __ldg(row + three + x1 + 1);
    const int n1 = two ? n0 + e1 - b1 : n0, n2 = three ? n1 + e2 - b2 : n1;   // members up to each row's end
#pragma unroll 2
    for (int t = sub; t < n2; t += kLanes) f(t < n0 ? b0 + t : t < n1 ? b1 + t - n0 : b2 + t - n1);
  }
}

// for_each_wall shared by kLanes consecutive lanes (one particle's): lane `sub` takes every
// kLanes-th wall of the cells.
template <int kLanes, typename F>
__device__ __forceinline__ void for_each_wall_lanes(const WallView& W, const sph_grid& g, int r, int cx, int cy,
                                                    float xf, float yf, float thr_b, int sub, F&& f, int coff = 0) {
  for_each_member<kLanes>(W.cell_start + coff, g, r, cx, cy, sub, [&](int b) {
    const float2 xb = __ldg(W.x + b);
    if (dist2_ref(xb.x, xb.y, xf, yf) <= thr_b) f(b, xb);
  });
}

// Sum of v over the kLanes consecutive lanes of one particle (every lane gets the sum; the
// whole warp must take part).
template <int kLanes>
__device__ __forceinline__ float lane_sum(float v) {
#pragma unroll
  for (int o = 1; o < kLanes; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Geometry of a query pair, src/modules/neighborSearch.py:244-251: d = x_q - x, r = |d|;
// e = d / r (0 when r < threshold); q = r / h_q.
__device__ __forceinline__ float2 query_geometry(float2 xq, float2 x, float hq, float threshold, float* radial) {
  const float dx = xq.x - x.x, dy = xq.y - x.y;
  const float d = sqrtf(dx * dx + dy * dy);
  *radial = d / hq;
  return d < threshold ? make_float2(0.f, 0.f) : make_float2(dx / d, dy / d);
}

// ---------------------------------------------------------------- candidate segments
// The candidates of a particle in one cell row are a contiguous sorted range; it is tested
// in segments of 32 candidates into bit masks (bit t: candidate c + t passes the pair test),
// and a particle keeps its non-empty segments, at most kMaxSegments, as (start, mask) pairs.
constexpr int kMaxSegments = 8;

// One candidate per step (the force passes' rare fallback for a particle whose segments
// did not fit).
__device__ __forceinline__ uint32_t segment_mask_scalar(const float2* __restrict__ x, int c, int e, float xi,
                                                        float yi, float thr) {
  const int len = min(e - c, 32);
  uint32_t m = 0;
  for (int t = 0; t < len; ++t) {
    const float2 pj = __ldg(x + c + t);
    m |= (uint32_t)(dist2_ref(xi, yi, pj.x, pj.y) <= thr) << t;
  }
  return m;
}

// The pair test on one paired float32 add: (x_j, y_j) + (-x_i, -y_i) of the candidate as it was
// loaded, which is minus dist2_ref's difference exactly, then its product and fused sum, so
// the value is dist2_ref's bit for bit.  (Pairs across two candidates, dx with dx and dy with dy,
// need both loads' halves moved into place and negated.)  The count of 2^20 lattice particles
// with densities takes 64 µs (69 across two candidates), a serving step's records 114 (120).
__device__ __forceinline__ float dist2_from(float2 neg_i, float2 pj) {
  const float2 d = __fadd2_rn(pj, neg_i);
  return __fmaf_rn(d.x, d.x, __fmul_rn(d.y, d.y));
}

// Two candidates per step.
__device__ __forceinline__ uint32_t segment_mask(const float2* __restrict__ x, int c, int e, float xi, float yi,
                                                 float thr) {
  const int len = min(e - c, 32);
  uint32_t m = 0;
  const float2 neg = make_float2(-xi, -yi);
  // unrolled over the segment's 16 candidate pairs, each guarded by the length: every bit
  // position is a constant, so a candidate costs its test and one predicated OR
#pragma unroll
  for (int t = 0; t < 32; t += 2) {
    if (t + 1 < len) {
      const float2 a = __ldg(x + c + t), b = __ldg(x + c + t + 1);
      if (dist2_from(neg, a) <= thr) m |= 1u << t;
      if (dist2_from(neg, b) <= thr) m |= 2u << t;
    } else if (t < len) {
      if (dist2_from(neg, __ldg(x + c + t)) <= thr) m |= 1u << t;
    }
  }
  return m;
}

// segment_mask when c + 32 <= n (the array's length): every candidate load is in bounds, so
// all 32 candidates are tested without per-pair guards (all loads can be in flight
// together) and the bits past the range are cleared; the bits inside it are segment_mask's.
__device__ __forceinline__ uint32_t segment_mask_full(const float2* __restrict__ x, int c, int e, float xi,
                                                      float yi, float thr) {
  const int len = min(e - c, 32);
  uint32_t m = 0;
  const float2 neg = make_float2(-xi, -yi);
#pragma unroll
  for (int t = 0; t < 32; ++t)
    if (dist2_from(neg, __ldg(x + c + t)) <= thr) m |= 1u << t;
  return len >= 32 ? m : m & ((1u << len) - 1u);
}

// segment_mask with the density terms of the accepted candidates added to acc in index
// order, in the same unrolled pass: the terms of a candidate pair are formed together on
// the paired float32 instructions and only the accepted ones are added (the caller scales
// the sum by c_w).  Distance r = v * rsqrt(max(v, 1e-30)): 0 for the particle itself,
// within a few ulp of sqrt(v) otherwise.  W(q) / c_w = (1-q)^4 (1+4q), src/kernels.py:20-24.
__device__ __forceinline__ uint32_t segment_mask_density(const float2* __restrict__ x, const float* __restrict__ sa,
                                                         int c, int e, float xi, float yi, float thr,
                                                         float inv_support, float& acc) {
  const int len = min(e - c, 32);
  uint32_t m = 0;
  const float2 neg = make_float2(-xi, -yi), is2 = make_float2(inv_support, inv_support);
  const float2 one = make_float2(1.f, 1.f);
#pragma unroll
  for (int t = 0; t < 32; t += 2) {
    if (t < len) {
      const bool two = t + 1 < len;
      float2 v;
      v.x = dist2_from(neg, __ldg(x + c + t));
      v.y = two ? dist2_from(neg, __ldg(x + c + t + 1)) : v.x;
      const bool in0 = v.x <= thr, in1 = two && v.y <= thr;
      if (in0) m |= 1u << t;
      if (in1) m |= 2u << t;
      if (in0 || in1) {
        const float2 rs = __fmul2_rn(make_float2(rsqrt_normal(fmaxf(v.x, 1e-30f)), rsqrt_normal(fmaxf(v.y, 1e-30f))), is2);
        const float2 q = __fmul2_rn(v, rs);
        const float2 am = __ffma2_rn(q, make_float2(-1.f, -1.f), one);   // 1 - q, rounded once
        const float2 a2 = __fmul2_rn(am, am);
        const float2 w = __fmul2_rn(__fmul2_rn(a2, a2), __ffma2_rn(make_float2(4.f, 4.f), q, one));
        if (in0) acc = fmaf(w.x, __ldg(sa + c + t), acc);
        if (in1) acc = fmaf(w.y, __ldg(sa + c + t + 1), acc);
      }
    }
  }
  return m;
}

// The bits of a stored segment that name a particle: none for a start outside [0, n),
// none at index n or past it.
__device__ __forceinline__ uint32_t clip_segment(uint32_t w, int b, int n) {
  if ((unsigned)b >= (unsigned)n) return 0;
  return n - b < 32 ? w & ((1u << (n - b)) - 1) : w;
}

struct FluidView {
  const float2* x;
  const float2* v;
  const float* rho;
  const float* area;
  const uint32_t* keys;
  const int32_t* offsets;
  const int32_t* cols;
  const int32_t* cell_start;
  int n;
  int pair_cap;  // 0: cols holds every row
};

// End of particle i's CSR row [offsets[i], end): a row that ends past the column buffer was
// not filled and reads as empty, so no kernel reads a column that was never written.
__device__ __forceinline__ int row_end(const FluidView& F, int i, int k0) {
  const int k1 = F.offsets[i + 1];
  return (F.pair_cap > 0 && k1 > F.pair_cap) ? k0 : k1;
}

// Cell coordinates of a grid key.  A key past the grid (a particle outside its grid) gives a
// row far below the grid, so that every +-r cell window around it is empty.
__device__ __forceinline__ void cell_of(uint32_t key, const sph_grid& g, int* cx, int* cy) {
  if (key >= (uint32_t)g.num_cells) {
    *cx = 0;
    *cy = -(1 << 20);
    return;
  }
  *cx = (int)(key % (uint32_t)g.cells_x);
  *cy = (int)(key / (uint32_t)g.cells_x);
}

// ---------------------------------------------------------------------------- cell-row pairs
// The pairs of particle i straight from the cell table, without a CSR list: its candidates
// are the contiguous sorted ranges of its 2r+1 cell rows (cells cx-r..cx+r of each row).
// A range is tested in segments of 32 candidates into a bit mask, and the accepted
// candidates are visited in increasing index: the CSR fill's order, so every sum is the
// same.  Visiting set bits keeps a warp's lanes together the way a CSR row does (a lane
// runs the pair body only for its own neighbors).
//
// The records pass stores each particle's non-empty segments in order, at most
// kMaxSegments: start seg_start[k * n + i] and mask seg_mask[k * n + i] for k < nseg[i]
// (nseg[i] = -1 when there are more; the force passes then test its cell rows
// themselves).  A force pass holds one segment and the next one, loaded ahead, so moving
// on to the next segment costs a lane a register move.
// Every row of the window, tested here (any r); with kTpp lanes per particle, lane `sub`
// takes rows y0 + sub, y0 + sub + kTpp, ...
// kPaired: the candidate tests two at a time (segment_mask) or one at a time; the sums are
// the same either way (which one a pass uses is a measured code-generation choice).
template <int kTpp = 1, bool kPaired = false, typename Fn>
__device__ __forceinline__ void cell_pairs(const FluidView& F, const sph_grid& g, int r, int coff, int cx, int cy,
                                           float xi, float yi, float thr, Fn&& fn, int sub = 0) {
  const int x0 = max(cx - r, 0), x1 = min(cx + r, g.cells_x - 1);
  if (x0 > x1) return;
  const int y0 = max(cy - r, 0), y1 = min(cy + r, g.cells_y - 1);
  const int32_t* cs = F.cell_start + coff;
  for (int yy = y0 + sub; yy <= y1; yy += kTpp) {
    const int row = yy * g.cells_x;
    const int b = __ldg(cs + row + x0), e = __ldg(cs + row + x1 + 1);
    for (int c = b; c < e; c += 32) {
      uint32_t w = kPaired ? segment_mask(F.x, c, e, xi, yi, thr) : segment_mask_scalar(F.x, c, e, xi, yi, thr);
      while (w) {
        const int j = c - 1 + __ffs(w);
        w &= w - 1;
        fn(j);
      }
    }
  }
}

// The segment list of particle i.
__device__ __forceinline__ void segments_body(int i, const FluidView& F, const sph_grid& g, int coff, int r,
                                              float thr, int32_t* __restrict__ nseg, int32_t* __restrict__ seg_start,
                                              uint32_t* __restrict__ seg_mask) {
  int cx, cy;
  cell_of(F.keys[i] - (uint32_t)coff, g, &cx, &cy);
  const float2 xi = F.x[i];
  const size_t n = (size_t)F.n;
  int k = 0;
  const int x0 = max(cx - r, 0), x1 = min(cx + r, g.cells_x - 1);
  const int y0 = max(cy - r, 0), y1 = min(cy + r, g.cells_y - 1);
  const int32_t* cs = F.cell_start + coff;
  if (x0 <= x1) {
    for (int yy = y0; yy <= y1; ++yy) {
      const int row = yy * g.cells_x;
      const int b = __ldg(cs + row + x0), e = __ldg(cs + row + x1 + 1);
      for (int c = b; c < e; c += 32) {
        const uint32_t w = c + 32 <= F.n ? segment_mask_full(F.x, c, e, xi.x, xi.y, thr)
                                         : segment_mask(F.x, c, e, xi.x, xi.y, thr);
        if (w == 0) continue;
        if (k < kMaxSegments) {
          seg_start[k * n + i] = c;
          seg_mask[k * n + i] = w;
        }
        ++k;
      }
    }
  }
  nseg[i] = k <= kMaxSegments ? k : -1;
}

// Lane `sub`'s candidates of a segment shared by kTpp lanes: every kTpp-th bit.
template <int kTpp>
__device__ __forceinline__ uint32_t lane_bits(uint32_t w, int sub) {
  static_assert(kTpp == 1 || kTpp == 2 || kTpp == 4 || kTpp == 8, "lanes per particle");
  constexpr uint32_t every = kTpp == 1 ? 0xffffffffu : kTpp == 2 ? 0x55555555u : kTpp == 4 ? 0x11111111u : 0x01010101u;
  return w & (every << sub);
}

// The pairs of particle i from its segment list (its cell rows when the list overflowed).
// With kTpp lanes per particle every lane walks all segments and takes its lane_bits of each
// (about 28 / kTpp pairs, however the accepted candidates fall into segments; rows are dealt
// on the overflow path); each lane holds its current segment and the next one, loaded ahead.
template <int kTpp = 1, bool kPaired = false, typename Fn>
__device__ __forceinline__ void stored_pairs(int i, const FluidView& F, const sph_grid& g, int coff, int r,
                                             const int32_t* __restrict__ nseg, const int32_t* __restrict__ seg_start,
                                             const uint32_t* __restrict__ seg_mask, float xi, float yi, float thr,
                                             Fn&& fn, int sub = 0) {
  const int ns = nseg[i];
  if (ns < 0 || ns > kMaxSegments) {
    int cx, cy;
    cell_of(F.keys[i] - (uint32_t)coff, g, &cx, &cy);
    cell_pairs<kTpp, kPaired>(F, g, r, coff, cx, cy, xi, yi, thr, fn, sub);
    return;
  }
  if (ns == 0) return;
  const size_t n = (size_t)F.n;
  int k = 0;
  int b = seg_start[i];
  uint32_t w = lane_bits<kTpp>(clip_segment(seg_mask[i], b, F.n), sub);
  int bn = 0;
  uint32_t wn = 0;
  if (1 < ns) {
    bn = seg_start[n + i];
    wn = seg_mask[n + i];
  }
  for (;;) {
    while (w == 0) {
      ++k;
      if (k >= ns) return;
      b = bn;
      w = lane_bits<kTpp>(clip_segment(wn, bn, F.n), sub);
      if (k + 1 < ns) {
        bn = seg_start[(k + 1) * n + i];
        wn = seg_mask[(k + 1) * n + i];
      }
    }
    const int j = b - 1 + __ffs(w);
    w &= w - 1;
    fn(j);
  }
}

// for_each_wall with the walls of a cell row tested 32 at a time and the accepted ones' records
// four in flight: use(load(b)) in the same order.
template <typename Load, typename Use>
__device__ __forceinline__ void for_each_wall_by_four(const WallView& W, const sph_grid& g, int r, int cx, int cy,
                                                      float xf, float yf, float thr_b, Load&& load, Use&& use,
                                                      int coff = 0) {
  const int x0 = max(cx - r, 0), x1 = min(cx + r, g.cells_x - 1);
  if (x0 > x1) return;
  const int y0 = max(cy - r, 0), y1 = min(cy + r, g.cells_y - 1);
  const int32_t* cs = W.cell_start + coff;
  for (int yy = y0; yy <= y1; ++yy) {
    const int32_t* row = cs + (int64_t)yy * g.cells_x;
    const int b0 = __ldg(row + x0), b1 = __ldg(row + x1 + 1);
    for (int c = b0; c < b1; c += 32) {
      uint32_t w = c + 32 <= W.n ? segment_mask_full(W.x, c, b1, xf, yf, thr_b)
                                 : segment_mask(W.x, c, b1, xf, yf, thr_b);
      while (w) {
        int j[4];
        bool ok[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          ok[t] = w != 0;
          j[t] = ok[t] ? c - 1 + __ffs(w) : c;
          w &= w - 1;   // 0 stays 0
        }
        const auto f0 = load(j[0]), f1 = load(j[1]), f2 = load(j[2]), f3 = load(j[3]);
        use(f0);
        if (ok[1]) use(f1);
        if (ok[2]) use(f2);
        if (ok[3]) use(f3);
      }
    }
  }
}

// stored_pairs in groups of four: use(load(j)) in the same order, the four records of a group in
// flight together.  For scenes too small to hide a load's latency behind other warps.
template <typename Load, typename Use>
__device__ __forceinline__ void stored_pairs_by_four(int i, const FluidView& F, const sph_grid& g, int coff, int r,
                                                     const int32_t* __restrict__ nseg,
                                                     const int32_t* __restrict__ seg_start,
                                                     const uint32_t* __restrict__ seg_mask, float xi, float yi,
                                                     float thr, Load&& load, Use&& use) {
  const int ns = nseg[i];
  if (ns < 0 || ns > kMaxSegments) {
    int cx, cy;
    cell_of(F.keys[i] - (uint32_t)coff, g, &cx, &cy);
    cell_pairs(F, g, r, coff, cx, cy, xi, yi, thr, [&](int j) { use(load(j)); });
    return;
  }
  const size_t n = (size_t)F.n;
  int j0 = i, j1 = i, j2 = i, j3 = i, k = 0, b = 0, bn = 0;
  uint32_t w = 0, wn = 0;
  if (ns > 0) {
    bn = seg_start[i];
    wn = seg_mask[i];
  }
  for (bool more = ns > 0; more;) {
    int q = 0;   // the group's pairs, the last of them in j3
    while (q < 4) {
      while (w == 0 && k < ns) {
        b = bn;
        w = clip_segment(wn, bn, F.n);
        if (++k < ns) {
          bn = seg_start[k * n + i];
          wn = seg_mask[k * n + i];
        }
      }
      if (w == 0) break;
      j0 = j1;
      j1 = j2;
      j2 = j3;
      j3 = b - 1 + __ffs(w);
      w &= w - 1;
      ++q;
    }
    more = q == 4;
    const auto r0 = load(j0), r1 = load(j1), r2 = load(j2), r3 = load(j3);
    if (q > 3) use(r0);
    if (q > 2) use(r1);
    if (q > 1) use(r2);
    if (q > 0) use(r3);
  }
}

// Pairs from the segment lists S (kCells) instead of the CSR row.
struct Segments {
  const int32_t* nseg;
  const int32_t* start;
  const uint32_t* mask;
};

}  // namespace sph

// Host-side conversions of the C-ABI views into the kernels' views.
namespace sph {
// One scene of a batch as the kernels see it: derived parameters, its search grid, its
// first slot in the concatenated cell tables and its time step.
struct SceneDev {
  SphParams P;
  sph_grid g;
  int coff;
  float dt;
};

static inline SphParams to_params(const sph_params* p) {
  SphParams P;
  P.h = p->support;
  P.inv_h = 1.0f / p->support;
  P.thr = sq_threshold(p->support);
  const double h = p->support;
  P.c_w = (float)(7.0 / 3.14159265358979323846 / (h * h));
  P.c_g = (float)(7.0 / 3.14159265358979323846 / (h * h * h));
  P.c_s = (float)(30.0 / 3.14159265358979323846 / (h * h * h));
  P.gk = (float)(-20.0 * 7.0 / 3.14159265358979323846 / (h * h * h * h));
  P.eps = (float)(h * h * 0.1);
  P.rho0 = p->rest_density;
  P.c0 = p->c0;
  P.gamma = p->gamma;
  P.tait_k = (float)((double)p->rest_density * p->c0 * p->c0 / p->gamma);
  P.visc_k = (float)(h * p->alpha * p->c0);
  P.diff_k = (float)(h * p->delta * p->c0);
  P.kinematic = p->kinematic;
  P.gx = p->gravity[0];
  P.gy = p->gravity[1];
  P.point_source = p->point_source;
  P.point_mag = p->point_magnitude;
  P.point_cx = p->point_center[0];
  P.point_cy = p->point_center[1];
  P.diffusion = p->density_diffusion;
  P.boundary_diffusion = p->boundary_diffusion;
  P.search_radius = p->search_radius;
  P.cell_capacity = p->cell_capacity;
  return P;
}

static inline FluidView to_fluid(const sph_fluid_view* f) {
  FluidView F;
  F.x = reinterpret_cast<const float2*>(f->x);
  F.v = reinterpret_cast<const float2*>(f->v);
  F.rho = f->rho;
  F.area = f->area;
  F.keys = f->keys;
  F.offsets = f->offsets;
  F.cols = f->cols;
  F.cell_start = f->cell_start;
  F.n = (int)f->n;
  F.pair_cap = f->pair_capacity > 0x7fffffff ? 0x7fffffff : (int)f->pair_capacity;
  return F;
}

static inline WallView to_walls(const sph_wall_view* w) {
  WallView W;
  W.x = reinterpret_cast<const float2*>(w->x);
  W.xg = reinterpret_cast<const float2*>(w->ghost);
  W.area = w->area;
  W.cell_start = w->cell_start;
  W.n = (int)w->n;
  W.rho = w->rho;
  W.vol = w->volume;
  W.p = w->pressure;
  return W;
}

}  // namespace sph

#define SPH_VIEW_CHECK(f) SPH_REQUIRE((f) && (f)->n >= 0 && (f)->n < (1LL << 31), "bad particle view")
