// Differentiable deltaSPH rollout of a free fluid (no walls): the right-hand side of
// src/deltaSPH.py:146-200 with MOG density diffusion and gravity or the point source, the
// semi-implicit Euler update (src/simulationBase.py:647-652), and the discrete adjoint of
// one step in closed form.
//
// Pairs are rows of columns in original particle order (CSR, or a rollout's rows of fixed slots);
// the list is symmetric because every particle has the same support.  Particle i's adjoint
// gathers over its own row both
//   (d f_ij / d in_i)^T lambda_out_i   (its own right-hand side)   and
//   (d f_ji / d in_i)^T lambda_out_j   (its neighbors' right-hand sides),
// so there are no atomics and the result does not depend on thread timing.  Scalars are float
// or double.
//
// What bounds it: in double the FP64 pipe (two operations a clock and SM), in float a small
// rollout's latency.  4 or 8 lanes share a row in both (drop_lanes).
//   double: every quantity that both particles' terms share is formed once per pair, with one
//     division for its three reciprocals, and the derivatives are written out (about 110
//     operations a pair, where two sweeps of 5-component dual numbers took some 2,000).
//   float: the pair function and its dual numbers, whose terms the lanes form side by side and
//     add one after another in row order: a float32 gradient with respect to alpha is a sum
//     that cancels to 1/70 of its terms, so its rounding is kept to that of one thread per
//     row, bit for bit.
// At 3,985 particles in double the right-hand side takes 23 µs (one thread per row: 179) and
// the adjoint 44 (dual numbers: 819); at 16,173 in float 9.4 (31) and 20 (40).
#include "sph_common.cuh"

namespace sph {

template <typename T>
struct DropParams {
  T inv_h, cg20;      // 1/h, 20 * 7/(pi h^3)
  T rho0, inv_rho0, tait_k;   // tait_k = rho0 c0^2 / gamma (gamma = 7)
  T eps;              // 0.1 h^2
  T visc_unit;        // h c0 (artificial viscosity factor without alpha)
  T alpha, nu;        // artificial and laminar (kinematic) viscosity
  T diff_k;           // h delta c0 (MOG)
  T gx, gy;           // constant gravity
  int point_source;
  T point_mag, cx, cy;
  int mog;
};

// ---------------------------------------------------------------- float: pair function and dual numbers
template <typename T, int K>
struct Dual {
  T v;
  T d[K];
};

template <typename T>
__device__ __forceinline__ T val(T a) {
  return a;
}
template <typename T, int K>
__device__ __forceinline__ T val(const Dual<T, K>& a) {
  return a.v;
}

template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator+(const Dual<T, K>& a, const Dual<T, K>& b) {
  Dual<T, K> r;
  r.v = a.v + b.v;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] + b.d[k];
  return r;
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator-(const Dual<T, K>& a, const Dual<T, K>& b) {
  Dual<T, K> r;
  r.v = a.v - b.v;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] - b.d[k];
  return r;
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator-(const Dual<T, K>& a) {
  Dual<T, K> r;
  r.v = -a.v;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = -a.d[k];
  return r;
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator*(const Dual<T, K>& a, const Dual<T, K>& b) {
  Dual<T, K> r;
  r.v = a.v * b.v;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] * b.v + a.v * b.d[k];
  return r;
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator/(const Dual<T, K>& a, const Dual<T, K>& b) {
  Dual<T, K> r;
  const T ib = T(1) / b.v;
  r.v = a.v * ib;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = (a.d[k] - r.v * b.d[k]) * ib;
  return r;
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator+(const Dual<T, K>& a, T b) {
  Dual<T, K> r = a;
  r.v += b;
  return r;
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator+(T b, const Dual<T, K>& a) {
  return a + b;
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator-(const Dual<T, K>& a, T b) {
  Dual<T, K> r = a;
  r.v -= b;
  return r;
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator-(T b, const Dual<T, K>& a) {
  return -(a - b);
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator*(const Dual<T, K>& a, T b) {
  Dual<T, K> r;
  r.v = a.v * b;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] * b;
  return r;
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator*(T b, const Dual<T, K>& a) {
  return a * b;
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator/(const Dual<T, K>& a, T b) {
  return a * (T(1) / b);
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> operator/(T b, const Dual<T, K>& a) {
  Dual<T, K> one;
  one.v = b;
#pragma unroll
  for (int k = 0; k < K; ++k) one.d[k] = T(0);
  return one / a;
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> sqrt_(const Dual<T, K>& a) {
  Dual<T, K> r;
  r.v = sqrt(a.v);
  const T f = T(0.5) / r.v;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = a.d[k] * f;
  return r;
}
template <typename T>
__device__ __forceinline__ T sqrt_(T a) {
  return sqrt(a);
}
template <typename T>
__device__ __forceinline__ T make_const(T c, T) {
  return c;
}
template <typename T, int K>
__device__ __forceinline__ Dual<T, K> make_const(T c, const Dual<T, K>&) {
  Dual<T, K> r;
  r.v = c;
#pragma unroll
  for (int k = 0; k < K; ++k) r.d[k] = T(0);
  return r;
}

template <typename S>
struct PairOut {
  S ax, ay, dp;
  S vx, vy;  // artificial viscosity part without alpha (for d/d alpha)
};

template <typename S, typename T>
__device__ __forceinline__ S tait7(const S& rt, const DropParams<T>& P) {
  const S r2 = rt * rt;
  const S r4 = r2 * r2;
  return P.tait_k * (r4 * r2 * rt - T(1));
}

// Row i's terms from neighbor j (x_i - x_j nonzero).  Reference formulas: pressure.py:31-38,
// diffusion.py:30-44, laminar.py:30-46 (its index choices), momentum.py:31-38,
// densityDiffusion.py:74-82, kernels.py:20-33.
template <typename S, typename T>
__device__ __forceinline__ PairOut<S> pair_terms(const S& xix, const S& xiy, const S& vix, const S& viy,
                                                 const S& rti, const S& xjx, const S& xjy, const S& vjx,
                                                 const S& vjy, const S& rtj, T Aj, const DropParams<T>& P) {
  const S dx = xix - xjx, dy = xiy - xjy;          // x_i - x_j
  const S r2 = dx * dx + dy * dy;
  const S r = sqrt_(r2);
  const S q = r * P.inv_h;
  const S a = T(1) - q;
  const S gwr = -(P.cg20 * q * a * a * a) / r;   // gradW = gwr * (x_i - x_j)
  const S gx = gwr * dx, gy = gwr * dy;
  const S rhoi = rti * P.rho0, rhoj = rtj * P.rho0;
  const S Vj = Aj / rtj;
  const S pi = tait7(rti, P), pj = tait7(rtj, P);
  const S ux = vjx - vix, uy = vjy - viy;          // u_j - u_i
  const S rx = -dx, ry = -dy;                      // x_j - x_i
  const S R2 = r2 + P.eps;
  const S rg = rx * gx + ry * gy;
  PairOut<S> o;
  const S pf = (pi + pj) * Vj / rhoi;
  o.ax = -(pf * gx);
  o.ay = -(pf * gy);
  S pij = ux * rx + uy * ry;
  if (val(pij) > T(0)) pij = make_const(T(0), pij);
  const S vf = P.visc_unit * pij / R2 * Vj * rhoj / (rhoi + rhoj);
  o.vx = vf * gx;
  o.vy = vf * gy;
  o.ax = o.ax + P.alpha * o.vx;
  o.ay = o.ay + P.alpha * o.vy;
  const S rs = rhoi + rhoj;
  const S term = T(8) * rhoj * Vj * rhoi * P.nu * rg / (rs * rs * R2);   // 4 m_j (mu_i + mu_j), mu = rho_i nu
  o.ax = o.ax - term * (vix - vjx);
  o.ay = o.ay - term * (viy - vjy);
  o.dp = -((ux * gx + uy * gy) * Vj * rhoj);
  if (P.mog) o.dp = o.dp + P.diff_k * T(2) * (rhoj - rhoi) / R2 * rg * Vj;
  return o;
}

template <typename T>
__device__ __forceinline__ bool apart(T xix, T xiy, T xjx, T xjy) {
  const T dx = xix - xjx, dy = xiy - xjy;
  return dx * dx + dy * dy >= T(1e-14);   // the reference's e_ij is 0 below r = 1e-7
}

// ---------------------------------------------------------------- lanes

// The columns of row i: a rollout's own rows of `room` slots each (row_info holds their counts), or
// with room 0 a CSR list (row_info holds its offsets).
template <typename Col>
struct DropRows {
  const int32_t* row_info;
  const Col* cols;
  int room;
  __device__ __forceinline__ const Col* row(int i, int& m) const {
    const int a = row_info[i];
    m = room ? min(a, room) : row_info[i + 1] - a;
    return cols + (room ? (int64_t)i * room : (int64_t)a);
  }
};

template <int kLanes, typename T>
__device__ __forceinline__ T drop_sum(T v) {
#pragma unroll
  for (int o = 1; o < kLanes; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// sum + the lanes' terms one after another (every lane of the group gets the result; the whole
// warp must take part).
template <int kLanes>
__device__ __forceinline__ float drop_add_in_order(float sum, float term) {
#pragma unroll
  for (int l = 0; l < kLanes; ++l) {
    const float v = __shfl_sync(0xffffffffu, term, l, kLanes);
    sum += v;
  }
  return sum;
}

// Pairs of the longest row among a warp's groups (the loops of the lanes that add in order are
// as long in the whole warp).
template <int kLanes>
__device__ __forceinline__ int drop_longest(int m) {
#pragma unroll
  for (int o = kLanes; o < 32; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}

// ---------------------------------------------------------------- double: closed form
// What both rows of a pair (i, j) share, d = x_i - x_j and w = v_i - v_j: the Wendland gradient
// gradW_ij = gd d with gd = -20 c_g (1 - q)^3 / h (kernels.py:20-33), r, s = w . d, and the
// reciprocals of r (one rsqrt), and of R2 = r^2 + eps, rho_i + rho_j and rho~_j (one division).
struct DropPair {
  double dx, dy, wx, wy, r2, ir, r, gd, s, iR, irs, irj;
};

// False for a pair closer than r = 1e-7, where the reference's e_ij is zero (the particle itself).
__device__ __forceinline__ bool drop_pair(double2 xi, double2 vi, double ri, double2 xj, double2 vj, double rj,
                                          const DropParams<double>& P, DropPair& o) {
  o.dx = xi.x - xj.x;
  o.dy = xi.y - xj.y;
  o.r2 = o.dx * o.dx + o.dy * o.dy;
  if (!(o.r2 >= 1e-14)) return false;
  o.ir = rsqrt(o.r2);
  o.r = o.r2 * o.ir;
  const double a = 1.0 - o.r * P.inv_h;
  o.gd = -(P.cg20 * P.inv_h) * (a * a * a);
  o.wx = vi.x - vj.x;
  o.wy = vi.y - vj.y;
  o.s = o.wx * o.dx + o.wy * o.dy;
  const double R2 = o.r2 + P.eps, rs = P.rho0 * (ri + rj);
  const double t = 1.0 / (R2 * rs * rj);
  o.iR = t * (rs * rj);
  o.irs = t * (R2 * rj);
  o.irj = t * (R2 * rs);
  return true;
}

// Sums of row i (m columns) over the lanes' pairs (double; pressure.py:31-38, diffusion.py:30-44,
// laminar.py:30-46 with its index choices, momentum.py:31-38, densityDiffusion.py:74-82): with
// rho = rho0 rho~, V = A / rho~, m = rho V = rho0 A,
//   a_i  = -1/rho_i sum (p_i + p_j) V_j gd d + alpha h c0 sum min(s, 0) m_j irs iR gd d
//          + 8 nu rho_i sum m_j gd r2 irs^2 iR w
//   dp_i = sum m_j gd s - 2 h delta c0 sum (rho_j - rho_i) V_j gd r2 iR
template <int kLanes, typename Col>
__device__ __forceinline__ void drop_row(int m, int sub, const Col* __restrict__ cols, double2 xi, double2 vi,
                                         double ri, const double2* __restrict__ x, const double2* __restrict__ v,
                                         const double* __restrict__ rt, const double* __restrict__ area,
                                         const DropParams<double>& P, double& ax, double& ay, double& dp) {
  using T = double;
  const T rhoi = P.rho0 * ri, pi = tait7(ri, P);
  T px = 0, py = 0, vx = 0, vy = 0, lx = 0, ly = 0, d1 = 0, d2 = 0;
  for (int k = sub; k < m; k += kLanes) {
    const int j = (int)__ldg(cols + k);
    const T rj = rt[j], Aj = area[j];
    DropPair e;
    if (!drop_pair(xi, vi, ri, x[j], v[j], rj, P, e)) continue;
    const T mg = P.rho0 * Aj * e.gd, Vg = Aj * e.irj * e.gd;   // m_j gd, V_j gd
    const T pf = (pi + tait7(rj, P)) * Vg;
    px += pf * e.dx;
    py += pf * e.dy;
    const T g = mg * e.irs * e.iR;
    const T vf = (e.s > T(0) ? T(0) : e.s) * g;
    vx += vf * e.dx;
    vy += vf * e.dy;
    const T lf = e.r2 * e.irs * g;
    lx += lf * e.wx;
    ly += lf * e.wy;
    d1 += mg * e.s;
    d2 += (rj - ri) * Vg * (e.r2 * e.iR);
  }
  px = drop_sum<kLanes>(px);
  py = drop_sum<kLanes>(py);
  vx = drop_sum<kLanes>(vx);
  vy = drop_sum<kLanes>(vy);
  lx = drop_sum<kLanes>(lx);
  ly = drop_sum<kLanes>(ly);
  d1 = drop_sum<kLanes>(d1);
  d2 = drop_sum<kLanes>(d2);
  const T fp = T(-1) / rhoi, fv = P.alpha * P.visc_unit, fl = T(8) * P.nu * rhoi;
  ax = fp * px + fv * vx + fl * lx;
  ay = fp * py + fv * vy + fl * ly;
  dp = P.mog ? d1 - P.diff_k * T(2) * P.rho0 * d2 : d1;
}

// The same sums in float, added in row order.
template <int kLanes, typename Col>
__device__ __forceinline__ void drop_row(int m, int sub, const Col* __restrict__ cols, float2 xi, float2 vi,
                                         float ri, const float2* __restrict__ x, const float2* __restrict__ v,
                                         const float* __restrict__ rt, const float* __restrict__ area,
                                         const DropParams<float>& P, float& ax, float& ay, float& dp) {
  ax = ay = dp = 0.f;
  const int longest = drop_longest<kLanes>(m);
  for (int q = 0; q < longest; q += kLanes) {
    float tx = 0.f, ty = 0.f, td = 0.f;   // adding 0 where a lane has no pair changes no sum's value
    if (q + sub < m) {
      const int j = (int)__ldg(cols + q + sub);
      const float2 xj = x[j], vj = v[j];
      if (apart(xi.x, xi.y, xj.x, xj.y)) {
        const PairOut<float> o =
            pair_terms<float, float>(xi.x, xi.y, vi.x, vi.y, ri, xj.x, xj.y, vj.x, vj.y, rt[j], area[j], P);
        tx = o.ax;
        ty = o.ay;
        td = o.dp;
      }
    }
    ax = drop_add_in_order<kLanes>(ax, tx);
    ay = drop_add_in_order<kLanes>(ay, ty);
    dp = drop_add_in_order<kLanes>(dp, td);
  }
}

// Right-hand side of every particle.  kStep: advance (x, v, rho) by semi-implicit Euler into xo, vo,
// ro, with the new positions in float32 in x32 (may be NULL) for the next search; else write
// acc and dpdt.
template <int kLanes, typename T, typename V2, typename Col, bool kStep>
__global__ void __launch_bounds__(128) k_drop_rhs(int n, DropRows<Col> rows,
                                                  const V2* __restrict__ x, const V2* __restrict__ v,
                                                  const T* __restrict__ rt, const T* __restrict__ area,
                                                  DropParams<T> P, T dt, V2* __restrict__ acc, T* __restrict__ dpdt,
                                                  V2* __restrict__ xo, V2* __restrict__ vo, T* __restrict__ ro,
                                                  float2* __restrict__ x32) {
  const int row = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes);
  const int sub = threadIdx.x % kLanes;
  const bool live = row < n;
  const int i = live ? row : n - 1;   // lanes past the last particle only take part in the sums
  const V2 xi = x[i], vi = v[i];
  const T ri = rt[i];
  int m;
  const Col* cols = rows.row(i, m);
  T ax, ay, dp;
  drop_row<kLanes>(m, sub, cols, xi, vi, ri, x, v, rt, area, P, ax, ay, dp);
  if (!live || sub != 0) return;
  if (P.point_source) {
    T dx = xi.x - P.cx, dy = xi.y - P.cy;
    const T d = sqrt(dx * dx + dy * dy);
    if (d > T(1e-7)) {
      dx /= d;
      dy /= d;
    }
    ax += -P.point_mag * dx * d;
    ay += -P.point_mag * dy * d;
  } else {
    ax += P.gx;
    ay += P.gy;
  }
  if constexpr (kStep) {
    V2 vn, xn;
    vn.x = vi.x + dt * ax;
    vn.y = vi.y + dt * ay;
    xn.x = xi.x + dt * (vi.x + dt * ax);
    xn.y = xi.y + dt * (vi.y + dt * ay);
    xo[i] = xn;
    vo[i] = vn;
    ro[i] = ri + dt * dp / P.rho0;
    if (x32) x32[i] = make_float2((float)xn.x, (float)xn.y);
  } else {
    acc[i].x = ax;
    acc[i].y = ay;
    dpdt[i] = dp;
  }
}

template <typename T, typename V2>
__global__ void k_drop_sie(int n, V2* __restrict__ x, V2* __restrict__ v, T* __restrict__ rt,
                           const V2* __restrict__ acc, const T* __restrict__ dpdt, T dt, T rho0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const V2 a = acc[i], vi = v[i], xi = x[i];
  V2 vn, xn;
  vn.x = vi.x + dt * a.x;
  vn.y = vi.y + dt * a.y;
  xn.x = xi.x + dt * (vi.x + dt * a.x);
  xn.y = xi.y + dt * (vi.y + dt * a.y);
  x[i] = xn;
  v[i] = vn;
  rt[i] = rt[i] + dt * dpdt[i] / rho0;
}

// Sums of particle i's adjoint over the lanes' pairs (double).  With la, ld the adjoints of a_i
// and dp_i (lb, le: of row j), the pair's terms of both rows sum to
//   F = gd (p_i + p_j) Q1 + alpha h c0 gd min(s, 0) irs iR Q2 + 8 nu gd r2 irs^2 iR Q3
//       + gd s Q4 - 2 h delta c0 gd r2 iR (rho_j - rho_i) Q5,
//   Q1 = V_i/rho_j (lb.d) - V_j/rho_i (la.d),  Q2 = m_j (la.d) - m_i (lb.d),
//   Q3 = m_j rho_i (la.w) - m_i rho_j (lb.w),  Q4 = m_j ld + m_i le,  Q5 = V_j ld - V_i le,
// whose gradient with respect to d, w and rho~_i is particle i's share (m does not depend on
// rho~; d gd / d r2 = 30 c_g (1 - q)^2 / (h^2 r)).
template <int kLanes, typename Col>
__device__ __forceinline__ void adjoint_row(int i, int m, int sub, const Col* __restrict__ cols, double2 xi,
                                            double2 vi, double ri, const double2* __restrict__ x,
                                            const double2* __restrict__ v, const double* __restrict__ rt,
                                            const double* __restrict__ area, const DropParams<double>& P, double dt,
                                            const double2* __restrict__ lx1, const double2* __restrict__ lv1,
                                            const double* __restrict__ lr1, double lax, double lay, double ld,
                                            double (&g)[5], double& da) {
  using T = double;
  using V2 = double2;
  const T dt2 = dt * dt, sdp = dt / P.rho0;
  const T rhoi = P.rho0 * ri, iri = T(1) / ri, Vi = area[i] * iri, mi = P.rho0 * area[i], irhoi = iri * P.inv_rho0;
  const T ri2 = ri * ri, ri6 = ri2 * ri2 * ri2, pi = P.tait_k * (ri6 * ri - T(1)), dpi = T(7) * P.tait_k * ri6;
  const T av = P.alpha * P.visc_unit, nu8 = T(8) * P.nu, df = P.mog ? T(-2) * P.diff_k * P.rho0 : T(0);
  T gx = 0, gy = 0, gvx = 0, gvy = 0, gr = 0;
  da = 0;
  for (int k = sub; k < m; k += kLanes) {
    const int j = (int)__ldg(cols + k);
    const T rj = rt[j], Aj = area[j];
    DropPair e;
    if (!drop_pair(xi, vi, ri, x[j], v[j], rj, P, e)) continue;
    const V2 lxj1 = lx1[j], lvj1 = lv1[j];
    const T lbx = dt * lvj1.x + dt2 * lxj1.x, lby = dt * lvj1.y + dt2 * lxj1.y, le = sdp * lr1[j];
    const T rhoj = P.rho0 * rj, Vj = Aj * e.irj, mj = P.rho0 * Aj;
    const T Pp = pi + tait7(rj, P);
    const T ea = lax * e.dx + lay * e.dy, eb = lbx * e.dx + lby * e.dy;   // la . d, lb . d
    const T fa = lax * e.wx + lay * e.wy, fb = lbx * e.wx + lby * e.wy;   // la . w, lb . w
    const T cij = Vj * irhoi, cji = Vi * (e.irj * P.inv_rho0);
    const T Q1 = cji * eb - cij * ea;
    const T Q2 = mj * ea - mi * eb;
    const T mri = mj * rhoi, mrj = mi * rhoj;
    const T Q3 = mri * fa - mrj * fb;
    const T Q4 = mj * ld + mi * le;
    const T Q5 = Vj * ld - Vi * le;
    const T a = T(1) - e.r * P.inv_h;
    const T g1 = T(1.5) * P.cg20 * P.inv_h * P.inv_h * (a * a) * e.ir;   // d gd / d r2
    const T gi = e.gd * e.iR, dgi = (g1 - gi) * e.iR;                   // gd iR and its d / d r2
    const T rgi = e.r2 * gi, drgi = gi + e.r2 * dgi;                    // gd r2 iR
    const bool closing = !(e.s > T(0));
    const T s = closing ? e.s : T(0);
    const T kv = av * e.irs, kl = nu8 * e.irs * e.irs, D = rj - ri;
    // d F / d r2 with d and w held, times two
    const T f2 = T(2) * (g1 * (Pp * Q1 + e.s * Q4) + kv * s * Q2 * dgi + (kl * Q3 + df * D * Q5) * drgi);
    // d F / d (la . d), d F / d (lb . d), d F / d s
    const T cp = e.gd * Pp, cv = kv * gi * s;
    const T wa = cv * mj - cp * cij, wb = cp * cji - cv * mi;
    const T ws = e.gd * Q4 + (closing ? kv * gi * Q2 : T(0));
    const T la3 = kl * rgi * mri, lb3 = -kl * rgi * mrj;   // d F / d (la . w), d F / d (lb . w)
    gx += f2 * e.dx + wa * lax + wb * lbx + ws * e.wx;
    gy += f2 * e.dy + wa * lay + wb * lby + ws * e.wy;
    gvx += ws * e.dx + la3 * lax + lb3 * lbx;
    gvy += ws * e.dy + la3 * lay + lb3 * lby;
    gr += e.gd * (dpi * Q1 + Pp * iri * (cij * ea - cji * eb)) - P.rho0 * e.irs * (cv * Q2) +
          kl * rgi * (mj * P.rho0 * fa - T(2) * P.rho0 * e.irs * Q3) + df * rgi * (D * (Vi * iri) * le - Q5);
    da += P.visc_unit * gi * e.irs * s * mj * ea;
  }
  gx = drop_sum<kLanes>(gx);
  gy = drop_sum<kLanes>(gy);
  gvx = drop_sum<kLanes>(gvx);
  gvy = drop_sum<kLanes>(gvy);
  gr = drop_sum<kLanes>(gr);
  da = drop_sum<kLanes>(da);
  g[0] = gx;
  g[1] = gy;
  g[2] = gvx;
  g[3] = gvy;
  g[4] = gr;
}

// The same sums in float by dual numbers, added in row order: of each pair the own row's share,
// then the neighbor row's.
template <int kLanes, typename Col>
__device__ __forceinline__ void adjoint_row(int i, int m, int sub, const Col* __restrict__ cols, float2 xi,
                                            float2 vi, float ri, const float2* __restrict__ x,
                                            const float2* __restrict__ v, const float* __restrict__ rt,
                                            const float* __restrict__ area, const DropParams<float>& P, float dt,
                                            const float2* __restrict__ lx1, const float2* __restrict__ lv1,
                                            const float* __restrict__ lr1, float lax, float lay, float ld,
                                            float (&g)[5], float& da) {
  using T = float;
  using D = Dual<T, 5>;
  const T dt2 = dt * dt, sdp = dt / P.rho0;
  D Xx, Xy, Vx, Vy, R;   // particle i's inputs, seeded
  Xx = make_const(xi.x, Xx);
  Xy = make_const(xi.y, Xy);
  Vx = make_const(vi.x, Vx);
  Vy = make_const(vi.y, Vy);
  R = make_const(ri, R);
  Xx.d[0] = T(1);
  Xy.d[1] = T(1);
  Vx.d[2] = T(1);
  Vy.d[3] = T(1);
  R.d[4] = T(1);
#pragma unroll
  for (int c = 0; c < 5; ++c) g[c] = 0.f;
  da = 0.f;
  const int longest = drop_longest<kLanes>(m);
  for (int q = 0; q < longest; q += kLanes) {
    T own[5] = {0, 0, 0, 0, 0}, other[5] = {0, 0, 0, 0, 0}, ta = 0;
    if (q + sub < m) {
      const int j = (int)__ldg(cols + q + sub);
      const float2 xj = x[j], vj = v[j];
      if (apart(xi.x, xi.y, xj.x, xj.y)) {
        const T rj = rt[j];
        const D Jx = make_const(xj.x, Xx), Jy = make_const(xj.y, Xx), Jvx = make_const(vj.x, Xx),
                Jvy = make_const(vj.y, Xx), Jr = make_const(rj, Xx);
        // row i, derivatives with respect to i
        const PairOut<D> o = pair_terms<D, T>(Xx, Xy, Vx, Vy, R, Jx, Jy, Jvx, Jvy, Jr, area[j], P);
#pragma unroll
        for (int c = 0; c < 5; ++c) own[c] = o.ax.d[c] * lax + o.ay.d[c] * lay + o.dp.d[c] * ld;
        ta = o.vx.v * lax + o.vy.v * lay;
        // row j, derivatives with respect to i (its column)
        const float2 lxj1 = lx1[j], lvj1 = lv1[j];
        const T lbx = dt * lvj1.x + dt2 * lxj1.x, lby = dt * lvj1.y + dt2 * lxj1.y, le = sdp * lr1[j];
        const PairOut<D> w = pair_terms<D, T>(Jx, Jy, Jvx, Jvy, Jr, Xx, Xy, Vx, Vy, R, area[i], P);
#pragma unroll
        for (int c = 0; c < 5; ++c) other[c] = w.ax.d[c] * lbx + w.ay.d[c] * lby + w.dp.d[c] * le;
      }
    }
#pragma unroll
    for (int l = 0; l < kLanes; ++l) {
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        const T a = __shfl_sync(0xffffffffu, own[c], l, kLanes);
        const T b = __shfl_sync(0xffffffffu, other[c], l, kLanes);
        g[c] += a;
        g[c] += b;
      }
    }
    da = drop_add_in_order<kLanes>(da, ta);
  }
}

// One step of the adjoint: from (lx', lv', lr') of step k+1 and the state of step k, the
// adjoint of step k and particle i's share of dL/d alpha (added to dalpha when accumulate).
template <int kLanes, typename T, typename V2, typename Col>
__global__ void __launch_bounds__(128) k_drop_adjoint(int n, DropRows<Col> rows,
                                                      const V2* __restrict__ x, const V2* __restrict__ v,
                                                      const T* __restrict__ rt, const T* __restrict__ area,
                                                      DropParams<T> P, T dt, const V2* __restrict__ lx1,
                                                      const V2* __restrict__ lv1, const T* __restrict__ lr1,
                                                      V2* __restrict__ lx0, V2* __restrict__ lv0,
                                                      T* __restrict__ lr0, T* __restrict__ dalpha, int accumulate) {
  const int row = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes);
  const int sub = threadIdx.x % kLanes;
  const bool live = row < n;
  const int i = live ? row : n - 1;
  const T dt2 = dt * dt, sdp = dt / P.rho0;
  const V2 xi = x[i], vi = v[i];
  const T ri = rt[i];
  // lambda of row i's outputs: acc via v' = v + dt a and x' = x + dt v + dt^2 a; dpdt via rho'
  const V2 lxi1 = lx1[i], lvi1 = lv1[i];
  const T lax = dt * lvi1.x + dt2 * lxi1.x, lay = dt * lvi1.y + dt2 * lxi1.y, ld = sdp * lr1[i];
  int m;
  const Col* cols = rows.row(i, m);
  T g[5], da;
  adjoint_row<kLanes>(i, m, sub, cols, xi, vi, ri, x, v, rt, area, P, dt, lx1, lv1, lr1, lax, lay, ld, g, da);
  if (!live || sub != 0) return;
  if (P.point_source) {  // a = -mag (x - c) away from the centre
    const T dx = xi.x - P.cx, dy = xi.y - P.cy;
    if (dx * dx + dy * dy > T(1e-14)) {
      g[0] += -P.point_mag * lax;
      g[1] += -P.point_mag * lay;
    }
  }
  V2 ox, ov;
  ox.x = lxi1.x + g[0];
  ox.y = lxi1.y + g[1];
  ov.x = lvi1.x + dt * lxi1.x + g[2];
  ov.y = lvi1.y + dt * lxi1.y + g[3];
  lx0[i] = ox;
  lv0[i] = ov;
  lr0[i] = lr1[i] + g[4];
  dalpha[i] = accumulate ? dalpha[i] + da : da;
}

// ---------------------------------------------------------------- pairs of one step
// The columns of the particles in cell-sorted order, kDropLanes lanes per particle, into rows of
// `room` slots: no count, no scan and no second test of the candidates (with those and a launch
// of its own for the order a search took 25 us more than its sort at 16,173 particles, this
// one 8).  The candidates are walked as one range per three cell rows, and a lane's hits are
// placed by the group's ballot, so a row
// comes in cell order whatever the timing.  kOrdered: through shared memory in increasing
// order, a column's place the number of the row's columns below it.  A row with more
// columns than slots is left empty and flags SPH_FLAG_PAIR_CAPACITY.
constexpr int kDropLanes = 8, kDropBlock = 128, kDropBlockRows = kDropBlock / kDropLanes;
constexpr int kDropOrderedRoom = 512;   // slots up to which a block's rows fit in shared memory

template <bool kOrdered>
__global__ void __launch_bounds__(kDropBlock) k_drop_pairs(const float2* __restrict__ xs,
                                                           const float* __restrict__ support, int n,
                                                           const uint32_t* __restrict__ keys,
                                                           const int32_t* __restrict__ cell_start,
                                                           const sph_grid* __restrict__ gp, int32_t cap,
                                                           const uint32_t* __restrict__ order, int room,
                                                           int32_t* __restrict__ counts, int32_t* __restrict__ cols,
                                                           int32_t* status) {
  extern __shared__ int32_t drop_stage[];   // kOrdered: kDropBlockRows rows of room + 1
  const int64_t particle = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kDropLanes;
  const bool live = particle < n;   // lanes past the last particle take part in the warp's votes
  const int s = live ? (int)particle : n - 1;
  const int lane = threadIdx.x & 31, sub = lane % kDropLanes, base = lane - sub;
  const sph_grid g = *gp;
  const uint32_t key = keys[s];
  const int i = (int)order[s];
  int32_t* const out = cols + (int64_t)i * room;
  int32_t* const row = kOrdered ? drop_stage + (threadIdx.x / kDropLanes) * (room + 1) : out;
  const float2 xi = xs[s];
  const float thr = grid_threshold(support[i], g);
  int b[3] = {}, n0 = 0, n1 = 0, n2 = 0;   // the cell rows' first candidates, and candidates up to each one's end
  if (live && grid_ok(g, cap) && key < (uint32_t)g.num_cells) {
    const int cx = (int)(key % (uint32_t)g.cells_x), cy = (int)(key / (uint32_t)g.cells_x);
    const int x0 = max(cx - 1, 0), x1 = min(cx + 1, g.cells_x - 1);
    const int y0 = max(cy - 1, 0), y1 = min(cy + 1, g.cells_y - 1);
    int e[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int32_t* first = cell_start + (int64_t)min(y0 + q, y1) * g.cells_x;
      b[q] = __ldg(first + x0);
      e[q] = y0 + q <= y1 ? __ldg(first + x1 + 1) : b[q];
    }
    n0 = e[0] - b[0];
    n1 = n0 + e[1] - b[1];
    n2 = n1 + e[2] - b[2];
  }
  int found = 0;
  const int longest = __reduce_max_sync(0xffffffffu, n2);
  for (int t0 = 0; t0 < longest; t0 += kDropLanes) {
    const int t = t0 + sub;
    const int j = t < n0 ? b[0] + t : t < n1 ? b[1] + t - n0 : b[2] + t - n1;
    bool hit = false;
    if (t < n2) {
      const float2 xj = __ldg(xs + j);
      hit = dist2_ref(xi.x, xi.y, xj.x, xj.y) <= thr;
    }
    const unsigned hits = __ballot_sync(0xffffffffu, hit) >> base & ((1u << kDropLanes) - 1u);
    const int at = found + __popc(hits & ((1u << sub) - 1u));
    if (hit && at < room) row[at] = (int32_t)order[j];
    found += __popc(hits);
  }
  if (found > room) {
    if (sub == 0) flag(status, SPH_FLAG_PAIR_CAPACITY);
    found = 0;
  }
  if (live && sub == 0) counts[i] = found;
  if constexpr (kOrdered) {
    constexpr int kKeep = 4;   // columns a lane places at a time
    const int most = __reduce_max_sync(0xffffffffu, found);
    __syncwarp();
    for (int t0 = 0; t0 < most; t0 += kKeep * kDropLanes) {
      int32_t v[kKeep];
      int place[kKeep] = {};
#pragma unroll
      for (int q = 0; q < kKeep; ++q) {
        const int t = t0 + q * kDropLanes + sub;
        v[q] = t < found ? row[t] : 0x7fffffff;
      }
#pragma unroll 4
      for (int u = 0; u < most; ++u) {
        const int32_t c = u < found ? row[u] : 0x7fffffff;
#pragma unroll
        for (int q = 0; q < kKeep; ++q) place[q] += c < v[q];
      }
#pragma unroll
      for (int q = 0; q < kKeep; ++q)
        if (t0 + q * kDropLanes + sub < found) out[place[q]] = v[q];
    }
  }
}

template <typename T>
DropParams<T> drop_params(const sph_params* p, int mog) {
  DropParams<T> P;
  const double h = p->support;
  P.inv_h = T(1.0 / h);
  P.cg20 = T(20.0 * 7.0 / 3.14159265358979323846 / (h * h * h));
  P.rho0 = T(p->rest_density);
  P.inv_rho0 = T(1.0 / p->rest_density);
  P.tait_k = T((double)p->rest_density * p->c0 * p->c0 / p->gamma);
  P.eps = T(h * h * 0.1);
  P.visc_unit = T(h * p->c0);
  P.alpha = T(p->alpha);
  P.nu = T(p->kinematic);
  P.diff_k = T(h * p->delta * p->c0);
  P.gx = T(p->gravity[0]);
  P.gy = T(p->gravity[1]);
  P.point_source = p->point_source;
  P.point_mag = T(p->point_magnitude);
  P.cx = T(p->point_center[0]);
  P.cy = T(p->point_center[1]);
  P.mog = mog;
  return P;
}

// The columns of every row in increasing order, in -> out (distinct columns): one warp per row, for
// rows of more slots than shared memory takes.
__global__ void __launch_bounds__(256) k_order_rows(int n, int room, const int32_t* __restrict__ counts,
                                                    const int32_t* __restrict__ in, int32_t* __restrict__ out) {
  const int i = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (i >= n) return;
  const int m = min(counts[i], room);
  const int32_t* const row = in + (int64_t)i * room;
  for (int t0 = 0; t0 < m; t0 += 32) {
    const int t = t0 + lane;
    const int j = t < m ? __ldg(row + t) : 0x7fffffff;
    int r = 0;
    for (int u0 = 0; u0 < m; u0 += 32) {
      const int u = u0 + lane;
      const int ju = u0 == t0 ? j : u < m ? __ldg(row + u) : 0x7fffffff;
      const int len = min(m - u0, 32);
      for (int k = 0; k < len; ++k) r += __shfl_sync(0xffffffffu, ju, k) < j;
    }
    if (t < m) out[(int64_t)i * room + r] = j;
  }
}

}  // namespace sph

using namespace sph;

// Lanes per row, 8 while the launch has few blocks per SM, then 4: a row's sums and end are paid once per
// lane.  The line lies where the two measured the same: in double (bound by the FP64 pipe) at one
// block per SM, in float at ten for the right-hand side and four for the adjoint.  us with 8 / 4
// lanes, right-hand side and adjoint:
//   double   1,917 particles 18.5 / 22.9, 27.5 / 43.9;   2,893: 31.2 / 23.8, 50.3 / 45.0;
//            5,877: 45.9 / 39.5, 74.7 / 82.2;  8,029: 60.3 / 40.9, 99 / 85;  16,173: 104 / 79, 172 / 165;
//            65,049: 393 / 264, 655 / 564
//   float    3,985 particles 7.4 / 10.2, 10.2 / 12.2;  8,029: 8.1 / 10.7, 13.5 / 14.3;
//            12,093: 8.4 / 11.0, 22.2 / 17.0;  16,173: 9.4 / 11.5, 24.9 / 20.2;  23,709: 12.2 / 12.1,
//            34.6 / 31.9;  65,049: 27.5 / 24.2, 81 / 67;  130,429: 52 / 43, 166 / 129
static int drop_lanes(bool fp64, bool adjoint, int64_t n) {
  const int blocks = fp64 ? 1 : adjoint ? 4 : 10;   // per SM
  return n * 8 <= (int64_t)blocks * 128 * kNumSMs ? 8 : 4;
}

template <int kLanes, typename T, typename V2, bool kStep, typename Col>
static void rhs_as(int64_t n, const DropRows<Col>& rows, const void* x, const void* v, const void* rho,
                   const void* area, const sph_params* params, double dt, void* acc, void* dpdt, void* xo, void* vo, void* ro, float* x32,
                   cudaStream_t st) {
  k_drop_rhs<kLanes, T, V2, Col, kStep><<<grid_for(n * kLanes, 128), 128, 0, st>>>(
      (int)n, rows, static_cast<const V2*>(x), static_cast<const V2*>(v), static_cast<const T*>(rho),
      static_cast<const T*>(area), drop_params<T>(params, params->density_diffusion == 1), (T)dt, static_cast<V2*>(acc),
      static_cast<T*>(dpdt), static_cast<V2*>(xo), static_cast<V2*>(vo), static_cast<T*>(ro),
      reinterpret_cast<float2*>(x32));
}

template <int kLanes, typename T, typename V2, typename Col>
static void adjoint_as(int64_t n, const DropRows<Col>& rows, const void* x, const void* v, const void* rho,
                       const void* area, const sph_params* params, double dt, const void* lx1, const void* lv1,
                       const void* lr1, void* lx0, void* lv0, void* lr0, void* dalpha, int accumulate,
                       cudaStream_t st) {
  k_drop_adjoint<kLanes, T, V2, Col><<<grid_for(n * kLanes, 128), 128, 0, st>>>(
      (int)n, rows, static_cast<const V2*>(x), static_cast<const V2*>(v), static_cast<const T*>(rho),
      static_cast<const T*>(area), drop_params<T>(params, params->density_diffusion == 1), (T)dt,
      static_cast<const V2*>(lx1), static_cast<const V2*>(lv1), static_cast<const T*>(lr1), static_cast<V2*>(lx0),
      static_cast<V2*>(lv0), static_cast<T*>(lr0), static_cast<T*>(dalpha), accumulate);
}

template <bool kStep, typename Col, typename... Args>
static void launch_rhs(int32_t fp64, int64_t n, Args... args) {
  const bool four = drop_lanes(fp64, false, n) == 4;
  if (fp64)
    four ? rhs_as<4, double, double2, kStep, Col>(n, args...) : rhs_as<8, double, double2, kStep, Col>(n, args...);
  else
    four ? rhs_as<4, float, float2, kStep, Col>(n, args...) : rhs_as<8, float, float2, kStep, Col>(n, args...);
}

template <typename Col, typename... Args>
static void launch_adjoint(int32_t fp64, int64_t n, Args... args) {
  const bool four = drop_lanes(fp64, true, n) == 4;
  if (fp64)
    four ? adjoint_as<4, double, double2, Col>(n, args...) : adjoint_as<8, double, double2, Col>(n, args...);
  else
    four ? adjoint_as<4, float, float2, Col>(n, args...) : adjoint_as<8, float, float2, Col>(n, args...);
}

// The scratch of sph_drop_search, in order: cell_count [cap + 1] (zero between calls), cell_start
// [cap + 2], keys, order, sorted keys [n], sorted positions float2 [n], the sort's scratch.
struct DropScratch {
  int32_t *cell_count, *cell_start;
  uint32_t *keys, *order, *skeys;
  float* xs;
  void* sort;
  size_t sort_bytes;
};

static size_t drop_scratch(int64_t n, int32_t cap, char* base, DropScratch* s) {
  size_t at = 0;
  const auto take = [&](size_t bytes) {
    char* p = base ? base + at : nullptr;
    at += (bytes + 255) & ~(size_t)255;
    return p;
  };
  DropScratch d;
  d.cell_count = reinterpret_cast<int32_t*>(take(((size_t)cap + 1) * 4));
  d.cell_start = reinterpret_cast<int32_t*>(take(((size_t)cap + 2) * 4));
  d.keys = reinterpret_cast<uint32_t*>(take((size_t)n * 4));
  d.order = reinterpret_cast<uint32_t*>(take((size_t)n * 4));
  d.skeys = reinterpret_cast<uint32_t*>(take((size_t)n * 4));
  d.xs = reinterpret_cast<float*>(take((size_t)n * 8));
  d.sort_bytes = sph_counting_sort_scratch_bytes(n, cap);
  d.sort = take(d.sort_bytes);
  if (s) *s = d;
  return at;
}

#define SPH_DROP_PARAMS(p)                                                \
  ((p) && (p)->support > 0.f && (p)->gamma == 7.f &&                      \
   ((p)->density_diffusion == 0 || (p)->density_diffusion == 1))

extern "C" {

size_t sph_drop_search_scratch_bytes(int64_t n, int32_t cell_capacity) {
  return drop_scratch(n > 0 ? n : 0, cell_capacity > 0 ? cell_capacity : 0, nullptr, nullptr) + 256;
}

sph_status_t sph_drop_search(const float* x32, const float* support, int64_t n, const sph_grid* grid,
                             int32_t cell_capacity, int32_t* counts, int32_t row_capacity, int32_t* cols,
                             int32_t ordered, int32_t* unordered, int32_t* status, void* scratch, size_t scratch_bytes,
                             void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && cell_capacity > 0 && grid && status && row_capacity > 0 &&
                  (n == 0 || (x32 && support && cols && counts)) &&
                  (!ordered || row_capacity <= kDropOrderedRoom || (unordered && unordered != cols)),
              "drop_search: bad arguments");
  if (!scratch || scratch_bytes < sph_drop_search_scratch_bytes(n, cell_capacity)) {
    set_error_text("drop_search: scratch smaller than sph_drop_search_scratch_bytes(n, cell_capacity)");
    return SPH_ERR_SCRATCH_TOO_SMALL;
  }
  if (n == 0) return SPH_OK;
  cudaStream_t st = as_stream(stream);
  DropScratch d;
  char* base = reinterpret_cast<char*>((reinterpret_cast<uintptr_t>(scratch) + 255) & ~(uintptr_t)255);
  drop_scratch(n, cell_capacity, base, &d);
  sph_status_t r = sph_cell_keys(x32, n, grid, cell_capacity, d.keys, nullptr, d.cell_count, status, stream);
  if (r != SPH_OK) return r;
  const int32_t eb[1] = {8};
  const void* in[1] = {x32};
  void* out[1] = {d.xs};
  r = sph_counting_sort_permute(d.keys, n, cell_capacity, d.cell_count, d.cell_start, nullptr, d.order, d.skeys, 1, eb,
                                in, out, status, d.sort, d.sort_bytes, stream);
  if (r != SPH_OK) return r;
  const int nb = grid_for(n * kDropLanes, kDropBlock);
  const float2* xs = reinterpret_cast<const float2*>(d.xs);
  const bool in_block = ordered && row_capacity <= kDropOrderedRoom;
  if (in_block)
    k_drop_pairs<true><<<nb, kDropBlock, kDropBlockRows * (row_capacity + 1) * sizeof(int32_t), st>>>(
        xs, support, (int)n, d.skeys, d.cell_start, grid, cell_capacity, d.order, row_capacity, counts, cols, status);
  else
    k_drop_pairs<false><<<nb, kDropBlock, 0, st>>>(xs, support, (int)n, d.skeys, d.cell_start, grid, cell_capacity,
                                                   d.order, row_capacity, counts, ordered ? unordered : cols, status);
  if (ordered && !in_block)
    k_order_rows<<<grid_for(n, 8), 256, 0, st>>>((int)n, row_capacity, counts, unordered, cols);
  SPH_CHECK_LAUNCH("drop_search");
  return SPH_OK;
}

sph_status_t sph_drop_step(int32_t fp64, int64_t n, const int32_t* row_info, const int32_t* cols,
                           int32_t row_capacity, const void* x, const void* v, const void* rho, const void* area,
                           const sph_params* params, double dt, void* x_out, void* v_out, void* rho_out, float* x32_out,
                           void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && SPH_DROP_PARAMS(params) && params->rest_density > 0 &&
                  (n == 0 || (row_capacity >= 0 && row_info && cols && x && v && rho && area && x_out && v_out &&
                              rho_out)),
              "drop_step: bad arguments (gamma 7, MOG or no density diffusion)");
  SPH_REQUIRE(n == 0 || (x_out != x && v_out != v && rho_out != rho), "drop_step: outputs must not alias inputs");
  if (n == 0) return SPH_OK;
  launch_rhs<true, int32_t>(fp64, n, DropRows<int32_t>{row_info, cols, row_capacity}, x, v, rho, area, params, dt,
                            nullptr, nullptr, x_out, v_out, rho_out, x32_out, as_stream(stream));
  SPH_CHECK_LAUNCH("drop_step");
  return SPH_OK;
}

sph_status_t sph_drop_adjoint_step(int32_t fp64, int64_t n, const int32_t* row_info, const int32_t* cols,
                                   int32_t row_capacity, const void* x, const void* v, const void* rho,
                                   const void* area, const sph_params* params, double dt, const void* lx1,
                                   const void* lv1, const void* lr1, void* lx0, void* lv0, void* lr0, void* dalpha,
                                   void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && SPH_DROP_PARAMS(params) &&
                  (n == 0 || (row_capacity >= 0 && row_info && cols && x && v && rho && area && lx1 && lv1 && lr1 &&
                              lx0 && lv0 && lr0 && dalpha)),
              "drop_adjoint_step: bad arguments (gamma 7, MOG or no density diffusion)");
  SPH_REQUIRE(lx0 != lx1 && lv0 != lv1 && lr0 != lr1, "drop_adjoint_step: outputs must not alias inputs");
  if (n == 0) return SPH_OK;
  launch_adjoint<int32_t>(fp64, n, DropRows<int32_t>{row_info, cols, row_capacity}, x, v, rho, area, params, dt, lx1,
                          lv1, lr1, lx0, lv0, lr0, dalpha, 1, as_stream(stream));
  SPH_CHECK_LAUNCH("drop_adjoint_step");
  return SPH_OK;
}

sph_status_t sph_drop_rhs(int32_t fp64, int64_t n, const int32_t* offsets, const int64_t* cols, const void* x,
                          const void* v, const void* rho, const void* area, const sph_params* params, void* acc,
                          void* dpdt, void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && params && params->support > 0.f && params->gamma == 7.f &&
                  (params->density_diffusion == 0 || params->density_diffusion == 1) &&
                  (n == 0 || (offsets && cols && x && v && rho && area && acc && dpdt)),
              "drop_rhs: bad arguments (gamma 7, MOG or no density diffusion)");
  if (n == 0) return SPH_OK;
  launch_rhs<false, int64_t>(fp64, n, DropRows<int64_t>{offsets, cols, 0}, x, v, rho, area, params, 0.0, acc, dpdt,
                             nullptr, nullptr, nullptr, nullptr, as_stream(stream));
  SPH_CHECK_LAUNCH("drop_rhs");
  return SPH_OK;
}

sph_status_t sph_drop_integrate(int32_t fp64, int64_t n, void* x, void* v, void* rho, const void* acc,
                                const void* dpdt, double dt, double rest_density, void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && (n == 0 || (x && v && rho && acc && dpdt)) && rest_density > 0,
              "drop_integrate: bad arguments");
  if (n == 0) return SPH_OK;
  cudaStream_t st = as_stream(stream);
  if (fp64)
    k_drop_sie<double, double2><<<grid_for(n, 256), 256, 0, st>>>(
        (int)n, static_cast<double2*>(x), static_cast<double2*>(v), static_cast<double*>(rho),
        static_cast<const double2*>(acc), static_cast<const double*>(dpdt), dt, rest_density);
  else
    k_drop_sie<float, float2><<<grid_for(n, 256), 256, 0, st>>>(
        (int)n, static_cast<float2*>(x), static_cast<float2*>(v), static_cast<float*>(rho),
        static_cast<const float2*>(acc), static_cast<const float*>(dpdt), (float)dt, (float)rest_density);
  SPH_CHECK_LAUNCH("drop_integrate");
  return SPH_OK;
}

sph_status_t sph_drop_adjoint(int32_t fp64, int64_t n, const int32_t* offsets, const int64_t* cols, const void* x,
                              const void* v, const void* rho, const void* area, const sph_params* params, double dt,
                              const void* lx1, const void* lv1, const void* lr1, void* lx0, void* lv0, void* lr0,
                              void* dalpha, void* stream) {
  SPH_REQUIRE(n >= 0 && n < (1LL << 31) && params && params->support > 0.f && params->gamma == 7.f &&
                  (params->density_diffusion == 0 || params->density_diffusion == 1) &&
                  (n == 0 || (offsets && cols && x && v && rho && area && lx1 && lv1 && lr1 && lx0 && lv0 && lr0 &&
                              dalpha)),
              "drop_adjoint: bad arguments (gamma 7, MOG or no density diffusion)");
  SPH_REQUIRE(lx0 != lx1 && lv0 != lv1 && lr0 != lr1, "drop_adjoint: outputs must not alias inputs");
  if (n == 0) return SPH_OK;
  launch_adjoint<int64_t>(fp64, n, DropRows<int64_t>{offsets, cols, 0}, x, v, rho, area, params, dt, lx1, lv1, lr1,
                          lx0, lv0, lr0, dalpha, 0, as_stream(stream));
  SPH_CHECK_LAUNCH("drop_adjoint");
  return SPH_OK;
}

}  // extern "C"
