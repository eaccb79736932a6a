// Shared device helpers of the GB300 SPH hot path (sm_103a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/sph_gb300.h"

namespace sph {

// Records the last CUDA error text for sph_last_error().
void set_error(const char* where, cudaError_t err);
void set_error_text(const char* text);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

#define SPH_CHECK_LAUNCH(where)                            \
  do {                                                     \
    cudaError_t e_ = cudaGetLastError();                   \
    if (e_ != cudaSuccess) {                               \
      ::sph::set_error(where, e_);                         \
      return SPH_ERR_CUDA;                                 \
    }                                                      \
  } while (0)

#define SPH_REQUIRE(cond, msg)                 \
  do {                                         \
    if (!(cond)) {                             \
      ::sph::set_error_text(msg);              \
      return SPH_ERR_INVALID_ARGUMENT;         \
    }                                          \
  } while (0)

constexpr int kNumSMs = 152;

inline int grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  return (int)(b < 1 ? 1 : b);
}

// The reference pair predicate, cppSrc/neighSearch.cpp:222-223 as compiled with the
// reference's flags (GCC contracts dx*dx + dy*dy into fmaf(dx, dx, dy*dy)):
//   sqrtf(fmaf(dx, dx, dy*dy)) < h_i,  dx = x_i - x_j (i = query).
// Every operation is spelled as a round-to-nearest intrinsic so nvcc can neither
// contract nor approximate it.
__device__ __forceinline__ float dist2_ref(float xi, float yi, float xj, float yj) {
  float dx = __fsub_rn(xi, xj);
  float dy = __fsub_rn(yi, yj);
  return __fmaf_rn(dx, dx, __fmul_rn(dy, dy));
}

// Square-root-free form of the same predicate.  For a float v >= 0 and a float h > 0,
// with IEEE round-to-nearest sqrt:  RN(sqrt(v)) < h  <=>  sqrt(v) < m, where m is the
// midpoint between h and its float predecessor (RN(x) <= pred(h) exactly when x < m; a tie
// x = m cannot occur because m^2 has an odd ~50-bit significand while v has 24 bits).
// m^2 is exact in double, so the predicate is  v <= F  with F the largest float below
// m^2.  F is computed once per query particle; the candidate loop then needs no sqrt.
// The double arithmetic is slow on GB300, so kernels take F from a table computed once
// (grid_threshold, SphParams::thr) whenever the support is the common one.
__host__ __device__ __forceinline__ float sq_threshold(float h) {
  if (!(h > 0.f)) return -1.0f;          // sqrt(v) >= 0 >= h: nothing passes (NaN h too)
  if (isinf(h)) return 3.40282347e38f;   // every finite v passes
  float p = nextafterf(h, 0.0f);
  double m = ((double)p + (double)h) * 0.5;
  double m2 = m * m;
#ifdef __CUDA_ARCH__
  float f = __double2float_rn(m2);
#else
  float f = (float)m2;                   // round to nearest, as on the device
#endif
  if ((double)f >= m2) f = nextafterf(f, 0.0f);
  return f;
}

// sq_threshold(h) for a query of support h in grid g: the grid carries the value for its
// largest support (threshold_support, or the cell size hmax when that is 0), computed once
// by sph_grid_build.
__device__ __forceinline__ float grid_threshold(float h, const sph_grid& g) {
  const float hs = g.threshold_support > 0.f ? g.threshold_support : g.hmax;
  return (h == hs && g.hmax_threshold > 0.f) ? g.hmax_threshold : sq_threshold(h);
}

// Reference predicate with the distance: true iff sqrtf(fmaf(dx,dx,dy*dy)) < h_i.
__device__ __forceinline__ bool pair_pred(float xi, float yi, float xj, float yj, float hi, float* dist) {
  float v = dist2_ref(xi, yi, xj, yj);
  float d = __fsqrt_rn(v);
  *dist = d;
  return d < hi;
}

// Cell coordinate of sortPositions, src/modules/neighborSearch.py:46:
//   ceil((x - qmin) / hmax) in float32, then int32 conversion.
__device__ __forceinline__ int cell_coord(float x, float qmin, float hmax) {
  return (int)ceilf(__fdiv_rn(__fsub_rn(x, qmin), hmax));
}

// Wendland C2 in 2D, src/kernels.py:20-24: W(q) = 7/(pi h^2) (1-q)^4 (1+4q).
// c_w = 7/(pi h^2) precomputed by the caller.
__device__ __forceinline__ float wendland(float q, float c_w) {
  float a = 1.0f - q;
  float a2 = a * a;
  return a2 * a2 * (1.0f + 4.0f * q) * c_w;
}

// A grid is usable only if its cells fit the cell table.
__device__ __forceinline__ bool grid_ok(const sph_grid& g, int32_t cap) {
  return g.num_cells <= cap && g.cells_x > 0 && g.cells_y > 0;
}

// Up to kMaxArrays per-particle arrays moved together into a new order (4-, 8- or 16-byte
// rows): the permute kernel and the counting sort's in-cell fix copy row src of every
// in[k] to row dst of out[k].
constexpr int kMaxArrays = 8;
struct ArraySet {
  const void* in[kMaxArrays];
  void* out[kMaxArrays];
  int32_t bytes[kMaxArrays];
  int32_t count;
};

// The set from host arrays of `count` entries; false for a count above kMaxArrays, a
// missing or shared in/out pointer, or a row size other than 4, 8 or 16 bytes.
inline bool array_set_from(int32_t count, const int32_t* elem_bytes, const void* const* in, void* const* out,
                           ArraySet* a) {
  if (count < 0 || count > kMaxArrays || (count > 0 && (!elem_bytes || !in || !out))) return false;
  a->count = count;
  for (int k = 0; k < kMaxArrays; ++k) {
    a->in[k] = nullptr;
    a->out[k] = nullptr;
    a->bytes[k] = 4;
  }
  for (int k = 0; k < count; ++k) {
    if (!in[k] || !out[k] || in[k] == out[k] || (elem_bytes[k] != 4 && elem_bytes[k] != 8 && elem_bytes[k] != 16))
      return false;
    a->in[k] = in[k];
    a->out[k] = out[k];
    a->bytes[k] = elem_bytes[k];
  }
  return true;
}

// Rows of arrays first .. first + 3, all four loads in flight before the first store: copied one
// after another each row waits for its own load.
struct FourRows {
  uint4 v[4];
};

__device__ __forceinline__ FourRows load_rows(const ArraySet& a, int first, int64_t src) {
  FourRows r;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = first + q;
    if (k >= a.count) break;
    switch (a.bytes[k]) {
      case 4:
        r.v[q].x = __ldg(static_cast<const uint32_t*>(a.in[k]) + src);
        break;
      case 8: {
        const uint2 w = __ldg(static_cast<const uint2*>(a.in[k]) + src);
        r.v[q].x = w.x;
        r.v[q].y = w.y;
        break;
      }
      default:
        r.v[q] = __ldg(static_cast<const uint4*>(a.in[k]) + src);
        break;
    }
  }
  return r;
}

__device__ __forceinline__ void store_rows(const ArraySet& a, int first, int64_t dst, const FourRows& r) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = first + q;
    if (k >= a.count) break;
    switch (a.bytes[k]) {
      case 4:
        static_cast<uint32_t*>(a.out[k])[dst] = r.v[q].x;
        break;
      case 8:
        static_cast<uint2*>(a.out[k])[dst] = make_uint2(r.v[q].x, r.v[q].y);
        break;
      default:
        static_cast<uint4*>(a.out[k])[dst] = r.v[q];
        break;
    }
  }
}

// Rows from array `first` on.
__device__ __forceinline__ void copy_rows(const ArraySet& a, int64_t dst, int64_t src, int first = 0) {
#pragma unroll
  for (int k = 0; k < kMaxArrays; k += 4)
    if (k >= first && k < a.count) store_rows(a, k, dst, load_rows(a, k, src));
}

// ---------------------------------------------------------------- bitonic sorts in shared memory
// One step of a bitonic sort of the p2 shared words s (a power of two) by `threads` threads, of which
// this is number t: each pair (a, a ^ x), a = the p-th index without the bit `half`, is put in
// increasing order.  x = 2 half - 1 (the step that begins a merge) or half.  A thread's
// kPairs pairs (p = t, t + threads, ..) are in flight together.
template <int kPairs, typename W>
__device__ __forceinline__ void compare_pairs(W* s, int p2, int half, int x, int t, int threads) {
  int a[kPairs];
  W lo[kPairs], hi[kPairs];
#pragma unroll
  for (int q = 0; q < kPairs; ++q) {
    const int p = t + q * threads;
    a[q] = p < p2 / 2 ? 2 * p - (p & (half - 1)) : -1;
    lo[q] = a[q] >= 0 ? s[a[q]] : 0;
    hi[q] = a[q] >= 0 ? s[a[q] ^ x] : 0;
  }
#pragma unroll
  for (int q = 0; q < kPairs; ++q)
    if (lo[q] > hi[q]) {   // (never without a pair)
      s[a[q]] = hi[q];
      s[a[q] ^ x] = lo[q];
    }
}

// The p2 words in increasing order, by a block (after a barrier; ends with one).
constexpr int kBlockSortWords = 2048;   // (more than two pairs of a thread in flight cost a block its registers)

template <typename W>
__device__ __forceinline__ void block_sort(W* s, int p2) {
  const auto step = [&](int half, int x) {
    if (p2 <= 2 * (int)blockDim.x)
      compare_pairs<1>(s, p2, half, x, threadIdx.x, blockDim.x);
    else
#pragma unroll 1
      for (int t = threadIdx.x; t < p2 / 2; t += 2 * blockDim.x) compare_pairs<2>(s, p2, half, x, t, blockDim.x);
    __syncthreads();
  };
  for (int size = 2; size <= p2; size <<= 1) {
    step(size >> 1, size - 1);
    for (int stride = size >> 2; stride > 0; stride >>= 1) step(stride, stride);
  }
}

// The columns in[0, len), renumbered by `order` (may be NULL), in increasing order to row[0, len), by
// a warp with kWarpSortWords shared words s.  Pieces of kWarpSortWords are sorted in s, then
// merged: steps over longer distances in `row` itself, the others in s again.  A place past the
// end of the row counts as the largest value and never moves.
constexpr int kWarpSortWords = 256;   // 4 pairs a lane

static __device__ __noinline__ void warp_sort_row(const int32_t* __restrict__ in, const uint32_t* __restrict__ order,
                                                  int len, int64_t* row, uint32_t* s) {
  constexpr int kW = kWarpSortWords;
  const int lane = threadIdx.x & 31;
  const auto step = [&](int half, int x) {
    compare_pairs<kW / 64>(s, kW, half, x, lane, 32);
    __syncwarp();
  };
  for (int base = 0; base < len; base += kW) {
#pragma unroll
    for (int q = 0; q < kW; q += 32) {
      const int t = base + q + lane;
      const uint32_t c = t < len ? (uint32_t)in[t] : 0u;
      s[q + lane] = t >= len ? 0xffffffffu : order ? __ldg(order + c) : c;
    }
    __syncwarp();
    for (int size = 2; size <= kW; size <<= 1) {
      step(size >> 1, size - 1);
      for (int stride = size >> 2; stride > 0; stride >>= 1) step(stride, stride);
    }
    for (int t = lane; t < min(len - base, kW); t += 32) row[base + t] = s[t];
    __syncwarp();
  }
  for (int64_t size = 2 * kW; size / 2 < len; size *= 2) {
    const int64_t pairs = (len + size - 1) / size * (size / 2);
    for (int64_t half = size / 2; half >= kW; half /= 2) {
      const int64_t x = half == size / 2 ? size - 1 : half;
#pragma unroll 4
      for (int64_t p = lane; p < pairs; p += 32) {
        const int64_t a = 2 * p - (p & (half - 1)), b = a ^ x;
        if (b < len) {
          const int64_t lo = row[a], hi = row[b];
          if (lo > hi) {
            row[a] = hi;
            row[b] = lo;
          }
        }
      }
      __syncwarp();
    }
    for (int base = 0; base < len; base += kW) {
#pragma unroll
      for (int q = 0; q < kW; q += 32) {
        const int t = base + q + lane;
        s[q + lane] = t < len ? (uint32_t)row[t] : 0xffffffffu;
      }
      __syncwarp();
      for (int stride = kW / 2; stride > 0; stride >>= 1) step(stride, stride);
      for (int t = lane; t < min(len - base, kW); t += 32) row[base + t] = s[t];
      __syncwarp();
    }
  }
}

// Rows past kLongRow columns are sorted by a kernel of their own: counting the smaller columns of each
// in a warp's registers, which the others do, is quadratic.  65,536 rows of 99 / 139 / 199 / 399
// columns with their distances take 212 / 348 / 671 / 2,376 us that way and 218 / 244 / 271 / 641
// sorted, 8,192 rows of 2,048 8.2 and 0.57 ms.  In the counting kernel itself the sort's shared words
// cost short rows 7 to 10 %; the launch without a long row takes 2.0 us at 65,536 rows, 3.3 at 260,017
// and 7.2 at 10^6 (2.9, 3.6 and 7.8 with twice the blocks).
constexpr int kLongRow = 112;
constexpr int kLongRowBlocks = 4 * kNumSMs;   // of 256 threads

// use(row, length) by a whole warp for every long row of n, by blocks of 256 threads: a block looks its
// share of the rows over, 256 at a time, and deals the long ones to its warps.
template <typename Length, typename Use>
__device__ __forceinline__ void for_long_rows(int64_t n, Length&& length, Use&& use) {
  __shared__ int at[256], lengths[256], count;
  const int64_t share = (n + gridDim.x - 1) / gridDim.x;
  const int64_t end = min((blockIdx.x + 1) * share, n);
  for (int64_t base = blockIdx.x * share; base < end; base += 256) {   // the same in the whole block
    const int64_t row = base + threadIdx.x;
    const int len = row < end ? length(row) : 0;
    if (!__syncthreads_or(len > kLongRow)) continue;
    if (threadIdx.x == 0) count = 0;
    __syncthreads();
    if (len > kLongRow) {
      const int q = atomicAdd(&count, 1);
      at[q] = threadIdx.x;
      lengths[q] = len;
    }
    __syncthreads();
    for (int q = threadIdx.x >> 5; q < count; q += 8) {
      use(base + at[q], lengths[q]);
      __syncwarp();
    }
  }
}

__device__ __forceinline__ void flag(int32_t* status, int32_t f) {
  if (status) atomicOr(status, f);
}

}  // namespace sph
