// Two-pass CSR neighbor list over particles in cell-sorted order (sm_103a).
//
// Layout: xy (float2, sorted), sorted support h, sorted area A, sorted cell keys, and the
// cell begin table cell_start[c] (cell c = [cell_start[c], cell_start[c+1])).  With the
// linear cell id ix + cells_x*iy, the cells (cx-r .. cx+r, yy) of one grid row are
// contiguous in the sorted order, so a particle scans 2r+1 contiguous index ranges.
//
// The pair test is the reference's sqrtf(fmaf(dx,dx,dy*dy)) < h_i in its square-root-free
// exact form v <= F_i (sq_threshold); the distance is taken only for accepted pairs that
// need it (density).
#include "sph_math.cuh"

namespace sph {

// Segments kept per particle by the one-scene search (the batch step's force passes keep
// kMaxSegments): a particle with more goes on the dense list.  24 covers three cell rows of
// up to 8 x 32 candidates each, ~9x the density of a jittered lattice at support 3 dx.
constexpr int kSearchSegments = 24;

template <typename F>
__device__ __forceinline__ void scan_candidates(const float2* __restrict__ xy, const int32_t* __restrict__ cell_start,
                                                const sph_grid& g, int r, int cx, int cy, float xi, float yi,
                                                float thr, F&& f) {
  const int x0 = max(cx - r, 0), x1 = min(cx + r, g.cells_x - 1);
  if (x0 > x1) return;
  const int y0 = max(cy - r, 0), y1 = min(cy + r, g.cells_y - 1);
  for (int yy = y0; yy <= y1; ++yy) {
    const int row = yy * g.cells_x;
    const int b = __ldg(cell_start + row + x0);
    const int e = __ldg(cell_start + row + x1 + 1);
    for (int j = b; j < e; ++j) {
      const float2 pj = __ldg(xy + j);
      const float v = dist2_ref(xi, yi, pj.x, pj.y);
      if (v <= thr) f(j, v);
    }
  }
}

__global__ void __launch_bounds__(256) k_nl_count(const float2* __restrict__ xy, const float* __restrict__ sh,
                                                  const float* __restrict__ sa, int64_t n,
                                                  const uint32_t* __restrict__ keys,
                                                  const int32_t* __restrict__ cell_start,
                                                  const sph_grid* __restrict__ gp, int32_t cap, int r,
                                                  float inv_support, float c_w, int32_t* __restrict__ counts,
                                                  float* __restrict__ rho) {
  int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const sph_grid g = *gp;
  const uint32_t key = keys[s];
  int cnt = 0;
  float acc = 0.f;
  if (grid_ok(g, cap) && key < (uint32_t)g.num_cells) {
    const float2 pi = xy[s];
    const float thr = grid_threshold(sh[s], g);
    const int cx = (int)(key % (uint32_t)g.cells_x), cy = (int)(key / (uint32_t)g.cells_x);
    if (rho) {   // the candidates in segments of 32, as k_nl_segments, so both give the same sums
      const int x0 = max(cx - r, 0), x1 = min(cx + r, g.cells_x - 1);
      const int y0 = max(cy - r, 0), y1 = min(cy + r, g.cells_y - 1);
      for (int yy = y0; yy <= y1 && x0 <= x1; ++yy) {
        const int row = yy * g.cells_x;
        const int b = __ldg(cell_start + row + x0), e = __ldg(cell_start + row + x1 + 1);
        for (int c = b; c < e; c += 32) {
          cnt += __popc(segment_mask_density(xy, sa, c, e, pi.x, pi.y, thr, inv_support, acc));
        }
      }
      acc *= c_w;
    } else {
      scan_candidates(xy, cell_start, g, r, cx, cy, pi.x, pi.y, thr, [&](int, float) { ++cnt; });
    }
  }
  counts[s] = cnt;
  if (rho) rho[s] = acc;
}

constexpr int kFillStage = 8192;  // CSR columns one 256-thread block builds in shared memory (32 KiB)

// Writes the row [offsets[s], offsets[s+1]) of particle s with the columns `scan` emits.
// The rows of one block are one contiguous span of cols, written through a shared-memory
// stage in windows of kFillStage columns: for each window the rows that reach into it emit
// their columns that fall inside it (a row across a window edge is emitted once per window
// it touches), and the block stores the window with coalesced stores.  A block whose span
// ends past the column buffer writes its rows in place instead, and a row that does not
// fit is skipped with SPH_FLAG_PAIR_CAPACITY set.  Every thread of the block must call
// this (inactive ones with active = false): it holds block barriers.
template <typename Scan>
__device__ __forceinline__ void staged_fill(int64_t s, int64_t n, bool active, const int32_t* __restrict__ offsets,
                                            int64_t pair_capacity, int32_t* __restrict__ cols, int32_t* status,
                                            Scan&& scan) {
  __shared__ int32_t stage[kFillStage];
  const int64_t b0 = (int64_t)blockIdx.x * blockDim.x;
  const int64_t b1 = min(b0 + (int64_t)blockDim.x, n);
  const int64_t span0 = offsets[b0], span1 = offsets[b1];
  const bool staged = span0 >= 0 && span1 >= span0 && span1 <= pair_capacity;  // the same in the whole block
  if (!staged) {
    if (!active) return;
    if ((int64_t)offsets[s + 1] <= pair_capacity) {
      int32_t o = offsets[s];
      const int32_t e = offsets[s + 1];
      if (o >= 0) scan([&](int j) {   // writes stay inside the row even if offsets disagree with the scan
        if (o < e) cols[o++] = j;
      });
    } else {
      flag(status, SPH_FLAG_PAIR_CAPACITY);
    }
    return;
  }
  if (span1 - span0 <= kFillStage) {   // one window
    if (active) {
      int32_t o = offsets[s] - (int32_t)span0;
      const int32_t e = offsets[s + 1] - (int32_t)span0;
      if (o >= 0) scan([&](int j) {
        if (o < e) stage[o++] = j;
      });
    }
    __syncthreads();
    for (int k = threadIdx.x; k < (int)(span1 - span0); k += blockDim.x) cols[span0 + k] = stage[k];
    return;
  }
  const int64_t r0 = active ? offsets[s] : 0, r1 = active ? offsets[s + 1] : 0;
  for (int64_t w0 = span0; w0 < span1; w0 += kFillStage) {
    const int64_t w1 = min(w0 + (int64_t)kFillStage, span1);
    if (active && r0 < w1 && r1 > w0) {
      int64_t o = r0;
      scan([&](int j) {
        if (o >= w0 && o < w1 && o < r1) stage[o - w0] = j;
        ++o;
      });
    }
    __syncthreads();
    for (int64_t k = threadIdx.x; k < w1 - w0; k += blockDim.x) cols[w0 + k] = stage[k];
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_nl_fill(const float2* __restrict__ xy, const float* __restrict__ sh, int64_t n,
                                                 const uint32_t* __restrict__ keys,
                                                 const int32_t* __restrict__ cell_start,
                                                 const sph_grid* __restrict__ gp, int32_t cap, int r,
                                                 const int32_t* __restrict__ offsets, int64_t pair_capacity,
                                                 int32_t* __restrict__ cols, int32_t* status) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const sph_grid g = *gp;
  const uint32_t key = s < n ? keys[s] : 0xffffffffu;
  const bool active = s < n && grid_ok(g, cap) && key < (uint32_t)g.num_cells;
  float2 pi = make_float2(0.f, 0.f);
  float thr = 0.f;
  if (active) {
    pi = xy[s];
    thr = grid_threshold(sh[s], g);
  }
  const int cx = active ? (int)(key % (uint32_t)g.cells_x) : 0, cy = active ? (int)(key / (uint32_t)g.cells_x) : 0;
  staged_fill(s, n, active, offsets, pair_capacity, cols, status, [&](auto&& emit) {
    scan_candidates(xy, cell_start, g, r, cx, cy, pi.x, pi.y, thr, [&](int j, float) { emit(j); });
  });
}

// One candidate pass for count, density and the CSR fill: particle s's cell rows are
// tested in segments of 32 candidates (segment_mask); the non-empty segments are stored for
// k_nl_fill_segments, the count is their bit count, and the density visits the set bits in
// order, the order of k_nl_count, so both give the same sums.  A particle with more than
// kSearchSegments segments gets nseg[s] = -1 and goes on the dense list, whose rows the fill
// writes one warp per particle.
__global__ void __launch_bounds__(256) k_nl_segments(const float2* __restrict__ xy, const float* __restrict__ sh,
                                                     const float* __restrict__ sa, int64_t n,
                                                     const uint32_t* __restrict__ keys,
                                                     const int32_t* __restrict__ cell_start,
                                                     const sph_grid* __restrict__ gp, int32_t cap, int r,
                                                     float inv_support, float c_w, int32_t* __restrict__ counts,
                                                     float* __restrict__ rho, int32_t* __restrict__ nseg,
                                                     int32_t* __restrict__ seg_start, uint32_t* __restrict__ seg_mask,
                                                     int32_t* __restrict__ dense_list, int32_t* __restrict__ dense_count) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const sph_grid g = *gp;
  const uint32_t key = keys[s];
  int cnt = 0, k = 0;
  float acc = 0.f;
  if (grid_ok(g, cap) && key < (uint32_t)g.num_cells) {
    const float2 pi = xy[s];
    const float thr = grid_threshold(sh[s], g);
    const int cx = (int)(key % (uint32_t)g.cells_x), cy = (int)(key / (uint32_t)g.cells_x);
    const int x0 = max(cx - r, 0), x1 = min(cx + r, g.cells_x - 1);
    const int y0 = max(cy - r, 0), y1 = min(cy + r, g.cells_y - 1);
    for (int yy = y0; yy <= y1 && x0 <= x1; ++yy) {
      const int row = yy * g.cells_x;
      const int b = __ldg(cell_start + row + x0), e = __ldg(cell_start + row + x1 + 1);
      for (int c = b; c < e; c += 32) {
        uint32_t w = rho ? segment_mask_density(xy, sa, c, e, pi.x, pi.y, thr, inv_support, acc)
                         : segment_mask(xy, c, e, pi.x, pi.y, thr);
        if (w == 0) continue;
        if (k < kSearchSegments) {
          seg_start[(int64_t)k * n + s] = c;
          seg_mask[(int64_t)k * n + s] = w;
        }
        ++k;
        cnt += __popc(w);
      }
    }
  }
  counts[s] = cnt;
  if (rho) rho[s] = acc * c_w;
  nseg[s] = k <= kSearchSegments ? k : -1;
  if (k > kSearchSegments) dense_list[atomicAdd(dense_count, 1)] = (int32_t)s;
}

// The rows of the dense list, one warp per particle: each sweep tests 32 candidates of a
// cell row at once, and the accepted ones are written in order through a ballot, so the row
// goes out in coalesced stores.  A row that does not fit the column buffer is skipped with
// SPH_FLAG_PAIR_CAPACITY set.
struct DenseRows {
  const float2* xy;
  const float* sh;
  const int32_t* cell_start;
  int r;
  const int32_t* list;
  const int32_t* count;
};

__device__ __noinline__ void fill_dense_rows(const DenseRows D, const uint32_t* __restrict__ keys, const sph_grid& g,
                                             const int32_t* __restrict__ offsets, int64_t pair_capacity,
                                             int32_t* __restrict__ cols, int32_t* status, int nd) {
  const int lane = threadIdx.x & 31;
  const int warps = gridDim.x * (blockDim.x >> 5);
  for (int q = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); q < nd; q += warps) {
    const int s = D.list[q];
    int o = offsets[s];
    const int end = offsets[s + 1];
    if ((int64_t)end > pair_capacity || o < 0) {
      if (lane == 0) flag(status, SPH_FLAG_PAIR_CAPACITY);
      continue;
    }
    const uint32_t key = keys[s];
    const float2 pi = D.xy[s];
    const float thr = grid_threshold(D.sh[s], g);
    const int cx = (int)(key % (uint32_t)g.cells_x), cy = (int)(key / (uint32_t)g.cells_x);
    const int x0 = max(cx - D.r, 0), x1 = min(cx + D.r, g.cells_x - 1);
    const int y0 = max(cy - D.r, 0), y1 = min(cy + D.r, g.cells_y - 1);
    for (int yy = y0; yy <= y1 && x0 <= x1; ++yy) {
      const int row = yy * g.cells_x;
      const int b = __ldg(D.cell_start + row + x0), e = __ldg(D.cell_start + row + x1 + 1);
      for (int c = b; c < e; c += 32) {
        const int j = c + lane;
        bool hit = false;
        if (j < e) {
          const float2 pj = __ldg(D.xy + j);
          hit = dist2_ref(pi.x, pi.y, pj.x, pj.y) <= thr;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, hit);
        const int pos = o + __popc(m & ((1u << lane) - 1u));
        if (hit && pos < end) cols[pos] = j;
        o += __popc(m);
      }
    }
  }
}

// The CSR columns from the stored segments (no pair tests), one warp per 32 rows and no block
// barrier.  The rows of a warp are one contiguous span of cols: it is built in the warp's
// shared stage and stored flat, in whole lines.  A span past the stage is taken in 2, 4 .. 32
// passes over as many fewer rows, and a row's segments are then dealt to that many lanes (the
// lanes' bit counts place them), so all lanes expand masks whatever the rows' length; a row of
// at most kSearchSegments x 32 columns always fits.  Bound by instruction issue (65 to 76 % of
// the slots).  2^20 lattice particles (29.6 M columns): 37 µs; 1,000,003 with half of them in a
// cluster (62 M): 99.  A stage of 8192 columns per block, and a warp per row for longer spans,
// took 45 and 186; rows staged apart per lane and stored one by one 45 and 146.
// A row that does not fit the column buffer is skipped with SPH_FLAG_PAIR_CAPACITY set.  The rows of
// the dense list are dealt to all warps at the end (a launch of their own took 2 us of every
// search, mostly for an empty list); a warp that has one among its rows takes those one by
// one, so that no span copies placeholders over it.
__device__ __forceinline__ int highest_bit(uint32_t w) {
  int b;
  asm("bfind.u32 %0, %1;" : "=r"(b) : "r"(w));
  return b;
}

// Blocks of a fill, at least (or one per four rows): the dense rows of a small set would otherwise be
// dealt to few warps, 32 rows each.  8,192 particles with rows of 1,024, all dense: 280 µs with the
// 64 blocks of the rows alone, 22 with these; 8,192 lattice particles 4.7 and 5.2.
constexpr int kFillBlocks = 8 * kNumSMs;

constexpr int kRowStage = 1280;   // 40 columns a row: the usual rows in one pass
static_assert(kRowStage >= kSearchSegments * 32, "one row has to fit");

__global__ void __launch_bounds__(128) k_nl_fill_segments(int64_t n, const uint32_t* __restrict__ keys,
                                                          const sph_grid* __restrict__ gp, int32_t cap,
                                                          const int32_t* __restrict__ offsets, int64_t pair_capacity,
                                                          int32_t* __restrict__ cols, int32_t* status,
                                                          const int32_t* __restrict__ nseg,
                                                          const int32_t* __restrict__ seg_start,
                                                          const uint32_t* __restrict__ seg_mask,
                                                          const DenseRows dense) {
  __shared__ __align__(16) int32_t stages[4][kRowStage + 4];
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const int64_t s0 = s - lane;
  int32_t* const stage = stages[threadIdx.x >> 5];
  const sph_grid g = *gp;
  const int nd = __ldg(dense.count);
  // this lane's row: first column, end, segments (none for a row that is not written)
  const int lo = offsets[min(s, n)], hi = offsets[min(s + 1, n)];
  int ns = 0;
  bool is_dense = false;
  if (s < n && grid_ok(g, cap) && keys[s] < (uint32_t)g.num_cells) {
    ns = nseg[s];
    is_dense = ns < 0;
    if ((int64_t)hi > pair_capacity) {
      flag(status, SPH_FLAG_PAIR_CAPACITY);
      ns = 0;
    }
    if (ns < 0 || ns > kSearchSegments || lo < 0 || hi < lo || hi - lo > kRowStage) ns = 0;
  }
  // lanes per row: 1 << sh, the fewest whose passes' spans all fit
  int sh = __any_sync(0xffffffffu, is_dense) ? 5 : 0, first = lo, last = hi;
  for (;; ++sh) {
    const int rows = 32 >> sh;
    first = __shfl_sync(0xffffffffu, lo, lane & -rows);
    last = __shfl_sync(0xffffffffu, hi, lane | (rows - 1));
    const bool fits = first >= 0 && last >= first && last - first <= kRowStage && (int64_t)last <= pair_capacity;
    if (sh == 5 || __all_sync(0xffffffffu, fits)) break;
  }
  const int sub = lane & ((1 << sh) - 1);
  for (int r0 = 0; r0 < 32; r0 += 32 >> sh) {
    const int t = r0 + (lane >> sh);   // this lane's row of the pass
    const int segs = __shfl_sync(0xffffffffu, ns, t);
    const int o = __shfl_sync(0xffffffffu, lo, t), e = __shfl_sync(0xffffffffu, hi, t);
    const int span0 = __shfl_sync(0xffffffffu, first, r0), span1 = __shfl_sync(0xffffffffu, last, r0);
    const int longest = __reduce_max_sync(0xffffffffu, segs);
    if (longest == 0) continue;
    // columns stay inside the row and the span even if offsets and masks disagree
    const int room = o >= span0 && e <= span1 ? e - o : 0;
    int32_t* const mine = stage + (o - (span0 & ~3));   // the stage begins on span0's 16 bytes
    int c_next = 0;
    uint32_t w_next = 0;
    const auto load = [&](int k) {
      c_next = 0;
      w_next = 0;
      if (k < segs) {
        c_next = seg_start[(int64_t)k * n + s0 + t];
        w_next = seg_mask[(int64_t)k * n + s0 + t];
      }
    };
    load(sub);
    int done = 0;   // columns of the row's earlier segments
    for (int k = 0; k < longest; k += 1 << sh) {
      const int c = c_next;
      uint32_t w = clip_segment(w_next, c, (int)n);
      load(k + (1 << sh) + sub);
      int cnt = __popc(w);
      int at = done;
      if (sh) {   // the segments of the row's lower lanes come first
        int incl = cnt;
        for (int d = 1; d < 1 << sh; d <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, incl, d, 1 << sh);
          if (sub >= d) incl += v;
        }
        at += incl - cnt;
        done += __shfl_sync(0xffffffffu, incl, (1 << sh) - 1, 1 << sh);
      } else {
        done += cnt;
      }
      for (; at + cnt > room && cnt > 0; --cnt) w &= ~(1u << highest_bit(w));
      for (int32_t* q = mine + at + cnt; w;) {   // from the last: the highest bit is one instruction
        const int bit = highest_bit(w);
        *--q = c + bit;
        w ^= 1u << bit;
      }
      __syncwarp();
    }
    if (span0 >= 0 && span1 - span0 <= kRowStage && (int64_t)span1 <= pair_capacity) {
      const int32_t* const from = stage - (span0 & ~3);
      int a = span0, b = span0;   // [a, b): by 16 bytes
      if ((reinterpret_cast<uintptr_t>(cols) & 15) == 0) {
        a = min((span0 + 3) & ~3, span1);
        b = max(span1 & ~3, a);
      }
      if (lane < a - span0) cols[span0 + lane] = from[span0 + lane];
      for (int j = a + 4 * lane; j < b; j += 128)
        *reinterpret_cast<int4*>(cols + j) = *reinterpret_cast<const int4*>(from + j);
      for (int j = b + lane; j < span1; j += 32) cols[j] = from[j];
    }
    __syncwarp();
  }
  if (nd > 0) fill_dense_rows(dense, keys, g, offsets, pair_capacity, cols, status, nd);
}

// Query points (any order, e.g. wall or ghost particles) against the sorted grid, with
// the query's own support in the predicate (dx = x_query - x_j): the pair set of
// buildNeighborListUnsortedPerParticle, cppSrc/neighSearch.cpp:261-331.
__device__ __forceinline__ bool query_cell(float x, float qmin, float hmax, int* c) {
  float v = ceilf(__fdiv_rn(__fsub_rn(x, qmin), hmax));
  if (!(v > -1.0e9f && v < 1.0e9f)) return false;
  *c = (int)v;
  return true;
}

// Where a query pair goes: sorted or original columns with 32-bit rows (sph_nl_query_fill), or
// searchExisting's own outputs, with the row offsets as int32 (sph_nl_query_pairs).
struct QueryPairs {
  const uint32_t* order;
  int32_t *rows, *cols;
  int64_t *rows64, *cols64;
  const float2* points;   // original order
  float threshold;
  float2* dist;
  float* radial;
  int32_t* row_offsets;
};

// Latency bounds the few thousand wall or ghost points of a scene, so kQueryLanes lanes share a
// point's candidates and place their hits by ballot, in the order of one thread; the points
// of a warp walk their cell rows in step.  The walls of a 30,621-particle block: 3.8 µs for
// counting and 6 for filling with the geometry (one thread each: 4.8, and 8 + 2 for it).
constexpr int kQueryLanes = 8;

enum { kQueryCount, kQueryRows, kQueryModule };

template <int kMode>
__global__ void __launch_bounds__(128) k_nl_query(const float2* __restrict__ qpos, const float* __restrict__ qh, int64_t m,
                                                  const float2* __restrict__ xy,
                                                  const int32_t* __restrict__ cell_start,
                                                  const sph_grid* __restrict__ gp, int32_t cap, int r,
                                                  int32_t* __restrict__ counts, const int64_t* __restrict__ offsets,
                                                  const QueryPairs out) {
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kQueryLanes;
  const bool live = row < m;   // lanes past the last point take part in the warp's votes
  const int64_t b = live ? row : m - 1;
  const int lane = threadIdx.x & 31, sub = lane % kQueryLanes, base = lane - sub;
  const sph_grid g = *gp;
  int cnt = 0;
  const int64_t o = kMode != kQueryCount ? offsets[b] : 0;
  const float2 xi = qpos[b];
  const float h = qh[b];
  const float thr = grid_threshold(h, g);
  int qx, qy, x0 = 0, x1 = -1, y0 = 0, y1 = -1;
  if (live && grid_ok(g, cap) && query_cell(xi.x, g.qmin[0], g.hmax, &qx) && query_cell(xi.y, g.qmin[1], g.hmax, &qy)) {
    x0 = max(qx - r, 0);
    x1 = min(qx + r, g.cells_x - 1);
    y0 = max(qy - r, 0);
    y1 = x0 <= x1 ? min(qy + r, g.cells_y - 1) : y0 - 1;
  }
  const int cell_rows = __reduce_max_sync(0xffffffffu, y1 - y0 + 1);
  for (int q = 0; q < cell_rows; ++q) {
    int j0 = 0, j1 = 0;
    if (y0 + q <= y1) {
      const int32_t* cells = cell_start + (int64_t)(y0 + q) * g.cells_x;
      j0 = __ldg(cells + x0);
      j1 = __ldg(cells + x1 + 1);
    }
    const int longest = __reduce_max_sync(0xffffffffu, j1 - j0);
    for (int t = 0; t < longest; t += kQueryLanes) {
      const int j = j0 + t + sub;
      bool hit = false;
      if (j < j1) {
        const float2 pj = __ldg(xy + j);
        hit = dist2_ref(xi.x, xi.y, pj.x, pj.y) <= thr;
      }
      const unsigned hits = __ballot_sync(0xffffffffu, hit) >> base & ((1u << kQueryLanes) - 1u);
      if (kMode != kQueryCount && hit) {
        const int64_t k = o + cnt + __popc(hits & ((1u << sub) - 1u));
        const int c = out.order ? (int)out.order[j] : j;
        if (kMode == kQueryRows) {
          out.rows[k] = (int32_t)b;
          out.cols[k] = c;
        } else {
          out.rows64[k] = b;
          out.cols64[k] = c;
          out.dist[k] = query_geometry(xi, out.points[c], h, out.threshold, out.radial + k);
        }
      }
      cnt += __popc(hits);
    }
  }
  if (kMode == kQueryCount && live && sub == 0) counts[b] = cnt;
  if (kMode == kQueryModule && live && sub == 0) {
    out.row_offsets[b] = (int32_t)o;
    if (b == m - 1) out.row_offsets[m] = (int32_t)offsets[m];
  }
}

// One warp per original particle i: its row of the (i, j)-ordered COO list, plus the
// reference's fluidDistances / fluidRadialDistances (src/modules/neighborSearch.py:218-223).
// A lane holds one pair.  Up to 32 columns are sorted in the lanes (bitonic; a column's sorted
// place comes back from rank); in a longer row a column's place is the number of the row's
// columns below it (they are distinct), counted over the warp's registers 32 columns at a
// time; rows past kLongRow are left to k_nl_to_coo_long.  No scratch, and the row's loads and four
// outputs are contiguous pieces, where one thread per row moved every column through global
// memory once per inversion: 558 us for 260,017 particles, 7.2 M pairs (201 MB of pairs and
// distances stored); counting in all rows 103, sorting the short ones 85.  Bound by instruction
// issue: the sort, and the correctly rounded root and divisions.
struct CooRows {
  const float2* xy;
  const uint32_t* order;
  const uint32_t* rank;
  const int32_t* offsets;
  const int32_t* cols;
  const int64_t* orig_offsets;
  float thr, support;
  int64_t *prow, *pcol;
  float *dist, *radial;
};

// Pair k: original particles i at pi and jo, which is c in sorted order.
__device__ __forceinline__ void write_pair(const CooRows& R, int64_t i, float2 pi, int64_t k, uint32_t jo, int32_t c) {
  R.prow[k] = i;
  R.pcol[k] = (int64_t)jo;
  if (R.dist || R.radial) {
    const float2 pj = __ldg(R.xy + c);
    const float dx = pi.x - pj.x, dy = pi.y - pj.y;
    const float rr = sqrtf(dx * dx + dy * dy);
    if (R.dist) {
      const float2 e = rr < R.thr ? make_float2(0.f, 0.f) : make_float2(dx / rr, dy / rr);
      if ((reinterpret_cast<uintptr_t>(R.dist) & 7) == 0) {
        reinterpret_cast<float2*>(R.dist)[k] = e;
      } else {
        R.dist[2 * k] = e.x;
        R.dist[2 * k + 1] = e.y;
      }
    }
    if (R.radial) R.radial[k] = rr / R.support;
  }
}

__global__ void __launch_bounds__(256) k_nl_to_coo(int64_t n, const CooRows R) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= n) return;
  const uint32_t s = __ldg(R.rank + i);
  const int32_t b = __ldg(R.offsets + s), m = __ldg(R.offsets + s + 1) - b;
  if (m > kLongRow) return;
  const int64_t o = __ldg(R.orig_offsets + i);
  const float2 pi = __ldg(R.xy + s);
  if (m <= 32) {
    uint32_t jo = lane < m ? __ldg(R.order + __ldg(R.cols + b + lane)) : 0xffffffffu;
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
      for (int d = k >> 1; d > 0; d >>= 1) {
        const uint32_t v = __shfl_xor_sync(0xffffffffu, jo, d);
        jo = ((lane & k) == 0) == ((lane & d) == 0) ? min(jo, v) : max(jo, v);
      }
    if (lane < m) write_pair(R, i, pi, o + lane, jo, (int32_t)__ldg(R.rank + jo));
    return;
  }
  for (int t0 = 0; t0 < m; t0 += 32) {
    const int t = t0 + lane;
    const int32_t c = t < m ? __ldg(R.cols + b + t) : 0;
    const uint32_t jo = t < m ? __ldg(R.order + c) : 0xffffffffu;
    int r = 0;
    for (int u0 = 0; u0 < m; u0 += 32) {
      const int u = u0 + lane;
      const uint32_t ju = u0 == t0 ? jo : (u < m ? __ldg(R.order + __ldg(R.cols + b + u)) : 0xffffffffu);
      const int len = min(m - u0, 32);
      for (int k = 0; k < len; ++k) r += __shfl_sync(0xffffffffu, ju, k) < jo;
    }
    if (t < m) write_pair(R, i, pi, o + r, jo, c);
  }
}

// The rows past kLongRow, a warp each.
__global__ void __launch_bounds__(256) k_nl_to_coo_long(int64_t n, const CooRows R) {
  __shared__ uint32_t words[8][kWarpSortWords];
  const int lane = threadIdx.x & 31;
  for_long_rows(n, [&](int64_t s) { return R.offsets[s + 1] - R.offsets[s]; }, [&](int64_t s, int m) {
    const int64_t i = R.order[s], o = R.orig_offsets[i];
    const float2 pi = R.xy[s];
    warp_sort_row(R.cols + R.offsets[s], R.order, m, R.pcol + o, words[threadIdx.x >> 5]);
    for (int t = lane; t < m; t += 32) {
      const uint32_t jo = (uint32_t)R.pcol[o + t];
      write_pair(R, i, pi, o + t, jo, (int32_t)__ldg(R.rank + jo));
    }
  });
}

// ---------------------------------------------------------------------------- batch of scenes
// Keys are global: scene s's cells occupy [coff_s, coff_s + num_cells_s) of the cell table.
__global__ void __launch_bounds__(256) k_batch_nl_count(const float2* __restrict__ xy, const float* __restrict__ sh,
                                                        int64_t n, const uint32_t* __restrict__ keys,
                                                        const int32_t* __restrict__ cell_start,
                                                        const SceneDev* __restrict__ scenes,
                                                        const int32_t* __restrict__ sid, int32_t* __restrict__ counts) {
  int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const SceneDev& S = scenes[sid[s]];
  const uint32_t key = keys[s] - (uint32_t)S.coff;
  int cnt = 0;
  if (keys[s] >= (uint32_t)S.coff && key < (uint32_t)S.g.num_cells) {
    const float2 pi = xy[s];
    const float thr = grid_threshold(sh[s], S.g);
    const int cx = (int)(key % (uint32_t)S.g.cells_x), cy = (int)(key / (uint32_t)S.g.cells_x);
    scan_candidates(xy, cell_start + S.coff, S.g, S.P.search_radius, cx, cy, pi.x, pi.y, thr,
                    [&](int, float) { ++cnt; });
  }
  counts[s] = cnt;
}

__global__ void __launch_bounds__(256) k_batch_nl_fill(const float2* __restrict__ xy, const float* __restrict__ sh,
                                                       int64_t n, const uint32_t* __restrict__ keys,
                                                       const int32_t* __restrict__ cell_start,
                                                       const SceneDev* __restrict__ scenes,
                                                       const int32_t* __restrict__ sid,
                                                       const int32_t* __restrict__ offsets, int64_t pair_capacity,
                                                       int32_t* __restrict__ cols, int32_t* status) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const SceneDev* S = s < n ? scenes + sid[s] : scenes;
  const uint32_t key = s < n ? keys[s] - (uint32_t)S->coff : 0xffffffffu;
  const bool active = s < n && keys[s] >= (uint32_t)S->coff && key < (uint32_t)S->g.num_cells;
  float2 pi = make_float2(0.f, 0.f);
  float thr = 0.f;
  int cx = 0, cy = 0;
  if (active) {
    pi = xy[s];
    thr = grid_threshold(sh[s], S->g);
    cx = (int)(key % (uint32_t)S->g.cells_x);
    cy = (int)(key / (uint32_t)S->g.cells_x);
  }
  staged_fill(s, n, active, offsets, pair_capacity, cols, status, [&](auto&& emit) {
    scan_candidates(xy, cell_start + S->coff, S->g, S->P.search_radius, cx, cy, pi.x, pi.y, thr,
                    [&](int j, float) { emit(j); });
  });
}

}  // namespace sph

using namespace sph;

extern "C" {

sph_status_t sph_batch_nl_count(const float* xy, const float* sorted_support, int64_t n, const uint32_t* sorted_keys,
                                const int32_t* cell_start, const void* scenes, const int32_t* sid, int32_t* counts,
                                void* stream) {
  SPH_REQUIRE(n >= 0 && xy && sorted_support && sorted_keys && cell_start && scenes && sid && counts,
              "batch_nl_count: bad arguments");
  if (n == 0) return SPH_OK;
  k_batch_nl_count<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(
      reinterpret_cast<const float2*>(xy), sorted_support, n, sorted_keys, cell_start,
      static_cast<const SceneDev*>(scenes), sid, counts);
  SPH_CHECK_LAUNCH("batch_nl_count");
  return SPH_OK;
}

sph_status_t sph_batch_nl_fill(const float* xy, const float* sorted_support, int64_t n, const uint32_t* sorted_keys,
                               const int32_t* cell_start, const void* scenes, const int32_t* sid, const int32_t* offsets,
                               int64_t pair_capacity, int32_t* cols, int32_t* status, void* stream) {
  SPH_REQUIRE(n >= 0 && xy && sorted_support && sorted_keys && cell_start && scenes && sid && offsets && cols,
              "batch_nl_fill: bad arguments");
  if (n == 0) return SPH_OK;
  k_batch_nl_fill<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(
      reinterpret_cast<const float2*>(xy), sorted_support, n, sorted_keys, cell_start,
      static_cast<const SceneDev*>(scenes), sid, offsets, pair_capacity, cols, status);
  SPH_CHECK_LAUNCH("batch_nl_fill");
  return SPH_OK;
}

sph_status_t sph_nl_count(const float* xy, const float* sorted_support, const float* sorted_area, int64_t n,
                          const uint32_t* sorted_keys, const int32_t* cell_start, const sph_grid* grid,
                          int32_t cell_capacity, int32_t search_radius, float kernel_support, int32_t* counts,
                          float* rho, void* stream) {
  SPH_REQUIRE(n >= 0 && xy && sorted_support && sorted_keys && cell_start && grid && counts && search_radius >= 0,
              "nl_count: bad arguments");
  SPH_REQUIRE(!rho || (kernel_support > 0.f && sorted_area), "nl_count: density needs kernel_support > 0 and areas");
  if (n == 0) return SPH_OK;
  float inv = rho ? 1.0f / kernel_support : 0.f;
  float cw = rho ? (float)(7.0 / 3.14159265358979323846) / (kernel_support * kernel_support) : 0.f;
  k_nl_count<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(reinterpret_cast<const float2*>(xy), sorted_support,
                                                               sorted_area, n, sorted_keys, cell_start, grid,
                                                               cell_capacity, search_radius, inv, cw, counts, rho);
  SPH_CHECK_LAUNCH("nl_count");
  return SPH_OK;
}

size_t sph_nl_segments_scratch_bytes(int64_t n) {
  return (size_t)(n > 0 ? n : 0) * (kSearchSegments * (sizeof(int32_t) + sizeof(uint32_t)) + 2 * sizeof(int32_t)) +
         256 + 16;
}

// seg_mask [kSearchSegments n], seg_start [kSearchSegments n], nseg [n], the dense list [n] and its
// count inside the scratch.
static bool segments_from_scratch(void* scratch, size_t bytes, int64_t n, int32_t** nseg, int32_t** start,
                                  uint32_t** mask, int32_t** dense_list, int32_t** dense_count) {
  if (!scratch || bytes < sph_nl_segments_scratch_bytes(n)) return false;
  const uintptr_t p = (reinterpret_cast<uintptr_t>(scratch) + 15) & ~(uintptr_t)15;
  *mask = reinterpret_cast<uint32_t*>(p);
  *start = reinterpret_cast<int32_t*>(*mask + (size_t)kSearchSegments * n);
  *nseg = *start + (size_t)kSearchSegments * n;
  *dense_list = *nseg + n;
  *dense_count = *dense_list + n;
  return true;
}

sph_status_t sph_nl_count_segments(const float* xy, const float* sorted_support, const float* sorted_area, int64_t n,
                                   const uint32_t* sorted_keys, const int32_t* cell_start, const sph_grid* grid,
                                   int32_t cell_capacity, int32_t search_radius, float kernel_support,
                                   int32_t* counts, float* rho, void* seg_scratch, size_t seg_bytes, void* stream) {
  SPH_REQUIRE(n >= 0 && n < ((int64_t)1 << 31) && xy && sorted_support && sorted_keys && cell_start && grid &&
                  counts && search_radius >= 0,
              "nl_count_segments: bad arguments");
  SPH_REQUIRE(!rho || (kernel_support > 0.f && sorted_area),
              "nl_count_segments: density needs kernel_support > 0 and areas");
  int32_t *nseg, *start, *dense_list, *dense_count;
  uint32_t* mask;
  SPH_REQUIRE(segments_from_scratch(seg_scratch, seg_bytes, n, &nseg, &start, &mask, &dense_list, &dense_count),
              "nl_count_segments: scratch smaller than sph_nl_segments_scratch_bytes(n)");
  if (n == 0) return SPH_OK;
  cudaMemsetAsync(dense_count, 0, sizeof(int32_t), as_stream(stream));
  float inv = rho ? 1.0f / kernel_support : 0.f;
  float cw = rho ? (float)(7.0 / 3.14159265358979323846) / (kernel_support * kernel_support) : 0.f;
  k_nl_segments<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(
      reinterpret_cast<const float2*>(xy), sorted_support, sorted_area, n, sorted_keys, cell_start, grid,
      cell_capacity, search_radius, inv, cw, counts, rho, nseg, start, mask, dense_list, dense_count);
  SPH_CHECK_LAUNCH("nl_count_segments");
  return SPH_OK;
}

sph_status_t sph_nl_fill_segments(const float* xy, const float* sorted_support, int64_t n,
                                  const uint32_t* sorted_keys, const int32_t* cell_start, const sph_grid* grid,
                                  int32_t cell_capacity, int32_t search_radius, const int32_t* offsets,
                                  int64_t pair_capacity, int32_t* cols, int32_t* status, const void* seg_scratch,
                                  size_t seg_bytes, void* stream) {
  SPH_REQUIRE(n >= 0 && n < ((int64_t)1 << 31) && xy && sorted_support && sorted_keys && cell_start && grid &&
                  offsets && cols,
              "nl_fill_segments: bad arguments");
  int32_t *nseg, *start, *dense_list, *dense_count;
  uint32_t* mask;
  SPH_REQUIRE(segments_from_scratch(const_cast<void*>(seg_scratch), seg_bytes, n, &nseg, &start, &mask,
                                    &dense_list, &dense_count),
              "nl_fill_segments: scratch smaller than sph_nl_segments_scratch_bytes(n)");
  if (n == 0) return SPH_OK;
  cudaStream_t st = as_stream(stream);
  const DenseRows dense{reinterpret_cast<const float2*>(xy), sorted_support, cell_start, search_radius, dense_list,
                        dense_count};
  const int blocks = std::max(grid_for(n, 128), std::min(grid_for(n, 4), kFillBlocks));
  k_nl_fill_segments<<<blocks, 128, 0, st>>>(n, sorted_keys, grid, cell_capacity, offsets, pair_capacity,
                                                       cols, status, nseg, start, mask, dense);
  SPH_CHECK_LAUNCH("nl_fill_segments");
  return SPH_OK;
}

sph_status_t sph_nl_fill(const float* xy, const float* sorted_support, int64_t n, const uint32_t* sorted_keys,
                         const int32_t* cell_start, const sph_grid* grid, int32_t cell_capacity, int32_t search_radius,
                         const int32_t* offsets, int64_t pair_capacity, int32_t* cols, int32_t* status, void* stream) {
  SPH_REQUIRE(n >= 0 && xy && sorted_support && sorted_keys && cell_start && grid && offsets && cols,
              "nl_fill: bad arguments");
  if (n == 0) return SPH_OK;
  k_nl_fill<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(reinterpret_cast<const float2*>(xy), sorted_support, n,
                                                              sorted_keys, cell_start, grid, cell_capacity,
                                                              search_radius, offsets, pair_capacity, cols, status);
  SPH_CHECK_LAUNCH("nl_fill");
  return SPH_OK;
}

sph_status_t sph_nl_to_coo(const float* xy, int64_t n, const uint32_t* order, const uint32_t* rank,
                           const int32_t* offsets, const int32_t* cols, const int64_t* orig_offsets,
                           float grad_threshold, float kernel_support, int64_t* pairs, int64_t num_pairs, float* dist,
                           float* radial, void* stream) {
  SPH_REQUIRE(n >= 0 && xy && order && rank && offsets && cols && orig_offsets && pairs, "nl_to_coo: bad arguments");
  if (n == 0) return SPH_OK;
  const CooRows R{reinterpret_cast<const float2*>(xy), order, rank, offsets, cols, orig_offsets, grad_threshold,
                  kernel_support, pairs, pairs + num_pairs, dist, radial};
  cudaStream_t st = as_stream(stream);
  k_nl_to_coo<<<grid_for(n, 8), 256, 0, st>>>(n, R);
  if (num_pairs > kLongRow) k_nl_to_coo_long<<<std::min(grid_for(n, 8), kLongRowBlocks), 256, 0, st>>>(n, R);
  SPH_CHECK_LAUNCH("nl_to_coo");
  return SPH_OK;
}

sph_status_t sph_nl_query_count(const float* query_pos, const float* query_support, int64_t m, const float* xy,
                                const int32_t* cell_start, const sph_grid* grid, int32_t cell_capacity,
                                int32_t search_radius, int32_t* counts, void* stream) {
  SPH_REQUIRE(m >= 0 && query_pos && query_support && xy && cell_start && grid && counts && search_radius >= 0,
              "nl_query: bad arguments");
  if (m == 0) return SPH_OK;
  k_nl_query<kQueryCount><<<grid_for(m * kQueryLanes, 128), 128, 0, as_stream(stream)>>>(
      reinterpret_cast<const float2*>(query_pos), query_support, m, reinterpret_cast<const float2*>(xy), cell_start,
      grid, cell_capacity, search_radius, counts, nullptr, QueryPairs{});
  SPH_CHECK_LAUNCH("nl_query_count");
  return SPH_OK;
}

sph_status_t sph_nl_query_fill(const float* query_pos, const float* query_support, int64_t m, const float* xy,
                               const int32_t* cell_start, const sph_grid* grid, int32_t cell_capacity,
                               int32_t search_radius, const uint32_t* order, const int64_t* offsets, int32_t* rows,
                               int32_t* cols, void* stream) {
  SPH_REQUIRE(m >= 0 && query_pos && query_support && xy && cell_start && grid && offsets && rows && cols &&
                  search_radius >= 0,
              "nl_query: bad arguments");
  if (m == 0) return SPH_OK;
  QueryPairs out{};
  out.order = order;
  out.rows = rows;
  out.cols = cols;
  k_nl_query<kQueryRows><<<grid_for(m * kQueryLanes, 128), 128, 0, as_stream(stream)>>>(
      reinterpret_cast<const float2*>(query_pos), query_support, m, reinterpret_cast<const float2*>(xy), cell_start,
      grid, cell_capacity, search_radius, nullptr, offsets, out);
  SPH_CHECK_LAUNCH("nl_query_fill");
  return SPH_OK;
}

sph_status_t sph_nl_query_pairs(const float* query_pos, const float* query_support, int64_t m, const float* xy,
                                const int32_t* cell_start, const sph_grid* grid, int32_t cell_capacity,
                                int32_t search_radius, const uint32_t* order, const int64_t* offsets,
                                const float* points, float threshold, int64_t* rows, int64_t* cols, float* dist,
                                float* radial, int32_t* row_offsets, void* stream) {
  SPH_REQUIRE(m >= 0 && query_pos && query_support && xy && cell_start && grid && order && offsets && points && rows &&
                  cols && dist && radial && row_offsets && search_radius >= 0 &&
                  (reinterpret_cast<uintptr_t>(dist) & 7) == 0,
              "nl_query_pairs: bad arguments");
  if (m == 0) return SPH_OK;
  QueryPairs out{};
  out.order = order;
  out.rows64 = rows;
  out.cols64 = cols;
  out.points = reinterpret_cast<const float2*>(points);
  out.threshold = threshold;
  out.dist = reinterpret_cast<float2*>(dist);
  out.radial = radial;
  out.row_offsets = row_offsets;
  k_nl_query<kQueryModule><<<grid_for(m * kQueryLanes, 128), 128, 0, as_stream(stream)>>>(
      reinterpret_cast<const float2*>(query_pos), query_support, m, reinterpret_cast<const float2*>(xy), cell_start,
      grid, cell_capacity, search_radius, nullptr, offsets, out);
  SPH_CHECK_LAUNCH("nl_query_pairs");
  return SPH_OK;
}

}  // extern "C"
