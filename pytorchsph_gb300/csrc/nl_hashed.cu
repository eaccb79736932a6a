// Drop-in neighbor-list kernels over the reference's own hash-table format
// (hashTable [L,2] = (first slot, #cells), cellIndices / cumCell (= counts) /
// cellSpan (= begins) in hash order; src/modules/neighborSearch.py:58-88).  They reproduce
// the pair sets of cppSrc/neighSearch.cpp:172-410 and cppSrc/neighSearch_cuda.cu:101-209,
// two passes each (count, then fill at scanned int64 offsets).
#include "sph_common.cuh"

namespace sph {

// queryHashMap, cppSrc/neighSearch.cpp:93-114 / cppSrc/neighSearch_cuda.cu:76-99.
__device__ __forceinline__ int2 query_hash(int qx, int qy, const int32_t* __restrict__ table,
                                           const int32_t* __restrict__ ci, const int32_t* __restrict__ cc,
                                           const int32_t* __restrict__ cs, int cells_x, int L) {
  if (qx < 0 || qy < 0) return make_int2(-1, -1);
  int qlin = qx + cells_x * qy;
  // the reference computes this in int32; int64 keeps far-away query cells from
  // overflowing into a negative (out-of-table) bucket
  // (32-bit division while 3 qx + 5 qy fits; the 64-bit one is a long sequence)
  int qh = (qx | qy) < (1 << 28) ? (int)((3u * (unsigned)qx + 5u * (unsigned)qy) % (unsigned)L)
                                 : (int)(((long long)qx * 3 + (long long)qy * 5) % L);
  int first = table[2 * qh];
  if (first == -1) return make_int2(-1, -1);
  int last = first + table[2 * qh + 1];
  // 3 x + 5 y puts some ten cells of a square grid in a bucket: four of them are in flight at a time
  for (int k = first; k < last; k += 4) {
    int at = -1;
#pragma unroll
    for (int u = 3; u >= 0; --u) {
      const int v = ci[min(k + u, last - 1)];
      if (v == qlin) at = min(k + u, last - 1);
    }
    if (at >= 0) return make_int2(cs[at], cs[at] + cc[at]);
  }
  return make_int2(-1, -1);
}

// A query point is (2r + 1)^2 dependent table lookups and some 80 candidates.  kQueryLanes lanes
// share it: they look up a chunk of kQueryCells cells (all of r = 1) at once and walk the chunk's
// candidates as one list, the eight points of a warp in step (loops over
// single cells come apart and run one group after another: 32 + 37 µs for counting and filling
// 65,537 points, as slow as one thread per point, 28 + 39; now 21.5 + 25).  Hits are placed by
// ballot, so a row keeps the reference's visiting order.
constexpr int kQueryLanes = 4, kQueryCells = 9;

template <bool kFill>
__global__ void __launch_bounds__(128) k_hashed_query(
    const float2* __restrict__ qpos, const float* __restrict__ qh, int64_t m, const float2* __restrict__ spos,
    const int32_t* __restrict__ table, const int32_t* __restrict__ ci, const int32_t* __restrict__ cc,
    const int32_t* __restrict__ cs, const int32_t* __restrict__ sort, const float* __restrict__ qmin, float hmax,
    float hmax_threshold, int cells_x, int L, int r, int32_t* __restrict__ counts, const int64_t* __restrict__ offsets,
    int32_t* __restrict__ rows, int32_t* __restrict__ cols) {
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kQueryLanes;
  const bool live = row < m;   // lanes past the last point take part in the warp's votes
  const int64_t b = live ? row : m - 1;
  const int lane = threadIdx.x & 31, sub = lane % kQueryLanes, base = lane - sub;
  const float2 xi = qpos[b];
  const float h = qh[b];
  const float thr = h == hmax ? hmax_threshold : sq_threshold(h);   // the usual support's, off the FP64 pipe
  const int qx = cell_coord(xi.x, qmin[0], hmax);
  const int qy = cell_coord(xi.y, qmin[1], hmax);
  int cnt = 0;
  const int64_t o = kFill ? offsets[b] : 0;
  const int64_t side = 2 * (int64_t)r + 1, cells = side * side;
  int64_t x0 = 0, y0 = 0;   // the chunk's first cell, y fastest
  for (int64_t c0 = 0; c0 < cells; c0 += kQueryCells) {
    int b0[(kQueryCells + kQueryLanes - 1) / kQueryLanes], len[(kQueryCells + kQueryLanes - 1) / kQueryLanes];
#pragma unroll
    for (int q = 0; q * kQueryLanes < kQueryCells; ++q) {
      b0[q] = len[q] = 0;
      const int at = q * kQueryLanes + sub;
      if (at < kQueryCells && c0 + at < cells) {
        int64_t xx = x0, yy = y0 + at;
        while (yy >= side) {
          yy -= side;
          ++xx;
        }
        const int2 rg = query_hash(qx + (int)(xx - r), qy + (int)(yy - r), table, ci, cc, cs, cells_x, L);
        if (live && rg.x != -1) {
          b0[q] = rg.x;
          len[q] = max(rg.y - rg.x, 0);
        }
      }
    }
    y0 += kQueryCells;
    while (y0 >= side) {
      y0 -= side;
      ++x0;
    }
    // candidate t of the chunk is particle t + shift[k] for the k with first[k] <= t < first[k + 1]
    int first[kQueryCells], shift[kQueryCells], total = 0;
#pragma unroll
    for (int k = 0; k < kQueryCells; ++k) {
      const int kb = __shfl_sync(0xffffffffu, b0[k / kQueryLanes], k % kQueryLanes, kQueryLanes);
      const int kl = __shfl_sync(0xffffffffu, len[k / kQueryLanes], k % kQueryLanes, kQueryLanes);
      first[k] = total;
      shift[k] = kb - total;
      total += kl;
    }
    const int longest = __reduce_max_sync(0xffffffffu, total);
    for (int t0 = 0; t0 < longest; t0 += kQueryLanes) {
      const int t = t0 + sub;
      int j = t + shift[0];
#pragma unroll
      for (int k = 1; k < kQueryCells; ++k)
        if (t >= first[k]) j = t + shift[k];
      bool hit = false;
      if (t < total) {
        const float2 xj = spos[j];
        hit = dist2_ref(xi.x, xi.y, xj.x, xj.y) <= thr;
      }
      const unsigned hits = __ballot_sync(0xffffffffu, hit) >> base & ((1u << kQueryLanes) - 1u);
      if (kFill && hit) {
        const int64_t k = o + cnt + __popc(hits & ((1u << sub) - 1u));
        if (rows) rows[k] = (int32_t)b;
        cols[k] = sort[j];
      }
      cnt += __popc(hits);
    }
  }
  if (!kFill && live && sub == 0) counts[b] = cnt;
}

// The pairs of m rows (row b's columns at [offsets[b], offsets[b + 1])) as int64 (row, column) in
// increasing order, one warp per row.  The rows are in order already, so two sorts of the
// whole pair list, by column and by row, come down to this.  Up to 32 columns are sorted in the
// lanes (bitonic, 15 exchanges); of a longer row each column's place is the number of the
// row's columns below it (equal columns by their place in the row), and rows past kLongRow are left
// to k_long_pairs_in_order: 24 µs for 65,537 rows of 28, 11.7 with the short rows in the lanes; the
// two sorts took some 280 with their copies.
__global__ void __launch_bounds__(256) k_pairs_in_order(int64_t m, const int64_t* __restrict__ offsets,
                                                        const int32_t* __restrict__ in, int64_t* __restrict__ rows,
                                                        int64_t* __restrict__ cols) {
  const int64_t b = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (b >= m) return;
  const int64_t o = offsets[b];
  const int len = (int)(offsets[b + 1] - o);
  if (len > kLongRow) return;
  if (len <= 32) {
    int32_t j = lane < len ? __ldg(in + o + lane) : 0x7fffffff;   // columns are below 2^31 - 1
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
      for (int d = k >> 1; d > 0; d >>= 1) {
        const int32_t v = __shfl_xor_sync(0xffffffffu, j, d);
        j = ((lane & k) == 0) == ((lane & d) == 0) ? min(j, v) : max(j, v);
      }
    if (lane < len) {
      rows[o + lane] = b;
      cols[o + lane] = j;
    }
    return;
  }
  for (int t0 = 0; t0 < len; t0 += 32) {
    const int t = t0 + lane;
    const int32_t j = t < len ? __ldg(in + o + t) : 0x7fffffff;
    int r = 0;
    for (int u0 = 0; u0 < len; u0 += 32) {
      const int u = u0 + lane;
      const int32_t ju = u0 == t0 ? j : (u < len ? __ldg(in + o + u) : 0x7fffffff);
      const int end = min(len - u0, 32);
      for (int k = 0; k < end; ++k) {
        const int32_t v = __shfl_sync(0xffffffffu, ju, k);
        r += v < j || (v == j && u0 + k < t);
      }
    }
    if (t < len) {
      rows[o + r] = b;
      cols[o + r] = j;
    }
  }
}

// The rows past kLongRow, a warp each.
__global__ void __launch_bounds__(256) k_long_pairs_in_order(int64_t m, const int64_t* __restrict__ offsets,
                                                             const int32_t* __restrict__ in,
                                                             int64_t* __restrict__ rows, int64_t* __restrict__ cols) {
  __shared__ uint32_t words[8][kWarpSortWords];
  for_long_rows(m, [&](int64_t b) { return (int)(offsets[b + 1] - offsets[b]); }, [&](int64_t b, int len) {
    const int64_t o = offsets[b];
    warp_sort_row(in + o, nullptr, len, cols + o, words[threadIdx.x >> 5]);
    for (int t = threadIdx.x & 31; t < len; t += 32) rows[o + t] = b;
  });
}

template <bool kFill>
__global__ void k_hashed_cells(const float2* __restrict__ spos, const float* __restrict__ sh,
                               const int32_t* __restrict__ table, const int32_t* __restrict__ ci,
                               const int32_t* __restrict__ cc, const int32_t* __restrict__ cs,
                               const int32_t* __restrict__ sort, int64_t C, int cells_x, int L, int r,
                               int32_t* __restrict__ counts, const int64_t* __restrict__ offsets,
                               int32_t* __restrict__ rows, int32_t* __restrict__ cols) {
  int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= C) return;
  int cell = ci[b];
  int qx = cell % cells_x, qy = cell / cells_x;
  int2 own = query_hash(qx, qy, table, ci, cc, cs, cells_x, L);
  int cnt = 0;
  int64_t o = kFill ? offsets[b] : 0;
  for (int xx = -r; xx <= r; ++xx)
    for (int yy = -r; yy <= r; ++yy) {
      int2 rg = query_hash(qx + xx, qy + yy, table, ci, cc, cs, cells_x, L);
      if (rg.x == -1) continue;
      for (int i = own.x; i < own.y; ++i) {
        float2 xi = spos[i];
        const float thr = sq_threshold(sh[i]);
        for (int j = rg.x; j < rg.y; ++j) {
          float2 xj = spos[j];
          if (dist2_ref(xi.x, xi.y, xj.x, xj.y) <= thr) {
            if (kFill) {
              rows[o + cnt] = sort[i];
              cols[o + cnt] = sort[j];
            }
            ++cnt;
          }
        }
      }
    }
  if (!kFill) counts[b] = cnt;
}

template <bool kFill>
__global__ void k_hashed_asym(const float2* __restrict__ pa, const float* __restrict__ ha,
                              const int32_t* __restrict__ ta, const int32_t* __restrict__ cia,
                              const int32_t* __restrict__ cca, const int32_t* __restrict__ csa,
                              const int32_t* __restrict__ sa, int64_t Ca, const float2* __restrict__ pb,
                              const int32_t* __restrict__ tb, const int32_t* __restrict__ cib,
                              const int32_t* __restrict__ ccb, const int32_t* __restrict__ csb,
                              const int32_t* __restrict__ sb, int cells_x, int L, int32_t* __restrict__ counts,
                              const int64_t* __restrict__ offsets, int32_t* __restrict__ rows,
                              int32_t* __restrict__ cols) {
  int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= Ca) return;
  int cell = cia[b];
  int qx = cell % cells_x, qy = cell / cells_x;
  int2 own = query_hash(qx, qy, ta, cia, cca, csa, cells_x, L);
  int cnt = 0;
  int64_t o = kFill ? offsets[b] : 0;
  for (int xx = -1; xx <= 1; ++xx)
    for (int yy = -1; yy <= 1; ++yy) {
      int2 rg = query_hash(qx + xx, qy + yy, tb, cib, ccb, csb, cells_x, L);
      if (rg.x == -1) continue;
      for (int i = own.x; i < own.y; ++i) {
        float2 xi = pa[i];
        const float thr = sq_threshold(ha[i]);
        for (int j = rg.x; j < rg.y; ++j) {
          float2 xj = pb[j];
          if (dist2_ref(xi.x, xi.y, xj.x, xj.y) <= thr) {
            if (kFill) {
              rows[o + cnt] = sa[i];
              cols[o + cnt] = sb[j];
            }
            ++cnt;
          }
        }
      }
    }
  if (!kFill) counts[b] = cnt;
}

}  // namespace sph

using namespace sph;

extern "C" {

sph_status_t sph_nl_hashed_query_count(const float* query_pos, const float* query_support, int64_t m,
                                       const float* sorted_pos, const int32_t* hash_table, const int32_t* cell_indices,
                                       const int32_t* cum_cell, const int32_t* cell_span, const float* qmin,
                                       float hmax, int32_t cells_x, int32_t hash_len, int32_t search_radius,
                                       int32_t* counts, void* stream) {
  SPH_REQUIRE(m >= 0 && hash_len > 0 && cells_x > 0 && hmax > 0.f && search_radius >= 0, "hashed_query: bad arguments");
  if (m == 0) return SPH_OK;
  k_hashed_query<false><<<grid_for(m * kQueryLanes, 128), 128, 0, as_stream(stream)>>>(
      reinterpret_cast<const float2*>(query_pos), query_support, m, reinterpret_cast<const float2*>(sorted_pos),
      hash_table, cell_indices, cum_cell, cell_span, nullptr, qmin, hmax, sq_threshold(hmax), cells_x, hash_len,
      search_radius, counts, nullptr, nullptr, nullptr);
  SPH_CHECK_LAUNCH("hashed_query_count");
  return SPH_OK;
}

sph_status_t sph_nl_hashed_query_fill(const float* query_pos, const float* query_support, int64_t m,
                                      const float* sorted_pos, const int32_t* hash_table, const int32_t* cell_indices,
                                      const int32_t* cum_cell, const int32_t* cell_span, const int32_t* sort,
                                      const float* qmin, float hmax, int32_t cells_x, int32_t hash_len,
                                      int32_t search_radius, const int64_t* offsets, int32_t* rows, int32_t* cols,
                                      void* stream) {
  SPH_REQUIRE(m >= 0 && hash_len > 0 && cells_x > 0 && hmax > 0.f && search_radius >= 0, "hashed_query: bad arguments");
  if (m == 0) return SPH_OK;
  k_hashed_query<true><<<grid_for(m * kQueryLanes, 128), 128, 0, as_stream(stream)>>>(
      reinterpret_cast<const float2*>(query_pos), query_support, m, reinterpret_cast<const float2*>(sorted_pos),
      hash_table, cell_indices, cum_cell, cell_span, sort, qmin, hmax, sq_threshold(hmax), cells_x, hash_len,
      search_radius, nullptr, offsets, rows, cols);
  SPH_CHECK_LAUNCH("hashed_query_fill");
  return SPH_OK;
}

sph_status_t sph_nl_pairs_in_order(int64_t m, const int64_t* offsets, const int32_t* cols, int64_t* rows_out,
                                   int64_t* cols_out, void* stream) {
  SPH_REQUIRE(m >= 0 && (m == 0 || (offsets && cols && rows_out && cols_out)), "nl_pairs_in_order: bad arguments");
  if (m == 0) return SPH_OK;
  cudaStream_t st = as_stream(stream);
  const int nb = grid_for(m, 8);
  k_pairs_in_order<<<nb, 256, 0, st>>>(m, offsets, cols, rows_out, cols_out);
  k_long_pairs_in_order<<<std::min(nb, kLongRowBlocks), 256, 0, st>>>(m, offsets, cols, rows_out, cols_out);
  SPH_CHECK_LAUNCH("nl_pairs_in_order");
  return SPH_OK;
}

sph_status_t sph_nl_hashed_cells_count(const float* sorted_pos, const float* sorted_support, const int32_t* hash_table,
                                       const int32_t* cell_indices, const int32_t* cum_cell, const int32_t* cell_span,
                                       int64_t num_cells, int32_t cells_x, int32_t hash_len, int32_t search_radius,
                                       int32_t* counts, void* stream) {
  SPH_REQUIRE(num_cells >= 0 && hash_len > 0 && cells_x > 0 && search_radius >= 0, "hashed_cells: bad arguments");
  if (num_cells == 0) return SPH_OK;
  k_hashed_cells<false><<<grid_for(num_cells, 64), 64, 0, as_stream(stream)>>>(
      reinterpret_cast<const float2*>(sorted_pos), sorted_support, hash_table, cell_indices, cum_cell, cell_span,
      nullptr, num_cells, cells_x, hash_len, search_radius, counts, nullptr, nullptr, nullptr);
  SPH_CHECK_LAUNCH("hashed_cells_count");
  return SPH_OK;
}

sph_status_t sph_nl_hashed_cells_fill(const float* sorted_pos, const float* sorted_support, const int32_t* hash_table,
                                      const int32_t* cell_indices, const int32_t* cum_cell, const int32_t* cell_span,
                                      const int32_t* sort, int64_t num_cells, int32_t cells_x, int32_t hash_len,
                                      int32_t search_radius, const int64_t* offsets, int32_t* rows, int32_t* cols,
                                      void* stream) {
  SPH_REQUIRE(num_cells >= 0 && hash_len > 0 && cells_x > 0 && search_radius >= 0, "hashed_cells: bad arguments");
  if (num_cells == 0) return SPH_OK;
  k_hashed_cells<true><<<grid_for(num_cells, 64), 64, 0, as_stream(stream)>>>(
      reinterpret_cast<const float2*>(sorted_pos), sorted_support, hash_table, cell_indices, cum_cell, cell_span,
      sort, num_cells, cells_x, hash_len, search_radius, nullptr, offsets, rows, cols);
  SPH_CHECK_LAUNCH("hashed_cells_fill");
  return SPH_OK;
}

sph_status_t sph_nl_hashed_asym_count(const float* pos_a, const float* support_a, const int32_t* table_a,
                                      const int32_t* cell_indices_a, const int32_t* cum_cell_a,
                                      const int32_t* cell_span_a, int64_t num_cells_a, const float* pos_b,
                                      const int32_t* table_b, const int32_t* cell_indices_b, const int32_t* cum_cell_b,
                                      const int32_t* cell_span_b, int32_t cells_x, int32_t hash_len, int32_t* counts,
                                      void* stream) {
  SPH_REQUIRE(num_cells_a >= 0 && hash_len > 0 && cells_x > 0, "hashed_asym: bad arguments");
  if (num_cells_a == 0) return SPH_OK;
  k_hashed_asym<false><<<grid_for(num_cells_a, 64), 64, 0, as_stream(stream)>>>(
      reinterpret_cast<const float2*>(pos_a), support_a, table_a, cell_indices_a, cum_cell_a, cell_span_a, nullptr,
      num_cells_a, reinterpret_cast<const float2*>(pos_b), table_b, cell_indices_b, cum_cell_b, cell_span_b, nullptr,
      cells_x, hash_len, counts, nullptr, nullptr, nullptr);
  SPH_CHECK_LAUNCH("hashed_asym_count");
  return SPH_OK;
}

sph_status_t sph_nl_hashed_asym_fill(const float* pos_a, const float* support_a, const int32_t* table_a,
                                     const int32_t* cell_indices_a, const int32_t* cum_cell_a,
                                     const int32_t* cell_span_a, const int32_t* sort_a, int64_t num_cells_a,
                                     const float* pos_b, const int32_t* table_b, const int32_t* cell_indices_b,
                                     const int32_t* cum_cell_b, const int32_t* cell_span_b, const int32_t* sort_b,
                                     int32_t cells_x, int32_t hash_len, const int64_t* offsets, int32_t* rows,
                                     int32_t* cols, void* stream) {
  SPH_REQUIRE(num_cells_a >= 0 && hash_len > 0 && cells_x > 0, "hashed_asym: bad arguments");
  if (num_cells_a == 0) return SPH_OK;
  k_hashed_asym<true><<<grid_for(num_cells_a, 64), 64, 0, as_stream(stream)>>>(
      reinterpret_cast<const float2*>(pos_a), support_a, table_a, cell_indices_a, cum_cell_a, cell_span_a, sort_a,
      num_cells_a, reinterpret_cast<const float2*>(pos_b), table_b, cell_indices_b, cum_cell_b, cell_span_b, sort_b,
      cells_x, hash_len, nullptr, offsets, rows, cols);
  SPH_CHECK_LAUNCH("hashed_asym_fill");
  return SPH_OK;
}

}  // extern "C"
