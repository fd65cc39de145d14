// entries.cu -- entry points: each query starts its search at the nearest of a
// set of entry vertices instead of vertex 0.
//
// The reference always starts at vertex 0 (warp_astar_accelerator.h:173, and
// graph.h:176 with its random start commented out); that stays the default.
// With entries set (song_index_set_entries), a pre-pass picks for every query
// the entry with the smallest search distance, ties to the smaller id, and
// the search starts there.  Nothing else in the search changes.
//
// The distance is the search kernel's, bit for bit, on the FP32 rows (partial
// p sums dims p, p+32, ... with fused multiply-adds, the 32 partials meet in
// the xor butterfly): the warp takes one query and eight rows at a time, or
// four queries and eight rows (entry_rows.cuh).  The entry rows are copied
// once into a contiguous block.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "entry_choice.cuh"
#include "entry_rows.cuh"
#include "entry_tiles.cuh"
#include "internal.h"
#include "song_gb300.h"

namespace song {
namespace {

// Gathers the FP32 rows of the entries into a contiguous block.
__global__ void gather_entry_rows_kernel(const float *rows, uint32_t row_floats, const uint32_t *ids, int n,
                                         int dpad, float *out) {
  const uint64_t total = static_cast<uint64_t>(n) * dpad;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint64_t e = i / dpad;
    out[i] = rows[static_cast<uint64_t>(ids[e]) * row_floats + (i - e * dpad)];
  }
}

// ---------------------------------------------------------------------------
// Two-level choice: the probes nearest coarse entries, then the ns nearest
// entries of their clusters.  The second phase runs cluster by cluster: the
// probe lists are inverted into one query list per cluster, and four queries
// share the cluster's rows.  Each query's per-cluster best lists are then
// merged.  Small batches take both phases query by query.
// ---------------------------------------------------------------------------

// 16-byte global-to-shared copies that complete without holding registers
// (cp.async, waited for by group).
__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
  const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Block shape of the two kernels: `warps` warps (4 queries each), row tiles
// of `rows` rows (a multiple of 8), nbuf tiles in flight.  Wide rows get
// smaller blocks and tiles so that a block fits its shared memory.
struct TileShape {
  int warps, rows, nbuf;
  size_t smem(int dpad) const {
    return sizeof(float) * static_cast<size_t>(dpad) * (4 * warps + static_cast<size_t>(nbuf) * rows);
  }
};

TileShape tile_shape(int dpad) {
  TileShape t{8, 32, 2};
  const size_t budget = 100u * 1024u;
  while (t.smem(dpad) > budget) {
    if (t.nbuf == 2) t.nbuf = 1;
    else if (t.rows > 8) t.rows /= 2;
    else if (t.warps > 1) t.warps /= 2;
    else break;
  }
  return t;
}

// Streams rows [r0, r1) of the row-major block `rows` (dpad floats each)
// through nbuf shared-memory tiles of tile_rows rows (the next tile's copies in
// flight while the current one is scored) and calls score(first_row, n, tile)
// for each; every thread of the block takes part.  Only rows below r1 are
// copied.
template <class F>
__device__ __forceinline__ void stream_rows(const float *rows, int dpad, int r0, int r1, int tile_rows, int nbuf,
                                            float *xb, F &&score) {
  const size_t tile = static_cast<size_t>(dpad) * tile_rows;
  auto issue = [&](int first, float *buf) {
    const int n = min(tile_rows, r1 - first);
    const float4 *src = reinterpret_cast<const float4 *>(rows + static_cast<size_t>(first) * dpad);
    float4 *dst = reinterpret_cast<float4 *>(buf);
    const int n4 = n * (dpad / 4);
    for (int i = threadIdx.x; i < n4; i += blockDim.x) cp_async16(dst + i, src + i);
    cp_async_commit();
  };
  if (nbuf == 2 && r0 < r1) issue(r0, xb);
  for (int first = r0, k = 0; first < r1; first += tile_rows, ++k) {
    float *cur = xb + (nbuf == 2 ? static_cast<size_t>(k & 1) * tile : 0);
    if (nbuf == 2) {
      // the other buffer was last read before the previous iteration's closing barrier
      if (first + tile_rows < r1) {
        issue(first + tile_rows, xb + static_cast<size_t>((k + 1) & 1) * tile);
      } else {
        cp_async_commit();
      }
      cp_async_wait<1>();
    } else {
      issue(first, cur);
      cp_async_wait<0>();
    }
    __syncthreads();  // every thread's copies (and the staged queries) are visible
    score(first, min(tile_rows, r1 - first), cur);
    __syncthreads();
  }
}

// Two-level choice, first kernel: each query's `probes` nearest coarse
// entries (positions in the coarse list, which is sorted by id, so the
// position is the tie order), and the number of probes of each cluster.
// A block takes 4 queries per warp and streams all coarse rows; lane l of a
// warp scores its query l >> 3 against rows l & 7 of each group of 8.
template <int METRIC, int NP>
__global__ void __launch_bounds__(256) heads_tiled_kernel(const float *queries, int nq, int dim, int dpad,
                                                          const float *coarse_rows, int n_coarse, int probes,
                                                          int tile_rows, int nbuf, uint32_t *probe_out,
                                                          uint32_t *cl_count) {
  extern __shared__ __align__(16) float smt[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int bq = 4 * (blockDim.x >> 5);  // queries per block
  const int q0 = blockIdx.x * bq;
  float *qs = smt;
  float *xb = smt + static_cast<size_t>(dpad) * bq;
  for (int i = threadIdx.x; i < bq * dpad; i += blockDim.x) {
    const int r = i / dpad, j = i - r * dpad;
    qs[i] = (q0 + r < nq && j < dim) ? queries[static_cast<size_t>(q0 + r) * dim + j] : 0.0f;
  }
  float pd[NP];
  uint32_t pi[NP];
#pragma unroll
  for (int m = 0; m < NP; ++m) {
    pd[m] = __int_as_float(0x7f800000);
    pi[m] = 0xffffffffu;
  }
  const float *qw = qs + static_cast<size_t>(4 * warp) * dpad;
  stream_rows(coarse_rows, dpad, 0, n_coarse, tile_rows, nbuf, xb, [&](int first, int n, const float *cur) {
    for (int g = 0; g < n; g += 8) {
      const float d = warp_tile_distance<METRIC>(qw, dpad, cur + static_cast<size_t>(g) * dpad, dpad, dpad, lane);
      const int r = g + (lane & 7);
      if (r < n) list_insert<NP>(pd, pi, d, static_cast<uint32_t>(first + r));
    }
  });
  const int q = q0 + 4 * warp + (lane >> 3);
  int h = 0;
  for (int r = 0; r < probes; ++r) {
    float wd;
    uint32_t wid;
    group8_take<NP>(pd, pi, h, wd, wid);
    if (wid >= static_cast<uint32_t>(n_coarse)) wid = 0;  // no finite distance (a query that is not finite)
    if ((lane & 7) == 0 && q < nq) {
      probe_out[static_cast<size_t>(q) * probes + r] = wid;
      atomicAdd(cl_count + wid, 1u);
    }
  }
}

// Exclusive block scan of one value per thread (1024 threads); returns this
// thread's exclusive prefix, and the total in *total.
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t s, uint32_t *warp_sum, uint32_t *total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = s;  // inclusive scan within the warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();  // warp_sum may still be read by a previous scan
  if (lane == 31) warp_sum[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < static_cast<int>(blockDim.x >> 5) ? warp_sum[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    warp_sum[lane] = w;
  }
  __syncthreads();
  *total = warp_sum[(blockDim.x >> 5) - 1];
  return x - s + (warp > 0 ? warp_sum[warp - 1] : 0u);
}

// Exclusive scans of the per-cluster probe counts (one block): offs[0..n],
// a copy of offs[0..n-1] as the scatter cursors, and task_offs[c], the first
// of cluster c's tasks (one per 4 of its queries) when the clusters are taken
// in the order `order`; *n_tasks tasks in all.
__global__ void __launch_bounds__(1024) cluster_scan_kernel(const uint32_t *count, int n, const uint32_t *order,
                                                            uint32_t *offs, uint32_t *cursor, uint32_t *task_offs,
                                                            uint32_t *n_tasks) {
  __shared__ uint32_t warp_sum[32];
  const int per = (n + blockDim.x - 1) / blockDim.x;
  const int b = threadIdx.x * per, e = min(n, b + per);
  uint32_t s = 0, st = 0;
  for (int i = b; i < e; ++i) {
    s += count[i];
    st += (count[order[i]] + 3u) / 4u;
  }
  uint32_t total, ttotal;
  uint32_t run = block_exclusive_scan(s, warp_sum, &total);
  uint32_t trun = block_exclusive_scan(st, warp_sum, &ttotal);
  for (int i = b; i < e; ++i) {
    offs[i] = run;
    cursor[i] = run;
    run += count[i];
    const uint32_t c = order[i];
    task_offs[c] = trun;
    trun += (count[c] + 3u) / 4u;
  }
  if (threadIdx.x == 0) {
    offs[n] = total;
    *n_tasks = ttotal;
  }
}

// Inverts the probe lists: list[cursor[c]++] = q * probes + r for every
// probe r of every query q that names cluster c.  The first of each four
// writes their task: (cluster, which four).
__global__ void cluster_scatter_kernel(const uint32_t *probe, int total, const uint32_t *offs,
                                       const uint32_t *task_offs, uint32_t *cursor, uint32_t *list, uint2 *tasks) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    const uint32_t c = probe[i], at = atomicAdd(cursor + c, 1u), k = at - offs[c];
    list[at] = static_cast<uint32_t>(i);
    if ((k & 3u) == 0u) tasks[task_offs[c] + (k >> 2)] = make_uint2(c, k >> 2);
  }
}

// Two-level choice, second kernel: tasks of (cluster, 4 of the queries that
// probe it), taken by persistent blocks of `warps` warps.  The block stages
// its 4 queries, its warps take the cluster's rows eight at a time in turn
// (tile_distance), and the lists of all warps meet in shared memory: each
// (query, probe) pair's NS nearest entries go to part_*.
// What bounds it: FP32 instructions while there are many tasks (a third of
// the issue slots at 10,000 queries; its rows' 282 MB come from DRAM once,
// prefetched a pass ahead: 360 -> 348 us for the choice), else the rows'
// latency, which four warps a task and 128 registers of loads in flight
// shorten: a block per cluster with its rows staged in shared memory took
// 2,150 us of the 960-d choice of 1000 queries, now 382 in all.
template <int METRIC, int NS>
__global__ void __launch_bounds__(128, 4) clusters_rows_kernel(const float *queries, int dim, int dpad, int qs,
                                                            const float *fine_rows, const uint32_t *fine_ids,
                                                            const uint32_t *row_offs, const uint32_t *q_offs,
                                                            const uint32_t *q_list, const uint2 *tasks,
                                                            const uint32_t *n_tasks, int probes, float *part_d,
                                                            uint32_t *part_i) {
  extern __shared__ __align__(16) float smt[];
  __shared__ float md[4][4][NS];
  __shared__ uint32_t mi[4][4][NS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
  const uint32_t total = *n_tasks;
  for (uint32_t t = blockIdx.x; t < total; t += gridDim.x) {
    const uint2 task = tasks[t];
    const uint32_t c = task.x, qb = q_offs[c] + 4u * task.y;
    const int nqg = static_cast<int>(min(4u, q_offs[c + 1] - qb));
    const int r0 = static_cast<int>(row_offs[c]), r1 = static_cast<int>(row_offs[c + 1]);
    __syncthreads();  // the previous task's queries and lists are no longer read
    stage_queries<4>(smt, qs, dim, nqg, threadIdx.x, blockDim.x, [&](int a) {
      return queries + static_cast<size_t>(q_list[qb + a] / static_cast<uint32_t>(probes)) * dim;
    });
    __syncthreads();
    float bd[NS];
    uint32_t bi[NS];
    clear_list<NS>(bd, bi);
    for (int first = r0 + 8 * warp; first < r1; first += 8 * warps) {
      // the rows of this warp's next pass start their way into L2: on a
      // large base they come from DRAM (each cluster is read once)
      const int ahead = first + 8 * warps;
      if (ahead < r1) {
        const char *nx = reinterpret_cast<const char *>(fine_rows + static_cast<size_t>(ahead) * dpad);
        const int bytes = min(8, r1 - ahead) * dpad * 4;
        for (int i = 128 * lane; i < bytes; i += 128 * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + i));
      }
      const float d = tile_distance<METRIC>(smt, qs, fine_rows + static_cast<size_t>(first) * dpad, r1 - 1 - first,
                                            dpad, lane);
      const int r = first + (lane & 7);
      const uint32_t id = r < r1 ? __ldg(fine_ids + r) : 0xffffffffu;
      if (r < r1 && closer(d, id, bd[NS - 1], bi[NS - 1])) list_insert<NS>(bd, bi, d, id);
    }
    const int a = lane >> 3;
    const uint32_t pair = a < nqg ? q_list[qb + a] : 0u;
    const size_t at = static_cast<size_t>(pair) * NS;
    int h = 0;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < NS; ++r) {
      float wd;
      uint32_t wid;
      group8_take<NS>(bd, bi, h, wd, wid);
      if ((lane & 7) == 0) {
        md[warp][a][r] = wd;
        mi[warp][a][r] = wid;
      }
    }
    __syncthreads();
    if (warp == 0) {
      const int i = lane & 7;  // lane l takes warp l & 7's list of query l / 8
      clear_list<NS>(bd, bi);
      if (i < warps) {
#pragma unroll
        for (int r = 0; r < NS; ++r) {
          bd[r] = md[i][a][r];
          bi[r] = mi[i][a][r];
        }
      }
      h = 0;
      __syncwarp();
#pragma unroll
      for (int r = 0; r < NS; ++r) {
        float wd;
        uint32_t wid;
        group8_take<NS>(bd, bi, h, wd, wid);
        if (i == 0 && a < nqg) {
          part_d[at + r] = wd;
          part_i[at + r] = wid;
        }
      }
    }
  }
}

// Small batches: the whole two-level choice in two kernels, every head scored
// exactly (the heads stay in L2, and a few hundred queries' exact scan takes
// less than the tensor-core phase's three launches and the grouping by
// cluster: one query of 1M x 128 takes 22 us for the choice, 90 there).
// First (and for the flat choice, over all entries), block (x, y): rows
// chunk * x .. against the NQ queries from NQ * y, eight warps; each query's
// NP nearest of the chunk, by the rows' ids or positions (ids null), to
// part_* (queries x chunks x NP).
template <int METRIC, int NP, int NQ>
__global__ void __launch_bounds__(256, 2) nearest_rows_kernel(const float *queries, int nq, int qstride, int dim,
                                                              int dpad, int qs, const float *heads,
                                                              const uint32_t *ids, int n_heads, int chunk,
                                                              float *part_d, uint32_t *part_i) {
  extern __shared__ __align__(16) float smt[];
  __shared__ float md[8][4][NP];
  __shared__ uint32_t mi[8][4][NP];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int q0 = NQ * blockIdx.y, nqg = min(NQ, nq - q0);
  stage_queries<NQ>(smt, qs, dim, nqg, threadIdx.x, blockDim.x,
                    [&](int a) { return queries + static_cast<size_t>(q0 + a) * qstride; });
  __syncthreads();
  float bd[NP];
  uint32_t bi[NP];
  clear_list<NP>(bd, bi);
  const int r0 = chunk * blockIdx.x, r1 = min(n_heads, r0 + chunk);
  for (int first = r0 + 8 * warp; first < r1; first += 64) {
    const float *row = heads + static_cast<size_t>(first) * dpad;
    float d;
    int r;
    if (NQ == 1) {  // four lanes a row; the first of them keeps it
      float one[1];
      r = first + (lane >> 2);
      rows8_distance<METRIC, 1>(row + static_cast<size_t>(min(lane >> 2, r1 - 1 - first)) * dpad, smt, qs, dpad, one,
                                lane);
      d = one[0];
      if ((lane & 3) != 0) r = r1;
    } else {
      d = tile_distance<METRIC>(smt, qs, row, r1 - 1 - first, dpad, lane);
      r = first + (lane & 7);
    }
    const uint32_t name = ids && r < r1 ? __ldg(ids + r) : static_cast<uint32_t>(r);
    if (r < r1 && closer(d, name, bd[NP - 1], bi[NP - 1])) list_insert<NP>(bd, bi, d, name);
  }
  // NQ = 1: one list over the warp; else query l >> 3's over eight lanes
  const int a = NQ == 1 ? 0 : lane >> 3;
  int h = 0;
  __syncwarp();
#pragma unroll
  for (int r = 0; r < NP; ++r) {
    float wd;
    uint32_t wid;
    if (NQ == 1) warp_list_take<NP>(bd, bi, h, wd, wid);
    else group8_take<NP>(bd, bi, h, wd, wid);
    if ((lane & 7) == 0) {
      md[warp][a][r] = wd;
      mi[warp][a][r] = wid;
    }
  }
  __syncthreads();
  if (warp == 0) {
    const int q = lane >> 3;  // lane l takes warp l & 7's list of query l >> 3
    clear_list<NP>(bd, bi);
    if (q < NQ) {
#pragma unroll
      for (int r = 0; r < NP; ++r) {
        bd[r] = md[lane & 7][q][r];
        bi[r] = mi[lane & 7][q][r];
      }
    }
    h = 0;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < NP; ++r) {
      float wd;
      uint32_t wid;
      group8_take<NP>(bd, bi, h, wd, wid);
      if ((lane & 7) == 0 && q < nqg) {
        const size_t at = (static_cast<size_t>(q0 + q) * gridDim.x + blockIdx.x) * NP + r;
        part_d[at] = wd;
        part_i[at] = wid;
      }
    }
  }
}

// The flat choice's end: a warp per query merges the chunks' lists.
template <int N>
__global__ void __launch_bounds__(256) merge_lists_kernel(const float *part_d, const uint32_t *part_i, int nq,
                                                          int chunks, int ns, uint32_t *out) {
  const int lane = threadIdx.x & 31, q = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (q >= nq) return;  // whole warps
  float bd[N];
  uint32_t bi[N];
  clear_list<N>(bd, bi);
  const size_t base = static_cast<size_t>(q) * chunks * N;
  for (int i = lane; i < chunks * N; i += 32) list_insert<N>(bd, bi, part_d[base + i], part_i[base + i]);
  int h = 0;
  __syncwarp();
  for (int r = 0; r < ns; ++r) {
    float wd;
    uint32_t wid;
    warp_list_take<N>(bd, bi, h, wd, wid);
    // no finite distance (a query that is not finite): vertex 0
    if (lane == 0) out[static_cast<size_t>(q) * ns + r] = wid == 0xffffffffu ? 0u : wid;
  }
}

// The flat choice of short rows or few entries: a warp takes QB queries and a
// lane a whole distance.  The block stages 32 entry rows at a time (coalesced
// 16-byte loads, rows padded to an odd number of 16-byte units, so that the
// lanes' reads of 32 different rows hit distinct banks), and lane e scores row e
// against the warp's queries: it keeps the 32 partial sums and adds them in the
// butterfly's pairs.  Padded elements add fma(0, 0, t).  No lane is idle however
// few dimensions there are, and no lists go through memory (nearest_rows_kernel
// spreads a row over 32 lanes and needs a second launch).
template <int METRIC, int QB, int NS>
__global__ void __launch_bounds__(256) flat_tiled_kernel(const float *queries, int nq, int qstride, int dim, int dpad,
                                                         const float *entry_rows, const uint32_t *entry_ids,
                                                         int n_entries, int ns, uint32_t *starts) {
  extern __shared__ float4 sm4[];
  constexpr int TILE = 32;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int q0 = (blockIdx.x * nwarps + wib) * QB;
  const bool active = q0 < nq;  // warp-uniform; idle warps still help load tiles
  const int d4 = dpad >> 2, rs4 = d4 + 1;
  float4 *tile = sm4;
  float *qw = reinterpret_cast<float *>(sm4 + TILE * rs4) + static_cast<size_t>(wib) * QB * dpad;
  for (int b = 0; b < QB; ++b)
    for (int j = lane; j < dpad; j += 32)
      qw[b * dpad + j] = (q0 + b < nq && j < dim) ? queries[static_cast<size_t>(q0 + b) * qstride + j] : 0.0f;
  const float4 *q4 = reinterpret_cast<const float4 *>(qw);
  float bd[QB][NS];
  uint32_t bi[QB][NS];
#pragma unroll
  for (int b = 0; b < QB; ++b) clear_list<NS>(bd[b], bi[b]);
  for (int t0 = 0; t0 < n_entries; t0 += TILE) {
    const int rows = min(TILE, n_entries - t0);
    __syncthreads();  // the previous tile is consumed (and, first time, the queries are staged)
    for (int i = threadIdx.x; i < rows * d4; i += blockDim.x) {
      const int r = i / d4, c = i - r * d4;
      tile[r * rs4 + c] = __ldg(reinterpret_cast<const float4 *>(entry_rows + static_cast<size_t>(t0 + r) * dpad) + c);
    }
    __syncthreads();
    if (!active || lane >= rows) continue;
    const float4 *x4 = tile + lane * rs4;
    float t[QB][32], l[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      l[i] = 0.0f;
#pragma unroll
      for (int b = 0; b < QB; ++b) t[b][i] = 0.0f;
    }
    for (int c0 = 0; c0 < d4; c0 += 8) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        if (c0 + i < d4) {
          const float4 xv = x4[c0 + i];
          const float xs[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
          for (int b = 0; b < QB; ++b) {
            const float4 qv = q4[b * d4 + c0 + i];
            const float qq[4] = {qv.x, qv.y, qv.z, qv.w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              if (METRIC == SONG_METRIC_L2) {
                const float d = __fsub_rn(qq[c], xs[c]);
                t[b][4 * i + c] = __fmaf_rn(d, d, t[b][4 * i + c]);
              } else {
                t[b][4 * i + c] = __fmaf_rn(qq[c], xs[c], t[b][4 * i + c]);
              }
            }
          }
          if (METRIC == SONG_METRIC_COS) {
#pragma unroll
            for (int c = 0; c < 4; ++c) l[4 * i + c] = __fmaf_rn(xs[c], xs[c], l[4 * i + c]);
          }
        }
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
      for (int i = 0; i < off; ++i) {
#pragma unroll
        for (int b = 0; b < QB; ++b) t[b][i] = __fadd_rn(t[b][i], t[b][i + off]);
        if (METRIC == SONG_METRIC_COS) l[i] = __fadd_rn(l[i], l[i + off]);
      }
    }
    const uint32_t id = entry_ids[t0 + lane];
#pragma unroll
    for (int b = 0; b < QB; ++b) {
      float d;
      if (METRIC == SONG_METRIC_L2) {
        d = t[b][0];
      } else if (METRIC == SONG_METRIC_IP) {
        d = -t[b][0];
      } else if (l[0] != 0.0f) {
        const float sign = t[b][0] < 0.0f ? 1.0f : -1.0f;
        d = __fdiv_rn(__fmul_rn(__fmul_rn(sign, t[b][0]), t[b][0]), l[0]);
      } else {
        d = 0.0f;
      }
      list_insert<NS>(bd[b], bi[b], d, id);
    }
  }
  if (!active) return;
#pragma unroll
  for (int b = 0; b < QB; ++b) {
    int h = 0;
    for (int r = 0; r < ns; ++r) {
      float wd;
      uint32_t wid;
      warp_list_take<NS>(bd[b], bi[b], h, wd, wid);
      // no finite distance (a query that is not finite): vertex 0
      if (lane == 0 && q0 + b < nq) starts[static_cast<size_t>(q0 + b) * ns + r] = wid == 0xffffffffu ? 0u : wid;
    }
  }
}

// The N smallest of the block's lists (16 warps), ascending, to out(r, d, id)
// on one lane of warp 0; ends with the lists no longer read.
template <int N, class Out>
__device__ __forceinline__ void block_lists(float (&bd)[N], uint32_t (&bi)[N], int n, float (*md)[8],
                                            uint32_t (*mi)[8], int warp, int lane, Out out) {
  int h = 0;
  for (int r = 0; r < n; ++r) {
    float wd;
    uint32_t wid;
    warp_list_take<N>(bd, bi, h, wd, wid);
    if (lane == 0) {
      md[warp][r] = wd;
      mi[warp][r] = wid;
    }
  }
  __syncthreads();
  if (warp == 0) {
    clear_list<N>(bd, bi);
#pragma unroll
    for (int r = 0; r < N; ++r)
      if (lane < 16 && r < n) {
        bd[r] = md[lane][r];
        bi[r] = mi[lane][r];
      }
    h = 0;
    for (int r = 0; r < n; ++r) {
      float wd;
      uint32_t wid;
      warp_list_take<N>(bd, bi, h, wd, wid);
      if (lane == 0) out(r, wid);
    }
  }
  __syncthreads();
}

// Then a block of 16 warps per query: its probed clusters from the chunks'
// lists, and its ns nearest entries over those clusters' rows, the warps
// taking eight rows in turn.
template <int METRIC, int NP, int NS>
__global__ void __launch_bounds__(512) query_starts_kernel(const float *queries, int dim, int dpad, int qs,
                                                           const float *part_d, const uint32_t *part_i, int chunks,
                                                           int n_heads, int probes, const float *fine_rows,
                                                           const uint32_t *fine_ids, const uint32_t *row_offs, int ns,
                                                           uint32_t *starts) {
  extern __shared__ __align__(16) float smt[];
  __shared__ float md[16][8];
  __shared__ uint32_t mi[16][8];
  __shared__ uint32_t probe[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t q = blockIdx.x;
  stage_queries<1>(smt, qs, dim, 1, threadIdx.x, blockDim.x, [&](int) { return queries + q * dim; });
  {
    float bd[NP];
    uint32_t bi[NP];
    clear_list<NP>(bd, bi);
    const size_t base = q * chunks * NP;
    for (int i = threadIdx.x; i < chunks * NP; i += blockDim.x)
      list_insert<NP>(bd, bi, part_d[base + i], part_i[base + i]);
    // (a query that is not finite has no nearest head: cluster 0)
    block_lists<NP>(bd, bi, probes, md, mi, warp, lane,
                    [&](int r, uint32_t id) { probe[r] = id < static_cast<uint32_t>(n_heads) ? id : 0u; });
  }
  float bd[NS];
  uint32_t bi[NS];
  clear_list<NS>(bd, bi);
  int turn = warp;  // passes until this warp's next one
  for (int i = 0; i < probes; ++i) {
    const int r0 = static_cast<int>(row_offs[probe[i]]), r1 = static_cast<int>(row_offs[probe[i] + 1]);
    scan_rows<METRIC, NS>(fine_rows, dpad, r0 + 8 * turn, 128, r1, smt, qs, bd, bi, lane,
                             [&](int row) { return __ldg(fine_ids + row); });
    turn = (turn + 15 * ((r1 - r0 + 7) / 8)) & 15;
  }
  block_lists<NS>(bd, bi, ns, md, mi, warp, lane,
                  [&](int r, uint32_t id) { starts[q * ns + r] = id == 0xffffffffu ? 0u : id; });
}

// Each query's ns nearest over its probes' lists, ascending by (distance, id).
template <int NS>
__global__ void merge_starts_kernel(const float *part_d, const uint32_t *part_i, int nq, int probes, int ns,
                                    uint32_t *starts) {
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < nq; q += gridDim.x * blockDim.x) {
    float bd[NS];
    uint32_t bi[NS];
#pragma unroll
    for (int m = 0; m < NS; ++m) {
      bd[m] = __int_as_float(0x7f800000);
      bi[m] = 0xffffffffu;
    }
    const size_t base = static_cast<size_t>(q) * probes * NS;
    for (int i = 0; i < probes * NS; ++i) list_insert<NS>(bd, bi, part_d[base + i], part_i[base + i]);
#pragma unroll
    for (int m = 0; m < NS; ++m)
      if (m < ns)  // no finite distance (a query that is not finite): vertex 0
        starts[static_cast<size_t>(q) * ns + m] = bi[m] == 0xffffffffu ? 0u : bi[m];
  }
}

// Work area of the choice, grown to `words`.
cudaError_t entry_work(song_index *ix, size_t words) {
  if (words <= ix->cap_entry_work) return cudaSuccess;
  cudaFree(ix->d_entry_work);
  ix->d_entry_work = nullptr;
  ix->cap_entry_work = 0;
  cudaError_t e = song::dev_malloc(&ix->d_entry_work, sizeof(uint32_t) * words);
  if (e == cudaSuccess) ix->cap_entry_work = words;
  return e;
}

// Template arguments for run-time list lengths 1, 2, 4 or 8.
#define SONG_BY_LEN(n, CALL)  \
  switch (n) {                \
    case 1: CALL(1); break;   \
    case 2: CALL(2); break;   \
    case 4: CALL(4); break;   \
    default: CALL(8); break;  \
  }

// Batches that take the two-kernel choice: up to 512 queries (1M x 128, 4096
// heads: 68 against 96 us at 257 queries, 112 against 109 at 512; 960-d rows,
// 1024 heads: 230 against 323 at 257, 355 against 349 at 600; 256-d rows, 126
// against 128 at 500), within 2^29 query x head x dimension products; with few
// short heads, 2^22 products (15k x 16, 128 heads: 44 against 94 us at 1000
// queries).
bool small_batch(int nq, int coarse, int dpad) {
  const double work = static_cast<double>(nq) * coarse * dpad;
  return (nq <= 512 && work <= 536870912.0) || work <= 4194304.0;
}

// nearest_rows_kernel's split: one query a block row while there are few, four
// afterwards; chunks of 64 rows (one pass a warp) until the grid fills the GPU
// some times over.
struct RowsSplit {
  int nqb, chunk;
};
RowsSplit rows_split(int nq, int n) {
  RowsSplit r{nq <= 4 ? 1 : 4, 64};
  const long long groups = (nq + r.nqb - 1) / r.nqb;
  while (r.chunk < n && groups * (n / r.chunk) > 2048) r.chunk *= 2;
  return r;
}

// Whether the flat choice takes flat_tiled_kernel (rows of up to 1 KB).  Both
// kernels' times in us, estimated: one warp's chain over the tiles of 32 rows,
// once or as often as the warps exceed the resident ones; one block's over the
// passes of 64 rows, and as often again as 200 blocks go into the grid.  The
// constants are fitted to 1,944 shapes (4 to 256 dimensions, 8 to 16,384
// entries, 1 to 50,000 queries, 1 to 8 starts, L2 and cosine): the kernel taken
// is the faster one or within 5 % of it in 96 of 100, at worst 1.4 times as long.
// 10,000 queries of 16-d L2 rows: 64 entries 15 us with the tiled kernel and 31
// with the other, 4096 entries 394 and 454; one query of 4096 entries 109 and 11.
bool flat_tiled(int metric, int nq, int n, int dpad, int len) {
  if (dpad > 256) return false;
  const bool cos = metric == SONG_METRIC_COS;
  const double lists = len <= 1 ? 0.0 : (len <= 4 ? 1.0 : 2.0), tiles = (n + 31) / 32;
  const double tile = cos ? 0.51 + 0.0145 * dpad + 0.23 * lists : 0.55 + 0.018 * dpad + 0.37 * lists;
  const double tiled = 6.8 + 0.9 * lists + tiles * tile * std::max(1.0, cos ? nq / 1840.0 : nq / (2.0 * 1640.0));
  const RowsSplit r = rows_split(nq, n);
  const double passes = (std::min(r.chunk, n) + 63) / 64, pass = (cos ? 0.54 : 0.41) + 0.0033 * std::max(dpad, 32) + 0.12 * lists;
  const double blocks = std::ceil(static_cast<double>(nq) / r.nqb) * ((n - 1) / r.chunk + 1);
  const double rows = 9.8 + 1.0 * lists + (0.87 + 0.77 * lists + passes * pass) * (1.0 + blocks / 200.0);
  return tiled < 0.97 * rows;
}

// The NP nearest of n rows for each of nq queries, chunk by chunk: *chunks
// lists a query in the work area.
template <int METRIC, int NP>
cudaError_t launch_nearest_rows(song_index *ix, const float *queries, int nq, int qstride, const float *rows,
                                const uint32_t *ids, int n, int *chunks, float **part_d, uint32_t **part_i,
                                cudaStream_t s) {
  const int dim = ix->dx.dim, dpad = static_cast<int>(ix->dx.f32_row_bytes / 4), qs = (dpad + 31) & ~31;
  const RowsSplit split = rows_split(nq, n);
  const int nqb = split.nqb, chunk = split.chunk;
  *chunks = (n + chunk - 1) / chunk;
  const size_t lists = static_cast<size_t>(nq) * *chunks * NP;
  cudaError_t e = entry_work(ix, 2 * lists);
  if (e != cudaSuccess) return e;
  *part_d = reinterpret_cast<float *>(ix->d_entry_work);
  *part_i = ix->d_entry_work + lists;
  auto k = nqb == 1 ? nearest_rows_kernel<METRIC, NP, 1> : nearest_rows_kernel<METRIC, NP, 4>;
  const size_t smem = sizeof(float) * nqb * qs;
  if ((e = allow_shared(k, smem)) != cudaSuccess) return e;
  // at most 65,535 block rows a launch
  for (int q0 = 0; q0 < nq; q0 += 65535 * nqb) {
    const int m = std::min(nq - q0, 65535 * nqb);
    const size_t at = static_cast<size_t>(q0) * *chunks * NP;
    k<<<dim3(*chunks, (m + nqb - 1) / nqb), 256, smem, s>>>(queries + static_cast<size_t>(q0) * qstride, m, qstride,
                                                           dim, dpad, qs, rows, ids, n, chunk, *part_d + at,
                                                           *part_i + at);
  }
  return cudaGetLastError();
}

// The ns nearest of n rows (ids) for each of nq queries (qstride floats
// apart), into out[q * ns ..]: the flat choice.  4096 entries of 256 floats:
// 1.19 ms for 10,000 queries (3.15 with a thread per distance), 18 us for one
// (773: one warp then took all the entries).
template <int METRIC, int N>
cudaError_t launch_flat(song_index *ix, const float *queries, int nq, int qstride, const float *rows,
                        const uint32_t *ids, int n, int ns, uint32_t *out, cudaStream_t s) {
  const int dpad = static_cast<int>(ix->dx.f32_row_bytes / 4);
  if (flat_tiled(METRIC, nq, n, dpad, N)) {
    constexpr int QB = METRIC == SONG_METRIC_COS ? 1 : 2;
    const int per_warp = static_cast<int>(sizeof(float)) * dpad * QB, tile_bytes = 32 * (dpad / 4 + 1) * 16;
    const int wpb = std::max(1, std::min(8, (48 * 1024 - tile_bytes) / per_warp));
    flat_tiled_kernel<METRIC, QB, N><<<(nq - 1) / (wpb * QB) + 1, 32 * wpb, tile_bytes + per_warp * wpb, s>>>(
        queries, nq, qstride, ix->dx.dim, dpad, rows, ids, n, ns, out);
    return cudaGetLastError();
  }
  int chunks = 0;
  float *part_d = nullptr;
  uint32_t *part_i = nullptr;
  cudaError_t e = launch_nearest_rows<METRIC, N>(ix, queries, nq, qstride, rows, ids, n, &chunks, &part_d, &part_i, s);
  if (e != cudaSuccess) return e;
  merge_lists_kernel<N><<<(nq + 7) / 8, 256, 0, s>>>(part_d, part_i, nq, chunks, ns, out);
  return cudaGetLastError();
}

cudaError_t launch_nearest(song_index *ix, const float *queries, int nq, int qstride, const float *rows,
                           const uint32_t *ids, int n, int ns, uint32_t *out, cudaStream_t s) {
  const int len = ns <= 1 ? 1 : (ns <= 2 ? 2 : (ns <= 4 ? 4 : 8));
  cudaError_t e = cudaSuccess;
#define SONG_FLAT_L2(N) e = launch_flat<SONG_METRIC_L2, N>(ix, queries, nq, qstride, rows, ids, n, ns, out, s)
#define SONG_FLAT_IP(N) e = launch_flat<SONG_METRIC_IP, N>(ix, queries, nq, qstride, rows, ids, n, ns, out, s)
#define SONG_FLAT_COS(N) e = launch_flat<SONG_METRIC_COS, N>(ix, queries, nq, qstride, rows, ids, n, ns, out, s)
  switch (ix->dx.metric) {
    case SONG_METRIC_L2: SONG_BY_LEN(len, SONG_FLAT_L2); break;
    case SONG_METRIC_IP: SONG_BY_LEN(len, SONG_FLAT_IP); break;
    default: SONG_BY_LEN(len, SONG_FLAT_COS); break;
  }
#undef SONG_FLAT_L2
#undef SONG_FLAT_IP
#undef SONG_FLAT_COS
  return e;
}

template <int METRIC, int NP>
cudaError_t launch_small(song_index *ix, const float *queries, int nq, int ns, uint32_t *out, cudaStream_t s) {
  const int dim = ix->dx.dim, dpad = static_cast<int>(ix->dx.f32_row_bytes / 4), qs = (dpad + 31) & ~31;
  const int n = ix->n_coarse;
  int chunks = 0;
  float *part_d = nullptr;
  uint32_t *part_i = nullptr;
  cudaError_t e = launch_nearest_rows<METRIC, NP>(ix, queries, nq, dim, ix->d_coarse_rows, nullptr, n, &chunks,
                                                  &part_d, &part_i, s);
  if (e != cudaSuccess) return e;
#define SONG_STARTS(NS)                                                                                       \
  do {                                                                                                        \
    auto k = query_starts_kernel<METRIC, NP, NS>;                                                             \
    if ((e = allow_shared(k, sizeof(float) * qs)) != cudaSuccess) return e;                                     \
    k<<<nq, 512, sizeof(float) * qs, s>>>(queries, dim, dpad, qs, part_d, part_i, chunks, n, ix->n_probes,    \
                                          ix->d_entry_rows, ix->d_entry_ids, ix->d_offsets, ns, out);         \
  } while (0)
  SONG_BY_LEN(ns <= 1 ? 1 : (ns <= 2 ? 2 : (ns <= 4 ? 4 : 8)), SONG_STARTS);
#undef SONG_STARTS
  return cudaGetLastError();
}

template <int METRIC>
cudaError_t launch_small_by_probes(song_index *ix, const float *queries, int nq, uint32_t *out, cudaStream_t s) {
  const int np = ix->n_probes;
  cudaError_t e = cudaSuccess;
#define SONG_SMALL(NP) e = launch_small<METRIC, NP>(ix, queries, nq, ix->n_starts, out, s)
  SONG_BY_LEN(np <= 1 ? 1 : (np <= 2 ? 2 : (np <= 4 ? 4 : 8)), SONG_SMALL);
#undef SONG_SMALL
  return e;
}

// The two-level choice on stream s.  `out` holds nq * (ns + probes) words:
// the starts, then the probed clusters.
cudaError_t launch_2level(song_index *ix, const float *queries, int nq, uint32_t *out, cudaStream_t s) {
  if (ix->head_path < 0 && small_batch(nq, ix->n_coarse, static_cast<int>(ix->dx.f32_row_bytes / 4))) {
    switch (ix->dx.metric) {
      case SONG_METRIC_L2: return launch_small_by_probes<SONG_METRIC_L2>(ix, queries, nq, out, s);
      case SONG_METRIC_IP: return launch_small_by_probes<SONG_METRIC_IP>(ix, queries, nq, out, s);
      default: return launch_small_by_probes<SONG_METRIC_COS>(ix, queries, nq, out, s);
    }
  }
  const int dim = ix->dx.dim, dpad = static_cast<int>(ix->dx.f32_row_bytes / 4), qs = (dpad + 31) & ~31;
  const int ns = ix->n_starts, np = ix->n_probes, coarse = ix->n_coarse;
  const TileShape ts = tile_shape(dpad);
  const size_t smem = ts.smem(dpad);
  const int bq = 4 * ts.warps;
  const int NSel = ns <= 1 ? 1 : (ns <= 2 ? 2 : (ns <= 4 ? 4 : 8));
  const int NPsel = np <= 1 ? 1 : (np <= 2 ? 2 : (np <= 4 ? 4 : 8));
  uint32_t *probes = out + static_cast<size_t>(nq) * ns;
  // work area: tasks (at most one per pair), cursors, offsets, the tasks'
  // offsets, inverted lists, per-(query, probe) lists
  const size_t pairs = static_cast<size_t>(nq) * np;
  cudaError_t e = entry_work(ix, 2 * pairs + static_cast<size_t>(coarse) * 3 + 2 + pairs + 2 * pairs * NSel);
  if (e != cudaSuccess) return e;
  uint2 *tasks = reinterpret_cast<uint2 *>(ix->d_entry_work);
  uint32_t *cursor = ix->d_entry_work + 2 * pairs;
  uint32_t *q_offs = cursor + coarse;
  uint32_t *task_offs = q_offs + coarse + 1;
  uint32_t *n_tasks = task_offs + coarse;
  uint32_t *q_list = n_tasks + 1;
  float *part_d = reinterpret_cast<float *>(q_list + pairs);
  uint32_t *part_i = q_list + pairs + pairs * NSel;
  // warps a task: four share a task's rows while there are few tasks, two
  // from 32768 pairs on (10,000 queries, 4 probes: 348 us for the whole choice
  // with two, 367 with four, 360 with one; 2501 queries of 256-d rows 313 us
  // with one, 187 with four)
  const int tw = pairs >= 32768 ? 2 : 4;
  e = cudaMemsetAsync(ix->d_cl_count, 0, sizeof(uint32_t) * coarse, s);
  if (e != cudaSuccess) return e;
  const unsigned grid_q = static_cast<unsigned>((nq + bq - 1) / bq);
#define SONG_HEADS(M, NP)                                                                                \
  do {                                                                                                   \
    auto k_ = heads_tiled_kernel<M, NP>;                                                                 \
    if ((e = allow_shared(k_, smem)) != cudaSuccess) return e;                                             \
    k_<<<grid_q, ts.warps * 32, smem, s>>>(queries, nq, dim, dpad, ix->d_coarse_rows, coarse, np, ts.rows, \
                                           ts.nbuf, probes, ix->d_cl_count);                             \
  } while (0)
#define SONG_CLUSTERS(M, NS)                                                                             \
  do {                                                                                                   \
    auto k_ = clusters_rows_kernel<M, NS>;                                                               \
    const size_t qsm = sizeof(float) * 4 * qs;                                                           \
    if ((e = allow_shared(k_, qsm)) != cudaSuccess) return e;                                              \
    int per_sm = 0, sms = 0, dev = 0;                                                                    \
    cudaGetDevice(&dev);                                                                                 \
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);                                   \
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_, 32 * tw, qsm)) != cudaSuccess)   \
      return e;                                                                                          \
    const size_t cap = static_cast<size_t>(std::max(1, per_sm)) * sms;                                   \
    k_<<<static_cast<unsigned>(std::min(cap, pairs)), 32 * tw, qsm, s>>>(                                \
        queries, dim, dpad, qs, ix->d_entry_rows, ix->d_entry_ids, ix->d_offsets, q_offs, q_list, tasks, \
        n_tasks, np, part_d, part_i);                                                                    \
    merge_starts_kernel<NS><<<(nq + 255) / 256, 256, 0, s>>>(part_d, part_i, nq, np, ns, out);           \
  } while (0)
#define SONG_HEADS_L2(NP) SONG_HEADS(SONG_METRIC_L2, NP)
#define SONG_HEADS_IP(NP) SONG_HEADS(SONG_METRIC_IP, NP)
#define SONG_HEADS_COS(NP) SONG_HEADS(SONG_METRIC_COS, NP)
#define SONG_CLUSTERS_L2(NS) SONG_CLUSTERS(SONG_METRIC_L2, NS)
#define SONG_CLUSTERS_IP(NS) SONG_CLUSTERS(SONG_METRIC_IP, NS)
#define SONG_CLUSTERS_COS(NS) SONG_CLUSTERS(SONG_METRIC_COS, NS)
  if (heads_mma_usable(ix, queries, np)) {  // tensor-core scores, exact re-scoring of a shortlist
    if ((e = launch_heads_mma(ix, queries, nq, np, probes, s)) != cudaSuccess) return e;
  } else {
    switch (ix->dx.metric) {
      case SONG_METRIC_L2: SONG_BY_LEN(NPsel, SONG_HEADS_L2); break;
      case SONG_METRIC_IP: SONG_BY_LEN(NPsel, SONG_HEADS_IP); break;
      default: SONG_BY_LEN(NPsel, SONG_HEADS_COS); break;
    }
  }
  cluster_scan_kernel<<<1, 1024, 0, s>>>(ix->d_cl_count, coarse, ix->d_cl_order, q_offs, cursor, task_offs,
                                         n_tasks);
  cluster_scatter_kernel<<<static_cast<unsigned>(std::min<size_t>((pairs + 255) / 256, 4096)), 256, 0, s>>>(
      probes, static_cast<int>(pairs), q_offs, task_offs, cursor, q_list, tasks);
  switch (ix->dx.metric) {
    case SONG_METRIC_L2: SONG_BY_LEN(NSel, SONG_CLUSTERS_L2); break;
    case SONG_METRIC_IP: SONG_BY_LEN(NSel, SONG_CLUSTERS_IP); break;
    default: SONG_BY_LEN(NSel, SONG_CLUSTERS_COS); break;
  }
#undef SONG_CLUSTERS_L2
#undef SONG_CLUSTERS_IP
#undef SONG_CLUSTERS_COS
#undef SONG_HEADS_L2
#undef SONG_HEADS_IP
#undef SONG_HEADS_COS
#undef SONG_CLUSTERS
#undef SONG_HEADS
  return cudaGetLastError();
}

}  // namespace

void clear_entries(song_index *ix) {
  cudaFree(ix->d_entry_ids);
  cudaFree(ix->d_entry_rows);
  cudaFree(ix->d_coarse_rows);
  cudaFree(ix->d_offsets);
  cudaFree(ix->d_cl_count);
  cudaFree(ix->d_cl_order);
  cudaFree(ix->d_entry_work);
  cudaFree(ix->d_head_n2);
  cudaFree(ix->d_head_scores);
  ix->d_head_n2 = nullptr;
  ix->d_head_scores = nullptr;
  ix->cap_head_scores = 0;
  ix->heads_mma = false;
  ix->d_entry_ids = nullptr;
  ix->d_entry_rows = nullptr;
  ix->d_coarse_rows = nullptr;
  ix->d_offsets = nullptr;
  ix->d_cl_count = nullptr;
  ix->d_cl_order = nullptr;
  ix->d_entry_work = nullptr;
  ix->cap_entry_work = 0;
  ix->n_entries = 0;
  ix->n_coarse = 0;
  ix->n_probes = 0;
  ix->n_starts = 1;
}

int prepare_starts(song_index *ix, SearchCall &c, cudaStream_t s) {
  c.starts = nullptr;
  c.n_starts = 1;
  if (ix->n_entries <= 0 || c.nq <= 0) return SONG_OK;
  if (ix->n_starts > c.pq) return fail(SONG_ERR_ARG, "%d start vertices need pq >= %d", ix->n_starts, ix->n_starts);
  // the starts, then (two-level choice) each query's probed clusters
  const size_t need = static_cast<size_t>(c.nq) * (ix->n_starts + (ix->n_coarse > 0 ? ix->n_probes : 0));
  if (need > ix->cap_starts) {
    if (ix->d_starts) cudaFree(ix->d_starts);
    ix->d_starts = nullptr;
    ix->cap_starts = 0;
    cudaError_t e = song::dev_malloc(&ix->d_starts, sizeof(uint32_t) * need);
    if (e != cudaSuccess) return fail(SONG_ERR_OOM, "entry starts: %s", cudaGetErrorString(e));
    ix->cap_starts = need;
  }
  const cudaError_t le =
      ix->n_coarse > 0 ? launch_2level(ix, c.queries, c.nq, ix->d_starts, s)
                       : launch_nearest(ix, c.queries, c.nq, ix->dx.dim, ix->d_entry_rows, ix->d_entry_ids,
                                        ix->n_entries, ix->n_starts, ix->d_starts, s);
  if (le != cudaSuccess)
    return fail(le == cudaErrorMemoryAllocation ? SONG_ERR_OOM : SONG_ERR_CUDA, "entry choice: %s",
                cudaGetErrorString(le));
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(SONG_ERR_CUDA, "entry launch: %s", cudaGetErrorString(e));
  c.starts = ix->d_starts;
  c.n_starts = ix->n_starts;
  return SONG_OK;
}

}  // namespace song

extern "C" int song_index_set_entries(song_index *ix, const uint64_t *ids, int count, int starts) {
  using namespace song;
  clear_error();
  if (!ix) return fail(SONG_ERR_ARG, "null index");
  if (count < 0 || count > SONG_MAX_ENTRIES) return fail(SONG_ERR_ARG, "entry count must be 0..%d", SONG_MAX_ENTRIES);
  if (count > 0 && (starts < 1 || starts > SONG_MAX_STARTS || starts > count))
    return fail(SONG_ERR_ARG, "starts must be 1..min(%d, entry count)", SONG_MAX_STARTS);
  if (count > 0 && !ids) return fail(SONG_ERR_ARG, "null entry ids");
  std::vector<uint32_t> h(static_cast<size_t>(count));
  for (int i = 0; i < count; ++i) {
    if (ids[i] >= ix->dx.n) return fail(SONG_ERR_ARG, "entry %d: id %llu >= n", i, (unsigned long long)ids[i]);
    h[i] = static_cast<uint32_t>(ids[i]);
  }
  {
    std::vector<uint32_t> u(h);
    std::sort(u.begin(), u.end());
    if (std::adjacent_find(u.begin(), u.end()) != u.end()) return fail(SONG_ERR_ARG, "entry ids must be distinct");
  }
  if (ix->servers > 0) return fail(SONG_ERR_ARG, "entries are in use by %d server(s)", ix->servers);
  DeviceGuard guard(ix->device);
  if (!guard.ok) return fail(SONG_ERR_CUDA, "cannot select device %d", ix->device);
  cudaError_t e = cudaSuccess;
  clear_entries(ix);
  if (count == 0) return SONG_OK;
  const int dpad = static_cast<int>(ix->dx.f32_row_bytes / 4);
  e = song::dev_malloc(&ix->d_entry_ids, sizeof(uint32_t) * count);
  if (e == cudaSuccess) e = song::dev_malloc(&ix->d_entry_rows, sizeof(float) * count * static_cast<size_t>(dpad));
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(ix->d_entry_ids, h.data(), sizeof(uint32_t) * count, cudaMemcpyHostToDevice, ix->stream);
  if (e == cudaSuccess) {
    gather_entry_rows_kernel<<<256, 256, 0, ix->stream>>>(ix->dx.rows_f32, static_cast<uint32_t>(dpad),
                                                          ix->d_entry_ids, count, dpad, ix->d_entry_rows);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(ix->stream);
  if (e != cudaSuccess) {
    cudaFree(ix->d_entry_ids);
    cudaFree(ix->d_entry_rows);
    ix->d_entry_ids = nullptr;
    ix->d_entry_rows = nullptr;
    return fail(e == cudaErrorMemoryAllocation ? SONG_ERR_OOM : SONG_ERR_CUDA, "entries: %s", cudaGetErrorString(e));
  }
  ix->n_entries = count;
  ix->n_starts = starts;
  return SONG_OK;
}

extern "C" int song_index_set_entries_2level(song_index *ix, const uint64_t *ids, int count, int coarse, int probes,
                                             int starts) {
  using namespace song;
  clear_error();
  if (!ix) return fail(SONG_ERR_ARG, "null index");
  if (count < 1 || count > SONG_MAX_ENTRIES_2LEVEL || !ids)
    return fail(SONG_ERR_ARG, "entry count must be 1..%d", SONG_MAX_ENTRIES_2LEVEL);
  if (coarse < 1 || coarse > count || coarse > SONG_MAX_COARSE)
    return fail(SONG_ERR_ARG, "coarse must be 1..min(count, %d)", SONG_MAX_COARSE);
  if (probes < 1 || probes > SONG_MAX_STARTS || probes > coarse)
    return fail(SONG_ERR_ARG, "probes must be 1..min(%d, coarse)", SONG_MAX_STARTS);
  if (starts < 1 || starts > probes) return fail(SONG_ERR_ARG, "starts must be 1..probes");
  const int dpad = static_cast<int>(ix->dx.f32_row_bytes / 4);
  // the smallest block shape (one warp, 4 queries, one tile of 8 rows) fits
  // a block's shared memory
  auto fits = [](int dp) { return TileShape{1, 8, 1}.smem(dp) <= 227u * 1024u; };
  if (!fits(dpad)) {
    int widest = 4;
    while (fits(widest + 4)) widest += 4;
    return fail(SONG_ERR_ARG, "two-level entries support rows of up to %d floats", widest);
  }
  std::vector<uint32_t> h(static_cast<size_t>(count));
  for (int i = 0; i < count; ++i) {
    if (ids[i] >= ix->dx.n) return fail(SONG_ERR_ARG, "entry %d: id %llu >= n", i, (unsigned long long)ids[i]);
    h[i] = static_cast<uint32_t>(ids[i]);
  }
  {
    std::vector<uint32_t> u(h);
    std::sort(u.begin(), u.end());
    if (std::adjacent_find(u.begin(), u.end()) != u.end()) return fail(SONG_ERR_ARG, "entry ids must be distinct");
  }
  if (ix->servers > 0) return fail(SONG_ERR_ARG, "entries are in use by %d server(s)", ix->servers);
  DeviceGuard guard(ix->device);
  if (!guard.ok) return fail(SONG_ERR_CUDA, "cannot select device %d", ix->device);
  cudaError_t e = cudaSuccess;
  clear_entries(ix);
  // 1. all entry rows in list order; the clusters of the non-coarse entries
  uint32_t *d_ids = nullptr, *d_assign = nullptr, *d_perm = nullptr;
  float *d_rows = nullptr;
  std::vector<uint32_t> assign(static_cast<size_t>(count - coarse));
  e = song::dev_malloc(&d_ids, sizeof(uint32_t) * count);
  if (e == cudaSuccess) e = song::dev_malloc(&d_rows, sizeof(float) * static_cast<size_t>(count) * dpad);
  if (e == cudaSuccess && count > coarse) e = song::dev_malloc(&d_assign, sizeof(uint32_t) * (count - coarse));
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_ids, h.data(), sizeof(uint32_t) * count, cudaMemcpyHostToDevice, ix->stream);
  if (e == cudaSuccess) {
    gather_entry_rows_kernel<<<256, 256, 0, ix->stream>>>(ix->dx.rows_f32, static_cast<uint32_t>(dpad), d_ids, count,
                                                          dpad, d_rows);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess && count > coarse)
    e = launch_nearest(ix, d_rows + static_cast<size_t>(coarse) * dpad, count - coarse, dpad, d_rows, d_ids, coarse, 1,
                       d_assign, ix->stream);
  if (e == cudaSuccess && count > coarse)
    e = cudaMemcpyAsync(assign.data(), d_assign, sizeof(uint32_t) * (count - coarse), cudaMemcpyDeviceToHost,
                        ix->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ix->stream);
  // 2. clusters numbered by coarse id; entries ordered by cluster
  std::vector<int> corder(static_cast<size_t>(coarse));
  for (int i = 0; i < coarse; ++i) corder[i] = i;
  std::sort(corder.begin(), corder.end(), [&](int a, int b) { return h[a] < h[b]; });
  std::vector<uint32_t> cl_of_id_sorted(static_cast<size_t>(coarse));  // sorted coarse ids
  std::vector<int> rank(static_cast<size_t>(coarse));
  for (int k = 0; k < coarse; ++k) {
    rank[corder[k]] = k;
    cl_of_id_sorted[k] = h[corder[k]];
  }
  std::vector<uint32_t> cluster(static_cast<size_t>(count));
  for (int f = 0; f < count && e == cudaSuccess; ++f) {
    if (f < coarse) {
      cluster[f] = static_cast<uint32_t>(rank[f]);
    } else {
      const auto it = std::lower_bound(cl_of_id_sorted.begin(), cl_of_id_sorted.end(), assign[f - coarse]);
      cluster[f] = static_cast<uint32_t>(it - cl_of_id_sorted.begin());
    }
  }
  std::vector<uint32_t> offsets(static_cast<size_t>(coarse) + 1, 0u), perm(static_cast<size_t>(count)),
      fine_ids(static_cast<size_t>(count)), cperm(static_cast<size_t>(coarse));
  for (int f = 0; f < count; ++f) ++offsets[cluster[f] + 1];
  for (int k = 0; k < coarse; ++k) offsets[k + 1] += offsets[k];
  {
    std::vector<uint32_t> fill(offsets.begin(), offsets.end() - 1);
    for (int f = 0; f < count; ++f) {
      const uint32_t pos = fill[cluster[f]]++;
      perm[pos] = static_cast<uint32_t>(f);  // row f of d_rows
      fine_ids[pos] = h[f];
    }
  }
  for (int k = 0; k < coarse; ++k) cperm[k] = static_cast<uint32_t>(corder[k]);
  // the clusters largest first: the cluster phase's warps take tasks in this
  // order, so that the long tasks start first and the last ones are short
  std::vector<uint32_t> by_size(static_cast<size_t>(coarse));
  for (int k = 0; k < coarse; ++k) by_size[k] = static_cast<uint32_t>(k);
  std::stable_sort(by_size.begin(), by_size.end(), [&](uint32_t a, uint32_t b) {
    return offsets[a + 1] - offsets[a] > offsets[b + 1] - offsets[b];
  });
  // 3. device copies: entries in cluster order, coarse rows by id, offsets
  uint32_t *d_cperm = nullptr;
  if (e == cudaSuccess) e = song::dev_malloc(&d_perm, sizeof(uint32_t) * count);
  if (e == cudaSuccess) e = song::dev_malloc(&d_cperm, sizeof(uint32_t) * coarse);
  if (e == cudaSuccess) e = song::dev_malloc(&ix->d_entry_rows, sizeof(float) * static_cast<size_t>(count) * dpad);
  if (e == cudaSuccess) e = song::dev_malloc(&ix->d_entry_ids, sizeof(uint32_t) * count);
  if (e == cudaSuccess) e = song::dev_malloc(&ix->d_coarse_rows, sizeof(float) * static_cast<size_t>(coarse) * dpad);
  if (e == cudaSuccess) e = song::dev_malloc(&ix->d_offsets, sizeof(uint32_t) * (coarse + 1));
  if (e == cudaSuccess) e = song::dev_malloc(&ix->d_cl_order, sizeof(uint32_t) * coarse);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(ix->d_cl_order, by_size.data(), sizeof(uint32_t) * coarse, cudaMemcpyHostToDevice, ix->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_perm, perm.data(), sizeof(uint32_t) * count, cudaMemcpyHostToDevice, ix->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(d_cperm, cperm.data(), sizeof(uint32_t) * coarse, cudaMemcpyHostToDevice, ix->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(ix->d_entry_ids, fine_ids.data(), sizeof(uint32_t) * count, cudaMemcpyHostToDevice, ix->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(ix->d_offsets, offsets.data(), sizeof(uint32_t) * (coarse + 1), cudaMemcpyHostToDevice,
                        ix->stream);
  if (e == cudaSuccess) {
    gather_entry_rows_kernel<<<256, 256, 0, ix->stream>>>(d_rows, static_cast<uint32_t>(dpad), d_perm, count, dpad,
                                                          ix->d_entry_rows);
    gather_entry_rows_kernel<<<64, 256, 0, ix->stream>>>(d_rows, static_cast<uint32_t>(dpad), d_cperm, coarse, dpad,
                                                         ix->d_coarse_rows);
    e = cudaGetLastError();
  }
  // 4. the per-cluster probe counters of the second kernel; the head rows'
  // tensor map and norms (the tensor-core head phase; without them the
  // CUDA-core kernel scores the heads)
  if (e == cudaSuccess) e = song::dev_malloc(&ix->d_cl_count, sizeof(uint32_t) * coarse);
  if (e == cudaSuccess) song::heads_mma_prepare(ix, coarse);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ix->stream);
  cudaFree(d_ids);
  cudaFree(d_rows);
  cudaFree(d_assign);
  cudaFree(d_perm);
  cudaFree(d_cperm);
  if (e != cudaSuccess) {
    clear_entries(ix);
    return fail(e == cudaErrorMemoryAllocation ? SONG_ERR_OOM : SONG_ERR_CUDA, "entries: %s", cudaGetErrorString(e));
  }
  ix->n_entries = count;
  ix->n_coarse = coarse;
  ix->n_probes = probes;
  ix->n_starts = starts;
  return SONG_OK;
}
