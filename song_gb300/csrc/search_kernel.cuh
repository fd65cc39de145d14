// search_kernel.cuh -- the batched best-first graph search kernel for sm_103a.
//
// It computes what warp_independent_search_kernel computes
// (warp_astar_accelerator.h:41-341): for each query, a best-first walk from
// vertex 0 over the fixed-degree graph with a candidate queue bounded at pq,
// a top-pq list of expanded vertices, a visited hash over queue and list, the
// select-insert rule (skip a candidate when the queue is full and its maximum
// is closer) and the finish rule (stop when the list is full and its maximum
// is <= the vertex just popped).  With FP32 storage the distances are the
// reference's bit for bit: lane l sums dims l, l+32, ... with fused
// multiply-add and the 32 partial sums meet in the xor butterfly 16,8,4,2,1.
//
// GB300 design:
//  * persistent warps pull queries from a work counter; warps never wait for
//    one another (the only block barrier is the model load at kernel start);
//  * per-query state: query vector, visited hash (the reference's FixHash,
//    8*pq slots) and, for large pq, the candidate queue's ring in the warp's
//    shared memory; smaller queues and the top-pq list in registers
//    (reg_queue.cuh);
//  * each hop's unvisited neighbour rows are read straight from global memory
//    into registers, eight rows at a time, four lanes a row (gather_rows);
//  * one hop's visited-hash calls run one lane each (visited_update);
//  * the next hop's adjacency row is loaded as soon as the next pop is known;
//  * batches that fit the GPU a block per query get one (Team).
//
// Template parameters: METRIC (0 L2, 1 IP, 2 COS), STORAGE (0 F32, 1 BF16,
// 2 FP8-E4M3 with a per-row scale, 3 256-bit codes), S (register queue
// segment, capacity 32*S >= pq+1), LEARNED (per-hop features: trace capture
// and/or the early-exit network), MULTI (the multi-probe knobs), LONG (rows of
// LONG_ROW bytes and more; with codes, vectors too wide for WarpLayout's usual
// order).
//
// What bounds it: instructions, in full batches and for a single query alike
// (about six cycles each on a dependent path).  A hop of the headline search
// (1M x 128 L2, pq 43 from entry points, 21 candidates) takes 1,790 of them
// (2,650 before its rows were read directly and its hash calls made side by
// side), one at pq 1000 from vertex 0 500 (5,900).
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "device_common.cuh"
#include "internal.h"
#include "reg_queue.cuh"
#include "row_read.cuh"

namespace song {

constexpr int MAX_WARPS_PER_BLOCK = 4;
constexpr int MAX_PROBES = 4;  // candidate list of the MULTI kernel: MAX_PROBES * 32 ids
constexpr int MLP_IN = 5, MLP_H = 32;
// FP32 parameters of the early-exit network, in this order.
constexpr int MLP_W1 = 0;                        // [MLP_H][MLP_IN]
constexpr int MLP_B1 = MLP_W1 + MLP_H * MLP_IN;  // [MLP_H]
constexpr int MLP_W2 = MLP_B1 + MLP_H;           // [MLP_H][MLP_H]
constexpr int MLP_B2 = MLP_W2 + MLP_H * MLP_H;   // [MLP_H]
constexpr int MLP_W3 = MLP_B2 + MLP_H;           // [MLP_H]
constexpr int MLP_B3 = MLP_W3 + MLP_H;           // [1]
constexpr int MLP_NPARAM = MLP_B3 + 1;
constexpr uint32_t MLP_BYTES = MLP_NPARAM * sizeof(__nv_bfloat16) + 64;  // a block's copy
constexpr int TRACE_FIELDS = 6;  // 5 features + top-k version

struct Params {
  const uint8_t *rows;
  uint32_t row_bytes;
  uint32_t scale_off;  // FP8: byte offset of the row's float scale
  const float *rows_f32;
  uint32_t f32_row_bytes;
  int rerank;  // final candidates re-ranked with FP32 distances (low-precision storage)
  const uint32_t *adj;
  int shift;
  int dim;
  const float *queries;
  int nq, pq, k;
  uint64_t *out;
  int32_t *hops;
  int32_t *evals;
  uint32_t *counter;
  int32_t *error;
  uint32_t warp_bytes;
  uint32_t off_mbar, off_cand, off_q, off_queue, off_hash;
  int width;       // elements of a stored row, zero padding included
  uint32_t wait_limit;  // polls of a bounded mbarrier wait
  uint32_t extra_tx;    // test hook: bytes a copy's barrier expects beyond its own (0 in use)
  // the reference's N_MULTIPROBE / FINISH_CNT knobs (MULTI kernel only)
  int probes;      // vertices popped per iteration, 1..MAX_PROBES
  int finish_cnt;  // finish tests that must hold before the search ends, >= 1
  int double_check;  // select-insert skips candidates already visited (__ENABLE_MULTIPROBE_DOUBLE_CHECK)
  // learned variant
  const __nv_bfloat16 *mlp;  // MLP_NPARAM weights (BF16), null = no early exit
  float exit_threshold;
  int exit_min_hops;
  int exit_every;
  int exit_max_hops;      // > 0: stop after this many hops (fixed-budget heuristic)
  float *trace;           // [nq][trace_hops][TRACE_FIELDS] or null
  int trace_hops;
  int32_t *trace_final;   // [nq]: final top-k version, hops traced
  const uint32_t *qcodes; // BITS storage: [nq][8] 256-bit codes of the queries
  const uint32_t *starts; // [nq][n_starts] start vertices of each query, or null: vertex 0
  int n_starts;
  // entry points chosen inside the server's persistent warps (entry_rows
  // null: vertex 0); the layout of song_index's entry fields
  const float *entry_rows;
  const uint32_t *entry_ids;
  int n_entries;
  const float *coarse_rows;
  int n_coarse;
  const uint32_t *entry_offsets;
  int n_probes;
  int entry_dpad;
};

// The 256-bit code of a query (BITS storage), in every lane.
struct Code8 {
  uint32_t w[8];
};

// 32-dimension steps of a row whose loads are in flight together: 16 (FP8) to
// 32 registers a lane, 64 for long FP32 rows.
template <int STORAGE, bool LONG>
constexpr int row_steps() {
  return STORAGE == 0 && !LONG ? 4 : 8;
}

// One pass: the distance of the row of vertex `id` (the same in a row's four
// lanes), in those lanes.  qv: the query, zero-padded to a multiple of 32
// floats.  `width` elements a row (zero-padded to the 16-byte load; a padded
// element adds fma(0, 0, t)).
template <int METRIC, int STORAGE, bool LONG>
__device__ __forceinline__ float rows_pass(const uint8_t *rows, uint32_t rb, uint32_t scale_off, int width,
                                           const float *qv, uint32_t id, int lane) {
  using Read = RowRead<STORAGE>;
  const int g = lane & 3;
  const ulonglong2 *q2 = reinterpret_cast<const ulonglong2 *>(qv) + (Read::HALVES ? g : 2 * g);
  constexpr int QB = Read::HALVES ? 4 : 1;  // the second half's offset in 16-byte units
  const uint8_t *row = rows + static_cast<uint64_t>(id) * rb;
  const float scale = STORAGE == 2 ? __ldg(reinterpret_cast<const float *>(row + scale_off)) : 1.0f;
  uint64_t acc[4], len[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) acc[i] = len[i] = 0ull;
  auto add = [&](const Read &r, int j) {
    uint64_t x[4];
    r.get(x, scale);
    const ulonglong2 qa = q2[j >> 2], qb = q2[(j >> 2) + QB];
    const uint64_t q[4] = {qa.x, qa.y, qb.x, qb.y};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (METRIC == 0) {
        const uint64_t d = f2_sub(q[i], x[i]);
        acc[i] = f2_fma(d, d, acc[i]);
      } else {
        acc[i] = f2_fma(q[i], x[i], acc[i]);
        if (METRIC == 2) len[i] = f2_fma(x[i], x[i], len[i]);
      }
    }
  };
  int j = 0;
  constexpr int U = row_steps<STORAGE, LONG>();
  for (; j + 32 * U <= width; j += 32 * U) {
    Read r[U];
#pragma unroll
    for (int i = 0; i < U; ++i) r[i].load_full(row, j + 32 * i, g);
#pragma unroll
    for (int i = 0; i < U; ++i) add(r[i], j + 32 * i);
  }
  for (; j < width; j += 32) {
    Read r;
    r.load(row, j, g, width);
    add(r, j);
  }
  const float t = row_butterfly<Read::HALVES>(acc, lane);
  const float ln = METRIC == 2 ? row_butterfly<Read::HALVES>(len, lane) : 0.0f;
  return finish_distance<METRIC>(t, ln);
}

// Distances of candidates 0..m-1 (candidate c's id in lane c) in lane c.
template <int METRIC, int STORAGE, bool LONG = false>
__device__ __forceinline__ float gather_rows(const uint8_t *rows, uint32_t rb, uint32_t scale_off, int width,
                                             const float *qv, int m, uint32_t cid, int lane) {
  float out = 0.0f;
  for (int first = 0; first < m; first += 8) {
    const uint32_t id = __shfl_sync(FULL, cid, min(first + (lane >> 2), m - 1));
    const float d = rows_pass<METRIC, STORAGE, LONG>(rows, rb, scale_off, width, qv, id, lane);
    const float mine = __shfl_sync(FULL, d, ((lane - first) & 7) * 4);
    if (lane >= first && lane < first + 8) out = mine;
  }
  return out;
}

// The index's stored rows.
template <int METRIC, int STORAGE, bool LONG>
__device__ __forceinline__ float gather_distances(const Params &p, const float *qv, int m, uint32_t cid, int lane,
                                                  const Code8 &qc) {
  if constexpr (STORAGE == 3) {
    // Hamming distance of 256-bit codes: lane c reads candidate c's 32-byte
    // code straight from global memory (two 16-byte loads) and sums the
    // popcounts of its xor with the query's code (an integer, exact as float)
    float out = 0.0f;
    if (lane < m) {
      const uint4 *r = reinterpret_cast<const uint4 *>(p.rows + static_cast<uint64_t>(cid) * 32u);
      const uint4 a = __ldg(r), b = __ldg(r + 1);
      const int h = __popc(a.x ^ qc.w[0]) + __popc(a.y ^ qc.w[1]) + __popc(a.z ^ qc.w[2]) + __popc(a.w ^ qc.w[3]) +
                    __popc(b.x ^ qc.w[4]) + __popc(b.y ^ qc.w[5]) + __popc(b.z ^ qc.w[6]) + __popc(b.w ^ qc.w[7]);
      out = static_cast<float>(h);
    }
    return out;
  } else {
    return gather_rows<METRIC, STORAGE, LONG>(p.rows, p.row_bytes, p.scale_off, p.width, qv, m, cid, lane);
  }
}

__device__ __forceinline__ float key_float(uint64_t k) {
  const uint32_t b = key_dist(k);
  return __uint_as_float((b & 0x80000000u) ? (b & 0x7fffffffu) : ~b);
}

// Early-exit network, warp-parallel: lane j owns hidden unit j of both layers.
// BF16 weights in shared memory, FP32 arithmetic.  Returns the logit.
__device__ __forceinline__ float mlp_logit(const __nv_bfloat16 *w, const float f[MLP_IN], int lane) {
  float h1 = __bfloat162float(w[MLP_B1 + lane]);
#pragma unroll
  for (int i = 0; i < MLP_IN; ++i) h1 = __fmaf_rn(__bfloat162float(w[MLP_W1 + lane * MLP_IN + i]), f[i], h1);
  h1 = fmaxf(h1, 0.0f);
  float h2 = __bfloat162float(w[MLP_B2 + lane]);
#pragma unroll
  for (int i = 0; i < MLP_H; ++i)
    h2 = __fmaf_rn(__bfloat162float(w[MLP_W2 + lane * MLP_H + i]), __shfl_sync(FULL, h1, i), h2);
  h2 = fmaxf(h2, 0.0f);
  float z = __fmul_rn(__bfloat162float(w[MLP_W3 + lane]), h2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) z = __fadd_rn(z, __shfl_xor_sync(FULL, z, o));
  return __fadd_rn(z, __bfloat162float(w[MLP_B3]));
}

// The plain kernel keeps the reference's FixHash (bit parity); the learned
// kernel, which makes no parity claim, uses the smaller exact set.  Both are
// sized per query from its pq.
template <bool LEARNED>
struct VisitedOf {
  using type = VisitedHash;
  __device__ static VisitedHash make(int32_t *tab, int pq) {
    const int cap = 8 * pq;
    return VisitedHash{tab, cap, ~0ull / static_cast<uint64_t>(cap)};
  }
};
template <>
struct VisitedOf<true> {
  using type = ExactVisited;
  __device__ static ExactVisited make(int32_t *tab, int pq) {
    int lg = 5;
    while ((1 << lg) < 4 * pq) ++lg;
    return ExactVisited{tab, 1 << lg, lg};
  }
};

// From this register-queue segment on (pq >= 16*S), the candidate queue is a
// BufQueue.  10,000 queries of 1M x 128: pq 150 (S 8) 4.30 ms with a BufQueue,
// 3.80 with a RegQueue; pq 1000 (S 32) 37.4 ms with a BufQueue, 60 with a
// RegQueue.
constexpr int BUF_S = 16;

template <int S>
struct QueueOf {
  using type = typename std::conditional<(S >= BUF_S), BufQueue, RegQueue<S>>::type;
};

// Shared memory of one warp, in this order: the first adjacency row (bulk
// copy), its barrier, the candidate ids and home slots, the query, the
// queue's ring, and the visited hash, which the answer's sort reuses (8 bytes
// for each of 32*S keys).  Codes leave the FP32 query for the re-rank only:
// where it does not fit beside the rest (50,000 floats and the ring of pq
// 1000), it is staged once the search is done, over all but the barrier, after
// the sort's keys (`late`: the LONG kernels of codes).  Not at every size: the
// pointers it needs to the end cost spills (5000 queries of 15k x 16 at pq 100
// 1440 -> 1500 us).
constexpr uint32_t MAX_BLOCK_BYTES = 227u * 1024u;
constexpr uint32_t LATE_ROW = 16;  // late: the row's place, after the barrier
struct WarpLayout {
  uint32_t warp_bytes, off_mbar, off_cand, off_q, off_queue, off_hash;
  bool late;
};
inline WarpLayout warp_layout(int dim, int pq, int S, int cap, int cands, bool codes) {
  auto up = [](uint32_t x, uint32_t a) { return (x + a - 1) / a * a; };
  const uint32_t query = 4u * up(static_cast<uint32_t>(dim), 32), ring = S >= BUF_S ? BufQueue::bytes(pq) : 0u;
  const uint32_t hash = 4u * static_cast<uint32_t>(cap), sort = 256u * static_cast<uint32_t>(S);
  WarpLayout L;
  L.off_mbar = 128;
  L.off_cand = L.off_mbar + 16;
  L.off_q = L.off_cand + 8u * static_cast<uint32_t>(cands);
  L.off_queue = up(L.off_q + query, 16);
  L.off_hash = up(L.off_queue + ring, 16);
  L.warp_bytes = up(L.off_hash + std::max(hash, sort), 128);
  L.late = codes && L.warp_bytes > MAX_BLOCK_BYTES;
  if (L.late) {
    L.off_mbar = 0;
    L.off_queue = up(L.off_q, 16);
    L.off_hash = up(L.off_queue + ring, 16);
    L.off_q = LATE_ROW + sort;
    L.warp_bytes = up(std::max(L.off_hash + hash, L.off_q + query), 128);
  }
  return L;
}

// The warp's shared-memory slice and barrier phase.
struct WarpCtx {
  uint32_t *row;    // first adjacency row
  uint64_t *mbar;
  uint32_t *cbuf;   // candidate ids
  int32_t *chome;   // and their home slots
  float *qv;
  uint64_t *ring;
  int32_t *tab;
  const __nv_bfloat16 *wmlp;
  uint32_t ph;

  __device__ __forceinline__ void init(uint8_t *ws, const Params &p, int cands, int lane, uint32_t row_at = 0) {
    row = reinterpret_cast<uint32_t *>(ws + row_at);
    mbar = reinterpret_cast<uint64_t *>(ws + p.off_mbar);
    cbuf = reinterpret_cast<uint32_t *>(ws + p.off_cand);
    chome = reinterpret_cast<int32_t *>(cbuf + cands);
    qv = reinterpret_cast<float *>(ws + p.off_q);
    ring = reinterpret_cast<uint64_t *>(ws + p.off_queue);
    tab = reinterpret_cast<int32_t *>(ws + p.off_hash);
    if (lane == 0) {
      mbar_init(mbar, 1);
      fence_mbar_init();
    }
    __syncwarp();
    ph = 0;
  }
};

// Small batches leave most of the GPU idle, and a query's time is the latency
// of one warp's hops.  There a query gets a block of TEAM_WARPS warps: warp 0
// runs the search, the others wait for its commands at a named barrier --
// take your eight of a hop's candidates (the passes of one gather then run
// side by side), or fetch into L2 the rows that the next vertex's neighbours
// name (they arrive while warp 0 takes in this hop's candidates).  Search
// alone, 1M x 128 from entry points: one query at pq 100 375 -> 307 us, 300 at
// pq 43 257 -> 174; 300 of 60k x 960 at pq 75 652 -> 338; 15k x 16, whose rows
// never leave L2, within 3 % either way.
constexpr int TEAM_WARPS = 4;
constexpr uint32_t TEAM_BYTES = 256;  // commands and distances

struct Team {
  int32_t *cmd;   // two slots of (command, argument), used in turn
  float *dist;    // distances of one gather
  int turn;
  static constexpr int STOP = 0, PREFETCH = -1;  // > 0: gather that many

  __device__ __forceinline__ void init(uint8_t *mem) {
    cmd = reinterpret_cast<int32_t *>(mem);
    dist = reinterpret_cast<float *>(mem + 128);
    turn = 0;
  }
  static __device__ __forceinline__ void barrier() {
    asm volatile("bar.sync 1, %0;" ::"n"(32 * TEAM_WARPS) : "memory");
  }
  // Warp 0: hands out a command.
  __device__ __forceinline__ void call(int c, int arg, int lane) {
    if (lane == 0) {
      cmd[2 * turn] = c;
      cmd[2 * turn + 1] = arg;
    }
    __syncwarp();
    barrier();
    turn ^= 1;
  }
  // The others: waits for a command.
  __device__ __forceinline__ int next(int *arg) {
    barrier();
    const int c = cmd[2 * turn];
    *arg = cmd[2 * turn + 1];
    turn ^= 1;
    return c;
  }
};

// Warp `wib`'s share of a gather: candidates 8 wib .. of the m listed from
// cbuf[at] on.
template <int METRIC, int STORAGE, bool LONG>
__device__ __forceinline__ void team_pass(const Params &p, const WarpCtx &w, const Team &t, int m, int at, int wib,
                                          int lane) {
  const int c = 8 * wib + (lane >> 2);
  if (8 * wib >= m) return;  // whole warp
  const float d = rows_pass<METRIC, STORAGE, LONG>(p.rows, p.row_bytes, p.scale_off, p.width, w.qv,
                                             w.cbuf[at + min(c, m - 1)], lane);
  if ((lane & 3) == 0 && c < m) t.dist[c] = d;
}

template <int METRIC, int STORAGE, bool LEARNED, bool LONG>
__device__ __forceinline__ void team_help(const Params &p, const WarpCtx &w, Team t, int wib, int lane) {
  const auto vh = VisitedOf<LEARNED>::make(w.tab, p.pq);
  for (;;) {
    int arg;
    const int c = t.next(&arg);
    if (c == Team::STOP) return;
    if (c > 0) {
      team_pass<METRIC, STORAGE, LONG>(p, w, t, c, arg, wib, lane);
      Team::barrier();
      continue;
    }
    // the visited table may be changing under this look: it only decides what
    // is worth fetching
    const uint32_t *adj = p.adj + (static_cast<uint64_t>(static_cast<uint32_t>(arg)) << p.shift);
    const uint32_t a = lane < (1 << p.shift) ? __ldg(adj + lane) : 0u;
    const int deg = static_cast<int>(__shfl_sync(FULL, a, 0));
    if (lane >= 1 && lane <= deg && !vh.test(a)) {
      const uint8_t *row = p.rows + static_cast<uint64_t>(a) * p.row_bytes;
      for (uint32_t b = 128u * (wib - 1); b < p.row_bytes; b += 128u * (TEAM_WARPS - 1))
        asm volatile("prefetch.global.L2 [%0];" ::"l"(row + b));
    }
    __syncwarp();
  }
}

struct QueryStats {
  int hops, evals, version;
};

// Select-insert (:297-322) of candidates 0..m-1 (key ck, home slot chome in
// lane c), in candidate order, in two passes.  The queue pass applies the
// select-insert rule and the insertions and notes, in lane c, the key that
// candidate c's insertion pushed out (~0: none, the queue was not full).
// Below pq live keys the queue's maximum is an infinite key, which leaves and
// is never below a candidate; at pq, the select-insert rule, then the larger
// of the key and the maximum leaves (:315-320).  The maximum only falls, so
// after each insertion the candidates beyond it are dropped.  The hash pass
// then makes the reference's visited-hash calls -- add(candidate),
// delete(pushed-out key) per inserted candidate.  (Queue and hash are
// independent, so splitting the passes changes neither.)
template <FullTable FULL_TABLE, class Queue, class VH>
__device__ __forceinline__ void select_insert(Queue &Q, VH &vh, int m, uint64_t ck, int chome, int pq, int &qn,
                                              int lane) {
  uint64_t my_ev = ~0ull;
  unsigned ins = 0u;
  uint64_t qmax = Q.max();
  unsigned live = __ballot_sync(FULL, lane < m && key_dist(ck) <= key_dist(qmax));
  while (live) {
    const int c = __ffs(live) - 1;
    const uint64_t key = __shfl_sync(FULL, ck, c);
    const uint64_t ev = key < qmax ? qmax : key;
    Q.insert_evict(key, lane);
    ins |= 1u << c;
    if (lane == c) my_ev = ev;
    if (qn < pq) ++qn;
    qmax = Q.max();
    live &= (live - 1u) & __ballot_sync(FULL, key_dist(ck) <= key_dist(qmax));
  }
  if (ins) {
    const bool del = my_ev != ~0ull;
    const int ehome = del ? vh.slot(key_id(my_ev)) : 0;
    visited_update<VH, FULL_TABLE>(vh, (ins >> lane & 1u) != 0u, key_id(ck), chome, del, key_id(my_ev), ehome, lane);
  }
}

// One query: the search of warp_astar_accelerator.h:111-335 with the query
// vector at qsrc, queue bound pq, k ids written ascending to o.  `trace`
// (LEARNED) receives the per-hop features or is null.  False if a bulk copy
// never completed.  MULTI: the reference's N_MULTIPROBE / FINISH_CNT knobs
// (p.probes, p.finish_cnt) as run-time values.
template <int METRIC, int STORAGE, int S, bool LEARNED, bool MULTI = false, bool TEAM = false, bool LONG = false>
__device__ __forceinline__ bool run_query(const Params &p, WarpCtx &w, const float *qsrc, const uint32_t *starts,
                                          int ns, int pq, int k, uint64_t *o, float *trace, QueryStats &st,
                                          int lane, const uint32_t *qcode = nullptr, Team *team = nullptr) {
  Code8 qc;
#pragma unroll
  for (int i = 0; i < 8; ++i) qc.w[i] = STORAGE == 3 ? qcode[i] : 0u;
  typename VisitedOf<LEARNED>::type vh = VisitedOf<LEARNED>::make(w.tab, pq);
  typename QueueOf<S>::type Q;
  RegQueue<S> TS;  // top-pq list of the learned kernels (they read its k-th key)
  PopList<S> T;    // and of the others
  // (see visited_update)
  constexpr FullTable FULL_TABLE = STORAGE == 3 ? FullTable::CALLED
                                   : STORAGE == 0 && !LONG ? FullTable::INLINED : FullTable::BY_DELETES;
  const int nslots = 1 << p.shift;
  auto adjacency = [&](uint32_t v) {
    return lane < nslots ? __ldg(p.adj + (static_cast<uint64_t>(v) << p.shift) + lane) : 0u;
  };
  // Start vertices: vertex 0 (the reference's), or the ns entry points the
  // pre-pass chose (lane i holds start i).  The first start's adjacency row
  // is copied while the hash is cleared and the starts are scored.
  if (!starts) ns = 1;
  const uint32_t sid = (starts && lane < ns) ? starts[lane] : 0u;
  uint32_t next_id = __shfl_sync(FULL, sid, 0);
  const bool bulk = p.shift >= 2;  // rows of 16 bytes and more
  if (bulk) {
    fence_proxy_async();  // the buffer was last read through the generic proxy
    __syncwarp();
    if (lane == 0) {
      mbar_arrive_expect_tx(w.mbar, (4u << p.shift) + p.extra_tx);
      bulk_g2s(w.row, p.adj + (static_cast<uint64_t>(next_id) << p.shift), 4u << p.shift, w.mbar);
    }
  }
  auto stage_query = [&] {
    for (int j = lane; j < ((p.dim + 31) & ~31); j += 32) w.qv[j] = j < p.dim ? qsrc[j] : 0.0f;
  };
  constexpr bool late = STORAGE == 3 && LONG;
  if (!late) stage_query();
  vh.clear(lane);

  // warp_astar_accelerator.h:115-176: distances to the starts, queue = {starts}.
  float cd = gather_distances<METRIC, STORAGE, LONG>(p, w.qv, ns, sid, lane, qc);
  const float d0 = __shfl_sync(FULL, cd, 0);
  uint32_t a_next;
  if (bulk) {
    if (!mbar_wait_warp(w.mbar, w.ph, p.wait_limit)) return false;
    w.ph ^= 1u;
    a_next = lane < nslots ? w.row[lane] : 0u;
  } else {
    a_next = adjacency(next_id);
  }
  int qn = 0, tn = 0;
  Q.init(w.ring, pq, lane);
  if constexpr (LEARNED) TS.init(nullptr, pq, lane);
  else T.init();
  for (int i = 0; i < ns; ++i) {  // in start order, as the oracle queues them
    const uint32_t id = __shfl_sync(FULL, sid, i);
    Q.insert_evict(make_key(__shfl_sync(FULL, cd, i), id), lane);
    vh.add(id, lane);
  }
  qn = ns;
  if (ns > 1) {  // the first pop is the nearest start: load its row instead
    const uint32_t mid = key_id(warp_min_u64(lane < ns ? make_key(cd, sid) : ~0ull));
    if (mid != next_id) {
      next_id = mid;
      a_next = adjacency(mid);
    }
  }
  int hops = 0, evals = ns;
  int version = 0;           // number of changes of the top-k set (LEARNED)
  int last_change = 0;       // hop of the latest change (LEARNED)
  uint64_t kth_key = ~0ull;  // k-th smallest key of the list, ~0 while tn < k (LEARNED)
  uint64_t tmax = 0ull;      // the full list's maximum

  // Moves a popped vertex to the top-pq list (:198-210): a full list drops
  // its maximum, or the vertex itself when that is above it (which only a
  // multi-probe pop can be).
  auto list_insert = [&](uint64_t now, uint32_t now_id, int now_home) {
    if constexpr (LEARNED) {
      const uint64_t top = TS.max();
      const uint64_t ev = now < top ? top : now;
      TS.insert_evict(now, lane);
      visited_refresh(vh, now_id, now_home, lane);
      if (tn < pq) ++tn;
      else vh.del(key_id(ev), lane);
      if (tn == pq) tmax = TS.max();
      return;
    }
    visited_refresh(vh, now_id, now_home, lane);
    if (tn < pq) {
      ++tn;
      T.append(now, pq, lane);
      if (tn == pq) tmax = T.max();
    } else if (now < tmax) {
      vh.del(key_id(tmax), lane);
      T.replace(tmax, now, lane);
      tmax = T.max();
    } else {
      vh.del(now_id, lane);
    }
  };

  // Distances of the m candidates listed from cbuf[at] on (cid in lane c),
  // the block's other warps helping when there is one (Team).
  auto gather = [&](int m, uint32_t cid, int at) {
    if constexpr (TEAM) {
      if (m > 8) {
        team->call(m, at, lane);
        team_pass<METRIC, STORAGE, LONG>(p, w, *team, m, at, 0, lane);
        Team::barrier();
        return lane < m ? team->dist[lane] : 0.0f;
      }
    }
    // What the first pass does not load at once starts its way into L2: the
    // rows past it (512-byte rows: 1M x 128, 10,000 queries at pq 43 1193 ->
    // 1161 us, at pq 100 from vertex 0 4.61 -> 4.41 ms; no gain on shorter
    // ones, and the learned and multi-probe kernels lose registers to it: 959
    // -> 1025 us), and of long rows, in every kernel, also the first eight's ends
    // (1000 queries of 960-d rows with the exit network 2853 -> 2421 us).
    if constexpr (!TEAM && STORAGE <= 1 && (LONG || (!LEARNED && !MULTI))) {
      constexpr uint32_t first = 32u * row_steps<STORAGE, LONG>() * (STORAGE == 0 ? 4u : 2u);
      if (lane < m && (LONG || (lane >= 8 && p.row_bytes >= 512))) {
        const uint8_t *row = p.rows + static_cast<uint64_t>(cid) * p.row_bytes;
        for (uint32_t b = LONG && lane < 8 ? first : 0u; b < p.row_bytes; b += 128)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(row + b));
      }
      __syncwarp();
    }
    return gather_distances<METRIC, STORAGE, LONG>(p, w.qv, m, cid, lane, qc);
  };

  int finished = 0;  // MULTI: finish tests that held (finished[cid], :190-192)
  while (qn > 0) {
    if constexpr (MULTI) {
      // :182-228 up to p.probes pops per iteration.  Only the first takes the
      // finish test, which counts; the search ends when p.finish_cnt tests
      // held.  Every pop goes to the top-pq list, and the unvisited
      // neighbours of all of them are listed, in pop and row order (a vertex
      // adjacent to two pops may be listed twice, as in the reference),
      // before any distance is computed.
      int m = 0;
      bool fin = false;
      const int avail = qn;
      for (int kp = 0; kp < p.probes && kp < avail; ++kp) {
        uint64_t qh;
        const uint64_t now = Q.pop(lane, &qh);
        --qn;
        const uint32_t now_id = key_id(now);
        const uint32_t a = (kp == 0 && now_id == next_id) ? a_next : adjacency(now_id);
        const int now_home = vh.slot(now_id);
        if (kp == 0 && tn == pq && key_dist(tmax) <= key_dist(now) && ++finished >= p.finish_cnt) {
          fin = true;
          break;
        }
        ++hops;
        list_insert(now, now_id, now_home);
        const int deg = static_cast<int>(__shfl_sync(FULL, a, 0));
        const int ahome = vh.slot(a);
        const bool fresh = lane >= 1 && lane <= deg && !vh.test_at(a, ahome);
        const unsigned fm = __ballot_sync(FULL, fresh);
        if (fresh) {
          const int at = m + __popc(fm & lanemask_lt());
          w.cbuf[at] = a;
          w.chome[at] = ahome;
        }
        m += __popc(fm);
      }
      if (fin) break;
      __syncwarp();
      // :237-322 distances and select-insert, 32 candidates at a time, in
      // list order (the distances do not depend on the queue, so this is the
      // reference's all-distances-then-all-inserts order).
      for (int r0 = 0; r0 < m; r0 += 32) {
        const int mr = min(32, m - r0);
        const uint32_t cid = lane < mr ? w.cbuf[r0 + lane] : 0u;
        const int chome = lane < mr ? w.chome[r0 + lane] : 0;
        cd = gather(mr, cid, r0);
        evals += mr;
        const uint64_t ck = lane < mr ? make_key(cd, cid) : ~0ull;
        if (p.double_check) {
          // :297-322 with :307-310: a candidate already in the visited hash
          // (listed by an earlier pop of this iteration, or twice in one row)
          // is skipped, so the hash calls interleave with the insertions.
          for (int c = 0; c < mr; ++c) {
            const uint64_t key = __shfl_sync(FULL, ck, c);
            const uint64_t qmax = Q.max();
            if (key_dist(qmax) < key_dist(key)) continue;
            const uint32_t id = key_id(key);
            const int home = __shfl_sync(FULL, chome, c);
            if (vh.test_at(id, home)) continue;
            const uint64_t ev = key < qmax ? qmax : key;
            Q.insert_evict(key, lane);
            if (qn < pq) ++qn;
            vh.add_at(id, home, lane);
            if (ev != ~0ull) vh.del(key_id(ev), lane);
          }
          __syncwarp();
          continue;
        }
        select_insert<FULL_TABLE>(Q, vh, mr, ck, chome, pq, qn, lane);
      }
      // the next iteration's first pop is the queue head: load its row now
      if (qn > 0) {
        next_id = key_id(Q.min());
        a_next = adjacency(next_id);
        if constexpr (TEAM) team->call(Team::PREFETCH, static_cast<int>(next_id), lane);
      }
      continue;
    }
    // :186-193 pop the minimum, drop it from the visited hash.
    uint64_t qh;  // queue minimum after the pop
    const uint64_t now = Q.pop(lane, &qh);
    --qn;
    const uint32_t now_id = key_id(now);
    uint32_t a = a_next;
    if (now_id != next_id) a = adjacency(now_id);  // not taken: the prefetch predicts the pop exactly
    // :191 finish test (<=) against the list maximum.
    if (tn == pq && key_dist(tmax) <= key_dist(now)) break;
    ++hops;
    // LEARNED: does `now` enter the current top-k?  (Only such an entry
    // changes the k-th key: the list drops its maximum, never a top-k key.)
    const bool enters = LEARNED && now < kth_key;
    if (enters) {
      ++version;
      last_change = hops;
    }
    list_insert(now, now_id, vh.slot(now_id));
    if constexpr (LEARNED) {
      if (enters && tn >= k) kth_key = TS.at(TS.start + k - 1);
    }
    // :211-224 neighbours not in the visited hash, in row order.
    const int deg = static_cast<int>(__shfl_sync(FULL, a, 0));
    const int ahome = vh.slot(a);
    const bool fresh = lane >= 1 && lane <= deg && !vh.test_at(a, ahome);
    const unsigned fm = __ballot_sync(FULL, fresh);
    const int m = __popc(fm);
    if (fresh) {
      const int at = __popc(fm & lanemask_lt());
      w.cbuf[at] = a;
      w.chome[at] = ahome;
    }
    __syncwarp();
    const uint32_t cid = lane < m ? w.cbuf[lane] : 0u;
    const int chome = lane < m ? w.chome[lane] : 0;
    // :237-287 distances.
    cd = gather(m, cid, 0);
    evals += m;
    // The next vertex popped is the smaller of the queue head and the best
    // candidate (the select-insert rule can only reject candidates above a
    // full queue's maximum); start loading its adjacency row now so that it
    // arrives while the candidates are inserted.
    const uint64_t ck = lane < m ? make_key(cd, cid) : ~0ull;
    const uint64_t cmin = warp_min_u64(ck);
    const uint64_t nk = cmin < qh ? cmin : qh;
    if (nk != ~0ull) {
      next_id = key_id(nk);
      a_next = adjacency(next_id);
      if constexpr (TEAM) team->call(Team::PREFETCH, static_cast<int>(next_id), lane);
    }
    select_insert<FULL_TABLE>(Q, vh, m, ck, chome, pq, qn, lane);
    if constexpr (LEARNED) {
      const bool check = p.mlp && hops >= p.exit_min_hops && (hops % p.exit_every) == 0 && tn >= k;
      if (trace || check) {
      // Per-hop state: hop count, k-th and best distance, queue-head gap,
      // hops since the top-k last changed, distance evaluations.  Distances
      // enter through scale-free, bounded quantities: the top-k spread and
      // the queue-head gap relative to the progress span d0 - best (signed
      // logs).
      const float kth = key_float(tn >= k ? kth_key : TS.at(TS.start + tn - 1));
      const float best = key_float(TS.min());
      const float head = nk != ~0ull ? key_float(nk) : kth;
      const float span = fabsf(d0 - best) + 1e-6f * (fabsf(d0) + fabsf(best)) + 1e-30f;
      const float r1 = (kth - best) / span;
      const float r3 = (head - kth) / span;
      float f[MLP_IN];
      f[0] = __log2f(1.0f + static_cast<float>(hops)) * 0.1f;
      f[1] = copysignf(log1pf(fabsf(r1)), r1);
      f[2] = __log2f(1.0f + static_cast<float>(hops - last_change)) * 0.1f;
      f[3] = copysignf(log1pf(fabsf(r3)), r3);
      f[4] = __log2f(1.0f + static_cast<float>(evals)) * 0.1f;
      if (trace && hops <= p.trace_hops && lane < TRACE_FIELDS) {
        float v = lane < MLP_IN ? f[0] : static_cast<float>(version);
#pragma unroll
        for (int i = 1; i < MLP_IN; ++i) v = lane == i ? f[i] : v;
        trace[static_cast<size_t>(hops - 1) * TRACE_FIELDS + lane] = v;
      }
      if (check && mlp_logit(w.wmlp, f, lane) >= p.exit_threshold) break;  // converged
      }
      if (p.exit_max_hops > 0 && hops >= p.exit_max_hops) break;
    }
  }

  // :331-335 the list's first k ids, ascending; slots past its length get
  // UINT64_MAX.  The keys are sorted where the visited hash was (late: from
  // the adjacency row on).
  uint64_t *keys = late ? reinterpret_cast<uint64_t *>(w.row) : reinterpret_cast<uint64_t *>(w.tab);
  int live = tn;  // keys that can be returned
  __syncwarp();
  if constexpr (LEARNED) {
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const int r = lane * S + j - TS.start;
      if (r >= 0) keys[r] = r < tn ? TS.v[j] : ~0ull;
    }
    for (int i = pq + lane; i < 32 * S; i += 32) keys[i] = ~0ull;
  } else {
    T.dump(keys, pq, lane);
  }
  __syncwarp();
  if (STORAGE != 0 && p.rerank > 0) {
    // FP32 re-rank of the best `rerank` entries of the list, then the first k.
    const int R = min(max(p.rerank, k), tn);
    if (late) {
      stage_query();
      __syncwarp();
    }
    if (!LEARNED && R < tn) warp_sort_shared(keys, 32 * S, lane);
    for (int base = 0; base < R; base += 32) {
      const int cnt = min(32, R - base);
      const uint32_t id = lane < cnt ? key_id(keys[base + lane]) : 0u;
      const float d = gather_rows<METRIC, 0>(reinterpret_cast<const uint8_t *>(p.rows_f32), p.f32_row_bytes, 0u,
                                             static_cast<int>(p.f32_row_bytes >> 2), w.qv, cnt, id, lane);
      if (lane < cnt) keys[base + lane] = make_key(d, id);
    }
    for (int i = R + lane; i < 32 * S; i += 32) keys[i] = ~0ull;
    live = R;
    __syncwarp();
  }
  if (k <= 32) {
    const uint64_t key = warp_smallest32(keys, 32 * S, lane);
    if (lane < k) o[lane] = lane < live ? static_cast<uint64_t>(key_id(key)) : ~0ull;
  } else {
    warp_sort_shared(keys, 32 * S, lane);
    for (int i = lane; i < k; i += 32) o[i] = i < live ? static_cast<uint64_t>(key_id(keys[i])) : ~0ull;
  }
  __syncwarp();
  st.hops = hops;
  st.evals = evals;
  st.version = version;
  return true;
}

// Resident blocks of four warps asked for.  Short rows: 5 while the queues are
// small (S <= 4: 96 registers; 6 blocks, at 80, cost 25 % of a small batch's
// time, 1000 queries of 1M x 128 from entry points at pq 43 287 -> 362 us, for
// 1 % of a full one's), 4 for the wider register queue of S = 8 and the lists
// of S = 16, 2 beyond, where shared memory holds few warps anyway (five at pq
// 1000 and 128 dimensions: hash and ring, 41,216 bytes each).  The multi-probe
// kernels, whose double check is one long chain, take 6 (10,000
// queries of 1M x 128, two probes: 1489 us with 5, 1414 with 6), the learned
// ones on BF16 rows 4 (their decoding spills at 96 registers: 1765 us with 5,
// 1511 with 4).  LONG rows (1 KB and more): 3, for the 64 registers that a
// pass's loads take: 10,000 queries of 256-d rows from vertex 0 at pq 75 3.13
// ms with 5 blocks and half the loads in flight, 2.53 with 4, 2.78 with 3; 1000
// of 960-d rows 2.51, 2.33 and 1.70; 10,000 of 128-d rows at pq 43 1.16 with 5
// blocks, 1.50 with 3.  Their multi-probe and learned kernels on FP32 rows take
// 4 while pq < 32, where loading is less of a hop (10,000 of 256-d rows at pq 30,
// four probes: 3.22 ms with 3, 2.79 with 4; at pq 55 3.82 and 3.97; 4000 of 960-d
// L2 rows at pq 30, four probes 1.14 and 1.03, exit network 0.67 and 0.69).  A
// batch that fits the GPU either way has only the loads in flight to gain and
// would rather have 3: 1000 of 960-d cosine rows, exit network 1.21 and 1.51 ms.
constexpr uint32_t LONG_ROW = 1024;

template <int STORAGE, int S, bool LEARNED, bool MULTI, bool LONG>
struct MinBlocks {
  static constexpr int value = S > 16 ? 2
                               : LONG ? (S == 1 && STORAGE == 0 && (MULTI || LEARNED) ? 4 : 3)
                               : S > 4 ? 4
                               : MULTI ? 6
                               : LEARNED && STORAGE == 1 ? 4 : 5;
};

// Query qid of the launch; false if a bulk copy never completed.
template <int METRIC, int STORAGE, int S, bool LEARNED, bool MULTI, bool TEAM, bool LONG>
__device__ __forceinline__ bool search_one(const Params &p, WarpCtx &w, uint32_t qid, int lane, Team *team) {
  float *trace = nullptr;
  if (LEARNED && p.trace) trace = p.trace + static_cast<size_t>(qid) * p.trace_hops * TRACE_FIELDS;
  QueryStats st;
  if (!run_query<METRIC, STORAGE, S, LEARNED, MULTI, TEAM, LONG>(
          p, w, p.queries + static_cast<size_t>(qid) * p.dim,
          p.starts ? p.starts + static_cast<size_t>(qid) * p.n_starts : nullptr, p.n_starts, p.pq, p.k,
          p.out + static_cast<size_t>(qid) * p.k, trace, st, lane,
          STORAGE == 3 ? p.qcodes + static_cast<size_t>(qid) * 8 : nullptr, team)) {
    if (lane == 0) atomicOr(p.error, 1);
    return false;
  }
  if (lane == 0) {
    if (p.hops) p.hops[qid] = st.hops;
    if (p.evals) p.evals[qid] = st.evals;
    if (LEARNED && p.trace_final) {
      p.trace_final[2 * qid] = st.version;
      p.trace_final[2 * qid + 1] = min(st.hops, p.trace_hops);
    }
  }
  __syncwarp();
  return true;
}

// The early-exit network's weights into the block's shared memory.
__device__ __forceinline__ void load_mlp(const Params &p, __nv_bfloat16 *wmlp) {
  if (p.mlp)
    for (int i = threadIdx.x; i < MLP_NPARAM; i += blockDim.x) wmlp[i] = p.mlp[i];
  __syncthreads();
}

template <int METRIC, int STORAGE, int S, bool LEARNED, bool MULTI, bool LONG>
__global__ void __launch_bounds__(MAX_WARPS_PER_BLOCK * 32, MinBlocks<STORAGE, S, LEARNED, MULTI, LONG>::value)
    search_kernel(const Params p) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  WarpCtx w;
  w.init(smem_raw + static_cast<size_t>(wib) * p.warp_bytes, p, (MULTI ? MAX_PROBES : 1) * 32, lane,
         STORAGE == 3 && LONG ? LATE_ROW : 0u);
  __nv_bfloat16 *wmlp = reinterpret_cast<__nv_bfloat16 *>(smem_raw + static_cast<size_t>(nwarps) * p.warp_bytes);
  w.wmlp = wmlp;
  if (LEARNED) load_mlp(p, wmlp);

  for (;;) {
    uint32_t qid = 0;
    if (lane == 0) qid = atomicAdd(p.counter, 1u);
    qid = __shfl_sync(FULL, qid, 0);
    if (qid >= static_cast<uint32_t>(p.nq)) break;
    if (!search_one<METRIC, STORAGE, S, LEARNED, MULTI, false, LONG>(p, w, qid, lane, nullptr)) return;
  }
}

// The search with a block per query (Team).
template <int METRIC, int STORAGE, int S, bool LEARNED, bool MULTI, bool LONG>
__global__ void __launch_bounds__(TEAM_WARPS * 32, S > 16 ? 2 : 4) search_team_kernel(const Params p) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  WarpCtx w;
  w.init(smem_raw, p, (MULTI ? MAX_PROBES : 1) * 32, wib == 0 ? lane : 1);  // lane 0 of warp 0 sets the barrier up
  Team team;
  team.init(smem_raw + p.warp_bytes);
  __nv_bfloat16 *wmlp = reinterpret_cast<__nv_bfloat16 *>(smem_raw + p.warp_bytes + TEAM_BYTES);
  w.wmlp = wmlp;
  if (LEARNED) load_mlp(p, wmlp);
  if (wib > 0) {
    team_help<METRIC, STORAGE, LEARNED, LONG>(p, w, team, wib, lane);
    return;
  }
  for (uint32_t qid = blockIdx.x; qid < static_cast<uint32_t>(p.nq); qid += gridDim.x)
    if (!search_one<METRIC, STORAGE, S, LEARNED, MULTI, true, LONG>(p, w, qid, lane, &team)) break;
  team.call(Team::STOP, 0, lane);
}

// ---------------------------------------------------------------------------
// Host-side launch helpers shared by the per-storage translation units.
// ---------------------------------------------------------------------------

// Launch shape per (kernel, bytes per block): warps per block in {4, 2, 1}
// that keeps the most warps resident per SM (search.cu).
int get_shape(const void *fn, uint32_t warp_bytes, uint32_t extra_bytes, int *wpb, int *grid_cap);
// The same for blocks of a fixed size and footprint: how many fit on the GPU.
int get_team_shape(const void *fn, uint32_t bytes, int *grid_cap);

template <int METRIC, int STORAGE, int S, bool LEARNED, bool MULTI, bool LONG>
int launch_kernel(const Params &p, cudaStream_t stream) {
  const uint32_t extra = LEARNED ? MLP_BYTES : 0u;
  if constexpr (STORAGE != 3) {
    // a block per query while all of them run at once
    auto team = search_team_kernel<METRIC, STORAGE, S, LEARNED, MULTI, LONG>;
    const uint32_t bytes = p.warp_bytes + TEAM_BYTES + extra;
    int cap = 0;
    int e = get_team_shape(reinterpret_cast<const void *>(team), bytes, &cap);
    if (e == 0 && p.nq <= cap) {
      team<<<p.nq, TEAM_WARPS * 32, bytes, stream>>>(p);
      return cudaGetLastError();
    }
  }
  auto kern = search_kernel<METRIC, STORAGE, S, LEARNED, MULTI, LONG>;
  int wpb = 0, cap = 0;
  int e = get_shape(reinterpret_cast<const void *>(kern), p.warp_bytes, extra, &wpb, &cap);
  if (e != 0) return e;
  const int want = (p.nq + wpb - 1) / wpb;
  const int grid = want < cap ? (want > 0 ? want : 1) : cap;
  cudaError_t ce = cudaMemsetAsync(p.counter, 0, sizeof(uint32_t), stream);
  if (ce != cudaSuccess) return ce;
  kern<<<grid, wpb * 32, static_cast<size_t>(p.warp_bytes) * wpb + extra, stream>>>(p);
  return cudaGetLastError();
}

template <int STORAGE, int METRIC, bool LEARNED, bool MULTI, bool LONG>
int launch_by_s(const Params &p, int S, cudaStream_t s) {
  switch (S) {
    case 1: return launch_kernel<METRIC, STORAGE, 1, LEARNED, MULTI, LONG>(p, s);
    case 2: return launch_kernel<METRIC, STORAGE, 2, LEARNED, MULTI, LONG>(p, s);
    case 4: return launch_kernel<METRIC, STORAGE, 4, LEARNED, MULTI, LONG>(p, s);
    case 8: return launch_kernel<METRIC, STORAGE, 8, LEARNED, MULTI, LONG>(p, s);
    case 16: return launch_kernel<METRIC, STORAGE, 16, LEARNED, MULTI, LONG>(p, s);
    case 32: return launch_kernel<METRIC, STORAGE, 32, LEARNED, MULTI, LONG>(p, s);
    default: return -1;
  }
}

template <int STORAGE, bool LEARNED, bool MULTI = false, bool LONG = false>
int launch_storage(const Params &p, int metric, int S, cudaStream_t s) {
  switch (metric) {
    case 0: return launch_by_s<STORAGE, 0, LEARNED, MULTI, LONG>(p, S, s);
    case 1: return launch_by_s<STORAGE, 1, LEARNED, MULTI, LONG>(p, S, s);
    case 2: return launch_by_s<STORAGE, 2, LEARNED, MULTI, LONG>(p, S, s);
    default: return -1;
  }
}

// One per translation unit (search_f32.cu, search_bf16.cu, search_fp8.cu,
// search_bits.cu, search_learned.cu, search_multi.cu, and search_*_long.cu for
// rows of LONG_ROW bytes and more, search_bits_wide.cu for WarpLayout's late
// query).
int launch_f32(const Params &p, int metric, int S, cudaStream_t s);
int launch_bf16(const Params &p, int metric, int S, cudaStream_t s);
int launch_fp8(const Params &p, int metric, int S, cudaStream_t s);
int launch_bits(const Params &p, int metric, int S, cudaStream_t s);
int launch_bits_wide(const Params &p, int metric, int S, cudaStream_t s);
int launch_learned(const Params &p, int storage, int metric, int S, cudaStream_t s);
int launch_multi(const Params &p, int metric, int S, cudaStream_t s);
int launch_f32_long(const Params &p, int metric, int S, cudaStream_t s);
int launch_bf16_long(const Params &p, int metric, int S, cudaStream_t s);
int launch_learned_long(const Params &p, int storage, int metric, int S, cudaStream_t s);
int launch_multi_long(const Params &p, int metric, int S, cudaStream_t s);

}  // namespace song
