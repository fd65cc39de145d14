// graph_build_gpu.cu -- the graph builder with each batch's searches on the GPU.
//
// The builder (graph_build.cpp) inserts vertices in batches; every new vertex
// runs the reference's CPU best-first search (graph.h:169-216) with result
// size `budget` against the graph as it stood before its batch.  This file
// runs those searches on the GPU (a warp, or a block of four, per new vertex)
// and leaves the edge bookkeeping (graph.h:116-167) to graph_build.cpp.  The GPU search is the CPU
// search restated exactly, so the GPU builder writes the same graph as the CPU
// builder with the same batch_div, bit for bit:
//
//  * distances as data.h:28-62 computes them: float differences / products
//    (no contraction), accumulated in double in dimension order; cosine
//    divides by the two squared norms, each a float sum in dimension order;
//  * the queue is unbounded and ordered by (distance, id) like
//    std::pair<double, size_t>, the result list keeps the `budget` smallest
//    popped vertices by the same order, the search stops when the list is full
//    and its largest distance is below the next queue distance, and a vertex
//    enters the visited set when it is queued and never leaves it.
//
// A candidate farther than the maximum of a full result list is marked
// visited but not queued: the list's maximum only falls, so such a candidate
// could only ever be popped to end the search, which the next larger queue
// entry (or an empty queue) does just the same.
//
// Two kernels do it.  beam_search_kernel (budgets up to BEAM_BUDGET) keeps
// queue and result list as one sorted list and sums the distances of a row
// over the whole warp, in integers where that is exact (below).  What it cannot
// finish (more equal distances at the list's end than its list holds, NaN
// distances) and larger budgets take build_search_kernel, which follows the CPU
// search step by step: one lane per candidate, lane 0 keeping the two heaps, the
// visited set and the queue heap in a device scratch region whose size is
// checked.  A search that must be repeated, or would overflow its region, says
// so in place of its result, and the host repeats these searches alone.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "graph_build.h"
#include "internal.h"
#include "song_gb300.h"

namespace song {
namespace {

constexpr unsigned FULLM = 0xffffffffu;
constexpr uint32_t VIS_EMPTY = 0xffffffffu;
constexpr int BUILD_WARPS = 4;  // warps per block

struct QE {
  double d;
  uint32_t id;
  uint32_t pad;
};

__device__ __forceinline__ bool qless(const QE &a, const QE &b) {
  return a.d < b.d || (a.d == b.d && a.id < b.id);
}

struct BuildArgs {
  const float *data;     // n x dim
  const float *norms;    // cos: per-row squared norm (float, dimension order); else null
  const uint32_t *adj;   // n << shift
  int dim, metric, shift;
  uint64_t first;        // new vertices first + t: t = todo[0 .. count - 1], or 0 .. count - 1 (todo null)
  uint32_t count;
  const uint32_t *todo;
  uint64_t limit;        // vertices inserted before the batch
  int budget;            // result size k of the search
  int out_k;             // ids written per vertex (search_degree)
  uint32_t *out;         // row t: vertex first + t's, out_k places
  int32_t *out_cnt;      // their number, or why the search must be repeated (NEED_*)
  uint32_t *vis;         // per warp: vis_cap slots
  uint32_t vis_cap;      // power of two
  int vis_log2;
  uint32_t vis_limit;    // a search that has visited more is repeated: at most 3/4 of the slots
  QE *q;                 // per warp: q_cap entries
  uint32_t q_cap;
  uint32_t *counter;
};

// Searches to be repeated, alone: with a larger visited set, with a larger
// queue, or by the step-by-step search.
constexpr int32_t NEED_VISITED = -1, NEED_QUEUE = -2, NEED_STEPS = -3;

// data.h:28-62 with a = base row, v = the query (in shared memory).
__device__ __forceinline__ double cpu_distance(const BuildArgs &p, const float *a, const float *v, float lena,
                                               float lenv) {
  double ret = 0.0;
  if (p.metric == SONG_METRIC_L2) {
    for (int i = 0; i < p.dim; ++i) {
      const float diff = __fsub_rn(__ldg(a + i), v[i]);
      ret = __dadd_rn(ret, static_cast<double>(__fmul_rn(diff, diff)));
    }
    return ret;
  }
  if (p.metric == SONG_METRIC_IP) {
    for (int i = 0; i < p.dim; ++i) ret = __dsub_rn(ret, static_cast<double>(__fmul_rn(__ldg(a + i), v[i])));
    return ret;
  }
  for (int i = 0; i < p.dim; ++i) ret = __dadd_rn(ret, static_cast<double>(__fmul_rn(__ldg(a + i), v[i])));
  const double sign = ret < 0 ? 1.0 : -1.0;
  return __dmul_rn(sign, __ddiv_rn(__ddiv_rn(__dmul_rn(ret, ret), static_cast<double>(lena)),
                                   static_cast<double>(lenv)));
}

// Insert-only visited set; true when id was not yet present.
__device__ __forceinline__ bool vis_insert(uint32_t *tab, uint32_t cap, int log2cap, uint32_t id) {
  uint32_t s = (id * 0x9E3779B1u) >> (32 - log2cap);
  for (uint32_t i = 0; i < cap; ++i) {
    const uint32_t old = atomicCAS(tab + s, VIS_EMPTY, id);
    if (old == VIS_EMPTY) return true;
    if (old == id) return false;
    s = (s + 1) & (cap - 1);
  }
  return false;  // unreachable: the fill is bounded below cap
}

// Min-heap (queue) and max-heap (result list) of QE, operated by one lane.
__device__ __forceinline__ void minheap_push(QE *h, uint32_t &n, const QE &e) {
  uint32_t i = n++;
  while (i > 0) {
    const uint32_t par = (i - 1) >> 1;
    const QE pe = h[par];
    if (!qless(e, pe)) break;
    h[i] = pe;
    i = par;
  }
  h[i] = e;
}

__device__ __forceinline__ void minheap_pop(QE *h, uint32_t &n) {
  const QE last = h[--n];
  uint32_t i = 0;
  for (;;) {
    uint32_t c = 2 * i + 1;
    if (c >= n) break;
    if (c + 1 < n && qless(h[c + 1], h[c])) ++c;
    const QE ce = h[c];
    if (!qless(ce, last)) break;
    h[i] = ce;
    i = c;
  }
  if (n > 0) h[i] = last;
}

__device__ __forceinline__ void maxheap_push(QE *h, int &n, const QE &e) {
  int i = n++;
  while (i > 0) {
    const int par = (i - 1) >> 1;
    const QE pe = h[par];
    if (!qless(pe, e)) break;
    h[i] = pe;
    i = par;
  }
  h[i] = e;
}

// Replace the maximum by e (e below it) and restore the heap.
__device__ __forceinline__ void maxheap_replace_top(QE *h, int n, const QE &e) {
  int i = 0;
  for (;;) {
    int c = 2 * i + 1;
    if (c >= n) break;
    if (c + 1 < n && qless(h[c], h[c + 1])) ++c;
    const QE ce = h[c];
    if (!qless(e, ce)) break;
    h[i] = ce;
    i = c;
  }
  h[i] = e;
}

__global__ void __launch_bounds__(BUILD_WARPS * 32) build_search_kernel(const BuildArgs p) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const size_t per_warp = static_cast<size_t>(p.budget) * sizeof(QE) + ((static_cast<size_t>(p.dim) * 4 + 15) & ~15ull);
  QE *T = reinterpret_cast<QE *>(smem + per_warp * wib);
  float *qv = reinterpret_cast<float *>(smem + per_warp * wib + static_cast<size_t>(p.budget) * sizeof(QE));
  const uint64_t gw = static_cast<uint64_t>(blockIdx.x) * BUILD_WARPS + wib;
  uint32_t *vis = p.vis + gw * p.vis_cap;
  QE *Q = p.q + gw * p.q_cap;
  const uint32_t nslots = 1u << p.shift;

  for (;;) {
    uint32_t t = 0;
    if (lane == 0) t = atomicAdd(p.counter, 1u);
    t = __shfl_sync(FULLM, t, 0);
    if (t >= p.count) break;
    if (p.todo) t = p.todo[t];
    const uint64_t v = p.first + t;
    if (p.limit == 0) {  // the first vertex: nothing to search
      if (lane == 0) p.out_cnt[t] = 0;
      continue;
    }
    for (uint32_t i = lane; i < p.vis_cap; i += 32) vis[i] = VIS_EMPTY;
    const float *vrow = p.data + v * static_cast<uint64_t>(p.dim);
    for (int i = lane; i < p.dim; i += 32) qv[i] = vrow[i];
    const float lenv = p.norms ? p.norms[v] : 0.0f;
    __syncwarp();

    uint32_t qn = 0, vis_n = 1;
    int tn = 0;
    bool overflow = false;
    if (lane == 0) {
      vis_insert(vis, p.vis_cap, p.vis_log2, 0u);
      QE e;
      e.d = cpu_distance(p, p.data, qv, p.norms ? p.norms[0] : 0.0f, lenv);
      e.id = 0;
      e.pad = 0;
      minheap_push(Q, qn, e);
    }
    qn = __shfl_sync(FULLM, qn, 0);
    // Every lane holds the same qn, tn, vis_n and overflow at every branch:
    // lane 0 changes the heaps, and each change is broadcast before any lane
    // tests them.  The iteration cap is the reference's (graph.h:186).
    for (int iter = 0; iter < 1000000 && qn > 0; ++iter) {
      // graph.h:186-195: stop, or pop the minimum into the result list.
      QE now;
      int stop = 0;
      if (lane == 0) {
        now = Q[0];
        if (tn == p.budget && T[0].d < now.d) {
          stop = 1;
        } else {
          minheap_pop(Q, qn);
          if (tn < p.budget) maxheap_push(T, tn, now);
          else if (qless(now, T[0])) maxheap_replace_top(T, tn, now);
        }
      }
      stop = __shfl_sync(FULLM, stop, 0);
      if (stop) break;
      tn = __shfl_sync(FULLM, tn, 0);
      qn = __shfl_sync(FULLM, qn, 0);
      const uint32_t now_id = __shfl_sync(FULLM, lane == 0 ? now.id : 0u, 0);
      // graph.h:196-205: unvisited neighbours, one per lane.
      const uint32_t *row = p.adj + (static_cast<uint64_t>(now_id) << p.shift);
      const uint32_t deg = __ldg(row);
      uint32_t s = 0;
      bool fresh = false;
      for (uint32_t base = 1; base <= deg; base += 32) {
        const uint32_t slot = base + lane;
        s = 0;
        fresh = false;
        if (slot <= deg && slot < nslots) {
          s = __ldg(row + slot);
          fresh = vis_insert(vis, p.vis_cap, p.vis_log2, s);
        }
        const unsigned fm = __ballot_sync(FULLM, fresh);
        vis_n += __popc(fm);
        if (vis_n > p.vis_limit) overflow = true;
        double d = 0.0;
        if (fresh) d = cpu_distance(p, p.data + static_cast<uint64_t>(s) * p.dim, qv, p.norms ? p.norms[s] : 0.0f, lenv);
        // Queue the fresh candidates (lane order; the heap order does not
        // depend on it), skipping those beyond a full list's maximum.
        const double tmax = __shfl_sync(FULLM, (lane == 0 && tn == p.budget) ? T[0].d : 0.0, 0);
        const bool full = tn == p.budget;
        unsigned qm = __ballot_sync(FULLM, fresh && !(full && tmax < d));
        if (qn + __popc(qm) > p.q_cap) {
          overflow = true;
          qm = 0;
        }
        while (qm) {
          const int src = __ffs(qm) - 1;
          qm &= qm - 1;
          const double dd = __shfl_sync(FULLM, d, src);
          const uint32_t ss = __shfl_sync(FULLM, s, src);
          if (lane == 0) {
            QE e;
            e.d = dd;
            e.id = ss;
            e.pad = 0;
            minheap_push(Q, qn, e);
          }
        }
        qn = __shfl_sync(FULLM, qn, 0);
      }
      if (overflow) break;
    }
    if (overflow) {
      if (lane == 0) p.out_cnt[t] = vis_n > p.vis_limit ? NEED_VISITED : NEED_QUEUE;
      continue;
    }
    // graph.h:207-215: the list in ascending order (in-place heap sort).
    if (lane == 0) {
      for (int i = tn - 1; i > 0; --i) {
        const QE top = T[0];
        maxheap_replace_top(T, i, T[i]);
        T[i] = top;
      }
    }
    __syncwarp();
    const int num = min(tn, p.out_k);
    for (int i = lane; i < num; i += 32) p.out[static_cast<uint64_t>(t) * p.out_k + i] = T[i].id;
    if (lane == 0) p.out_cnt[t] = tn;
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// The search with one sorted list.
//
// The list holds queued and popped vertices together, ordered by (distance,
// id), each with a flag.  The next pop is its first vertex not popped.  A
// vertex with `budget` or more listed vertices strictly below it can be
// dropped: those below it pop first, and the result list is then full with
// a maximum below it, which is the stop rule.  So the list keeps its first
// `budget` vertices and those at the distance of the last of them, the search
// ends when all of them are popped, and they are the result list.
//
// Distances.  The CPU adds the products (floats) in double, in dimension
// order.  A product is M * 2^(e - 150) with a 24-bit M; with E the largest e
// of a row's products, M << (e - E + K) is an integer when no nonzero product
// lies more than K binades below the largest, and with dim * 2^(24 + K) <=
// 2^53 every partial sum, in any order, is such an integer that a double
// holds exactly.  So the sum is the CPU's whatever the order: a warp takes a
// row's dimensions side by side and adds in 64-bit integers (the GB300 adds
// two FP64 lanes a clock per SM).  Rows that fail the test (a wide range of
// products, infinities, NaNs, denormal products) are summed in dimension
// order, one lane each.
// ---------------------------------------------------------------------------

constexpr int BEAM_CAP = 256;     // list places
constexpr int BEAM_BUDGET = 192;  // largest budget
constexpr int BEAM_VIS_LOG2 = 13; // visited slots in shared memory (a block per vertex)

struct BeamList {
  uint64_t d[BEAM_CAP];   // order-preserving bits of the distance
  uint32_t w[BEAM_CAP];   // id << 1 | popped
};

__device__ __forceinline__ uint64_t ordered(double d) {
  if (d == 0.0) d = 0.0;  // -0 and +0 compare equal
  const uint64_t u = static_cast<uint64_t>(__double_as_longlong(d));
  return (u >> 63) ? ~u : (u | (1ull << 63));
}

// A row's products summed as integers: the sum and the largest exponent, the
// same in all lanes; false when the sum is not exact.  K: see above.
__device__ __forceinline__ bool exact_sum(const float *row, const float *qv, int dim, int metric, int K, int lane,
                                          int64_t &sum, int &emax) {
  constexpr int R = 8;  // products kept in registers (rows of up to 256 floats are read once)
  uint32_t b[R];
  uint32_t top = 0u;
  auto product = [&](int j) {
    const float x = __ldg(row + j), q = qv[j];
    if (metric == SONG_METRIC_L2) {
      const float diff = __fsub_rn(x, q);
      return __float_as_uint(__fmul_rn(diff, diff));
    }
    return __float_as_uint(__fmul_rn(x, q));
  };
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int j = lane + 32 * r;
    b[r] = j < dim ? product(j) : 0u;
    top = max(top, b[r] & 0x7f800000u);
  }
  for (int j = lane + 32 * R; j < dim; j += 32) top = max(top, product(j) & 0x7f800000u);
  emax = static_cast<int>(__reduce_max_sync(FULLM, top) >> 23);
  const int base = emax - K;
  bool ok = emax != 255;
  int64_t s = 0;
  auto take = [&](uint32_t bits) {
    const int e = static_cast<int>((bits >> 23) & 255u);
    const int sh = e - base;
    const bool zero = (bits & 0x7fffffffu) == 0u;
    ok = ok && (zero || (e > 0 && sh >= 0));
    const int64_t m = zero ? 0 : static_cast<int64_t>((bits & 0x7fffffu) | 0x800000u) << max(sh, 0);
    s += (bits & 0x80000000u) ? -m : m;
  };
#pragma unroll
  for (int r = 0; r < R; ++r) take(b[r]);
  for (int j = lane + 32 * R; j < dim; j += 32) take(product(j));
  if (__any_sync(FULLM, !ok)) return false;
  // the warp's magnitudes sum to dim * 2^(24 + K) <= 2^53 at most: the sum of
  // the parts s >> 24 stays within 2^29 + 32, that of the low 24 bits below 2^29
  const int hi = __reduce_add_sync(FULLM, static_cast<int>(s >> 24));
  const int lo = __reduce_add_sync(FULLM, static_cast<int>(s & 0xffffff));
  sum = (static_cast<int64_t>(hi) << 24) + lo;
  return true;
}

// W warps a vertex: 4, with the visited set in the block's shared memory, for
// batches that fill the GPU that way at most once (what counts there is the
// latency of one search); 1, with it in the scratch region, beyond, and for a
// search that fills a block's set.
template <int W>
__global__ void __launch_bounds__(BUILD_WARPS * 32) beam_search_kernel(const BuildArgs p, const int K) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int team = W == 1 ? wib : 0, rank = W == 1 ? 0 : wib;  // this vertex's slice, this warp's place in it
  const size_t qbytes = (static_cast<size_t>(p.dim) * 4 + 15) & ~size_t(15);
  const size_t slice = sizeof(BeamList) + 32 * 8 + 32 * 4 + 16 + qbytes;
  unsigned char *mem = smem + slice * team;
  BeamList &L = *reinterpret_cast<BeamList *>(mem);
  double *cd = reinterpret_cast<double *>(mem + sizeof(BeamList));        // candidates' distances
  uint32_t *cid = reinterpret_cast<uint32_t *>(cd + 32);                  // and ids
  volatile int *ctl = reinterpret_cast<volatile int *>(cid + 32);         // candidates of the hop, -1: done
  float *qv = reinterpret_cast<float *>(mem + sizeof(BeamList) + 32 * 8 + 32 * 4 + 16);
  const uint64_t gw = static_cast<uint64_t>(blockIdx.x) * BUILD_WARPS + wib;
  uint32_t *vis = W == 1 ? p.vis + gw * p.vis_cap : reinterpret_cast<uint32_t *>(smem + slice);
  const uint32_t vis_cap = W == 1 ? p.vis_cap : 1u << BEAM_VIS_LOG2;
  const int vis_log2 = W == 1 ? p.vis_log2 : BEAM_VIS_LOG2;
  const uint32_t nslots = 1u << p.shift;
  auto sync = [&] {
    if (W == 1) __syncwarp();
    else __syncthreads();
  };

  for (;;) {
    uint32_t t = 0;
    if (rank == 0 && lane == 0) t = atomicAdd(p.counter, 1u);
    if (W == 1) {
      t = __shfl_sync(FULLM, t, 0);
    } else {
      if (threadIdx.x == 0) ctl[1] = static_cast<int>(t);
      __syncthreads();
      t = static_cast<uint32_t>(ctl[1]);
    }
    if (t >= p.count) break;
    if (p.todo) t = p.todo[t];
    const uint64_t v = p.first + t;
    if (p.limit == 0) {  // the first vertex: nothing to search
      if (rank == 0 && lane == 0) p.out_cnt[t] = 0;
      sync();
      continue;
    }
    for (uint32_t i = rank * 32 + lane; i < vis_cap; i += 32 * W) vis[i] = VIS_EMPTY;
    const float *vrow = p.data + v * static_cast<uint64_t>(p.dim);
    for (int i = rank * 32 + lane; i < p.dim; i += 32 * W) qv[i] = vrow[i];
    const float lenv = p.norms ? p.norms[v] : 0.0f;
    sync();
    if (rank == 0 && lane == 0) {
      vis_insert(vis, vis_cap, vis_log2, 0u);
      cid[0] = 0u;
      ctl[0] = 1;
    }
    sync();
    int n = 0;             // listed vertices (rank 0)
    uint32_t vis_n = 1;    // visited ones (rank 0)
    bool overflow = false; // the search must be repeated (rank 0)
    for (;;) {
      // distances of this hop's candidates, the warps taking them in turn
      const int m = ctl[0];
      if (m < 0) break;
      int64_t sum = 0;
      int emax = 0;
      bool have = false, ok = false;
      for (int c = rank; c < m; c += W) {
        int64_t s = 0;
        int e = 0;
        const bool good =
            exact_sum(p.data + static_cast<uint64_t>(cid[c]) * p.dim, qv, p.dim, p.metric, K, lane, s, e);
        if (lane == c) {
          sum = s;
          emax = e;
          ok = good;
          have = true;
        }
      }
      if (have) {
        const uint32_t id = cid[lane];
        double d;
        if (ok) {
          // 2^(emax - K - 150): the integers' unit
          const double unit = __longlong_as_double(static_cast<int64_t>(emax - K - 150 + 1023) << 52);
          d = __dmul_rn(static_cast<double>(sum), unit);
          if (p.metric == SONG_METRIC_IP) d = __dsub_rn(0.0, d);
          if (p.metric == SONG_METRIC_COS) {
            const double sign = d < 0 ? 1.0 : -1.0;
            d = __dmul_rn(sign, __ddiv_rn(__ddiv_rn(__dmul_rn(d, d), static_cast<double>(p.norms[id])),
                                          static_cast<double>(lenv)));
          }
        } else {
          d = cpu_distance(p, p.data + static_cast<uint64_t>(id) * p.dim, qv, p.norms ? p.norms[id] : 0.0f, lenv);
        }
        cd[lane] = d;
      }
      sync();
      if (rank == 0) {
        // the candidates into the list: each one's place is the number of
        // listed vertices and of candidates below it
        uint64_t key = ~0ull;
        uint32_t id = 0xffffffffu;
        bool in = lane < m;
        if (in) {
          key = ordered(cd[lane]);
          id = cid[lane];
          if (n >= p.budget && key > L.d[p.budget - 1]) in = false;
        }
        const bool bad = lane < m && isnan(cd[min(lane, 31)]);  // no order: for the step-by-step search
        if (__any_sync(FULLM, bad)) overflow = true;
        unsigned live = __ballot_sync(FULLM, in);
        const int add = __popc(live);
        if (n + add > BEAM_CAP) overflow = true;
        if (add > 0 && !overflow) {
          int lo = 0;
          if (in) {
            int hi = n;
            while (lo < hi) {
              const int mid = (lo + hi) >> 1;
              const uint64_t x = L.d[mid];
              if (x < key || (x == key && (L.w[mid] >> 1) < id)) lo = mid + 1;
              else hi = mid;
            }
          }
          uint64_t od[BEAM_CAP / 32];
          uint32_t ow[BEAM_CAP / 32];
          int up[BEAM_CAP / 32];
#pragma unroll
          for (int j = 0; j < BEAM_CAP / 32; ++j) {
            od[j] = L.d[32 * j + lane];
            ow[j] = L.w[32 * j + lane];
            up[j] = 0;
          }
          int before = 0;
          __syncwarp();
          while (live) {
            const int c = __ffs(live) - 1;
            live &= live - 1u;
            const uint64_t ok_ = __shfl_sync(FULLM, key, c);
            const uint32_t oid = __shfl_sync(FULLM, id, c);
            const int at = __shfl_sync(FULLM, lo, c);
            before += (ok_ < key || (ok_ == key && oid < id)) ? 1 : 0;
#pragma unroll
            for (int j = 0; j < BEAM_CAP / 32; ++j) up[j] += at <= 32 * j + lane ? 1 : 0;
          }
#pragma unroll
          for (int j = 0; j < BEAM_CAP / 32; ++j) {
            const int i = 32 * j + lane;
            if (i < n && up[j] > 0) {
              L.d[i + up[j]] = od[j];
              L.w[i + up[j]] = ow[j];
            }
          }
          if (in) {
            L.d[lo + before] = key;
            L.w[lo + before] = id << 1;
          }
          n += add;
          __syncwarp();
          if (n > p.budget) {  // beyond the first `budget`, only their last one's equals stay
            const uint64_t last = L.d[p.budget - 1];
            int keep = p.budget;
            for (int b = p.budget; b < n; b += 32)
              keep += __popc(__ballot_sync(FULLM, b + lane < n && L.d[min(b + lane, BEAM_CAP - 1)] <= last));
            n = keep;
          }
        }
        // the next pop: the first listed vertex not popped
        int at = -1;
        for (int b = 0; b < n && at < 0; b += 32) {
          const unsigned o = __ballot_sync(FULLM, b + lane < n && (L.w[min(b + lane, BEAM_CAP - 1)] & 1u) == 0u);
          if (o) at = b + __ffs(o) - 1;
        }
        int next = -1;
        if (at >= 0 && !overflow) {
          const uint32_t now = L.w[at] >> 1;
          __syncwarp();
          if (lane == 0) L.w[at] |= 1u;
          // graph.h:196-205: its unvisited neighbours
          const uint32_t *row = p.adj + (static_cast<uint64_t>(now) << p.shift);
          const uint32_t a = static_cast<uint32_t>(lane) < nslots ? __ldg(row + lane) : 0u;
          const uint32_t deg = __shfl_sync(FULLM, a, 0);
          const bool fresh = lane >= 1 && static_cast<uint32_t>(lane) <= deg && vis_insert(vis, vis_cap, vis_log2, a);
          const unsigned fm = __ballot_sync(FULLM, fresh);
          next = __popc(fm);
          vis_n += next;
          if (vis_n > p.vis_limit) overflow = true;
          if (fresh) cid[__popc(fm & ((1u << lane) - 1u))] = a;
        }
        if (lane == 0) ctl[0] = overflow ? -1 : next;
      }
      sync();
    }
    if (rank == 0) {
      if (overflow) {
        if (lane == 0) p.out_cnt[t] = vis_n > p.vis_limit ? NEED_VISITED : NEED_STEPS;
      } else {
        // graph.h:207-215: the list in ascending order
        const int num = min(min(n, p.budget), p.out_k);
        for (int i = lane; i < num; i += 32) p.out[static_cast<uint64_t>(t) * p.out_k + i] = L.w[i] >> 1;
        if (lane == 0) p.out_cnt[t] = min(n, p.budget);
      }
    }
    sync();
  }
}

// Squared norms of all rows, each a float sum in dimension order (data.h:50-62).
__global__ void row_norms_kernel(const float *data, uint64_t n, int dim, float *out) {
  for (uint64_t r = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; r < n;
       r += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const float *a = data + r * static_cast<uint64_t>(dim);
    float len = 0.0f;
    for (int i = 0; i < dim; ++i) len = __fadd_rn(len, __fmul_rn(a[i], a[i]));
    out[r] = len;
  }
}

// Scatter of changed adjacency rows: rows[i] (uint32 x 2^shift) goes to row ids[i].
__global__ void scatter_rows_kernel(const uint32_t *rows, const uint64_t *ids, uint64_t count, int shift,
                                    uint32_t *adj) {
  const uint32_t w = 1u << shift;
  const uint64_t total = count * w;
  for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < total;
       i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint64_t r = i >> shift;
    adj[(ids[r] << shift) + (i & (w - 1))] = rows[i];
  }
}

struct DevBuf {
  void *p = nullptr;
  ~DevBuf() {
    if (p) cudaFree(p);
  }
};

// song_debug_build: of the calling thread.
struct BuildDebug {
  int visited_log2 = 0;
  uint64_t searches[3] = {0, 0, 0};
};
thread_local BuildDebug g_build_debug;

struct HostPinned {
  void *p = nullptr;
  ~HostPinned() {
    if (p) cudaFreeHost(p);
  }
};

}  // namespace
}  // namespace song

extern "C" int song_debug_build(int visited_log2, uint64_t *searches) {
  using namespace song;
  clear_error();
  if (visited_log2 != 0 && (visited_log2 < 6 || visited_log2 > BEAM_VIS_LOG2))
    return fail(SONG_ERR_ARG, "visited_log2 must be 0 or in [6, %d]", BEAM_VIS_LOG2);
  if (searches)
    for (int i = 0; i < 3; ++i) searches[i] = g_build_debug.searches[i];
  g_build_debug = BuildDebug{};
  g_build_debug.visited_log2 = visited_log2;
  return SONG_OK;
}

extern "C" int song_graph_build_gpu(const float *data, uint64_t n, int dim, int metric, int shift,
                                    int search_degree, int fixed_degree, int budget, int batch_div,
                                    int device, int nthreads, uint64_t *graph_out) {
  using namespace song;
  clear_error();
  if (!data || !graph_out || n == 0 || dim <= 0) return fail(SONG_ERR_ARG, "graph build: null buffer or empty data");
  if (metric < SONG_METRIC_L2 || metric > SONG_METRIC_COS) return fail(SONG_ERR_ARG, "graph build: bad metric");
  if (shift < 1 || shift > 10) return fail(SONG_ERR_ARG, "graph build: shift must be 1..10");
  if (fixed_degree < 1 || fixed_degree > (1 << shift) - 1)
    return fail(SONG_ERR_ARG, "graph build: fixed_degree must be 1..2^shift-1");
  if (search_degree < 1 || search_degree > fixed_degree || budget < search_degree)
    return fail(SONG_ERR_ARG, "graph build: need 1 <= search_degree <= fixed_degree and budget >= search_degree");
  if (budget > 1024) return fail(SONG_ERR_ARG, "graph build: budget above 1024");
  if (batch_div < 0) return fail(SONG_ERR_ARG, "graph build: batch_div < 0");
  if (n >= (1ull << 32) - 1) return fail(SONG_ERR_ARG, "graph build: more than 2^32-2 vertices");
  if (nthreads < 1) nthreads = 1;
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return fail(SONG_ERR_CUDA, "graph build: cudaSetDevice: %s", cudaGetErrorString(e));
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (sms <= 0) sms = 1;

  GraphBuilder *gb = graph_builder_create(data, n, dim, metric, shift, search_degree, fixed_degree, budget);
  if (!gb) return fail(SONG_ERR_OOM, "graph build: host edge arrays");
  struct Guard {
    GraphBuilder *g;
    ~Guard() { graph_builder_free(g); }
  } guard{gb};

  const size_t per_warp_smem = static_cast<size_t>(budget) * sizeof(QE) + ((static_cast<size_t>(dim) * 4 + 15) & ~15ull);
  const size_t smem = per_warp_smem * BUILD_WARPS;
  int optin = 0;
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  if (smem > static_cast<size_t>(optin)) return fail(SONG_ERR_ARG, "graph build: dim/budget need too much shared memory");
  e = allow_shared(build_search_kernel, smem);
  if (e != cudaSuccess) return fail(SONG_ERR_CUDA, "graph build: %s", cudaGetErrorString(e));
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, build_search_kernel, BUILD_WARPS * 32, smem);
  if (per_sm < 1) return fail(SONG_ERR_ARG, "graph build: kernel does not fit on an SM");
  per_sm = std::min(per_sm, 8);  // 32 warps per SM: enough to hide the heap latency, bounded scratch
  const uint64_t blocks = static_cast<uint64_t>(sms) * per_sm;
  const uint64_t warps = blocks * BUILD_WARPS;

  // the one-list search: list, candidates and query per vertex, and with a
  // block per vertex the visited set
  const size_t beam_slice = sizeof(BeamList) + 32 * 8 + 32 * 4 + 16 + ((static_cast<size_t>(dim) * 4 + 15) & ~size_t(15));
  const size_t beam_smem1 = beam_slice * BUILD_WARPS, beam_smem4 = beam_slice + (sizeof(uint32_t) << BEAM_VIS_LOG2);
  int log2dim = 0;
  while ((1ull << log2dim) < static_cast<uint64_t>(dim)) ++log2dim;
  const int beam_k = 53 - 24 - log2dim;
  int beam1 = 0, beam4 = 0;  // resident blocks per SM
  const bool beam = budget <= BEAM_BUDGET && shift <= 5 && n < (1ull << 31) && beam_smem1 <= static_cast<size_t>(optin) &&
                    beam_smem4 <= static_cast<size_t>(optin) && beam_k > 0;
  if (beam) {
    e = allow_shared(beam_search_kernel<1>, beam_smem1);
    if (e == cudaSuccess) e = allow_shared(beam_search_kernel<4>, beam_smem4);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&beam1, beam_search_kernel<1>, BUILD_WARPS * 32, beam_smem1);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&beam4, beam_search_kernel<4>, BUILD_WARPS * 32, beam_smem4);
    if (e != cudaSuccess) return fail(SONG_ERR_CUDA, "graph build: %s", cudaGetErrorString(e));
    beam1 = std::max(1, std::min(beam1, per_sm));  // (the scratch has room for per_sm blocks)
    beam4 = std::max(1, beam4);
  }

  cudaStream_t st;
  e = cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking);
  if (e != cudaSuccess) return fail(SONG_ERR_CUDA, "graph build: %s", cudaGetErrorString(e));
  struct StreamGuard {
    cudaStream_t s;
    ~StreamGuard() { cudaStreamDestroy(s); }
  } sg{st};

  const uint64_t max_batch = batch_div == 0 ? 1 : std::max<uint64_t>(1, n / batch_div) + 1;
  const uint32_t w = 1u << shift;
  DevBuf d_data, d_norms, d_adj, d_out, d_cnt, d_ctl, d_vis, d_q, d_rows, d_ids, d_todo;
  HostPinned h_out, h_cnt, h_rows, h_ids;
  const size_t rows_cap = static_cast<size_t>(max_batch) * (search_degree + 1);
#define SONG_GB_CK(call)                                                          \
  do {                                                                            \
    cudaError_t e_ = (call);                                                      \
    if (e_ != cudaSuccess)                                                        \
      return fail(e_ == cudaErrorMemoryAllocation ? SONG_ERR_OOM : SONG_ERR_CUDA, \
                  "graph build: %s: %s", #call, cudaGetErrorString(e_));          \
  } while (0)
  SONG_GB_CK(song::dev_malloc(&d_data.p, sizeof(float) * n * dim));
  SONG_GB_CK(song::dev_malloc(&d_adj.p, sizeof(uint32_t) * (n << shift)));
  SONG_GB_CK(song::dev_malloc(&d_out.p, sizeof(uint32_t) * max_batch * search_degree));
  SONG_GB_CK(song::dev_malloc(&d_cnt.p, sizeof(int32_t) * max_batch));
  SONG_GB_CK(song::dev_malloc(&d_ctl.p, 256));
  SONG_GB_CK(song::dev_malloc(&d_rows.p, sizeof(uint32_t) * rows_cap * w));
  SONG_GB_CK(song::dev_malloc(&d_ids.p, sizeof(uint64_t) * rows_cap));
  SONG_GB_CK(cudaMallocHost(&h_out.p, sizeof(uint32_t) * max_batch * search_degree));
  SONG_GB_CK(cudaMallocHost(&h_cnt.p, sizeof(int32_t) * max_batch));
  SONG_GB_CK(cudaMallocHost(&h_rows.p, sizeof(uint32_t) * rows_cap * w));
  SONG_GB_CK(cudaMallocHost(&h_ids.p, sizeof(uint64_t) * rows_cap));
  SONG_GB_CK(cudaMemcpyAsync(d_data.p, data, sizeof(float) * n * dim, cudaMemcpyHostToDevice, st));
  SONG_GB_CK(cudaMemsetAsync(d_adj.p, 0, sizeof(uint32_t) * (n << shift), st));
  if (metric == SONG_METRIC_COS) {
    SONG_GB_CK(song::dev_malloc(&d_norms.p, sizeof(float) * n));
    row_norms_kernel<<<sms * 8, 256, 0, st>>>(static_cast<const float *>(d_data.p), n, dim,
                                              static_cast<float *>(d_norms.p));
    SONG_GB_CK(cudaGetLastError());
  }
  // scratch of the searches that keep their sets in device memory, allocated
  // when the first of them comes; grown when one overflows
  const int set_log2 = g_build_debug.visited_log2 > 0 ? g_build_debug.visited_log2 : BEAM_VIS_LOG2;
  int vis_log2 = set_log2, q_log2 = 12;
  auto alloc_scratch = [&](bool queue) -> int {
    if (d_vis.p) cudaFree(d_vis.p);
    if (d_q.p) cudaFree(d_q.p);
    d_vis.p = d_q.p = nullptr;
    cudaError_t e1 = song::dev_malloc(&d_vis.p, sizeof(uint32_t) * (warps << vis_log2));
    if (e1 == cudaSuccess && queue) e1 = song::dev_malloc(&d_q.p, sizeof(QE) * (warps << q_log2));
    if (e1 != cudaSuccess)
      return fail(e1 == cudaErrorMemoryAllocation ? SONG_ERR_OOM : SONG_ERR_CUDA, "graph build: scratch: %s",
                  cudaGetErrorString(e1));
    return SONG_OK;
  };
  int rc = SONG_OK;

  uint32_t *h_out32 = static_cast<uint32_t *>(h_out.p);
  int32_t *h_cnt32 = static_cast<int32_t *>(h_cnt.p);
  const uint64_t *edges = graph_builder_edges(gb);
  uint64_t a = 0;
  // Where most searches end up step by step (many equal distances, NaNs) they
  // go there at once: for the next 15 batches, when of the last 32 vertices or
  // more that tried the one list most did (20,000 corners of a 32-d cube: 778 ms
  // with both searches for every batch, 671 so).
  uint64_t tried = 0, repeated = 0;
  int steps_first = 0;
  std::vector<uint32_t> todo[2];  // searches to be repeated: by a warp with one list, step by step
  while (a < n) {
    const uint64_t bs = batch_div == 0 ? 1 : std::max<uint64_t>(1, a / static_cast<uint64_t>(batch_div));
    const uint64_t end = std::min<uint64_t>(n, a + bs);
    const uint64_t fit4 = static_cast<uint64_t>(sms) * beam4, fit1 = static_cast<uint64_t>(sms) * beam1;
    enum { BLOCK, WARP, STEPS } how = !beam || steps_first > 0 ? STEPS : (end - a <= fit4 ? BLOCK : WARP);
    if (steps_first > 0) --steps_first;
    const uint32_t *list = nullptr;  // of the vertices searched, on the device (null: all)
    uint64_t count = end - a;
    for (int grown = 0;;) {
      const uint64_t grid = std::min<uint64_t>(blocks, (count + BUILD_WARPS - 1) / BUILD_WARPS);
      if ((how != BLOCK && !d_vis.p) || (how == STEPS && !d_q.p))
        if ((rc = alloc_scratch(how == STEPS)) != SONG_OK) return rc;
      BuildArgs p;
      p.data = static_cast<const float *>(d_data.p);
      p.norms = static_cast<const float *>(d_norms.p);
      p.adj = static_cast<const uint32_t *>(d_adj.p);
      p.dim = dim;
      p.metric = metric;
      p.shift = shift;
      p.first = a;
      p.count = static_cast<uint32_t>(count);
      p.todo = list;
      p.limit = a;
      p.budget = budget;
      p.out_k = search_degree;
      p.out = static_cast<uint32_t *>(d_out.p);
      p.out_cnt = static_cast<int32_t *>(d_cnt.p);
      p.vis = static_cast<uint32_t *>(d_vis.p);
      p.vis_log2 = vis_log2;
      p.vis_cap = 1u << vis_log2;
      p.vis_limit = 3u << ((how == BLOCK ? set_log2 : vis_log2) - 2);
      p.q = static_cast<QE *>(d_q.p);
      p.q_cap = 1u << q_log2;
      p.counter = static_cast<uint32_t *>(d_ctl.p);
      SONG_GB_CK(cudaMemsetAsync(d_ctl.p, 0, 8, st));
      if (how == BLOCK)
        beam_search_kernel<4><<<static_cast<unsigned>(count), BUILD_WARPS * 32, beam_smem4, st>>>(p, beam_k);
      else if (how == WARP)
        beam_search_kernel<1><<<static_cast<unsigned>(std::min<uint64_t>(fit1, grid)), BUILD_WARPS * 32, beam_smem1, st>>>(
            p, beam_k);
      else
        build_search_kernel<<<static_cast<unsigned>(grid), BUILD_WARPS * 32, smem, st>>>(p);
      SONG_GB_CK(cudaGetLastError());
      SONG_GB_CK(cudaMemcpyAsync(h_cnt32, d_cnt.p, sizeof(int32_t) * (end - a), cudaMemcpyDeviceToHost, st));
      SONG_GB_CK(cudaMemcpyAsync(h_out32, d_out.p, sizeof(uint32_t) * (end - a) * search_degree,
                                 cudaMemcpyDeviceToHost, st));
      SONG_GB_CK(cudaStreamSynchronize(st));
      g_build_debug.searches[how] += count;
      // (those not yet repeated still hold their mark)
      bool more_visited = false, more_queue = false;
      todo[0].clear();
      todo[1].clear();
      for (uint32_t t = 0; t < end - a; ++t) {
        const int32_t c = h_cnt32[t];
        if (c >= 0) continue;
        more_visited = more_visited || (c == NEED_VISITED && how != BLOCK);
        more_queue = more_queue || c == NEED_QUEUE;
        todo[c == NEED_VISITED && how != STEPS ? 0 : 1].push_back(t);
      }
      if (!list && how != STEPS) {
        tried += count;
        repeated += todo[1].size();
        if (tried >= 32) {
          if (2 * repeated > tried) steps_first = 15;
          tried = repeated = 0;
        }
      }
      if (todo[0].empty() && todo[1].empty()) break;
      if (more_visited || more_queue) {
        if (++grown > 7) return fail(SONG_ERR_OOM, "graph build: search scratch still too small after growing");
        if (more_visited) ++vis_log2;
        if (more_queue) ++q_log2;
        if ((rc = alloc_scratch(d_q.p != nullptr)) != SONG_OK) return rc;
      }
      how = todo[0].empty() ? STEPS : WARP;
      const std::vector<uint32_t> &next = todo[todo[0].empty() ? 1 : 0];
      if (!d_todo.p) SONG_GB_CK(song::dev_malloc(&d_todo.p, sizeof(uint32_t) * max_batch));
      count = next.size();
      list = static_cast<const uint32_t *>(d_todo.p);
      SONG_GB_CK(cudaMemcpyAsync(d_todo.p, next.data(), sizeof(uint32_t) * count, cudaMemcpyHostToDevice, st));
    }
    // the edges, and the changed rows straight into the upload buffer: <= (end - a) * (search_degree + 1) <= rows_cap
    uint32_t *hr = static_cast<uint32_t *>(h_rows.p);
    uint64_t *hi = static_cast<uint64_t *>(h_ids.p);
    const uint64_t nt = graph_builder_apply(gb, a, end, h_out32, h_cnt32, search_degree, nthreads, hr, hi);
    SONG_GB_CK(cudaMemcpyAsync(d_rows.p, hr, sizeof(uint32_t) * nt * w, cudaMemcpyHostToDevice, st));
    SONG_GB_CK(cudaMemcpyAsync(d_ids.p, hi, sizeof(uint64_t) * nt, cudaMemcpyHostToDevice, st));
    const uint64_t blocks_s = std::min<uint64_t>(4096, (nt * w + 255) / 256);
    if (nt > 0) {
      scatter_rows_kernel<<<static_cast<unsigned>(blocks_s), 256, 0, st>>>(
          static_cast<const uint32_t *>(d_rows.p), static_cast<const uint64_t *>(d_ids.p), nt, shift,
          static_cast<uint32_t *>(d_adj.p));
      SONG_GB_CK(cudaGetLastError());
    }
    a = end;
  }
  SONG_GB_CK(cudaStreamSynchronize(st));
#undef SONG_GB_CK
  std::memcpy(graph_out, edges, sizeof(uint64_t) * (static_cast<size_t>(n) << shift));
  return SONG_OK;
}
