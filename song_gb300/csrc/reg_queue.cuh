// reg_queue.cuh -- the per-query sorted structures of the search, one warp
// each.  Keys are (distance, id) in 64 bits, ascending; every operation is
// warp-uniform.
//
//   RegQueue   a sorted array in registers: the candidate queue (the
//              reference's serial min-max heap, smmh2.h) for small bounds, and
//              the top-pq list of the learned kernels, which read its k-th key.
//   BufQueue   the candidate queue for large bounds: a sorted ring in shared
//              memory behind a 32-key insertion buffer in registers.
//   PopList    the top-pq list (the binary heap, bin_heap.h) of the other
//              kernels: an unsorted register array.
#pragma once

#include <cstdint>

#include "device_common.cuh"

namespace song {

__device__ __forceinline__ uint64_t warp_max_u64(uint64_t x) {
  const uint32_t hi = __reduce_max_sync(FULL, static_cast<uint32_t>(x >> 32));
  const uint32_t lo = __reduce_max_sync(FULL, static_cast<uint32_t>(x >> 32) == hi ? static_cast<uint32_t>(x) : 0u);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}
__device__ __forceinline__ uint64_t warp_min_u64(uint64_t x) {
  const uint32_t hi = __reduce_min_sync(FULL, static_cast<uint32_t>(x >> 32));
  const uint32_t lo =
      __reduce_min_sync(FULL, static_cast<uint32_t>(x >> 32) == hi ? static_cast<uint32_t>(x) : 0xffffffffu);
  return (static_cast<uint64_t>(hi) << 32) | lo;
}

// Layout: capacity C = 32*S positions, lane-blocked (lane l holds positions
// l*S .. l*S+S-1 in v[0..S-1]), ascending, in the WINDOW form: positions
// C-pq .. C-1 always hold pq keys, the live keys first and then "infinite"
// keys (~0); every position left of the window holds 0, smaller than any
// real key (real keys carry order-preserving distance bits >= 0x007fffff in
// their high word).  Consequences:
//   * an insertion is always "insert and drop the window's maximum": keys not
//     below the new key move one place right and an infinite key (or, when
//     all pq are live, the real maximum) falls off -- one code path, per-slot
//     compares and selects, one shuffle at the lane boundary;
//   * the maximum is always at position C-1 (lane 31, v[S-1]): O(1);
//   * the minimum is at position C-pq; removing it shifts the window one
//     place left and appends an infinite key;
//   * reads at a run-time (warp-uniform) position are a binary tree of
//     selects on the slot bits; nothing is indexed at run time, so the array
//     never goes to local memory.
template <int S>
struct RegQueue {
  static constexpr int C = 32 * S;
  uint64_t v[S];
  int start;  // C - pq

  __device__ __forceinline__ void init(uint64_t *, int pq, int lane) {
    start = C - pq;
#pragma unroll
    for (int j = 0; j < S; ++j) v[j] = (lane * S + j) >= start ? ~0ull : 0ull;
  }

  // The window's maximum: an infinite key while fewer than pq keys are live.
  __device__ __forceinline__ uint64_t max() const { return __shfl_sync(FULL, v[S - 1], 31); }

  // The minimum (an infinite key when empty).
  __device__ __forceinline__ uint64_t min() const { return at(start); }

  // Key at the warp-uniform position pos (broadcast).  (Selections never
  // index v[] with a run-time value: the compiler would move the array to
  // local memory.)
  __device__ __forceinline__ uint64_t at(int pos) const {
    const int owner = pos / S;
    return __shfl_sync(FULL, slot(pos - owner * S), owner);
  }

  // Insert and drop the window's maximum: keys not below `key` move one
  // place right and the old maximum falls off.  If key >= the maximum nothing
  // changes (the key itself is dropped).
  __device__ __forceinline__ void insert_evict(uint64_t key, int lane) {
    uint64_t prv = __shfl_up_sync(FULL, v[S - 1], 1);
    if (lane == 0) prv = 0ull;
#pragma unroll
    for (int j = S - 1; j >= 0; --j) {
      const uint64_t left = j > 0 ? v[j - 1] : prv;
      v[j] = v[j] < key ? v[j] : (left < key ? key : left);
    }
  }

  // v[r] for a warp-uniform slot r in [0, S): a binary tree of selects on
  // the bits of r (S - 1 selects, depth log2 S; a chain of S compares would
  // serialise S dependent selects).
  __device__ __forceinline__ uint64_t slot(int r) const {
    uint64_t t[S];
#pragma unroll
    for (int j = 0; j < S; ++j) t[j] = v[j];
#pragma unroll
    for (int w = 1; w < S; w <<= 1) {
      const bool b = (r & w) != 0;
#pragma unroll
      for (int j = 0; j + w < S; j += 2 * w) t[j] = b ? t[j + w] : t[j];
    }
    return t[0];
  }

  // Removes the minimum (returned); *next gets the new minimum.
  __device__ __forceinline__ uint64_t pop(int lane, uint64_t *next) {
    const int owner = start / S, r = start - owner * S;
    const uint64_t m = __shfl_sync(FULL, slot(r), owner);
    uint64_t nxt = __shfl_down_sync(FULL, v[0], 1);
    if (lane == 31) nxt = ~0ull;
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const uint64_t right = j + 1 < S ? v[j + 1] : nxt;
      v[j] = (lane * S + j) >= start ? right : v[j];
    }
    *next = __shfl_sync(FULL, slot(r), owner);
    return m;
  }
};

// Candidate queue of up to pq keys: `n` of them sorted in a ring of pq + 32
// places in shared memory, `bn` sorted across the lanes of one register
// (infinite keys past them).  An insertion goes to the register (a compare,
// two selects and a shuffle whatever pq is); the minimum and the maximum are
// the smaller and the larger of both parts' ends, so a pop or an eviction
// moves an index or one register.  A full register is merged into the ring:
// every ring key moves up by the number of buffered keys below it, 32 keys a
// step from the top until a step moves nothing.  RegQueue's insertion touches
// all 32*S places instead; the line between the two is BUF_S in
// search_kernel.cuh.
struct BufQueue {
  uint64_t *m;   // ring of `size` places
  int size, pq;
  int head, n;   // ring position of the minimum, keys in the ring
  uint64_t b;
  int bn;
  uint64_t lo, hi;  // ring minimum (infinite when empty) and maximum (0 when empty)

  static __host__ __device__ uint32_t bytes(int pq) { return 8u * static_cast<uint32_t>(pq + 32); }

  __device__ __forceinline__ void init(uint64_t *ring, int bound, int) {
    m = ring;
    pq = bound;
    size = bound + 32;
    head = n = bn = 0;
    b = ~0ull;
    lo = ~0ull;
    hi = 0ull;
  }
  __device__ __forceinline__ int place(int i) const {  // 0 <= i < size
    const int c = head + i;
    return c >= size ? c - size : c;
  }
  __device__ __forceinline__ uint64_t buf_max() const { return bn > 0 ? __shfl_sync(FULL, b, bn - 1) : 0ull; }

  __device__ __forceinline__ uint64_t max() const {
    if (n + bn < pq) return ~0ull;
    const uint64_t x = buf_max();
    return x > hi ? x : hi;
  }
  __device__ __forceinline__ uint64_t min() const {
    const uint64_t x = __shfl_sync(FULL, b, 0);
    return x < lo ? x : lo;
  }

  __device__ __forceinline__ uint64_t pop(int lane, uint64_t *next) {
    uint64_t x = __shfl_sync(FULL, b, 0);
    uint64_t r;
    if (x < lo) {
      r = x;
      b = __shfl_down_sync(FULL, b, 1);
      if (lane == 31) b = ~0ull;
      --bn;
      x = __shfl_sync(FULL, b, 0);
    } else {
      r = lo;
      head = place(1);
      --n;
      lo = n > 0 ? m[head] : ~0ull;
      if (n == 0) hi = 0ull;
    }
    *next = x < lo ? x : lo;
    return r;
  }

  // Inserts `key`; a full queue drops its maximum first (which the caller
  // has seen to be above the key).
  __device__ __forceinline__ void insert_evict(uint64_t key, int lane) {
    if (n + bn >= pq) {
      const uint64_t x = buf_max();
      if (!((x > hi ? x : hi) > key)) return;
      if (x > hi) {
        --bn;
        if (lane == bn) b = ~0ull;
      } else {
        --n;
        hi = n > 0 ? m[place(n - 1)] : 0ull;
        if (n == 0) lo = ~0ull;
      }
    }
    if (bn == 32) merge(lane);
    uint64_t prv = __shfl_up_sync(FULL, b, 1);
    if (lane == 0) prv = 0ull;
    b = b < key ? b : (prv < key ? key : prv);
    ++bn;
  }

  // Moves the bn buffered keys into the ring (n + bn <= pq <= size - 32).
  __device__ __forceinline__ void merge(int lane) {
    // buffered key `lane` goes above the ring keys not above it
    int rank = 0;
    {
      int l = 0, h = n;
      while (l < h) {
        const int mid = (l + h) >> 1;
        if (m[place(mid)] <= b) l = mid + 1;
        else h = mid;
      }
      rank = l;
    }
    for (int top = n; top > 0; top -= 32) {
      const int i = top - 32 + lane;
      const uint64_t key = i >= 0 ? m[place(i)] : 0ull;
      int cnt = 0;  // buffered keys below `key`
#pragma unroll
      for (int s = 16; s > 0; s >>= 1)
        if (__shfl_sync(FULL, b, cnt + s - 1) < key) cnt += s;
      if (__shfl_sync(FULL, b, cnt) < key) ++cnt;
      if (!__any_sync(FULL, cnt > 0)) break;
      __syncwarp();
      if (cnt > 0) m[place(i + cnt)] = key;
      __syncwarp();
    }
    if (lane < bn) m[place(rank + lane)] = b;
    __syncwarp();
    n += bn;
    bn = 0;
    b = ~0ull;
    lo = m[head];
    hi = m[place(n - 1)];
  }
};

// The top-pq list: popped vertices in the order they arrive, element i in
// lane i % 32's register i / 32.  Only its maximum is ever asked for, and
// only once pq vertices are in it, so nothing is kept sorted: an arrival is
// one predicated move (whole registers go to the array 32 arrivals at a
// time), the maximum a scan of S registers and two warp reductions, and the
// answer is sorted once at the end.  (A sorted array costs an insertion over
// 32*S places per hop: 20 instructions per register pair of S.)
template <int S>
struct PopList {
  uint64_t v[S];
  uint64_t cur;  // the 32 latest arrivals, not yet in v
  int n;

  __device__ __forceinline__ void init() {
#pragma unroll
    for (int j = 0; j < S; ++j) v[j] = 0ull;
    cur = 0ull;
    n = 0;
  }
  __device__ __forceinline__ void flush(int j) {
#pragma unroll
    for (int i = 0; i < S; ++i) v[i] = i == j ? cur : v[i];
    cur = 0ull;
  }
  // Arrival number n (n < pq).
  __device__ __forceinline__ void append(uint64_t key, int pq, int lane) {
    if (lane == (n & 31)) cur = key;
    ++n;
    if ((n & 31) == 0 || n == pq) flush((n - 1) >> 5);
  }
  // n == pq.
  __device__ __forceinline__ uint64_t max() const {
    uint64_t x = 0ull;
#pragma unroll
    for (int j = 0; j < S; ++j) x = v[j] > x ? v[j] : x;
    return warp_max_u64(x);
  }
  // Replaces one element equal to `old`.
  __device__ __forceinline__ void replace(uint64_t old, uint64_t key, int lane) {
    bool has = false;
#pragma unroll
    for (int j = 0; j < S; ++j) has = has || v[j] == old;
    const unsigned who = __ballot_sync(FULL, has);
    bool todo = lane == __ffs(who) - 1;
#pragma unroll
    for (int j = 0; j < S; ++j) {
      const bool here = todo && v[j] == old;
      v[j] = here ? key : v[j];
      todo = todo && !here;
    }
  }
  // Writes the n elements and then infinite keys, 32*S in all.
  __device__ __forceinline__ void dump(uint64_t *out, int pq, int lane) {
    if ((n & 31) != 0 && n < pq) flush(n >> 5);
#pragma unroll
    for (int j = 0; j < S; ++j) out[32 * j + lane] = 32 * j + lane < n ? v[j] : ~0ull;
  }
};

// Ascending across the lanes.
__device__ __forceinline__ uint64_t warp_sort(uint64_t x, int lane) {
#pragma unroll
  for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      const uint64_t y = __shfl_xor_sync(FULL, x, j);
      const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
      x = (x < y) == keep_min ? x : y;
    }
  return x;
}

// The 32 smallest of count (a multiple of 32) keys in shared memory, ascending
// across the lanes.
__device__ __forceinline__ uint64_t warp_smallest32(const uint64_t *keys, int count, int lane) {
  uint64_t x = warp_sort(keys[lane], lane);
  for (int a = 32; a < count; a += 32) {
    const uint64_t y = warp_sort(keys[a + lane], lane);
    const uint64_t z = __shfl_sync(FULL, y, 31 - lane);  // descending: min() leaves a bitonic sequence
    x = z < x ? z : x;
#pragma unroll
    for (int j = 16; j > 0; j >>= 1) {
      const uint64_t o = __shfl_xor_sync(FULL, x, j);
      x = (x < o) == ((lane & j) == 0) ? x : o;
    }
  }
  return x;
}

// Sorts count (a power of two >= 32) keys in shared memory, ascending.
__device__ __forceinline__ void warp_sort_shared(uint64_t *keys, int count, int lane) {
  for (int k = 2; k <= count; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      for (int t = lane; t < count / 2; t += 32) {
        const int i = ((t & ~(j - 1)) << 1) | (t & (j - 1));
        const uint64_t a = keys[i], c = keys[i | j];
        if ((a > c) == ((i & k) == 0)) {
          keys[i] = c;
          keys[i | j] = a;
        }
      }
      __syncwarp();
    }
}

}  // namespace song
