// device_common.cuh -- warp-cooperative building blocks of the search kernel:
// bulk-copy / mbarrier wrappers (inline PTX, sm_90+ forms valid on sm_103a),
// the sort keys of the candidate / top-pq queues, and the visited hashes held
// in the shared memory slice of one warp.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace song {

constexpr unsigned FULL = 0xffffffffu;
constexpr int32_t FH_EMPTY = -1;     // fixhash.h:3 EMPTY
constexpr int32_t FH_DELETION = -2;  // fixhash.h:3 DELETION (never written with backward-shift delete)
// fixhash.h:9, the first multiplier / xor pair used by hash(0, x).
constexpr uint64_t FH_R0 = 0x4bcb391f924ed183ULL;
constexpr uint64_t FH_R1 = 0xa0ab69ccd854fc0aULL;

// Bounded waits: an mbarrier that does not complete within this many polls
// (each poll may itself suspend in hardware) sets the error flag and returns.
// The default of an index; song_debug_set_wait changes it per index.
constexpr uint32_t WAIT_LIMIT = 1u << 24;

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
}

// 1-D bulk copy global -> shared, completion counted on `bar` in bytes.
// dst, src and bytes must be multiples of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait for phase `parity` of `bar`; false on timeout.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, uint32_t limit) {
  for (uint32_t i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

// The same with one decision for the whole warp: a lane that gave up alone
// would leave the others shuffling with a lane that is gone, and lanes that see
// the phase at different polls, with a return between them and the code they
// share, would go through all of it apart (in the server one query of 15k x 16
// took 1363 us that way, 299 so).
__device__ __forceinline__ bool mbar_wait_warp(uint64_t *bar, uint32_t parity, uint32_t limit) {
  const bool done = mbar_wait(bar, parity, limit);
  __syncwarp();
  return __ballot_sync(FULL, done) == FULL;
}

// Two FP32 lanes in one 64-bit register, for the paired FP32 instructions of
// sm_100-family GPUs (sub/fma .rn.f32x2: each half rounded to nearest even,
// exactly the scalar __fsub_rn / __fmaf_rn).
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_unpack(uint64_t r, float &lo, float &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(r));
}
__device__ __forceinline__ uint64_t f2_sub(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// The xor butterfly 16, 8, 4, 2, 1 over the 32 lanes' partial sums of H rows
// at once.  At the first log2(H) levels each lane keeps half of its rows and
// sends its partner the other half, so one shuffle serves two rows; every
// row still meets its partials in the butterfly's pairs (each pair sum is
// the same two floats, and a + b == b + a), so the sums are bit for bit the
// per-row butterfly's.  Returns, in lane l, the sum of row l / (32 / H).
template <int H>
__device__ __forceinline__ float butterfly_rows(float (&v)[H], int lane) {
  static_assert(H >= 1 && H <= 32 && (H & (H - 1)) == 0, "H must be a power of two");
  int o = 16;
#pragma unroll
  for (int n = H; n > 1; n >>= 1, o >>= 1) {
    const bool hi = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const float keep = hi ? v[i + n / 2] : v[i];
      const float send = hi ? v[i] : v[i + n / 2];
      v[i] = __fadd_rn(keep, __shfl_xor_sync(FULL, send, o));
    }
  }
#pragma unroll
  for (; o > 0; o >>= 1) v[0] = __fadd_rn(v[0], __shfl_xor_sync(FULL, v[0], o));
  return v[0];
}

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// ---------------------------------------------------------------------------
// Keys of the sorted queues: (distance, id) in one uint64 whose unsigned
// order is (distance ascending, id ascending).  The distance is mapped to an
// order-preserving uint32 after -0 is folded onto +0, so that the reference's
// float comparisons (which treat -0 == +0) and key comparisons agree.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t dist_bits(float d) {
  if (d == 0.0f) d = 0.0f;
  uint32_t u = __float_as_uint(d);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ uint64_t make_key(float d, uint32_t id) {
  return (static_cast<uint64_t>(dist_bits(d)) << 32) | id;
}
__device__ __forceinline__ uint32_t key_dist(uint64_t k) { return static_cast<uint32_t>(k >> 32); }
__device__ __forceinline__ uint32_t key_id(uint64_t k) { return static_cast<uint32_t>(k); }

// ---------------------------------------------------------------------------
// A walk along a visited set's slots reads the first few at once (the table
// is at most a quarter full, so most walks end there): one shared-memory
// latency instead of one per slot, and no loop whose lanes leave at different
// times.
// ---------------------------------------------------------------------------

// One lane, own key: is it in the set?
template <class VH>
__device__ __forceinline__ bool visited_test(const VH &vh, uint32_t id, int home) {
  constexpr int W = 4;
  int32_t v[W];
#pragma unroll
  for (int i = 0; i < W; ++i) v[i] = vh.tab[vh.ahead(home, i)];
  bool found = false, open = true;  // open: no empty slot so far
#pragma unroll
  for (int i = 0; i < W; ++i) {
    found = found || (open && v[i] == static_cast<int32_t>(id));
    open = open && v[i] != FH_EMPTY;
  }
  if (open && !found) {
    int c = vh.ahead(home, W);
    for (int i = W; i < vh.cap; ++i) {
      const int32_t x = vh.tab[c];
      if (x == FH_EMPTY) break;
      if (x == static_cast<int32_t>(id)) return true;
      c = vh.next(c);
    }
  }
  return found;
}

// One lane: the first empty slot from `home` on; -1 in a table without one.
template <class VH>
__device__ __forceinline__ int visited_end(const VH &vh, int home) {
  constexpr int W = 4;
  int32_t v[W];
#pragma unroll
  for (int i = 0; i < W; ++i) v[i] = vh.tab[vh.ahead(home, i)];
  int at = W;
#pragma unroll
  for (int i = W - 1; i >= 0; --i) at = v[i] == FH_EMPTY ? i : at;
  int c = vh.ahead(home, at);
  if (at == W) {
    int i = W;
    while (vh.tab[c] != FH_EMPTY) {
      c = vh.next(c);
      if (++i > vh.cap) return -1;
    }
  }
  return c;
}

// One lane: where key id sits (-1: nowhere) and the first empty slot after it
// (or, when it is absent, on its walk); false in a table without empty slots.
template <class VH>
__device__ __forceinline__ bool visited_find(const VH &vh, uint32_t id, int home, int &at, int &end) {
  constexpr int W = 6;
  int32_t v[W];
#pragma unroll
  for (int i = 0; i < W; ++i) v[i] = vh.tab[vh.ahead(home, i)];
  int m = W, t = W;
#pragma unroll
  for (int i = W - 1; i >= 0; --i) {
    m = v[i] == static_cast<int32_t>(id) ? i : m;
    t = v[i] == FH_EMPTY ? i : t;
  }
  at = m < t ? vh.ahead(home, m) : -1;
  end = vh.ahead(home, t);
  if (t == W) {
    int i = W;
    for (;;) {
      const int32_t x = vh.tab[end];
      if (x == FH_EMPTY) break;
      if (at < 0 && x == static_cast<int32_t>(id)) at = end;
      end = vh.next(end);
      if (++i > vh.cap) return false;
    }
  }
  return true;
}

// ---------------------------------------------------------------------------
// Visited hash: the reference's FixHash<int, 8*pq> (fixhash.h) in the warp's
// shared memory, with the same slot function, linear probing and
// backward-shift delete, so that membership answers (including the rare
// entries its delete loses) are the reference's.
// ---------------------------------------------------------------------------
struct VisitedHash {
  static constexpr bool FILLS = true;
  int32_t *tab;
  int cap;        // 8 * pq
  uint64_t magic; // floor((2^64 - 1) / cap): v % cap by one high multiply and one correction

  // hash(0, x) = (x ^ (x >> 16) * r0 ^ r1) % cap (fixhash.h:20-24).  x is the
  // stored int widened to 64 bits; ids are < 2^31 so that is the id itself.
  __device__ __forceinline__ int slot(uint32_t id) const {
    uint64_t x = id;
    uint64_t v = x ^ ((x >> 16) * FH_R0) ^ FH_R1;
    uint64_t q = __umul64hi(v, magic);
    // v - q * cap < 2 * cap: the low words hold it
    const uint32_t c = static_cast<uint32_t>(cap);
    uint32_t r = static_cast<uint32_t>(v) - static_cast<uint32_t>(q) * c;
    if (r >= c) r -= c;
    return static_cast<int>(r);
  }

  // s < cap + 32 <= 3 * cap (every caller adds at most 32 to a slot, and
  // cap = 8 * pq >= 16): two conditional subtractions, no branch
  __device__ __forceinline__ int wrap(int s) const {
    s = s >= cap ? s - cap : s;
    return s >= cap ? s - cap : s;
  }

  __device__ __forceinline__ int next(int c) const { return c + 1 == cap ? 0 : c + 1; }
  // slot c + i, 0 <= i < 16 <= cap
  __device__ __forceinline__ int ahead(int c, int i) const { return c + i >= cap ? c + i - cap : c + i; }

  __device__ __forceinline__ void clear(int lane) {
    for (int i = lane; i < cap; i += 32) tab[i] = FH_EMPTY;
    __syncwarp();
  }

  // One lane, own key, `home` = slot(id) (fixhash.h:49-57).
  __device__ __forceinline__ bool test_at(uint32_t id, int home) const {
    return visited_test(*this, id, home);
  }
  __device__ __forceinline__ bool test(uint32_t id) const { return test_at(id, slot(id)); }

  // The case analysis of the backward-shift delete (fixhash.h:64-90): does
  // the entry at slot nxt, whose home is ncode, move into the hole r left by
  // an entry whose home is code?
  __device__ __forceinline__ bool moves(int code, int r, int nxt, int ncode) const {
    const bool cond1 = code <= r, cond2 = r < nxt;
    if (cond1 && cond2) return ncode <= r;
    if (cond1) return nxt < ncode && ncode <= r;
    return nxt < ncode || ncode <= r;
  }

  // Whole warp, one key (fixhash.h:38-47): first EMPTY/DELETION slot on the
  // probe sequence, found 32 slots at a time with a ballot.  `home` is
  // slot(id), computed by the caller (often in parallel, one lane per key).
  __device__ __forceinline__ void add_at(uint32_t id, int home, int lane) {
    int base = home;
    for (int w = 0; w * 32 < cap + 32; ++w) {
      int s = wrap(base + lane);
      int32_t v = tab[s];
      unsigned b = __ballot_sync(FULL, v == FH_EMPTY || v == FH_DELETION);
      if (b) {
        if (lane == __ffs(b) - 1) tab[s] = static_cast<int32_t>(id);
        break;
      }
      base = wrap(base + 32);
    }
    __syncwarp();
  }

  __device__ __forceinline__ void add(uint32_t id, int lane) { add_at(id, slot(id), lane); }

  // Whole warp, one key (fixhash.h:59-93), `home` = slot(id).  The run after
  // the removed entry is read 32 slots at a time; the reference's sequential
  // case analysis then runs uniformly over it, with each lane's slot value
  // and home slot fetched by shuffle.  Home slots of the run are computed
  // only when the slot after the removed entry is occupied.
  __device__ __forceinline__ void del_at(uint32_t id, int home, int lane) {
    const int32_t x = static_cast<int32_t>(id);
    int code = home;
    int r = -1;
    int base = code;
    for (int w = 0; w * 32 < cap + 32; ++w) {
      int s = wrap(base + lane);
      int32_t v = tab[s];
      unsigned be = __ballot_sync(FULL, v == FH_EMPTY);
      unsigned bm = __ballot_sync(FULL, v == x);
      unsigned before = be ? ((1u << (__ffs(be) - 1)) - 1u) : FULL;
      unsigned hit = bm & before;
      if (hit) {
        r = wrap(base + __ffs(hit) - 1);
        break;
      }
      if (be) return;  // not present
      base = wrap(base + 32);
    }
    if (r < 0) return;
    int nbase = wrap(r + 1);
    for (int w = 0; w * 32 < cap + 32; ++w) {
      int s = wrap(nbase + lane);
      int32_t v = tab[s];
      unsigned be = __ballot_sync(FULL, v == FH_EMPTY);
      int run = be ? __ffs(be) - 1 : 32;
      int hv = 0;
      if (run > 0) hv = v >= 0 ? slot(static_cast<uint32_t>(v)) : 0;  // warp-uniform branch
      for (int i = 0; i < run; ++i) {
        int nxt = wrap(nbase + i);
        int ncode = __shfl_sync(FULL, hv, i);
        int32_t val = __shfl_sync(FULL, v, i);
        if (moves(code, r, nxt, ncode)) {
          if (lane == 0) tab[r] = val;
          r = nxt;
          code = ncode;
        }
      }
      __syncwarp();
      if (be) break;
      nbase = wrap(nbase + 32);
    }
    if (lane == 0) tab[r] = FH_EMPTY;
    __syncwarp();
  }

  __device__ __forceinline__ void del(uint32_t id, int lane) { del_at(id, slot(id), lane); }
};

// ---------------------------------------------------------------------------
// Exact visited set for the learned / low-precision path, which makes no
// bit-parity claim with the reference: power-of-two capacity (>= 4*pq), a
// multiplicative slot function, linear probing and the textbook
// backward-shift delete (an entry moves into the hole when its home slot is
// not cyclically inside (hole, position]), so no entry is ever lost.  Half the
// shared memory of VisitedHash at the same pq, and a two-instruction slot.
// ---------------------------------------------------------------------------
struct ExactVisited {
  static constexpr bool FILLS = false;
  int32_t *tab;
  int cap;       // power of two
  int log2cap;

  __device__ __forceinline__ int slot(uint32_t id) const {
    return static_cast<int>((id * 0x9E3779B1u) >> (32 - log2cap));  // cap >= 32
  }
  __device__ __forceinline__ int wrap(int s) const { return s & (cap - 1); }
  __device__ __forceinline__ int next(int c) const { return (c + 1) & (cap - 1); }
  __device__ __forceinline__ int ahead(int c, int i) const { return (c + i) & (cap - 1); }

  __device__ __forceinline__ void clear(int lane) {
    for (int i = lane; i < cap; i += 32) tab[i] = FH_EMPTY;
    __syncwarp();
  }

  __device__ __forceinline__ bool test_at(uint32_t id, int home) const {
    return visited_test(*this, id, home);
  }
  __device__ __forceinline__ bool test(uint32_t id) const { return test_at(id, slot(id)); }

  // An entry moves into the hole r when its home is not cyclically inside (r, nxt].
  __device__ __forceinline__ bool moves(int, int r, int nxt, int ncode) const {
    return ((nxt - ncode) & (cap - 1)) >= ((nxt - r) & (cap - 1));
  }

  __device__ __forceinline__ void add_at(uint32_t id, int home, int lane) {
    int base = home;
    for (int w = 0; w * 32 < cap + 32; ++w) {
      const int s = wrap(base + lane);
      const int32_t v = tab[s];
      const unsigned b = __ballot_sync(FULL, v == FH_EMPTY);
      if (b) {
        if (lane == __ffs(b) - 1) tab[s] = static_cast<int32_t>(id);
        break;
      }
      base = wrap(base + 32);
    }
    __syncwarp();
  }

  __device__ __forceinline__ void add(uint32_t id, int lane) { add_at(id, slot(id), lane); }

  __device__ __forceinline__ void del_at(uint32_t id, int home, int lane) {
    const int32_t x = static_cast<int32_t>(id);
    int base = home, h = -1;
    for (int w = 0; w * 32 < cap + 32; ++w) {
      const int s = wrap(base + lane);
      const int32_t v = tab[s];
      const unsigned be = __ballot_sync(FULL, v == FH_EMPTY);
      const unsigned bm = __ballot_sync(FULL, v == x);
      const unsigned before = be ? ((1u << (__ffs(be) - 1)) - 1u) : FULL;
      const unsigned hit = bm & before;
      if (hit) {
        h = wrap(base + __ffs(hit) - 1);
        break;
      }
      if (be) return;
      base = wrap(base + 32);
    }
    if (h < 0) return;
    int nbase = wrap(h + 1);
    for (int w = 0; w * 32 < cap + 32; ++w) {
      const int s = wrap(nbase + lane);
      const int32_t v = tab[s];
      const int home = v >= 0 ? slot(static_cast<uint32_t>(v)) : 0;
      const unsigned be = __ballot_sync(FULL, v == FH_EMPTY);
      const int run = be ? __ffs(be) - 1 : 32;
      for (int i = 0; i < run; ++i) {
        const int j = wrap(nbase + i);
        const int hm = __shfl_sync(FULL, home, i);
        const int32_t val = __shfl_sync(FULL, v, i);
        if (moves(0, h, j, hm)) {
          if (lane == 0) tab[h] = val;
          h = j;
        }
      }
      __syncwarp();
      if (be) break;
      nbase = wrap(nbase + 32);
    }
    if (lane == 0) tab[h] = FH_EMPTY;
    __syncwarp();
  }

  __device__ __forceinline__ void del(uint32_t id, int lane) { del_at(id, slot(id), lane); }
};

// ---------------------------------------------------------------------------
// Whole-warp operations over either visited set (VH), bit for bit the
// reference's one-at-a-time calls.
// ---------------------------------------------------------------------------

// del(id) followed by add(id) (a popped vertex leaves the queue and enters
// the list, warp_astar_accelerator.h:188-200).  The delete fills the hole
// with later entries of the run, hole after hole, and the add finds every
// slot before the last hole taken and lands in that one.  With an empty slot
// behind the entry (three pops of four) nothing changes at all.
template <class VH>
__device__ __forceinline__ void visited_refresh(VH &vh, uint32_t id, int home, int lane) {
  const int32_t v = vh.tab[vh.wrap(home + lane)];
  const unsigned be = __ballot_sync(FULL, v == FH_EMPTY);
  const unsigned bm = __ballot_sync(FULL, v == static_cast<int32_t>(id));
  const int end = __ffs(be) - 1, at = __ffs(bm) - 1;  // lowest empty slot, lowest match (-1: none)
  if (be && bm && at < end) {
    if (at + 1 == end) return;
    int r = at, code = home;
    const int hv = v >= 0 ? vh.slot(static_cast<uint32_t>(v)) : 0;
    for (int i = at + 1; i < end; ++i) {
      const int ncode = __shfl_sync(FULL, hv, i);
      if (vh.moves(code, vh.wrap(home + r), vh.wrap(home + i), ncode)) {
        if (lane == i) vh.tab[vh.wrap(home + r)] = v;
        r = i;
        code = ncode;
      }
    }
    if (r != at && lane == 0) vh.tab[vh.wrap(home + r)] = static_cast<int32_t>(id);
    __syncwarp();
    return;
  }
  vh.del_at(id, home, lane);
  vh.add_at(id, home, lane);
}

// Calls on a table without an empty slot, one after another, lane by lane.
template <class VH>
__device__ __forceinline__ void visited_in_order(VH &vh, unsigned adds, unsigned dels, uint32_t id, int home, uint32_t eid,
                                              int ehome, int lane) {
  for (unsigned left = adds | dels; left; left &= left - 1u) {
    const int l = __ffs(left) - 1;
    const uint32_t add = __shfl_sync(FULL, id, l), del = __shfl_sync(FULL, eid, l);
    const int ahome = __shfl_sync(FULL, home, l), dhome = __shfl_sync(FULL, ehome, l);
    if (adds >> l & 1u) vh.add_at(add, ahome, lane);
    if (dels >> l & 1u) vh.del_at(del, dhome, lane);
  }
}

template <class VH>
__device__ __noinline__ void visited_in_order_call(VH vh, unsigned adds, unsigned dels, uint32_t id, int home,
                                                   uint32_t eid, int ehome, int lane) {
  visited_in_order(vh, adds, dels, id, home, eid, ehome, lane);
}

// The visited-set calls of one select-insert pass
// (warp_astar_accelerator.h:311-320), in the reference's order -- lane 0's
// add(id), lane 0's del(eid), lane 1's add, ... -- each lane naming its own
// calls (padd / pdel).  One call changes the table only inside its cluster
// (the occupied slots around its home up to the first empty one), so calls
// with different terminating empty slots commute, and all of them run at
// once, one lane each.  Every round the lanes find their calls' terminating
// slots in the table as it stands and mark them; a call that finds another
// call's mark waits, together with every later call, for the next round.
// The first pending call always runs, which bounds the rounds; there are 1.4
// to 3.3 of them a hop (pq 1000, pq 100).
//
// FixHash's lost entries stay, and a small table fills up with them in a long
// walk (40 slots at pq 5 within some 400 hops): without an empty slot the calls
// run one after another.  That code hardly ever runs; what it costs is registers
// around it, which differ by kernel, so there are three forms of it:
//   INLINED     visited_in_order in place.  Short FP32 rows: 0 to 4 % of a
//               search's time (the next form 1 to 4 %: 1M x 128 at pq 150 -0.2
//               and +1.5 %, at pq 75 from vertex 0 +1.0 and +4.4 %).
//   BY_DELETES  the first delete in place, what is left in another round (adds
//               do nothing before a delete makes room).  BF16, FP8 and long
//               rows: 0 to 3 % (INLINED up to 8 %: 15k x 16 FP8 rows).
//   CALLED      visited_in_order as a call.  Codes: 1 to 2 % (BY_DELETES 9 % at
//               pq 100); 12 % for cosine vectors.
enum class FullTable { INLINED, CALLED, BY_DELETES };
template <class VH, FullTable FULL_TABLE>
__device__ __forceinline__ void visited_update(VH &vh, bool padd, uint32_t id, int home, bool pdel, uint32_t eid,
                                               int ehome, int lane) {
  const uint32_t ia = 2u * lane, id2 = ia + 1u;  // the calls' places in the order
  constexpr uint32_t MARK = 0x80000000u, NONE = 64u;
  int32_t *tab = vh.tab;
  for (;;) {
    int ta = 0, td = 0, r = -1;
    bool ok = true;
    if (padd) {
      ta = visited_end(vh, home);
      ok = ta >= 0;
    }
    if (pdel) ok = visited_find(vh, eid, ehome, r, td) && ok;
    if (__any_sync(FULL, !ok)) {
      if constexpr (!VH::FILLS) return;
      const unsigned adds = __ballot_sync(FULL, padd), dels = __ballot_sync(FULL, pdel);
      if constexpr (FULL_TABLE == FullTable::CALLED) {
        visited_in_order_call(vh, adds, dels, id, home, eid, ehome, lane);
        return;
      }
      if constexpr (FULL_TABLE == FullTable::INLINED) {
        visited_in_order(vh, adds, dels, id, home, eid, ehome, lane);
        return;
      }
      if (dels == 0u) return;
      const int l = __ffs(dels) - 1;
      vh.del_at(__shfl_sync(FULL, eid, l), __shfl_sync(FULL, ehome, l), lane);
      padd = padd && lane > l;
      pdel = pdel && lane > l;
      continue;
    }
    __syncwarp();
    if (padd) tab[ta] = static_cast<int32_t>(MARK + ia);
    if (pdel) tab[td] = static_cast<int32_t>(MARK + id2);
    __syncwarp();
    const bool la = padd && tab[ta] != static_cast<int32_t>(MARK + ia);
    const bool ld = pdel && tab[td] != static_cast<int32_t>(MARK + id2);
    bool ea = padd, ed = pdel;
    __syncwarp();
    const bool clash = __any_sync(FULL, la || ld);
    if (clash) {
      const uint32_t lost = __reduce_min_sync(FULL, la ? ia : (ld ? id2 : NONE));
      const uint32_t first = __reduce_min_sync(FULL, padd ? ia : (pdel ? id2 : NONE));
      const uint32_t end = max(lost, first + 1u);  // calls below `end` run in this round
      if (padd) tab[ta] = FH_EMPTY;
      if (pdel) tab[td] = FH_EMPTY;
      __syncwarp();
      ea = padd && ia < end;
      ed = pdel && id2 < end;
    }
    if (ea) tab[ta] = static_cast<int32_t>(id);
    if (ed) {
      tab[td] = FH_EMPTY;
      if (r >= 0) {
        int code = ehome;
        for (int c = vh.next(r); c != td; c = vh.next(c)) {
          const int32_t v = tab[c];
          const int nh = vh.slot(static_cast<uint32_t>(v));
          if (vh.moves(code, r, c, nh)) {
            tab[r] = v;
            r = c;
            code = nh;
          }
        }
        tab[r] = FH_EMPTY;
      }
    }
    __syncwarp();
    if (!clash) break;
    padd = padd && !ea;
    pdel = pdel && !ed;
    if (!__any_sync(FULL, padd || pdel)) break;
  }
}

}  // namespace song
