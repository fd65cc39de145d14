// entry_rows.cuh -- the two-level entry choice's scoring of contiguous FP32
// rows (heads, or a cluster's entries) against up to four queries at once,
// with the search's exact distances: a warp takes eight rows a pass, four
// lanes a row, read straight from global memory into the register pairs of
// the paired FP32 instructions (row_read.cuh), and every row's registers
// serve all the queries.
#pragma once

#include <cstdint>

#include "entry_choice.cuh"
#include "row_read.cuh"
#include "song_gb300.h"

namespace song {

// Distances of the row at `row` (dpad floats; four lanes share a row) to NQ
// queries staged `qs` floats apart (zero-padded to a multiple of 32 floats):
// out[a] in all four lanes.
template <int METRIC, int NQ>
__device__ __forceinline__ void rows8_distance(const float *row, const float *q, int qs, int dpad, float (&out)[NQ],
                                               int lane) {
  const int g = lane & 3;
  const uint8_t *x8 = reinterpret_cast<const uint8_t *>(row);
  uint64_t acc[NQ][4], len[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    len[i] = 0ull;
#pragma unroll
    for (int a = 0; a < NQ; ++a) acc[a][i] = 0ull;
  }
  auto add = [&](const RowRead<0> &r, int j) {
    uint64_t x[4];
    r.get(x, 1.0f);
#pragma unroll
    for (int a = 0; a < NQ; ++a) {
      const ulonglong2 *q2 = reinterpret_cast<const ulonglong2 *>(q + a * qs + j) + g;
      const ulonglong2 lo = q2[0], hi = q2[4];
      const uint64_t qv[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (METRIC == SONG_METRIC_L2) {
          const uint64_t d = f2_sub(qv[i], x[i]);
          acc[a][i] = f2_fma(d, d, acc[a][i]);
        } else {
          acc[a][i] = f2_fma(qv[i], x[i], acc[a][i]);
        }
      }
    }
    if (METRIC == SONG_METRIC_COS) {
#pragma unroll
      for (int i = 0; i < 4; ++i) len[i] = f2_fma(x[i], x[i], len[i]);
    }
  };
  constexpr int U = NQ == 1 ? 4 : 2;  // 32-float steps in flight
  int j = 0;
  for (; j + 32 * U <= dpad; j += 32 * U) {
    RowRead<0> r[U];
#pragma unroll
    for (int i = 0; i < U; ++i) r[i].load_full(x8, j + 32 * i, g);
#pragma unroll
    for (int i = 0; i < U; ++i) add(r[i], j + 32 * i);
  }
  for (; j < dpad; j += 32) {
    RowRead<0> r;
    r.load(x8, j, g, dpad);
    add(r, j);
  }
  const float ln = METRIC == SONG_METRIC_COS ? row_butterfly<true>(len, lane) : 0.0f;
#pragma unroll
  for (int a = 0; a < NQ; ++a) out[a] = finish_distance<METRIC>(row_butterfly<true>(acc[a], lane), ln);
}

// Stages n (<= NQ) query rows, gathered through row(a), zero-padded to qs
// floats (a multiple of 32); the missing ones repeat the first.
template <int NQ, class Row>
__device__ __forceinline__ void stage_queries(float *q, int qs, int dim, int n, int tid, int nthreads, Row row) {
#pragma unroll
  for (int a = 0; a < NQ; ++a) {
    const float *src = row(a < n ? a : 0);
    for (int j = tid; j < qs; j += nthreads) q[a * qs + j] = j < dim ? src[j] : 0.0f;
  }
}

// Distances of a tile of four queries (staged qs floats apart, zero-padded to
// a multiple of 32) x the eight rows from `row` on, `last` the index of the
// last one there is (rows past it repeat it): lane l gets query l >> 3 to row
// l & 7.  Lane l of the warp keeps partial l of all 32 pairs, so that a
// dimension costs the lane eight loads from global memory and four from
// shared memory for 32 pairs -- rows8_distance's 16-byte query loads, one per
// pair and four dimensions, would take four times the shared-memory
// bandwidth -- and the pairs meet in one transposed butterfly.
template <int METRIC>
__device__ __forceinline__ float tile_distance(const float *q, int qs, const float *row, int last, int dpad,
                                               int lane) {
  constexpr bool COS = METRIC == SONG_METRIC_COS;
  uint64_t acc[4][4], ln[4];  // query a, rows (2p, 2p + 1)
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    ln[p] = 0ull;
#pragma unroll
    for (int a = 0; a < 4; ++a) acc[a][p] = 0ull;
  }
  int off[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) off[i] = min(i, last) * dpad;
  auto add = [&](const float (&x)[8], int j) {
    uint64_t xx[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) xx[p] = f2_pack(x[2 * p], x[2 * p + 1]);
#pragma unroll
    for (int a = 0; a < 4; ++a) {
      const float qv = q[a * qs + j];
      const uint64_t qq = f2_pack(qv, qv);
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        if (METRIC == SONG_METRIC_L2) {
          const uint64_t d = f2_sub(qq, xx[p]);
          acc[a][p] = f2_fma(d, d, acc[a][p]);
        } else {
          acc[a][p] = f2_fma(qq, xx[p], acc[a][p]);
        }
      }
    }
    if (COS) {
#pragma unroll
      for (int p = 0; p < 4; ++p) ln[p] = f2_fma(xx[p], xx[p], ln[p]);
    }
  };
  constexpr int U = 4;  // 32-float steps in flight
  int j = lane;
  for (; j - lane + 32 * U <= dpad; j += 32 * U) {
    float x[U][8];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int i = 0; i < 8; ++i) x[u][i] = __ldg(row + off[i] + j + 32 * u);
#pragma unroll
    for (int u = 0; u < U; ++u) add(x[u], j + 32 * u);
  }
  for (; j - lane < dpad; j += 32) {
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = j < dpad ? __ldg(row + off[i] + j) : 0.0f;
    add(x, j);
  }
  float v[32];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int p = 0; p < 4; ++p) f2_unpack(acc[a][p], v[8 * a + 2 * p], v[8 * a + 2 * p + 1]);
  const float t = butterfly_rows<32>(v, lane);  // pair `lane`
  float len = 0.0f;
  if (COS) {
    float lv[8];
#pragma unroll
    for (int p = 0; p < 4; ++p) f2_unpack(ln[p], lv[2 * p], lv[2 * p + 1]);
    const float lsum = butterfly_rows<8>(lv, lane);  // row lane / 4
    len = __shfl_sync(FULL, lsum, 4 * (lane & 7));   // row lane & 7
  }
  return finish_distance<METRIC>(t, len);
}

template <int N>
__device__ __forceinline__ void clear_list(float (&bd)[N], uint32_t (&bi)[N]) {
#pragma unroll
  for (int m = 0; m < N; ++m) {
    bd[m] = __int_as_float(0x7f800000);
    bi[m] = 0xffffffffu;
  }
}

// Rows first .. first + 7, first + step, ... below end against one query: the
// first of a row's four lanes keeps it in its list.  id(row) names a row.
template <int METRIC, int N, class Id>
__device__ __forceinline__ void scan_rows(const float *rows, int dpad, int first, int step, int end, const float *q,
                                          int qs, float (&bd)[N], uint32_t (&bi)[N], int lane, Id id) {
  for (int r0 = first; r0 < end; r0 += step) {
    const int row = r0 + (lane >> 2);
    const int at = min(row, end - 1);
    float d[1];
    rows8_distance<METRIC, 1>(rows + static_cast<size_t>(at) * dpad, q, qs, dpad, d, lane);
    if (row < end && (lane & 3) == 0) list_insert<N>(bd, bi, d[0], id(at));
  }
  __syncwarp();
}

}  // namespace song
