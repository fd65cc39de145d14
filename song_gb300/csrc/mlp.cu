// mlp.cu -- training of the early-exit network (no counterpart in the
// reference).  Network 5 -> 32 -> 32 -> 1 with ReLU, trained with a weighted
// binary cross-entropy on logits by hand-written kernels, two a step:
//
//   chunk_kernel     a block of 16 warps per chunk of 32 samples: each warp
//                    runs two samples forward and backward, lane j owning
//                    hidden unit j of both layers; then each thread sums its
//                    parameters' gradient over the chunk's samples in order.
//                    One partial gradient per chunk (no atomics, so results
//                    are deterministic).
//   update_kernel    sums the partial gradients in chunk order, scales by
//                    1 / (sum of sample weights in the batch) and, in
//                    training, applies Adam to the FP32 parameters.
//
// What bounds a step is latency: 256 chunks at batch 8192 are a fraction of a
// wave.  Batch 8192, 6 epochs of 300,001 samples: 12.2 ms with a warp per
// chunk, its samples one after another, and a third launch for Adam; 4.8 with
// eight warps a chunk; 4.4 with 16 and the update's loads in flight together;
// 3.4 (14 us a step) with programmatic dependence between the launches.
//
// Parameter layout (MLP_NPARAM FP32): W1[32][5], b1[32], W2[32][32], b2[32],
// w3[32], b3 -- the same layout the search kernel reads (as BF16).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "internal.h"
#include "search_kernel.cuh"
#include "song_gb300.h"

namespace song {
namespace {

constexpr int CHUNK = 32;         // samples per block per step
constexpr int CHUNK_WARPS = 16;
constexpr int PER_WARP = CHUNK / CHUNK_WARPS;
constexpr int PARTIAL = MLP_NPARAM + 2;  // gradient + loss + weight sum

// The kernels of a step are launched with programmatic dependence: one may
// start, and load what does not depend on it, before the kernel ahead has
// ended; it waits here for that kernel's end (and so for all earlier ones')
// before it reads or writes anything they share.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

struct Samples {
  const float *x, *y, *w;  // n x MLP_IN; labels; weights (null: 1)
  const int32_t *idx;      // order (null: as they come)
};

// One sample's forward pass in a warp: lane j's hidden units and the logit.
// w1, b1 .. : lane j's parameters; w2r: its row of W2; hs: 32 floats of the
// warp's own shared memory for the first layer.
__device__ __forceinline__ float forward(const float (&xi)[MLP_IN], const float (&w1)[MLP_IN], float b1,
                                         const float (&w2r)[MLP_H], float b2, float w3, float b3, float *hs,
                                         float &a1, float &h1, float &a2, float &h2, int lane) {
  a1 = b1;
#pragma unroll
  for (int i = 0; i < MLP_IN; ++i) a1 = fmaf(w1[i], xi[i], a1);
  h1 = fmaxf(a1, 0.0f);
  hs[lane] = h1;
  __syncwarp();
  a2 = b2;
#pragma unroll
  for (int i = 0; i < MLP_H; i += 4) {
    const float4 h = *reinterpret_cast<const float4 *>(hs + i);
    a2 = fmaf(w2r[i], h.x, a2);
    a2 = fmaf(w2r[i + 1], h.y, a2);
    a2 = fmaf(w2r[i + 2], h.z, a2);
    a2 = fmaf(w2r[i + 3], h.w, a2);
  }
  h2 = fmaxf(a2, 0.0f);
  float z = __fmul_rn(w3, h2);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) z = __fadd_rn(z, __shfl_xor_sync(FULL, z, o));
  return __fadd_rn(z, b3);
}

// Stages W2 with rows padded to 33 floats (its rows and its columns are then
// read without bank conflicts) and loads the lane's other parameters.
__device__ __forceinline__ void stage_w2(const float *params, float *w2, int tid, int nthreads) {
  for (int i = tid; i < MLP_H * MLP_H; i += nthreads) w2[(i >> 5) * 33 + (i & 31)] = params[MLP_W2 + i];
}

__global__ void __launch_bounds__(CHUNK_WARPS * 32, 2)
    chunk_kernel(const Samples in, int64_t first, int64_t count, const float *params, float *partial) {
  __shared__ __align__(16) float w2[MLP_H * 33];
  // per sample of the chunk: both layers' outputs, the deltas, the inputs
  __shared__ __align__(16) float h1s[CHUNK][MLP_H], h2s[CHUNK][MLP_H], d1s[CHUNK][MLP_H], d2s[CHUNK][MLP_H];
  __shared__ float xs[CHUNK][MLP_IN], dzs[CHUNK], wws[CHUNK], ls[CHUNK];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t s0 = static_cast<int64_t>(blockIdx.x) * CHUNK;
  const int n = static_cast<int>(min(static_cast<int64_t>(CHUNK), count - s0));
  // the samples first: two dependent loads that the parameters' staging hides
  float xi2[PER_WARP][MLP_IN], yy2[PER_WARP], ww2[PER_WARP];
#pragma unroll
  for (int k = 0; k < PER_WARP; ++k) {
    const int s = min(warp + k * CHUNK_WARPS, n - 1);
    const int64_t r = in.idx ? static_cast<int64_t>(in.idx[first + s0 + s]) : first + s0 + s;
#pragma unroll
    for (int i = 0; i < MLP_IN; ++i) xi2[k][i] = in.x[r * MLP_IN + i];
    yy2[k] = in.y[r];
    ww2[k] = in.w ? in.w[r] : 1.0f;
  }
  after_previous();
  stage_w2(params, w2, tid, blockDim.x);
  float w1[MLP_IN];
#pragma unroll
  for (int i = 0; i < MLP_IN; ++i) w1[i] = params[MLP_W1 + lane * MLP_IN + i];
  const float b1 = params[MLP_B1 + lane], b2 = params[MLP_B2 + lane];
  const float w3 = params[MLP_W3 + lane], b3 = params[MLP_B3];
  __syncthreads();
  float w2r[MLP_H];
#pragma unroll
  for (int i = 0; i < MLP_H; ++i) w2r[i] = w2[lane * 33 + i];
#pragma unroll
  for (int k = 0; k < PER_WARP; ++k) {
    const int s = warp + k * CHUNK_WARPS;
    if (s >= n) break;
    const float(&xi)[MLP_IN] = xi2[k];
    const float yy = yy2[k], ww = ww2[k];
    float a1, h1, a2, h2;
    const float z = forward(xi, w1, b1, w2r, b2, w3, b3, h1s[s], a1, h1, a2, h2, lane);
    // weighted BCE on the logit: softplus(z) - y z; d/dz = sigmoid(z) - y
    const float sp = fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z)));
    const float p = 1.0f / (1.0f + expf(-z));
    const float dz = ww * (p - yy);
    const float da2 = a2 > 0.0f ? dz * w3 : 0.0f;
    h2s[s][lane] = h2;
    d2s[s][lane] = da2;
    __syncwarp();
    float dh1 = 0.0f;
#pragma unroll
    for (int i = 0; i < MLP_H; i += 4) {  // column `lane` of W2
      const float4 d = *reinterpret_cast<const float4 *>(d2s[s] + i);
      dh1 = fmaf(w2[i * 33 + lane], d.x, dh1);
      dh1 = fmaf(w2[(i + 1) * 33 + lane], d.y, dh1);
      dh1 = fmaf(w2[(i + 2) * 33 + lane], d.z, dh1);
      dh1 = fmaf(w2[(i + 3) * 33 + lane], d.w, dh1);
    }
    d1s[s][lane] = a1 > 0.0f ? dh1 : 0.0f;
    if (lane < MLP_IN) {
      float v = xi[0];
#pragma unroll
      for (int i = 1; i < MLP_IN; ++i) v = lane == i ? xi[i] : v;
      xs[s][lane] = v;
    }
    if (lane == 0) {
      dzs[s] = dz;
      wws[s] = ww;
      ls[s] = fmaf(-yy, z, sp);
    }
  }
  __syncthreads();
  // every parameter's sum over the chunk's samples, in order
  float *out = partial + static_cast<int64_t>(blockIdx.x) * PARTIAL;
  if (tid < 256) {
    const int j = tid >> 3, i = (tid & 7) * 4;  // W2[j][i .. i + 3]
    float g[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
    for (int s = 0; s < n; ++s) {
      const float d = d2s[s][j];
      const float4 h = *reinterpret_cast<const float4 *>(&h1s[s][i]);
      g[0] = fmaf(d, h.x, g[0]);
      g[1] = fmaf(d, h.y, g[1]);
      g[2] = fmaf(d, h.z, g[2]);
      g[3] = fmaf(d, h.w, g[3]);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) out[MLP_W2 + j * MLP_H + i + e] = g[e];
  }
  if (tid < 256) return;
  const int u = tid - 256;  // the other half of the block: the rest
  float g = 0.0f;
  if (u < 160) {
    const int j = u / MLP_IN, i = u - j * MLP_IN;
#pragma unroll 4
    for (int s = 0; s < n; ++s) g = fmaf(d1s[s][j], xs[s][i], g);
    out[MLP_W1 + u] = g;
  } else if (u < 192) {
#pragma unroll 4
    for (int s = 0; s < n; ++s) g = __fadd_rn(g, d1s[s][lane]);
    out[MLP_B1 + lane] = g;
  } else if (u < 224) {
#pragma unroll 4
    for (int s = 0; s < n; ++s) g = __fadd_rn(g, d2s[s][lane]);
    out[MLP_B2 + lane] = g;
  } else {
#pragma unroll 4
    for (int s = 0; s < n; ++s) g = fmaf(dzs[s], h2s[s][lane], g);
    out[MLP_W3 + lane] = g;
  }
  if (u < 3) {
    g = 0.0f;
    for (int s = 0; s < n; ++s)
      g = u == 0 ? __fadd_rn(g, dzs[s]) : (u == 1 ? fmaf(wws[s], ls[s], g) : __fadd_rn(g, wws[s]));
    out[MLP_B3 + u] = g;  // b3, then the loss, then the weight sum
  }
}

// Logits of n samples, a warp each.
__global__ void logits_kernel(const float *__restrict__ x, int64_t n, const float *__restrict__ params,
                              float *__restrict__ logits) {
  __shared__ __align__(16) float w2[MLP_H * 33], hs[4][MLP_H];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  stage_w2(params, w2, threadIdx.x, blockDim.x);
  float w1[MLP_IN], w2r[MLP_H];
#pragma unroll
  for (int i = 0; i < MLP_IN; ++i) w1[i] = params[MLP_W1 + lane * MLP_IN + i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < MLP_H; ++i) w2r[i] = w2[lane * 33 + i];
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * 4 + warp; r < n; r += static_cast<int64_t>(gridDim.x) * 4) {
    float xi[MLP_IN], a1, h1, a2, h2;
#pragma unroll
    for (int i = 0; i < MLP_IN; ++i) xi[i] = x[r * MLP_IN + i];
    const float z = forward(xi, w1, params[MLP_B1 + lane], w2r, params[MLP_B2 + lane], params[MLP_W3 + lane],
                            params[MLP_B3], hs[warp], a1, h1, a2, h2, lane);
    if (lane == 0) logits[r] = z;
    __syncwarp();
  }
}

// grad[p] = sum_c partial[c][p] / sum_c weight[c], the sums in chunk order;
// loss likewise.  A block takes UPD_COLS columns: it brings them to shared
// memory UPD_ROWS chunks at a time, one thread sums each.  With m, Adam's
// step on the block's parameters (grad may then be null).
constexpr int UPD_COLS = 16, UPD_ROWS = 256;

struct Adam {
  float *params, *m, *v;  // m null: no step
  float lr, b1, b2, eps, c1, c2;
};

__global__ void __launch_bounds__(256)
    update_kernel(const float *partial, int chunks, float *grad, float *loss_out, const Adam adam) {
  __shared__ float cols[UPD_ROWS][UPD_COLS + 1];  // the last column: the chunks' weight sums
  __shared__ float wtot;
  const int tid = threadIdx.x, c0 = blockIdx.x * UPD_COLS, p = c0 + tid;
  const bool step = adam.m && tid < UPD_COLS && p < MLP_NPARAM;
  after_previous();
  float pm = 0.0f, pv = 0.0f, pp = 0.0f;
  if (step) {
    pm = adam.m[p];
    pv = adam.v[p];
    pp = adam.params[p];
  }
  // this thread brings column tid % 16 of rows tid / 16, + 16, ..., and the
  // weight sum of row tid: all loads in flight together
  constexpr int PER = UPD_ROWS * UPD_COLS / 256;
  const int col = tid & (UPD_COLS - 1), row = tid / UPD_COLS;
  float t = 0.0f;
  for (int base = 0; base < chunks; base += UPD_ROWS) {
    const int n = min(UPD_ROWS, chunks - base);
    const float *src = partial + static_cast<int64_t>(base) * PARTIAL;
    float x[PER], wsum = 0.0f;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int r = row + k * (256 / UPD_COLS);
      x[k] = r < n && c0 + col <= MLP_NPARAM ? src[static_cast<int64_t>(r) * PARTIAL + c0 + col] : 0.0f;
    }
    if (tid < n) wsum = src[static_cast<int64_t>(tid) * PARTIAL + MLP_NPARAM + 1];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < PER; ++k) cols[row + k * (256 / UPD_COLS)][col] = x[k];
    cols[tid][UPD_COLS] = wsum;
    __syncthreads();
    if (tid <= UPD_COLS)
#pragma unroll 16
      for (int r = 0; r < n; ++r) t = __fadd_rn(t, cols[r][tid]);
  }
  if (tid == UPD_COLS) wtot = t > 0.0f ? t : 1.0f;
  __syncthreads();
  if (tid >= UPD_COLS || p > MLP_NPARAM) return;
  const float g = __fdiv_rn(t, wtot);
  if (p == MLP_NPARAM) {
    if (loss_out) *loss_out = g;
    return;
  }
  if (grad) grad[p] = g;
  if (!step) return;
  const float mi = fmaf(1.0f - adam.b1, g, __fmul_rn(adam.b1, pm));
  const float vi = fmaf(__fmul_rn(1.0f - adam.b2, g), g, __fmul_rn(adam.b2, pv));
  adam.m[p] = mi;
  adam.v[p] = vi;
  adam.params[p] = pp - adam.lr * (mi / adam.c1) / (sqrtf(vi / adam.c2) + adam.eps);
}

// Mean of the steps' losses, summed in FP64 in order.
__global__ void mean_loss_kernel(const float *loss, int64_t steps, float *out) {
  double acc = 0.0;
  for (int64_t i = 0; i < steps; ++i) acc = __dadd_rn(acc, static_cast<double>(loss[i]));
  *out = static_cast<float>(acc / static_cast<double>(steps));
}

int64_t chunks_of(int64_t count) { return (count + CHUNK - 1) / CHUNK; }

cudaError_t run_step(const Samples &in, int64_t first, int64_t count, const float *params, float *partial,
                     float *grad, float *loss, const Adam &adam, cudaStream_t s) {
  const int64_t chunks = chunks_of(count);
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  cfg.gridDim = dim3(static_cast<unsigned>(chunks));
  cfg.blockDim = dim3(CHUNK_WARPS * 32);
  cudaError_t e = cudaLaunchKernelEx(&cfg, chunk_kernel, in, first, count, params, partial);
  if (e != cudaSuccess) return e;
  cfg.gridDim = dim3((MLP_NPARAM + UPD_COLS) / UPD_COLS);
  cfg.blockDim = dim3(256);
  e = cudaLaunchKernelEx(&cfg, update_kernel, static_cast<const float *>(partial), static_cast<int>(chunks), grad, loss,
                         adam);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

}  // namespace
}  // namespace song

using song::MLP_NPARAM;

extern "C" {

int song_mlp_train_device(const float *d_x, const float *d_y, const float *d_w, int64_t n,
                          const int32_t *d_perm, int epochs, int batch, float lr, float *d_params,
                          float *d_loss, void *stream) {
  song::clear_error();
  if (!d_x || !d_y || !d_params || n < 1 || epochs < 1 || batch < 1 || lr <= 0.0f)
    return song::fail(SONG_ERR_ARG, "bad training arguments");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t steps = (n + batch - 1) / batch;
  // one block: partial gradients, Adam's moments, the epoch's step losses
  const int64_t words = song::chunks_of(batch) * song::PARTIAL;
  float *work = nullptr;
  cudaError_t e = song::dev_malloc(&work, sizeof(float) * (words + 2 * MLP_NPARAM + steps));
  float *partial = work, *m = work + words, *v = m + MLP_NPARAM, *lossbuf = v + MLP_NPARAM;
  if (e == cudaSuccess) e = cudaMemsetAsync(m, 0, sizeof(float) * 2 * MLP_NPARAM, s);
  song::Adam adam{d_params, m, v, lr, 0.9f, 0.999f, 1e-8f, 0.0f, 0.0f};
  int64_t t = 0;
  for (int ep = 0; ep < epochs && e == cudaSuccess; ++ep) {
    const song::Samples in{d_x, d_y, d_w, d_perm ? d_perm + static_cast<int64_t>(ep) * n : nullptr};
    for (int64_t st = 0; st < steps && e == cudaSuccess; ++st) {
      const int64_t first = st * batch;
      const int64_t count = first + batch <= n ? batch : n - first;
      ++t;
      adam.c1 = 1.0f - std::pow(adam.b1, static_cast<float>(t));
      adam.c2 = 1.0f - std::pow(adam.b2, static_cast<float>(t));
      e = song::run_step(in, first, count, d_params, partial, nullptr, lossbuf + st, adam, s);
    }
    if (e == cudaSuccess && d_loss) {
      song::mean_loss_kernel<<<1, 1, 0, s>>>(lossbuf, steps, d_loss + ep);
      e = cudaGetLastError();
    }
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  cudaFree(work);
  if (e != cudaSuccess)
    return song::fail(e == cudaErrorMemoryAllocation ? SONG_ERR_OOM : SONG_ERR_CUDA, "mlp training: %s",
                      cudaGetErrorString(e));
  return SONG_OK;
}

int song_mlp_grad(const float *x, const float *y, const float *w, int n, const float *params,
                  float *grad_out, float *loss_out) {
  song::clear_error();
  if (!x || !y || !params || !grad_out || n < 1) return song::fail(SONG_ERR_ARG, "bad arguments");
  float *dx = nullptr, *dy = nullptr, *dw = nullptr, *dp = nullptr, *partial = nullptr, *grad = nullptr,
        *loss = nullptr;
  cudaError_t e = song::dev_malloc(&dx, sizeof(float) * n * song::MLP_IN);
  if (e == cudaSuccess) e = song::dev_malloc(&dy, sizeof(float) * n);
  if (e == cudaSuccess && w) e = song::dev_malloc(&dw, sizeof(float) * n);
  if (e == cudaSuccess) e = song::dev_malloc(&dp, sizeof(float) * MLP_NPARAM);
  if (e == cudaSuccess) e = song::dev_malloc(&partial, sizeof(float) * song::chunks_of(n) * song::PARTIAL);
  if (e == cudaSuccess) e = song::dev_malloc(&grad, sizeof(float) * MLP_NPARAM);
  if (e == cudaSuccess) e = song::dev_malloc(&loss, sizeof(float));
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, sizeof(float) * n * song::MLP_IN, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dy, y, sizeof(float) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess && w) e = cudaMemcpy(dw, w, sizeof(float) * n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dp, params, sizeof(float) * MLP_NPARAM, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    e = song::run_step(song::Samples{dx, dy, dw, nullptr}, 0, n, dp, partial, grad, loss, song::Adam{}, 0);
  }
  if (e == cudaSuccess) e = cudaMemcpy(grad_out, grad, sizeof(float) * MLP_NPARAM, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && loss_out) e = cudaMemcpy(loss_out, loss, sizeof(float), cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dy);
  cudaFree(dw);
  cudaFree(dp);
  cudaFree(partial);
  cudaFree(grad);
  cudaFree(loss);
  if (e != cudaSuccess) return song::fail(SONG_ERR_CUDA, "mlp grad: %s", cudaGetErrorString(e));
  return SONG_OK;
}

int song_mlp_forward(const float *x, int n, const float *params, float *logits_out) {
  song::clear_error();
  if (!x || !params || !logits_out || n < 1) return song::fail(SONG_ERR_ARG, "bad arguments");
  float *dx = nullptr, *dp = nullptr, *dl = nullptr;
  cudaError_t e = song::dev_malloc(&dx, sizeof(float) * n * song::MLP_IN);
  if (e == cudaSuccess) e = song::dev_malloc(&dp, sizeof(float) * MLP_NPARAM);
  if (e == cudaSuccess) e = song::dev_malloc(&dl, sizeof(float) * n);
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, sizeof(float) * n * song::MLP_IN, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dp, params, sizeof(float) * MLP_NPARAM, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    song::logits_kernel<<<static_cast<unsigned>(std::min<int64_t>((static_cast<int64_t>(n) + 3) / 4, 4096)), 128>>>(dx, n, dp, dl);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(logits_out, dl, sizeof(float) * n, cudaMemcpyDeviceToHost);
  cudaFree(dx);
  cudaFree(dp);
  cudaFree(dl);
  if (e != cudaSuccess) return song::fail(SONG_ERR_CUDA, "mlp forward: %s", cudaGetErrorString(e));
  return SONG_OK;
}

}  // extern "C"
