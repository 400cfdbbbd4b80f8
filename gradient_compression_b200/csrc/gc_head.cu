// The classifier head of the CIFAR models as one forward kernel and two backward kernels: global average pool over the
// last feature map, linear layer, softmax cross-entropy (mean over the batch) and the batch's top-1 / top-5 hit rates.
// The reference runs avg_pool2d + nn.Linear + CrossEntropyLoss + a second CrossEntropyLoss + topk / eq / sum with three
// .item() reads (models/resnet.py:106-108, model_dispatcher.py:127-128,140-164 of the reference): about twenty small
// kernels and three device synchronisations per step.  Here the metrics stay on the device.
//
//   head_fwd_kernel      one block per sample: pooled[n, :] = mean over positions of x[n, :, :] (NHWC), logits = pooled W^T + b,
//                        log-softmax, loss_n, rank of the true class; dlogits[n, :] = (softmax - onehot) / N is written for the
//                        backward pass.  The block that draws the last ticket adds the per-sample values in sample order
//                        (deterministic) into out[0:3] = {mean loss, top-1 rate, top-5 rate}.
//   head_bwd_dx_kernel   dx[n, p, c] = g * sum_k dlogits[n, k] W[k, c] / positions, the same value at every position
//   head_bwd_dw_kernel   dW[k, c] = g * sum_n dlogits[n, k] pooled[n, c], db[k] = g * sum_n dlogits[n, k]
//   head_eval_kernel     inference: pooling and linear layer only (labels come later, with evaluate_predictions)
//   logit_metrics_kernel cross-entropy, top-1 and top-5 of given logits, one block, one thread per sample: a dozen torch launches
//                        took 66 of 470 microseconds of a small evaluation batch, and more of its host time.  Bound by the latency of
//                        rows read by a thread each, so for small batches or few classes (ops/head.py has the line and its figures)
// g is the gradient that reaches the loss (a device scalar, 1 for a plain loss.backward()).
#include <cuda_runtime.h>
#include <stdint.h>

#include "gc_device.cuh"

using namespace gc;

namespace {

constexpr int HEAD_THREADS = 256;
constexpr int HEAD_MAX_CLASSES = 32;
constexpr int HEAD_MAX_CHANNELS = 4096;

struct HeadShared {
  float __align__(16) pooled[HEAD_MAX_CHANNELS];
  float logit[HEAD_MAX_CLASSES];
  float part[HEAD_THREADS / 32][HEAD_MAX_CLASSES];
};

// Pooling and linear layer of sample n, by a whole block: sh.logit[0:K].  pooled (may be NULL), logits: of all samples.
__device__ __forceinline__ void pooled_logits(HeadShared& sh, const float* __restrict__ x, int n, int positions, int C, const float* __restrict__ W,
                                              const float* __restrict__ bias, int K, float* __restrict__ pooled, float* __restrict__ logits) {
  const float* xn = x + (int64_t)n * positions * C;
  const float inv_pos = 1.0f / (float)positions;
  for (int q = threadIdx.x; q < (C >> 2); q += HEAD_THREADS) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 16
    for (int p = 0; p < positions; ++p) {
      const float4 v = *reinterpret_cast<const float4*>(xn + (int64_t)p * C + 4 * q);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    acc.x *= inv_pos; acc.y *= inv_pos; acc.z *= inv_pos; acc.w *= inv_pos;
    *reinterpret_cast<float4*>(sh.pooled + 4 * q) = acc;
    if (pooled != nullptr) *reinterpret_cast<float4*>(pooled + (int64_t)n * C + 4 * q) = acc;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // every warp takes 128-channel slices of the pooled vector and all K classes at once (K independent 16-byte loads of
  // W in flight per lane); the eight warps' partial dot products meet in shared memory in a fixed order
  float acc[HEAD_MAX_CLASSES];
#pragma unroll
  for (int k = 0; k < HEAD_MAX_CLASSES; ++k) acc[k] = 0.f;
  for (int c = warp * 128 + lane * 4; c < C; c += (HEAD_THREADS / 32) * 128) {
    const float4 pv = *reinterpret_cast<const float4*>(sh.pooled + c);
#pragma unroll
    for (int k = 0; k < HEAD_MAX_CLASSES; ++k)
      if (k < K) {
        const float4 wv = *reinterpret_cast<const float4*>(W + (int64_t)k * C + c);
        acc[k] = fmaf(pv.x, wv.x, fmaf(pv.y, wv.y, fmaf(pv.z, wv.z, fmaf(pv.w, wv.w, acc[k]))));
      }
  }
#pragma unroll
  for (int k = 0; k < HEAD_MAX_CLASSES; ++k)
    if (k < K) {
      const float v = warp_sum(acc[k]);
      if (lane == 0) sh.part[warp][k] = v;
    }
  __syncthreads();
  if (threadIdx.x < K) {
    float v = bias != nullptr ? bias[threadIdx.x] : 0.f;
#pragma unroll
    for (int w = 0; w < HEAD_THREADS / 32; ++w) v += sh.part[w][threadIdx.x];
    sh.logit[threadIdx.x] = v;
    logits[(int64_t)n * K + threadIdx.x] = v;
  }
}

__global__ void __launch_bounds__(HEAD_THREADS) head_eval_kernel(const float* __restrict__ x, int positions, int C, const float* __restrict__ W,
                                                                 const float* __restrict__ bias, int K, float* __restrict__ logits) {
  __shared__ HeadShared sh;
  pooled_logits(sh, x, blockIdx.x, positions, C, W, bias, K, nullptr, logits);
}

// out = {mean cross-entropy, top-1 rate, top-5 rate} of logits[N, K].  Samples labelled -100 do not count in the loss
// (nn.CrossEntropyLoss's ignore_index); any other label outside the classes makes it NaN.  A NaN ranks above every number and
// ties go to the lower class.
constexpr int METRIC_THREADS = 1024, METRIC_MAX_CLASSES = 1024;
__global__ void __launch_bounds__(METRIC_THREADS) logit_metrics_kernel(const float* __restrict__ logits, const int64_t* __restrict__ labels, int N, int K,
                                                                       float* __restrict__ out) {
  __shared__ double part[METRIC_THREADS / 32][4];
  double loss = 0.0;
  int counted = 0, top1 = 0, top5 = 0;
  for (int n = threadIdx.x; n < N; n += METRIC_THREADS) {
    const float* z = logits + (int64_t)n * K;
    const int64_t label = labels[n];
    const bool known = label >= 0 && label < K;
    const float zl = known ? z[label] : NAN;
    float zmax = -INFINITY;
    int ahead = 0;
#pragma unroll 8
    for (int k = 0; k < K; ++k) {
      const float v = z[k];
      zmax = fmaxf(zmax, v);
      ahead += v > zl || (isnan(v) && !isnan(zl)) || ((v == zl || (isnan(v) && isnan(zl))) && k < label);
    }
    float sum = 0.f;
#pragma unroll 8
    for (int k = 0; k < K; ++k) sum += expf(z[k] - zmax);
    if (label != -100) {
      loss += (double)(logf(sum) + zmax - zl);
      ++counted;
    }
    top1 += known && ahead == 0;
    top5 += known && ahead < 5;
  }
  double v[4] = {loss, (double)counted, (double)top1, (double)top5};
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    for (int o = 16; o > 0; o >>= 1) v[j] += __shfl_xor_sync(FULL, v[j], o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5][j] = v[j];
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = 0.0;
    for (int w = 0; w < (int)blockDim.x / 32; ++w) t += part[w][threadIdx.x];
    part[0][threadIdx.x] = t;
  }
  __syncwarp();
  if (threadIdx.x == 0) out[0] = (float)(part[0][0] / part[0][1]);
  if (threadIdx.x == 1 || threadIdx.x == 2) out[threadIdx.x] = (float)part[0][threadIdx.x + 1] * (1.0f / (float)N);     // as a tensor divided by a number
}

__global__ void __launch_bounds__(HEAD_THREADS) head_fwd_kernel(const float* __restrict__ x, int positions, int C,
                                                                const float* __restrict__ W, const float* __restrict__ bias, int K,
                                                                const int64_t* __restrict__ labels, int N,
                                                                float* __restrict__ pooled, float* __restrict__ logits,
                                                                float* __restrict__ dlogits, float* __restrict__ per_sample,
                                                                unsigned int* __restrict__ ticket, float* __restrict__ out3, float* __restrict__ loss) {
  __shared__ HeadShared sh;
  __shared__ int last;
  const int n = blockIdx.x;
  pdl_wait();
  pdl_launch_dependents();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int label = warp == 0 ? (int)labels[n] : 0;                // on its way while the block pools
  pooled_logits(sh, x, n, positions, C, W, bias, K, pooled, logits);
  __syncthreads();
  if (warp == 0) {
    const float z = lane < K ? sh.logit[lane] : -INFINITY;
    const float zmax = warp_max(z);
    const float e = lane < K ? __expf(z - zmax) : 0.f;
    const float denom = warp_sum(e);
    const float zl = (label >= 0 && label < K) ? sh.logit[label] : 0.f;
    // position of the true class in the descending order (ties go to the lower class index, as a stable sort would)
    const int ahead = (lane < K && (z > zl || (z == zl && lane < label))) ? 1 : 0;
    const int rank = __reduce_add_sync(FULL, ahead);
    if (lane < K) dlogits[(int64_t)n * K + lane] = (e / denom - (lane == label ? 1.f : 0.f)) / (float)N;
    if (lane == 0) {
      per_sample[3 * n] = __logf(denom) + zmax - zl;
      per_sample[3 * n + 1] = rank == 0 ? 1.f : 0.f;
      per_sample[3 * n + 2] = rank < 5 ? 1.f : 0.f;
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(ticket, 1u) == gridDim.x - 1u ? 1 : 0;
  __syncthreads();
  if (!last) return;
  __threadfence();
  if (warp < 3) {                          // one warp per value: a single thread's N loads in a row took 3 us at 128 samples
    float acc = 0.f;
    for (int i = lane; i < N; i += 32) acc += __ldcg(per_sample + 3 * i + warp);
    acc = warp_sum(acc);
    if (lane == 0) {
      out3[warp] = acc / (float)N;
      if (warp == 0 && loss != nullptr) *loss = acc / (float)N;
    }
  }
  if (threadIdx.x == 0) *ticket = 0u;
}

__global__ void __launch_bounds__(HEAD_THREADS) head_bwd_dx_kernel(const float* __restrict__ dlogits, const float* __restrict__ W,
                                                                   const float* __restrict__ g, int positions, int C, int K,
                                                                   float* __restrict__ dx) {
  __shared__ float sd[HEAD_MAX_CLASSES];
  const int n = blockIdx.y;
  pdl_wait();
  pdl_launch_dependents();
  if (threadIdx.x < K) sd[threadIdx.x] = dlogits[(int64_t)n * K + threadIdx.x] * (g != nullptr ? *g : 1.f) / (float)positions;
  __syncthreads();
  const int q = blockIdx.x * HEAD_THREADS + threadIdx.x;
  if (q >= (C >> 2)) return;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k = 0; k < K; ++k) {
    const float4 w = *reinterpret_cast<const float4*>(W + (int64_t)k * C + 4 * q);
    const float d = sd[k];
    acc.x = fmaf(d, w.x, acc.x); acc.y = fmaf(d, w.y, acc.y); acc.z = fmaf(d, w.z, acc.z); acc.w = fmaf(d, w.w, acc.w);
  }
  float* dn = dx + (int64_t)n * positions * C + 4 * q;
  for (int p = 0; p < positions; ++p) *reinterpret_cast<float4*>(dn + (int64_t)p * C) = acc;
}

// One block per 32 channels: warp w sums the samples w, w + 8, ... for its lane's channel and all classes, the eight partial
// sums meet in shared memory.  Bound by latency: eight samples' values are loaded together (128 samples of 512 channels, one at a time: 11 us).
// beside: the launch in front is head_bwd_dx_kernel, which writes nothing that is read here and let this one start only when the kernels before it
// were complete; the two run side by side and this one ends after the other.
constexpr int HEAD_DW_CHANNELS = 32, HEAD_DW_AHEAD = 8;

__global__ void __launch_bounds__(HEAD_THREADS) head_bwd_dw_kernel(const float* __restrict__ dlogits, const float* __restrict__ pooled,
                                                                   const float* __restrict__ g, int N, int C, int K,
                                                                   float* __restrict__ dW, float* __restrict__ db, int beside) {
  extern __shared__ float sdl[];                 // dlogits [N, K], then partial sums [8 warps][K][32 channels]
  if (!beside) pdl_wait();
  pdl_launch_dependents();
  float* part = sdl + N * K;
  for (int i = threadIdx.x; i < N * K; i += HEAD_THREADS) sdl[i] = dlogits[i];
  __syncthreads();
  const float gs = g != nullptr ? *g : 1.f;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * HEAD_DW_CHANNELS + lane;
  float acc[HEAD_MAX_CLASSES];
#pragma unroll
  for (int k = 0; k < HEAD_MAX_CLASSES; ++k) acc[k] = 0.f;
  if (c < C) {
    for (int n0 = warp; n0 < N; n0 += HEAD_DW_AHEAD * (HEAD_THREADS / 32)) {
      float pv[HEAD_DW_AHEAD];
#pragma unroll
      for (int u = 0; u < HEAD_DW_AHEAD; ++u) {
        const int n = n0 + u * (HEAD_THREADS / 32);
        pv[u] = n < N ? pooled[(int64_t)n * C + c] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < HEAD_DW_AHEAD; ++u) {
        const int n = n0 + u * (HEAD_THREADS / 32);
        if (n >= N) break;
#pragma unroll
        for (int k = 0; k < HEAD_MAX_CLASSES; ++k)
          if (k < K) acc[k] = fmaf(sdl[n * K + k], pv[u], acc[k]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < HEAD_MAX_CLASSES; ++k)
    if (k < K) part[(warp * K + k) * HEAD_DW_CHANNELS + lane] = acc[k];
  __syncthreads();
  for (int i = threadIdx.x; i < K * HEAD_DW_CHANNELS; i += HEAD_THREADS) {
    const int k = i / HEAD_DW_CHANNELS, cc = blockIdx.x * HEAD_DW_CHANNELS + (i % HEAD_DW_CHANNELS);
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < HEAD_THREADS / 32; ++w) sum += part[(w * K + k) * HEAD_DW_CHANNELS + (i % HEAD_DW_CHANNELS)];   // fixed order
    if (cc < C) dW[(int64_t)k * C + cc] = sum * gs;
  }
  if (blockIdx.x == 0 && threadIdx.x < K && db != nullptr) {
    float sum = 0.f;
#pragma unroll 8
    for (int n = 0; n < N; ++n) sum += sdl[n * K + threadIdx.x];
    db[threadIdx.x] = sum * gs;
  }
  if (beside) pdl_wait();
}

}  // namespace

extern "C" {

// 1 when the head kernels cover the shape: C a multiple of 4 up to 4096, at most 32 classes, a batch whose dlogits fit the
// backward kernel's shared memory.
int gc_cuda_head_supported(int N, int positions, int C, int K) {
  return N >= 1 && positions >= 1 && C >= 4 && (C & 3) == 0 && C <= HEAD_MAX_CHANNELS && K >= 1 && K <= HEAD_MAX_CLASSES &&
         (int64_t)N * K * 4 + (HEAD_THREADS / 32) * K * HEAD_DW_CHANNELS * 4 <= 96 * 1024 ? 1 : 0;
}

// logits [N, K] of the feature map x [N, positions, C].  C a multiple of 4 up to 4096, at most 32 classes.
int gc_cuda_head_eval(const float* x, int N, int positions, int C, const float* W, const float* bias, int K, float* logits, void* cs) {
  if (N < 1 || positions < 1 || C < 4 || (C & 3) || C > HEAD_MAX_CHANNELS || K < 1 || K > HEAD_MAX_CLASSES) return (int)cudaErrorInvalidValue;
  head_eval_kernel<<<N, HEAD_THREADS, 0, (cudaStream_t)cs>>>(x, positions, C, W, bias, K, logits);
  return (int)cudaGetLastError();
}

// out[0:3] of logits [N, K], labels [N].
int gc_cuda_logit_metrics(const float* logits, const int64_t* labels, int N, int K, float* out, void* cs) {
  if (N < 1 || K < 1 || K > METRIC_MAX_CLASSES) return (int)cudaErrorInvalidValue;
  const int threads = N < METRIC_THREADS ? (N + 31) / 32 * 32 : METRIC_THREADS;
  logit_metrics_kernel<<<1, threads, 0, (cudaStream_t)cs>>>(logits, labels, N, K, out);
  return (int)cudaGetLastError();
}

// Bytes of the zero-initialised scratch (ticket + per-sample values) for batches of up to max_batch samples.
int64_t gc_cuda_head_scratch_bytes(int max_batch) { return 256 + (int64_t)max_batch * 3 * 4; }

// x [N, positions, C] (NHWC feature map), W [K, C], bias [K] or NULL, labels [N] int64.  Writes pooled [N, C], logits [N, K],
// dlogits [N, K], out3 = {mean cross-entropy, top-1 rate, top-5 rate} and, when given, loss = out3[0] (a tensor of its own for autograd).
// scratch: gc_cuda_head_scratch_bytes(N), zeroed once.
int gc_cuda_head_forward(const float* x, int N, int positions, int C, const float* W, const float* bias, int K,
                         const int64_t* labels, float* pooled, float* logits, float* dlogits, void* scratch, float* out3, float* loss, void* cs) {
  if (!gc_cuda_head_supported(N, positions, C, K)) return (int)cudaErrorInvalidValue;
  unsigned int* ticket = static_cast<unsigned int*>(scratch);
  float* per_sample = reinterpret_cast<float*>(static_cast<uint8_t*>(scratch) + 256);
  launch_pdl(head_fwd_kernel, dim3((unsigned)N), dim3(HEAD_THREADS), 0, (cudaStream_t)cs, x, positions, C, W, bias, K, labels, N, pooled, logits, dlogits, per_sample,
             ticket, out3, loss);
  return (int)cudaGetLastError();
}

// dx [N, positions, C], dW [K, C], db [K] (NULL: no bias) from what the forward kernel saved; g: device scalar (NULL = 1).
int gc_cuda_head_backward(const float* dlogits, const float* pooled, const float* W, const float* g, int N, int positions, int C,
                          int K, float* dx, float* dW, float* db, void* cs) {
  if (!gc_cuda_head_supported(N, positions, C, K)) return (int)cudaErrorInvalidValue;
  cudaStream_t st = (cudaStream_t)cs;
  if (dx != nullptr) {
    dim3 grid((unsigned)(((C >> 2) + HEAD_THREADS - 1) / HEAD_THREADS), (unsigned)N);
    launch_pdl(head_bwd_dx_kernel, grid, dim3(HEAD_THREADS), 0, st, dlogits, W, g, positions, C, K, dx);
  }
  if (dW != nullptr) {
    static bool configured = false;
    if (!configured) {
      cudaFuncSetAttribute(head_bwd_dw_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
      configured = true;
    }
    const size_t smem = (size_t)N * K * 4 + (size_t)(HEAD_THREADS / 32) * K * HEAD_DW_CHANNELS * 4;
    launch_pdl(head_bwd_dw_kernel, dim3((unsigned)((C + HEAD_DW_CHANNELS - 1) / HEAD_DW_CHANNELS)), dim3(HEAD_THREADS), smem, st, dlogits, pooled, g, N, C, K, dW, db,
               dx != nullptr ? 1 : 0);
  }
  return (int)cudaGetLastError();
}

}  // extern "C"
