// Batch norm (+ residual) (+ ReLU) (+ 2x2 max-pool) of NHWC fp32 activations in ONE launch per direction.
//
//   bn_fused_fwd_kernel   batch statistics (from the convolution's partial sums, or from the activation itself), running
//                         statistics, and the apply pass
//   bn_fused_bwd_kernel   both gradient sums, and the input gradient (+ the residual's)
//
// The activation [M, C] is cut into G = C / 32 groups of 32 channels (128 bytes of a row) times R runs of rows, G * R blocks of
// 1024 threads, one per SM at most.  A channel's totals only need the R blocks of its group: they leave 64 partial sums each and
// meet at a barrier of their own (monotonic arrival counts, bounded waits), so nothing is added up across the whole grid
// and no second or third kernel is launched: a reduction, a finalize and an apply kernel took about 4 microseconds of launch and
// drain a layer for work that is 3 to 20.  A thread keeps its four channels for the whole kernel, parameters in registers.
//
// What bounds it: DRAM.  The backward reads dy and x (and the saved output behind a residual) twice and writes dx (and the
// residual's gradient); the second reading runs over the block's rows backwards, and is served by the 126 MB L2 for
// everything but the widest first-stage layers.
#include <cuda_runtime.h>
#include <stdint.h>

#include "gc_device.cuh"

using namespace gc;

namespace {

constexpr int THREADS = 1024, CH = 32, QUADS = CH / 4, LANES = THREADS / QUADS;       // 128 rows at once
constexpr int MAX_BLOCKS = 148;          // groups x runs of rows; also the most groups
constexpr int VALUES = 2 * CH;

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ld4_last(const float* p) { return __ldcs(reinterpret_cast<const float4*>(p)); }     // nobody reads it again soon
__device__ __forceinline__ void st4(float* p, const float4& v) { *reinterpret_cast<float4*>(p) = v; }

struct PoolGeom { int H, W, Hp, Wp; };

// Rows (in units of C floats) of the four pixels of pooled pixel r.  (32-bit divisions: 2^31 rows of 32 channels are 256 GB, and the host refuses them.)
__device__ __forceinline__ void pool_rows(const PoolGeom& g, int64_t r, int64_t (&row)[4]) {
  const uint32_t line = (uint32_t)r / (uint32_t)g.Wp, n = line / (uint32_t)g.Hp;       // the pooled line, its image
  const uint32_t wp = (uint32_t)r - line * (uint32_t)g.Wp, hp = line - n * (uint32_t)g.Hp;
  row[0] = ((int64_t)n * g.H + 2 * hp) * g.W + 2 * wp;
  row[1] = row[0] + 1;
  row[2] = row[0] + g.W;
  row[3] = row[2] + 1;
}

// Arrival counts of the groups' barriers: they only ever grow.  `passed` is what earlier launches account for.
struct GroupSync {
  uint32_t arrived[MAX_BLOCKS], passed[MAX_BLOCKS];
};

struct Shape {
  int64_t M;               // rows the kernel walks (pooled pixels with a pool)
  int C, G, R;
  int64_t per;             // rows of a block
  PoolGeom pool;
  GroupSync* sync;
  float* parts;            // [R][G][VALUES]
  int* error_flag;
};

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// All R blocks of group g have arrived (their partial sums are visible).  A wait gives up after two seconds and reports.
__device__ __forceinline__ void group_barrier(const Shape& s, int g, int r, uint32_t passed) {
  __syncthreads();
  if (threadIdx.x == 0) {
    const uint32_t target = passed + (uint32_t)s.R;
    __threadfence();
    atomicAdd(&s.sync->arrived[g], 1u);
    const unsigned long long limit = now_ns() + 2000000000ull;
    int it = 0;
    while ((int32_t)(ld_acquire_gpu(&s.sync->arrived[g]) - target) < 0)
      if ((++it & 63) == 0 && now_ns() > limit) { atomicExch(s.error_flag, 2); break; }
    if (r == 0) s.sync->passed[g] = target;            // every block of the group has read it
  }
  __syncthreads();
}

// Sum of (a, b) over all rows of the group.  tot[4 * (channel quad) ...]: a's and b's totals, [quad][a.xyzw b.xyzw].
__device__ __forceinline__ void group_totals(const Shape& s, int g, int r, uint32_t passed, float4 a, float4 b, float (*warp_part)[VALUES],
                                             double (*lane_part)[VALUES], float* tot) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] += __shfl_xor_sync(FULL, v[j], 8);
    v[j] += __shfl_xor_sync(FULL, v[j], 16);
  }
  if (lane < QUADS)
#pragma unroll
    for (int j = 0; j < 8; ++j) warp_part[wid][lane * 8 + j] = v[j];
  __syncthreads();
  if (s.R == 1) {
    if (threadIdx.x < VALUES) {
      double t = 0.0;
#pragma unroll
      for (int w = 0; w < THREADS / 32; ++w) t += (double)warp_part[w][threadIdx.x];
      tot[threadIdx.x] = (float)t;
    }
    __syncthreads();
    return;
  }
  if (threadIdx.x < VALUES) {
    float t = 0.0f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) t += warp_part[w][threadIdx.x];
    __stcg(s.parts + ((int64_t)r * s.G + g) * VALUES + threadIdx.x, t);
  }
  group_barrier(s, g, r, passed);
  {
    const int value = threadIdx.x % VALUES, part = threadIdx.x / VALUES;
    double t = 0.0;
    for (int i = part; i < s.R; i += THREADS / VALUES) t += (double)__ldcg(s.parts + ((int64_t)i * s.G + g) * VALUES + value);
    lane_part[part][value] = t;
  }
  __syncthreads();
  if (threadIdx.x < VALUES) {
    double t = 0.0;
#pragma unroll
    for (int i = 0; i < THREADS / VALUES; ++i) t += lane_part[i][threadIdx.x];
    tot[threadIdx.x] = (float)t;
  }
  __syncthreads();
}

struct Channels { float4 mu, rs, gm, bt; };

__device__ __forceinline__ float4 normalized(const float4& v, const Channels& c) {
  return make_float4((v.x - c.mu.x) * c.rs.x, (v.y - c.mu.y) * c.rs.y, (v.z - c.mu.z) * c.rs.z, (v.w - c.mu.w) * c.rs.w);
}
__device__ __forceinline__ float4 affine(const float4& xh, const Channels& c) {
  return make_float4(fmaf(xh.x, c.gm.x, c.bt.x), fmaf(xh.y, c.gm.y, c.bt.y), fmaf(xh.z, c.gm.z, c.bt.z), fmaf(xh.w, c.gm.w, c.bt.w));
}
__device__ __forceinline__ float4 keep_positive(const float4& d, const float4& o) {
  return make_float4(o.x > 0.f ? d.x : 0.f, o.y > 0.f ? d.y : 0.f, o.z > 0.f ? d.z : 0.f, o.w > 0.f ? d.w : 0.f);
}
__device__ __forceinline__ float4 relu4(const float4& o) { return make_float4(fmaxf(o.x, 0.f), fmaxf(o.y, 0.f), fmaxf(o.z, 0.f), fmaxf(o.w, 0.f)); }

// ------------------------------------------------------------------------------------------ forward
struct FwdArgs {
  const float* x;
  const float* partials;   // [nparts][2][C] sums and sums of squares of x (NULL: computed here)
  int nparts;
  const float *gamma, *beta, *residual;
  int relu;
  float *running_mean, *running_var;
  float momentum, eps;
  float *stats, *y;
};

template <bool POOL, bool SUMS>
__global__ void __launch_bounds__(THREADS, 1) bn_fused_fwd_kernel(const Shape s, const FwdArgs a) {
  __shared__ float warp_part[SUMS ? THREADS / 32 : 1][VALUES];
  __shared__ double lane_part[THREADS / VALUES][VALUES];
  __shared__ __align__(16) float tot[VALUES], shift[CH], mean_s[CH], rstd_s[CH];
  const int g = blockIdx.x % s.G, r = blockIdx.x / s.G;
  const int q = threadIdx.x % QUADS, rl = threadIdx.x / QUADS;
  const int c4 = g * CH + 4 * q, C = s.C;
  const int64_t lo = (int64_t)r * s.per, hi = lo + s.per < s.M ? lo + s.per : s.M;
  pdl_launch_dependents();
  // The first rows of the apply pass are on their way while the statistics come together (a layer of few rows per thread is latency, not bandwidth).
  constexpr int U = 4;                       // rows in flight per thread: 64 KB a block (twice that with a residual)
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  int64_t i = hi - 1 - rl;
  float4 v[U];
  auto load_rows = [&]() {
    if (POOL) {
      int64_t row[4];
      if (i >= lo) {
        pool_rows(s.pool, i, row);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = ld4(a.x + row[j] * C + c4);
      }
    } else {
#pragma unroll
      for (int j = 0; j < U; ++j) v[j] = i - j * LANES >= lo ? ld4_last(a.x + (i - j * LANES) * C + c4) : zero;
    }
  };
  if (!SUMS) load_rows();
  if (SUMS) {
    // sums shifted by the channel's value in row 0: no cancellation when |mean| is large against the standard deviation
    const uint32_t passed = threadIdx.x == 0 ? *((volatile uint32_t*)&s.sync->passed[g]) : 0u;
    const float4 k = ld4(a.x + c4);
    float4 u = make_float4(0.f, 0.f, 0.f, 0.f), w = u;
    auto add = [&](float4 v) {
      v.x -= k.x; v.y -= k.y; v.z -= k.z; v.w -= k.w;
      u.x += v.x; u.y += v.y; u.z += v.z; u.w += v.w;
      w.x = fmaf(v.x, v.x, w.x); w.y = fmaf(v.y, v.y, w.y); w.z = fmaf(v.z, v.z, w.z); w.w = fmaf(v.w, v.w, w.w);
    };
    for (int64_t i = lo + rl; i < hi; i += LANES) {
      if (POOL) {
        int64_t row[4];
        pool_rows(s.pool, i, row);
        float4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = ld4(a.x + row[j] * C + c4);
#pragma unroll
        for (int j = 0; j < 4; ++j) add(v[j]);
      } else {
        add(ld4(a.x + i * C + c4));
      }
    }
    if (rl == 0) st4(shift + 4 * q, k);
    group_totals(s, g, r, passed, u, w, warp_part, lane_part, tot);
  } else {
    // the convolution's partial sums of this group's channels
    const int value = threadIdx.x % VALUES, part = threadIdx.x / VALUES;
    const float* base = a.partials + (int64_t)(value / CH) * C + g * CH + value % CH;
    constexpr int P = THREADS / VALUES;
    double t = 0.0;
    int i = part;
    for (; i + 7 * P < a.nparts; i += 8 * P) {
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = base[(int64_t)(i + j * P) * 2 * C];
      t += (((double)v[0] + (double)v[1]) + ((double)v[2] + (double)v[3])) + (((double)v[4] + (double)v[5]) + ((double)v[6] + (double)v[7]));
    }
    for (; i < a.nparts; i += P) t += (double)base[(int64_t)i * 2 * C];
    lane_part[part][value] = t;
    __syncthreads();
  }
  if (threadIdx.x < CH) {
    const int c = threadIdx.x;
    const double rows = (double)s.M * (POOL ? 4.0 : 1.0);
    double sum = 0.0, sq = 0.0;
    if (SUMS) {
      sum = (double)tot[(c / 4) * 8 + c % 4];
      sq = (double)tot[(c / 4) * 8 + 4 + c % 4];
    } else {
#pragma unroll
      for (int i = 0; i < THREADS / VALUES; ++i) { sum += lane_part[i][c]; sq += lane_part[i][CH + c]; }
    }
    const double dmean = sum / rows;
    double var = sq / rows - dmean * dmean;
    if (var < 0.0) var = 0.0;
    const double mean = (SUMS ? (double)shift[c] : 0.0) + dmean;
    mean_s[c] = (float)mean;
    rstd_s[c] = (float)(1.0 / sqrt(var + (double)a.eps));
    if (r == 0) {
      const int gc = g * CH + c;
      a.stats[gc] = mean_s[c];
      a.stats[C + gc] = rstd_s[c];
      if (a.running_mean != nullptr) {
        const double unbiased = rows > 1.0 ? var * rows / (rows - 1.0) : var;
        a.running_mean[gc] = (1.0f - a.momentum) * a.running_mean[gc] + a.momentum * (float)mean;
        a.running_var[gc] = (1.0f - a.momentum) * a.running_var[gc] + a.momentum * (float)unbiased;
      }
    }
  }
  __syncthreads();
  const Channels ch{ld4(mean_s + 4 * q), ld4(rstd_s + 4 * q), ld4(a.gamma + c4), ld4(a.beta + c4)};
  if (SUMS) load_rows();
  if (POOL) {
    while (i >= lo) {
      float4 o = affine(normalized(v[0], ch), ch);
      if (a.relu) o = relu4(o);
#pragma unroll
      for (int j = 1; j < 4; ++j) {
        float4 p = affine(normalized(v[j], ch), ch);
        if (a.relu) p = relu4(p);
        o = make_float4(fmaxf(o.x, p.x), fmaxf(o.y, p.y), fmaxf(o.z, p.z), fmaxf(o.w, p.w));
      }
      const int64_t at = i * C + c4;
      i -= LANES;
      load_rows();
      st4(a.y + at, o);
    }
    return;
  }
  while (i >= lo) {
    float4 res[U];
#pragma unroll
    for (int j = 0; j < U; ++j) res[j] = a.residual != nullptr && i - j * LANES >= lo ? ld4_last(a.residual + (i - j * LANES) * C + c4) : zero;
#pragma unroll
    for (int j = 0; j < U; ++j) {
      if (i - j * LANES < lo) break;
      float4 o = affine(normalized(v[j], ch), ch);
      o.x += res[j].x; o.y += res[j].y; o.z += res[j].z; o.w += res[j].w;
      st4(a.y + (i - j * LANES) * C + c4, a.relu ? relu4(o) : o);
    }
    i -= U * LANES;
    load_rows();
  }
}

// ------------------------------------------------------------------------------------------ backward
struct BwdArgs {
  const float *dy, *x, *y; // y: saved output (NULL: the ReLU's mask is found again from x)
  const float *stats, *gamma, *beta;
  int relu;
  float *sums, *dx, *dres;
  int64_t stream;          // rows of a block (whole pairs of rows of all threads) whose first reading leaves no trace in L2
  int masks;               // pairs of rows per thread whose ReLU masks fit the dynamic shared memory
};

// One channel of one window: position of the pooled gradient (the first maximum of the activations, -1 if the ReLU stops it) and
// that position's normalised value.
__device__ __forceinline__ int pool_route(float x0, float x1, float x2, float x3, float gm, float bt, int relu, float& xh_win) {
  const float xh[4] = {x0, x1, x2, x3};
  int which = 0;
  float best = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float o = fmaf(xh[j], gm, bt), act = relu ? fmaxf(o, 0.f) : o;
    if (j == 0 || act > best) { best = act; which = j; }
  }
  xh_win = which == 0 ? x0 : which == 1 ? x1 : which == 2 ? x2 : x3;
  return (relu && !(best > 0.f)) ? -1 : which;
}

__device__ __forceinline__ uint32_t positive_bits(const float4& o) {
  return (o.x > 0.f ? 1u : 0u) | (o.y > 0.f ? 2u : 0u) | (o.z > 0.f ? 4u : 0u) | (o.w > 0.f ? 8u : 0u);
}
__device__ __forceinline__ float4 keep_bits(const float4& d, uint32_t m) {
  return make_float4(m & 1u ? d.x : 0.f, m & 2u ? d.y : 0.f, m & 4u ? d.z : 0.f, m & 8u ? d.w : 0.f);
}

// A thread's rows are lo + rl + 128 k; pass 1 takes k upwards in pairs, pass 2 downwards.  Behind a residual the ReLU's mask comes
// from the saved output; pass 1 leaves it in shared memory, a byte per pair of rows and thread, so that the output is read once.
//
// STREAM: dy and x are more than L2 keeps between the passes.  Pass 2 starts with the rows that pass 1 read last, and finds them only if neither the rows in
// front of them nor its own results push them out: the first a.stream rows of a block are read, and everything is stored, with evict-first priority.
// 32x32x256 at batch 128 106.7 -> 101.5 us, behind a residual 162.0 -> 153.0, 16x16x512 50.4 -> 47.2 and 76.5 -> 72.4; ResNet-50's step 5760 -> 5724 us with
// 64 MB of both left to stay, 5729 with 96, 5739 with 128, 5736 with 48, 5760 with 32 (of 126 MB of L2; the next kernels read the results).
//
// KEEP: no thread has more than two rows, and what pass 1 read of dy and x stays in registers for pass 2 (8x8x256 at batch 31: 6.4 -> 6.1 us, 4x4x512
// at 128: 6.5 -> 6.1; four and six rows in shared memory gained nothing: 8x8x256 at batch 128 8.0 -> 8.3).  With a pool: no more than one pooled row, its four
// pixels and the winners stay (with 32-bit divisions and a row per thread instead of two: 4x4x512 at batch 128 12.3 -> 7.5 us, forward 5.4 -> 4.4).
template <bool POOL, bool KEEP, bool STREAM>
__global__ void __launch_bounds__(THREADS, 1) bn_fused_bwd_kernel(const Shape s, const BwdArgs a) {
  extern __shared__ uint8_t masks[];       // [a.masks][THREADS]
  __shared__ float warp_part[THREADS / 32][VALUES];
  __shared__ double lane_part[THREADS / VALUES][VALUES];
  __shared__ __align__(16) float tot[VALUES];
  const int g = blockIdx.x % s.G, r = blockIdx.x / s.G;
  const int q = threadIdx.x % QUADS, rl = threadIdx.x / QUADS;
  const int c4 = g * CH + 4 * q, C = s.C;
  const int64_t lo = (int64_t)r * s.per, hi = lo + s.per < s.M ? lo + s.per : s.M;
  pdl_launch_dependents();
  const uint32_t passed = threadIdx.x == 0 ? *((volatile uint32_t*)&s.sync->passed[g]) : 0u;
  const Channels ch{ld4(a.stats + c4), ld4(a.stats + C + c4), ld4(a.gamma + c4), ld4(a.beta + c4)};
  const bool from_y = a.relu && a.y != nullptr;
  float4 sg = make_float4(0.f, 0.f, 0.f, 0.f), sx = sg;
  float4 kw[4] = {sg, sg, sg, sg};                     // KEEP with a pool: the window's pixels normalised, the winner's index per channel (-1: none)
  int kwin[4] = {-1, -1, -1, -1};
  float4 kd0 = sg, kd1 = sg, kv0 = sg, kv1 = sg;       // KEEP: dy behind the ReLU and x normalised of both rows, zeros beyond the last one

  if (POOL && KEEP) {
    const int64_t i = lo + rl;
    if (i < hi) {
      int64_t row[4];
      pool_rows(s.pool, i, row);
      kd0 = ld4_last(a.dy + i * C + c4);
#pragma unroll
      for (int j = 0; j < 4; ++j) kw[j] = ld4_last(a.x + row[j] * C + c4);
#pragma unroll
      for (int j = 0; j < 4; ++j) kw[j] = normalized(kw[j], ch);
      float xh;
      kwin[0] = pool_route(kw[0].x, kw[1].x, kw[2].x, kw[3].x, ch.gm.x, ch.bt.x, a.relu, xh);
      if (kwin[0] >= 0) { sg.x = kd0.x; sx.x = kd0.x * xh; }
      kwin[1] = pool_route(kw[0].y, kw[1].y, kw[2].y, kw[3].y, ch.gm.y, ch.bt.y, a.relu, xh);
      if (kwin[1] >= 0) { sg.y = kd0.y; sx.y = kd0.y * xh; }
      kwin[2] = pool_route(kw[0].z, kw[1].z, kw[2].z, kw[3].z, ch.gm.z, ch.bt.z, a.relu, xh);
      if (kwin[2] >= 0) { sg.z = kd0.z; sx.z = kd0.z * xh; }
      kwin[3] = pool_route(kw[0].w, kw[1].w, kw[2].w, kw[3].w, ch.gm.w, ch.bt.w, a.relu, xh);
      if (kwin[3] >= 0) { sg.w = kd0.w; sx.w = kd0.w * xh; }
    }
  } else if (POOL) {
    for (int64_t i = lo + rl; i < hi; i += LANES) {
      int64_t row[4];
      pool_rows(s.pool, i, row);
      const float4 d = ld4(a.dy + i * C + c4);
      float4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = normalized(ld4(a.x + row[j] * C + c4), ch);
      float xh;
      if (pool_route(v[0].x, v[1].x, v[2].x, v[3].x, ch.gm.x, ch.bt.x, a.relu, xh) >= 0) { sg.x += d.x; sx.x = fmaf(d.x, xh, sx.x); }
      if (pool_route(v[0].y, v[1].y, v[2].y, v[3].y, ch.gm.y, ch.bt.y, a.relu, xh) >= 0) { sg.y += d.y; sx.y = fmaf(d.y, xh, sx.y); }
      if (pool_route(v[0].z, v[1].z, v[2].z, v[3].z, ch.gm.z, ch.bt.z, a.relu, xh) >= 0) { sg.z += d.z; sx.z = fmaf(d.z, xh, sx.z); }
      if (pool_route(v[0].w, v[1].w, v[2].w, v[3].w, ch.gm.w, ch.bt.w, a.relu, xh) >= 0) { sg.w += d.w; sx.w = fmaf(d.w, xh, sx.w); }
    }
  } else if (KEEP) {
    const int64_t i = lo + rl, at = i * C + c4, next = at + (int64_t)LANES * C;
    const bool one = i < hi, two = i + LANES < hi;
    float4 y0 = sg, y1 = sg;
    if (one) { kd0 = ld4_last(a.dy + at); kv0 = ld4_last(a.x + at); }
    if (two) { kd1 = ld4_last(a.dy + next); kv1 = ld4_last(a.x + next); }
    if (from_y && one) y0 = ld4_last(a.y + at);
    if (from_y && two) y1 = ld4_last(a.y + next);
    kv0 = normalized(kv0, ch);
    kv1 = normalized(kv1, ch);
    if (a.relu) {
      kd0 = keep_positive(kd0, from_y ? y0 : affine(kv0, ch));
      kd1 = keep_positive(kd1, from_y ? y1 : affine(kv1, ch));
    }
    auto add = [&](const float4& d, const float4& xh) {
      sg.x += d.x; sg.y += d.y; sg.z += d.z; sg.w += d.w;
      sx.x = fmaf(d.x, xh.x, sx.x); sx.y = fmaf(d.y, xh.y, sx.y); sx.z = fmaf(d.z, xh.z, sx.z); sx.w = fmaf(d.w, xh.w, sx.w);
    };
    if (one) add(kd0, kv0);
    if (two) add(kd1, kv1);
  } else {
    auto add = [&](float4 d, const float4& v, uint32_t m) {
      const float4 xh = normalized(v, ch);
      if (a.relu) d = from_y ? keep_bits(d, m) : keep_positive(d, affine(xh, ch));
      sg.x += d.x; sg.y += d.y; sg.z += d.z; sg.w += d.w;
      sx.x = fmaf(d.x, xh.x, sx.x); sx.y = fmaf(d.y, xh.y, sx.y); sx.z = fmaf(d.z, xh.z, sx.z); sx.w = fmaf(d.w, xh.w, sx.w);
    };
    int64_t i = lo + rl;
    int pair = 0;
    auto pairs_until = [&](int64_t end, auto load) {
      for (; i + LANES < end; i += 2 * LANES, ++pair) {
        const int64_t at = i * C + c4, next = at + (int64_t)LANES * C;
        const float4 d0 = load(a.dy + at), v0 = load(a.x + at), d1 = load(a.dy + next), v1 = load(a.x + next);
        uint32_t m = 0;
        if (from_y) {
          m = positive_bits(ld4_last(a.y + at)) | positive_bits(ld4_last(a.y + next)) << 4;
          if (pair < a.masks) masks[pair * THREADS + threadIdx.x] = (uint8_t)m;
        }
        add(d0, v0, m);
        add(d1, v1, m >> 4);
      }
    };
    if (STREAM) pairs_until(lo + a.stream < hi ? lo + a.stream : hi, [](const float* p) { return ld4_last(p); });
    pairs_until(hi, [](const float* p) { return ld4(p); });
    if (i < hi) {
      const int64_t at = i * C + c4;
      uint32_t m = 0;
      if (from_y) {
        m = positive_bits(ld4(a.y + at));
        if (pair < a.masks) masks[pair * THREADS + threadIdx.x] = (uint8_t)m;
      }
      add(ld4(a.dy + at), ld4(a.x + at), m);
    }
  }
  group_totals(s, g, r, passed, sg, sx, warp_part, lane_part, tot);
  const float4 db = ld4(tot + 8 * q), dg = ld4(tot + 8 * q + 4);
  if (r == 0 && rl == 0) {
    st4(a.sums + c4, db);
    st4(a.sums + C + c4, dg);
  }
  // dx = gamma * rstd * (g - dbeta / M - xhat * dgamma / M)
  const float inv_m = 1.0f / (float)(s.M * (POOL ? 4 : 1));
  const float4 mb = make_float4(db.x * inv_m, db.y * inv_m, db.z * inv_m, db.w * inv_m);
  auto input_gradient = [&](const float4& d, const float4& xh) {
    return make_float4(ch.gm.x * ch.rs.x * (d.x - mb.x - xh.x * dg.x * inv_m), ch.gm.y * ch.rs.y * (d.y - mb.y - xh.y * dg.y * inv_m),
                       ch.gm.z * ch.rs.z * (d.z - mb.z - xh.z * dg.z * inv_m), ch.gm.w * ch.rs.w * (d.w - mb.w - xh.w * dg.w * inv_m));
  };
  if (POOL && KEEP) {
    const int64_t i = lo + rl;
    if (i >= hi) return;
    int64_t row[4];
    pool_rows(s.pool, i, row);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      st4(a.dx + row[j] * C + c4, input_gradient(make_float4(kwin[0] == j ? kd0.x : 0.f, kwin[1] == j ? kd0.y : 0.f, kwin[2] == j ? kd0.z : 0.f, kwin[3] == j ? kd0.w : 0.f), kw[j]));
    return;
  }
  if (POOL) {
    for (int64_t i = hi - 1 - rl; i >= lo; i -= LANES) {
      int64_t row[4];
      pool_rows(s.pool, i, row);
      const float4 d = ld4(a.dy + i * C + c4);
      float4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = normalized(ld4(a.x + row[j] * C + c4), ch);
      float xw;
      const int wx = pool_route(v[0].x, v[1].x, v[2].x, v[3].x, ch.gm.x, ch.bt.x, a.relu, xw);
      const int wy = pool_route(v[0].y, v[1].y, v[2].y, v[3].y, ch.gm.y, ch.bt.y, a.relu, xw);
      const int wz = pool_route(v[0].z, v[1].z, v[2].z, v[3].z, ch.gm.z, ch.bt.z, a.relu, xw);
      const int ww = pool_route(v[0].w, v[1].w, v[2].w, v[3].w, ch.gm.w, ch.bt.w, a.relu, xw);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        st4(a.dx + row[j] * C + c4,
            input_gradient(make_float4(wx == j ? d.x : 0.f, wy == j ? d.y : 0.f, wz == j ? d.z : 0.f, ww == j ? d.w : 0.f), v[j]));
    }
    return;
  }
  if (KEEP) {
    const int64_t i = lo + rl, at = i * C + c4, next = at + (int64_t)LANES * C;
    if (i < hi) {
      if (a.dres != nullptr) st4(a.dres + at, kd0);
      st4(a.dx + at, input_gradient(kd0, kv0));
    }
    if (i + LANES < hi) {
      if (a.dres != nullptr) st4(a.dres + next, kd1);
      st4(a.dx + next, input_gradient(kd1, kv1));
    }
    return;
  }
  auto store = [](float* p, const float4& v) {
    if (STREAM) __stcs(reinterpret_cast<float4*>(p), v);
    else st4(p, v);
  };
  auto finish = [&](float4 d, const float4& v, uint32_t m, int64_t at) {
    const float4 xh = normalized(v, ch);
    if (a.relu) d = from_y ? keep_bits(d, m) : keep_positive(d, affine(xh, ch));
    if (a.dres != nullptr) store(a.dres + at, d);
    store(a.dx + at, input_gradient(d, xh));
  };
  const int rows = hi - lo > rl ? (int)((hi - lo - rl + LANES - 1) / LANES) : 0;       // this thread's
  auto mask_of = [&](int pair, int64_t at, int64_t next, bool two) {
    if (!from_y) return 0u;
    if (pair < a.masks) return (uint32_t)masks[pair * THREADS + threadIdx.x];
    return positive_bits(ld4(a.y + at)) | (two ? positive_bits(ld4(a.y + next)) << 4 : 0u);
  };
  int pair = rows / 2;
  if (rows & 1) {
    const int64_t at = (lo + rl + (int64_t)(rows - 1) * LANES) * C + c4;
    finish(ld4_last(a.dy + at), ld4_last(a.x + at), mask_of(pair, at, at, false), at);
  }
  for (--pair; pair >= 0; --pair) {
    const int64_t at = (lo + rl + (int64_t)pair * 2 * LANES) * C + c4, next = at + (int64_t)LANES * C;
    const float4 d0 = ld4_last(a.dy + at), v0 = ld4_last(a.x + at), d1 = ld4_last(a.dy + next), v1 = ld4_last(a.x + next);
    const uint32_t m = mask_of(pair, at, next, true);
    finish(d1, v1, m >> 4, next);
    finish(d0, v0, m, at);
  }
}

int sm_count() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
}

// Blocks of a launch: one per SM, and no more than the scratch has partial sums for, whatever the chip's size.
int block_limit(int sms) { return sms < MAX_BLOCKS ? sms : MAX_BLOCKS; }

// Runs of rows per channel group: as many as blocks allow, two hundred and some rows each at least (two per thread; one where a row is a
// pooled one with its four pixels).
void plan(Shape& s, int sms, int pool) {
  s.G = s.C / CH;
  const int64_t least = pool ? LANES : 2 * LANES;
  int64_t most = block_limit(sms) / s.G, want = (s.M + least - 1) / least;
  if (most < 1) most = 1;
  int64_t r = want < most ? want : most;
  s.per = (s.M + r - 1) / r;
  s.R = (int)((s.M + s.per - 1) / s.per);
}

bool shape_ok(int64_t M, int C, int sms) { return M >= 1 && C >= CH && C % CH == 0 && C / CH <= block_limit(sms); }

// Launched the ordinary way, without programmatic overlap: the backward is cooperative, and the forward, started while the convolution still holds
// its shared memory, keeps the SM's split between shared memory and L1 and has too few loads in flight (ResNet-50's step: 5857 -> 6112 us; 6580 with the
// smallest L1 asked for in both directions).  Their successors are released at the start.
template <typename A>
int launch(const void* kernel, const Shape& s, const A& a, bool barrier, size_t smem, cudaStream_t st) {
  void* args[2] = {(void*)&s, (void*)&a};
  const dim3 grid((unsigned)(s.G * s.R));
  if (barrier && s.R > 1) return (int)cudaLaunchCooperativeKernel(kernel, grid, dim3(THREADS), args, smem, st);
  return (int)cudaLaunchKernel(kernel, grid, dim3(THREADS), args, smem, st);
}

}  // namespace

extern "C" {

int gc_cuda_bn_fused_supported(int64_t M, int C) { return shape_ok(M, C, sm_count()) ? 1 : 0; }

// Blocks a launch on M rows of C channels takes on a chip of `sms` SMs, each of which has a row of partial sums (0: not taken).
static int planned_blocks(int64_t M, int C, int sms, int pool) {
  if (!shape_ok(M, C, sms)) return 0;
  Shape s{};
  s.M = M;
  s.C = C;
  plan(s, sms, pool);
  return s.G * s.R;
}
int gc_cuda_bn_fused_blocks(int64_t M, int C, int sms) { return planned_blocks(M, C, sms, 0); }
int gc_cuda_bn_fused_pool_blocks(int64_t M, int C, int sms) { return planned_blocks(M, C, sms, 1); }      // M pooled rows

// Scratch of both directions: barrier counts (zeroed once when allocated; every launch leaves them ready) and partial sums.
int64_t gc_cuda_bn_fused_scratch_bytes() { return (int64_t)sizeof(GroupSync) + (int64_t)MAX_BLOCKS * VALUES * 4; }

// y = act(gamma * (x - mean) * rstd + beta [+ residual]) of the batch statistics of x, which come from partials[nparts][2][C] when
// given.  pool (then no residual): x is [N, H, W, C], H and W even, and y the 2x2 max-pool of the activation.  Writes
// stats[0:C] = mean, stats[C:2C] = rstd and updates the running statistics (may be NULL).
int gc_cuda_bn_fused_forward(const float* x, int N, int H, int W, int C, int pool, const float* partials, int nparts, const float* gamma, const float* beta,
                             const float* residual, int relu, float* running_mean, float* running_var, float momentum, float eps, float* stats, float* y,
                             void* scratch, int* error_flag, void* cs) {
  Shape s{};
  s.M = (int64_t)N * H * W / (pool ? 4 : 1);
  s.C = C;
  if (!shape_ok(s.M, C, sm_count()) || (pool && ((H | W) & 1 || residual != nullptr || s.M > 0x3fffffff))) return (int)cudaErrorInvalidValue;
  s.pool = PoolGeom{H, W, H / 2, W / 2};
  s.sync = (GroupSync*)scratch;
  s.parts = (float*)((uint8_t*)scratch + sizeof(GroupSync));
  s.error_flag = error_flag;
  plan(s, sm_count(), pool);
  const FwdArgs a{x, partials, nparts, gamma, beta, residual, relu, running_mean, running_var, momentum, eps, stats, y};
  const void* k = partials != nullptr ? (pool ? (const void*)bn_fused_fwd_kernel<true, false> : (const void*)bn_fused_fwd_kernel<false, false>)
                                      : (pool ? (const void*)bn_fused_fwd_kernel<true, true> : (const void*)bn_fused_fwd_kernel<false, true>);
  return launch(k, s, a, partials == nullptr, 0, (cudaStream_t)cs);
}

// sums[0:C] = dbeta, sums[C:2C] = dgamma, dx, and dres (may be NULL) = the masked gradient.  y: saved output (needed when a
// residual was added).  pool: dy is the gradient of the pooled map.
int gc_cuda_bn_fused_backward(const float* dy, const float* x, const float* y, int N, int H, int W, int C, int pool, const float* stats, const float* gamma,
                              const float* beta, int relu, float* sums, float* dx, float* dres, void* scratch, int* error_flag, void* cs) {
  Shape s{};
  s.M = (int64_t)N * H * W / (pool ? 4 : 1);
  s.C = C;
  if (!shape_ok(s.M, C, sm_count()) || (pool && ((H | W) & 1 || dres != nullptr || s.M > 0x3fffffff))) return (int)cudaErrorInvalidValue;
  s.pool = PoolGeom{H, W, H / 2, W / 2};
  s.sync = (GroupSync*)scratch;
  s.parts = (float*)((uint8_t*)scratch + sizeof(GroupSync));
  s.error_flag = error_flag;
  plan(s, sm_count(), pool);
  const int64_t pairs = (s.per + 2 * LANES - 1) / (2 * LANES);
  const bool keep = s.per <= (pool ? 1 : 2) * LANES;
  // masks of as many row pairs as shared memory holds (192 KB: 49 K rows of 32 channels a block)
  constexpr int most = 192;
  const int masks = y == nullptr || pool || keep ? 0 : (int)(pairs < most ? pairs : most);
  // dy and x together beyond 64 MB: what exceeds it, the first rows of every block, is read the first time as data that is not needed again
  const int64_t both = s.M * C * 8, stay = (int64_t)64 << 20;
  const int64_t stream = pool || both <= stay ? 0 : (int64_t)((double)s.per * (double)(both - stay) / (double)both) / (2 * LANES) * (2 * LANES);
  const BwdArgs a{dy, x, y, stats, gamma, beta, relu, sums, dx, dres, stream, masks};
  const void* k = pool ? (keep ? (const void*)bn_fused_bwd_kernel<true, true, false> : (const void*)bn_fused_bwd_kernel<true, false, false>) : keep ? (const void*)bn_fused_bwd_kernel<false, true, false> :
                  stream > 0 ? (const void*)bn_fused_bwd_kernel<false, false, true> : (const void*)bn_fused_bwd_kernel<false, false, false>;
  if (masks * THREADS > 24 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most * THREADS);
    if (e != cudaSuccess) return (int)e;
  }
  return launch(k, s, a, true, (size_t)masks * THREADS, (cudaStream_t)cs);
}

}  // extern "C"
