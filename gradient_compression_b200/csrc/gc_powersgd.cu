// PowerSGD rank-r pipeline on the flat gradient (reference: reducer.py:1718-1858, there ~5 Python loops
// over 54 layers of cuBLAS GEMV calls and ~5 tiny kernels per Gram-Schmidt column):
//   psgd_p     P = (G + E) Q for every matrix in ONE launch (warp per matrix row); E <- G + E in place;
//              1-D tensors are packed behind P so that one exchange carries both
//   psgd_gs    classical Gram-Schmidt of every P in one launch (block per matrix)
//   psgd_q     Q' = M^T P for every matrix in one launch (block per 128-column tile, no atomics)
//   psgd_out   G <- P Q'^T, E <- M - P Q'^T; 1-D tensors get the plain mean
// All products are bandwidth-bound at r <= 4 (each streams the 94 MB gradient once), so they run on the
// CUDA cores with 16-byte loads; the two all-reduces in between use the one-shot peer-memory sum.
// A single worker has nothing to sum: gc_cuda_psgd_solo runs the chain without the exchanges and without the copies in
// front of them, on the gradient tensors where they lie (their pointers travel in the kernels' parameters).
// The error memory is written by psgd_p first row first, read by psgd_q last row first and by psgd_out first row first again,
// while the gradient passes through with streaming loads and stores: what the last kernel touched last is in L2 (VGG-16's 59 MB
// all of it: psgd_q 32 -> 13 us).
// Matrix table: int64 rows of {off, n, m, r, p_off, q_off, first row block, first Q' block, tensor}.
// Vector table: int64 rows of {off, len, dst, tensor}.
#include <cuda_runtime.h>
#include <stdint.h>

#include "gc_device.cuh"
#include "gc_segs.cuh"

extern "C" int gc_cuda_psgd_q_chunks(int max_rows);
extern "C" int gc_cuda_philox_fill(int kind, uint64_t seed, uint32_t stream_id, uint32_t step, const uint32_t* step_offset, int64_t n, void* out, void* cs);

using namespace gc;

namespace {

constexpr int RMAX = 4;
constexpr int MAT_FIELDS = 9, VEC_FIELDS = 4;

// Where the gradients lie: CAP == 1: one flat vector; otherwise a pointer per tensor.
template <int CAP>
struct GradPtrs {
  const float* in[CAP];
  float* out[CAP];
  __device__ __forceinline__ const float* src(int tensor, int64_t off) const { return CAP == 1 ? in[0] + off : in[tensor]; }
  __device__ __forceinline__ float* dst(int tensor, int64_t off) const { return CAP == 1 ? out[0] + off : out[tensor]; }
};

// Rows of an n x m matrix that one block of the P and output kernels takes: about 32 KB, so that looking the matrix up is paid
// once per block (once per row, ResNet-50's 26 K mostly short rows spent more time on it than on their data: 86 us for P).
__host__ __device__ inline int rows_per_block(int m) {
  const int r = (8192 / (m > 0 ? m : 1) + 7) / 8 * 8;
  return r < 8 ? 8 : (r > 256 ? 256 : r);
}
// A warp works on ROWS rows at once while a block has that many for each of its warps: with one row of a few hundred floats it
// had two loads in flight, and read the query block again for every row.  Longer rows (1024 floats and more) are taken one at
// a time, PIECES pieces of 128 floats in flight.  Two of each: four need 128 to 190 registers a thread and leave an SM with one
// or two blocks (VGG-16, rank 2: 25 us against 63 to 88 us for P).
constexpr int ROWS = 2, PIECES = 2;
// Rows per block of the Q' kernel: at most MAX_CHUNKS partial sums per matrix, and 64 KB or more for a block to read.
constexpr int MAX_CHUNKS = 16, MIN_CHUNK = 128;
__host__ __device__ inline int rows_per_chunk(int n) {
  const int r = ((n + MAX_CHUNKS - 1) / MAX_CHUNKS + 31) / 32 * 32;
  return r < MIN_CHUNK ? MIN_CHUNK : r;
}

struct Mat { int64_t off; int n, m, r; int64_t p_off, q_off; int tensor; };

__device__ __forceinline__ Mat load_mat(const int64_t* __restrict__ tab, int i) {
  const int64_t* t = tab + (int64_t)i * MAT_FIELDS;
  Mat m;
  m.off = t[0]; m.n = (int)t[1]; m.m = (int)t[2]; m.r = (int)t[3]; m.p_off = t[4]; m.q_off = t[5]; m.tensor = (int)t[8];
  return m;
}

// Largest i with tab[i][field] <= key.
__device__ __forceinline__ int find_mat(const int64_t* __restrict__ tab, int n_mats, int field, int64_t key) {
  int lo = 0, hi = n_mats - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (tab[(int64_t)mid * MAT_FIELDS + field] <= key) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// ------------------------------------------------------------------------------------------ P = (G + E) Q
// Four columns of a block of 128 for every lane: neighbours up to rank 2, 32 apart above.  There the query rows are what the L1 is busy
// with: four neighbouring rows of 16 bytes a lane make one load of the warp touch 16 lines, with columns 32 apart 4 (rank 4: L1 80 % busy,
// DRAM 30 %; VGG-16 P 51 -> 31 us and output 50 -> 30 us, ResNet-50 78 -> 60 and 80 -> 57 us).  At rank 2 the 16-byte loads of the gradient are worth
// more (VGG-16: P 25 us against 34 us with columns apart).  A lane's first column is `k`; the others may lie beyond the matrix when apart.
template <int R>
constexpr bool APART = R > 2;
template <int R>
__device__ __forceinline__ int first_column(int lane) { return APART<R> ? lane : lane * 4; }

template <int R, bool STREAM>
__device__ __forceinline__ void load4(const float* __restrict__ x, int k, int m, float (&v)[4]) {
  if constexpr (APART<R>) {
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = k + 32 * t >= m ? 0.f : STREAM ? __ldcs(x + k + 32 * t) : x[k + 32 * t];
  } else {
    const float4 o = STREAM ? __ldcs(reinterpret_cast<const float4*>(x + k)) : *reinterpret_cast<const float4*>(x + k);
    v[0] = o.x; v[1] = o.y; v[2] = o.z; v[3] = o.w;
  }
}

template <int R, bool STREAM>
__device__ __forceinline__ void store4(float* __restrict__ x, int k, int m, const float (&v)[4]) {
  if constexpr (APART<R>) {
#pragma unroll
    for (int t = 0; t < 4; ++t)
      if (k + 32 * t < m) {
        if (STREAM) __stcs(x + k + 32 * t, v[t]);
        else x[k + 32 * t] = v[t];
      }
  } else {
    const float4 o = make_float4(v[0], v[1], v[2], v[3]);
    if (STREAM) __stcs(reinterpret_cast<float4*>(x + k), o);
    else *reinterpret_cast<float4*>(x + k) = o;
  }
}

// Their query rows, [t][j] (zero beyond the matrix).
template <int R>
__device__ __forceinline__ void load_q4(const float* __restrict__ qm, int k, int m, float (&q)[4][R]) {
  if constexpr (!APART<R>) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const float4 v = *reinterpret_cast<const float4*>(qm + (int64_t)k * R + 4 * i);
      (&q[0][0])[4 * i] = v.x; (&q[0][0])[4 * i + 1] = v.y; (&q[0][0])[4 * i + 2] = v.z; (&q[0][0])[4 * i + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      const bool in = k + 32 * t < m;
      const float* row = qm + (int64_t)(k + 32 * t) * R;
      if constexpr (R == 4) {
        const float4 v = in ? *reinterpret_cast<const float4*>(row) : make_float4(0.f, 0.f, 0.f, 0.f);
        q[t][0] = v.x; q[t][1] = v.y; q[t][2] = v.z; q[t][3] = v.w;
      } else {
#pragma unroll
        for (int j = 0; j < R; ++j) q[t][j] = in ? row[j] : 0.f;
      }
    }
  }
}

// Sums N (a power of two, at most 32) values per lane over the warp; lane l ends up with the total of value l % N.  Halving
// the number of values a lane carries at every step takes N - 1 + 5 - log2(N) shuffles instead of 5 N.
template <int N>
__device__ __forceinline__ float warp_sum_many(float (&v)[N], int lane) {
  int o = 1;
#pragma unroll
  for (int h = N / 2; h >= 1; h >>= 1, o <<= 1) {
    const bool upper = (lane & o) != 0;
    // lanes with bit o set keep the values of odd index, the others the even ones (value index bit by bit equals lane bits)
#pragma unroll
    for (int i = 0; i < h; ++i) {
      const float keep = upper ? v[2 * i + 1] : v[2 * i], give = upper ? v[2 * i] : v[2 * i + 1];
      v[i] = keep + __shfl_xor_sync(FULL, give, o);
    }
  }
  float r = v[0];
#pragma unroll
  for (int s = N; s < 32; s <<= 1) r += __shfl_xor_sync(FULL, r, s);
  return r;
}

// One long row of P and of E <- G + E.
template <int R>
__device__ __forceinline__ void p_long_row(const float* __restrict__ g, float* __restrict__ e, int m, const float* __restrict__ qm, float* __restrict__ p,
                                           int lane) {
  float acc[R];
#pragma unroll
  for (int j = 0; j < R; ++j) acc[j] = 0.f;
  for (int k0 = first_column<R>(lane); k0 < m; k0 += 128 * PIECES) {
    float a[PIECES][4], b[PIECES][4];
#pragma unroll
    for (int u = 0; u < PIECES; ++u) {
      if (k0 + 128 * u >= m) continue;
      load4<R, true>(g, k0 + 128 * u, m, a[u]);
      load4<R, false>(e, k0 + 128 * u, m, b[u]);
    }
#pragma unroll
    for (int u = 0; u < PIECES; ++u) {
      if (k0 + 128 * u >= m) continue;
      float q[4][R];
      load_q4<R>(qm, k0 + 128 * u, m, q);
#pragma unroll
      for (int t = 0; t < 4; ++t) a[u][t] += b[u][t];
      store4<R, false>(e, k0 + 128 * u, m, a[u]);
#pragma unroll
      for (int j = 0; j < R; ++j) acc[j] = fmaf(a[u][0], q[0][j], fmaf(a[u][1], q[1][j], fmaf(a[u][2], q[2][j], fmaf(a[u][3], q[3][j], acc[j]))));
    }
  }
#pragma unroll
  for (int j = 0; j < R; ++j) {
    const float s = warp_sum(acc[j]);
    if (lane == 0) p[j] = s;
  }
}

// ROWS rows of P (fewer at the matrix' end) and of E <- G + E; R padded to a power of two in the sums.
template <int R>
__device__ __forceinline__ void p_rows(const float* __restrict__ g, float* __restrict__ e, int m, int rows, const float* __restrict__ qm,
                                       float* __restrict__ p, int lane) {
  constexpr int RP = R == 3 ? 4 : R;
  float acc[ROWS * RP];
#pragma unroll
  for (int i = 0; i < ROWS * RP; ++i) acc[i] = 0.f;
  for (int k = first_column<R>(lane); k < m; k += 128) {
    float a[ROWS][4], b[ROWS][4];
#pragma unroll
    for (int u = 0; u < ROWS; ++u)
      if (u < rows) {
        load4<R, true>(g + (int64_t)u * m, k, m, a[u]);
        load4<R, false>(e + (int64_t)u * m, k, m, b[u]);
      }
    float q[4][R];
    load_q4<R>(qm, k, m, q);
#pragma unroll
    for (int u = 0; u < ROWS; ++u)
      if (u < rows) {
#pragma unroll
        for (int t = 0; t < 4; ++t) a[u][t] += b[u][t];
        store4<R, false>(e + (int64_t)u * m, k, m, a[u]);
#pragma unroll
        for (int j = 0; j < R; ++j)
          acc[u * RP + j] = fmaf(a[u][0], q[0][j], fmaf(a[u][1], q[1][j], fmaf(a[u][2], q[2][j], fmaf(a[u][3], q[3][j], acc[u * RP + j]))));
      }
  }
  const float s = warp_sum_many<ROWS * RP>(acc, lane);
  const int u = lane / RP, j = lane % RP;
  if (lane < ROWS * RP && u < rows && j < R) p[u * R + j] = s;
}

template <int CAP, int R>
__global__ void __launch_bounds__(256) psgd_p_kernel(const __grid_constant__ GradPtrs<CAP> gp, float* __restrict__ e,
                                                     const int64_t* __restrict__ tab, int n_mats,
                                                     const float* __restrict__ q, float* __restrict__ p, uint32_t* step) {
  const int lane = threadIdx.x & 31;
  const int mi = find_mat(tab, n_mats, 6, (int64_t)blockIdx.x);      // (the tables are older than the kernel in front)
  const Mat mt = load_mat(tab, mi);
  pdl_wait();
  pdl_launch_dependents();
  if (step != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *step += 1u;      // the query matrices of this step have been drawn
  const int rpb = rows_per_block(mt.m), row0 = (int)((int64_t)blockIdx.x - tab[(int64_t)mi * MAT_FIELDS + 6]) * rpb;
  const int row1 = row0 + rpb < mt.n ? row0 + rpb : mt.n;
  const float* qm = q + mt.q_off;
  const int group = rpb < ROWS * 8 ? rpb / 8 : ROWS;
  for (int row = row0 + (threadIdx.x >> 5) * group; row < row1; row += 8 * group) {
    const float* g = gp.src(mt.tensor, mt.off) + (int64_t)row * mt.m;
    float* er = e + mt.off + (int64_t)row * mt.m;
    float* pr = p + mt.p_off + (int64_t)row * mt.r;
    const int rows = row1 - row < group ? row1 - row : group;
    // 16-byte path: row starts, row length and the query block must all be 16-byte aligned (and the rank the launch's own: matrices
    // with fewer rows or columns than that are small)
    const bool vec = (((reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(er)) & 15u) == 0) && ((mt.m & 3) == 0) && ((mt.q_off & 3) == 0) && mt.r == R;
    if (vec && group == 1) p_long_row<R>(g, er, mt.m, qm, pr, lane);
    else if (vec) p_rows<R>(g, er, mt.m, rows, qm, pr, lane);
    else
      for (int u = 0; u < rows; ++u, g += mt.m, er += mt.m, pr += mt.r) {
        float acc[RMAX] = {0.f, 0.f, 0.f, 0.f};
        for (int k = lane; k < mt.m; k += 32) {
          float a = g[k] + er[k];
          er[k] = a;
          for (int j = 0; j < mt.r; ++j) acc[j] = fmaf(a, qm[(int64_t)k * mt.r + j], acc[j]);
        }
        for (int j = 0; j < mt.r; ++j) {
          float s = warp_sum(acc[j]);
          if (lane == 0) pr[j] = s;
        }
      }
  }
}

// 1-D tensors: stage[dst + i] = g[off + i] (their error memory is identically zero).
__global__ void psgd_pack_vec_kernel(const float* __restrict__ g, const int64_t* __restrict__ vtab, int n_vecs,
                                     float* __restrict__ stage) {
  for (int v = blockIdx.x; v < n_vecs; v += gridDim.x) {
    int64_t off = vtab[v * VEC_FIELDS], len = vtab[v * VEC_FIELDS + 1], dst = vtab[v * VEC_FIELDS + 2];
    for (int64_t i = threadIdx.x; i < len; i += blockDim.x) stage[dst + i] = g[off + i];
  }
}

// ------------------------------------------------------------------------------------------ Gram-Schmidt
// Sums of up to RMAX values per thread over the block at once; every thread gets the totals.
template <int N>
__device__ __forceinline__ void block_sums(float (&v)[N], float (*smem)[32]) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
  for (int j = 0; j < N; ++j) v[j] = warp_sum(v[j]);
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int j = 0; j < N; ++j) smem[j][wid] = v[j];
  __syncthreads();
#pragma unroll
  for (int j = 0; j < N; ++j) v[j] = warp_sum(lane < nw ? smem[j][lane] : 0.0f);
}

// One block per matrix.  Up to GS_ROWS rows per thread stay in registers: a column costs two block-wide sums (its norm, and
// its products with all later columns together) and no memory traffic (n = 8192, r = 4: 49 -> 17.5 us a call).
constexpr int GS_THREADS = 1024, GS_ROWS = 8;

template <int R>
__device__ __forceinline__ void gs_registers(float* __restrict__ pm, int n, float eps, float (*smem)[32]) {
  float c[GS_ROWS][R];
#pragma unroll
  for (int u = 0; u < GS_ROWS; ++u) {
    const int row = threadIdx.x + u * GS_THREADS;
#pragma unroll
    for (int j = 0; j < R; ++j) c[u][j] = row < n ? pm[(int64_t)row * R + j] : 0.0f;
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    float ss[1] = {0.0f};
#pragma unroll
    for (int u = 0; u < GS_ROWS; ++u) ss[0] = fmaf(c[u][i], c[u][i], ss[0]);
    block_sums<1>(ss, smem);
    const float inv = 1.0f / (sqrtf(ss[0]) + eps);
#pragma unroll
    for (int u = 0; u < GS_ROWS; ++u) c[u][i] *= inv;
    if (i + 1 < R) {
      float dot[R];
#pragma unroll
      for (int j = 0; j < R; ++j) {
        dot[j] = 0.0f;
        if (j > i)
#pragma unroll
          for (int u = 0; u < GS_ROWS; ++u) dot[j] = fmaf(c[u][i], c[u][j], dot[j]);
      }
      block_sums<R>(dot, smem);
#pragma unroll
      for (int j = i + 1; j < R; ++j)
#pragma unroll
        for (int u = 0; u < GS_ROWS; ++u) c[u][j] = fmaf(-dot[j], c[u][i], c[u][j]);
    }
  }
#pragma unroll
  for (int u = 0; u < GS_ROWS; ++u) {
    const int row = threadIdx.x + u * GS_THREADS;
    if (row < n)
#pragma unroll
      for (int j = 0; j < R; ++j) pm[(int64_t)row * R + j] = c[u][j];
  }
}

__global__ void __launch_bounds__(GS_THREADS) psgd_gs_kernel(float* __restrict__ p, const int64_t* __restrict__ tab, float eps) {
  __shared__ float smem[RMAX][32];
  Mat mt = load_mat(tab, blockIdx.x);
  float* pm = p + mt.p_off;
  pdl_wait();
  pdl_launch_dependents();
  if (mt.n <= GS_THREADS * GS_ROWS) {
    if (mt.r == 1) gs_registers<1>(pm, mt.n, eps, smem);
    else if (mt.r == 2) gs_registers<2>(pm, mt.n, eps, smem);
    else if (mt.r == 3) gs_registers<3>(pm, mt.n, eps, smem);
    else gs_registers<4>(pm, mt.n, eps, smem);
    return;
  }
  for (int i = 0; i < mt.r; ++i) {
    float ss[1] = {0.f};
    for (int row = threadIdx.x; row < mt.n; row += blockDim.x) { float v = pm[(int64_t)row * mt.r + i]; ss[0] = fmaf(v, v, ss[0]); }
    block_sums<1>(ss, smem);
    float inv = 1.0f / (sqrtf(ss[0]) + eps);
    for (int row = threadIdx.x; row < mt.n; row += blockDim.x) pm[(int64_t)row * mt.r + i] *= inv;
    for (int j = i + 1; j < mt.r; ++j) {                    // (a thread only ever touches its own rows)
      float dot[1] = {0.f};
      for (int row = threadIdx.x; row < mt.n; row += blockDim.x)
        dot[0] = fmaf(pm[(int64_t)row * mt.r + i], pm[(int64_t)row * mt.r + j], dot[0]);
      block_sums<1>(dot, smem);
      for (int row = threadIdx.x; row < mt.n; row += blockDim.x)
        pm[(int64_t)row * mt.r + j] = fmaf(-dot[0], pm[(int64_t)row * mt.r + i], pm[(int64_t)row * mt.r + j]);
    }
  }
}

// ------------------------------------------------------------------------------------------ Q' = M^T P
// Block = one 128-column tile of one row chunk of one matrix; lane c owns columns 4c..4c+3 of the tile, the eight warps take
// every eighth row, eight rows in flight each (32 KB per block), and are combined through shared memory in a fixed order.
// The rank is a template parameter: with a run-time rank the accumulators were indexed in a loop and the kernel was bound by
// its instructions (VGG-16, rank 2: 32 us for 59 MB that were in L2).
template <int R>
__device__ __forceinline__ void q_tile(const float* __restrict__ base, const Mat& mt, int k0, int row_lo, int row_hi, const float* __restrict__ pm,
                                       bool vec, float (&acc)[4][RMAX]) {
  const int w = threadIdx.x >> 5;
  if (vec) {
    for (int row = row_lo + w; row < row_hi; row += 64) {
      float4 a[8];
      float pv[8][R];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int rr = row + 8 * u;
        a[u] = rr < row_hi ? __ldcg(reinterpret_cast<const float4*>(base + (int64_t)rr * mt.m + k0)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int j = 0; j < R; ++j) pv[u][j] = rr < row_hi ? __ldg(pm + (int64_t)rr * R + j) : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
#pragma unroll
        for (int j = 0; j < R; ++j) {
          acc[0][j] = fmaf(a[u].x, pv[u][j], acc[0][j]);
          acc[1][j] = fmaf(a[u].y, pv[u][j], acc[1][j]);
          acc[2][j] = fmaf(a[u].z, pv[u][j], acc[2][j]);
          acc[3][j] = fmaf(a[u].w, pv[u][j], acc[3][j]);
        }
    }
  } else {
    for (int row = row_lo + w; row < row_hi; row += 8)
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const float v = k0 + t < mt.m ? base[(int64_t)row * mt.m + k0 + t] : 0.f;
#pragma unroll
        for (int j = 0; j < R; ++j) acc[t][j] = fmaf(v, pm[(int64_t)row * R + j], acc[t][j]);
      }
  }
}

// a matrix whose rank is not the launch's (fewer rows or columns): small
__device__ __noinline__ void q_tile_any(const float* __restrict__ base, const Mat& mt, int k0, int row_lo, int row_hi, const float* __restrict__ pm,
                                        float (&acc)[4][RMAX]) {
  for (int row = row_lo + (threadIdx.x >> 5); row < row_hi; row += 8)
    for (int t = 0; t < 4; ++t) {
      const float v = k0 + t < mt.m ? base[(int64_t)row * mt.m + k0 + t] : 0.f;
      for (int j = 0; j < mt.r; ++j) acc[t][j] = fmaf(v, pm[(int64_t)row * mt.r + j], acc[t][j]);
    }
}

template <int R>
__global__ void __launch_bounds__(256) psgd_q_kernel(const float* __restrict__ e /* holds M = G + E */,
                                                     const int64_t* __restrict__ tab, int n_mats,
                                                     const float* __restrict__ p, float* __restrict__ qout,
                                                     int64_t q_total) {
  __shared__ float red[8][4 * RMAX][32];
  const int64_t block = (int64_t)gridDim.x - 1 - blockIdx.x;
  int mi = find_mat(tab, n_mats, 7, block);
  Mat mt = load_mat(tab, mi);
  pdl_wait();
  pdl_launch_dependents();
  // the table counts, per matrix, column tiles x row chunks (a grid over tiles x the largest chunk count left two thirds of
  // ResNet-50's blocks without rows: 57 us for a 94 MB read)
  const int local = (int)(block - tab[(int64_t)mi * MAT_FIELDS + 7]);
  const int tiles_m = (mt.m + 127) / 128;
  const int tile = local % tiles_m, chunk = local / tiles_m;
  const int c = threadIdx.x & 31, rl = threadIdx.x >> 5;
  const int k0 = tile * 128 + c * 4;
  float acc[4][RMAX];
#pragma unroll
  for (int t = 0; t < 4; ++t)
#pragma unroll
    for (int j = 0; j < RMAX; ++j) acc[t][j] = 0.f;
  const float* pm = p + mt.p_off;
  const bool vec = ((reinterpret_cast<uintptr_t>(e + mt.off) & 15u) == 0) && ((mt.m & 3) == 0);
  const int rpc = rows_per_chunk(mt.n), row_lo = chunk * rpc;
  const int row_hi = row_lo + rpc < mt.n ? row_lo + rpc : mt.n;
  float* qdst = qout + (int64_t)chunk * q_total;          // a chunk writes its own partial copy (copies of chunks a matrix
                                                          // does not have stay zero: the buffer is zeroed once)
  if (k0 < mt.m) {
    if (mt.r == R) q_tile<R>(e + mt.off, mt, k0, row_lo, row_hi, pm, vec, acc);
    else q_tile_any(e + mt.off, mt, k0, row_lo, row_hi, pm, acc);
  }
#pragma unroll
  for (int t = 0; t < 4; ++t)
#pragma unroll
    for (int j = 0; j < RMAX; ++j)
      if (j < mt.r) red[rl][t * RMAX + j][c] = acc[t][j];
  __syncthreads();
  // value (t, j) of column 4c + t by warp: 4 r values over eight warps
  for (int v = rl; v < 4 * RMAX; v += 8) {
    const int t = v / RMAX, j = v % RMAX;
    if (j >= mt.r || k0 + t >= mt.m) continue;
    float s = 0.f;
#pragma unroll
    for (int l = 0; l < 8; ++l) s += red[l][v][c];
    qdst[mt.q_off + (int64_t)(k0 + t) * mt.r + j] = s;
  }
}

// Sum of the row-chunk partials (only launched when some matrix has more than MIN_CHUNK rows).
__global__ void psgd_q_sum_kernel(float* q, const float* parts, int64_t q_total, int chunks) {
  pdl_wait();
  pdl_launch_dependents();
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < q_total; i += stride) {
    float s = parts[i];
#pragma unroll 8
    for (int c = 1; c < chunks; ++c) s += parts[(int64_t)c * q_total + i];
    q[i] = s;
  }
}

// ------------------------------------------------------------------------------------------ G = P Q'^T ; E = M - G
template <int R>
__device__ __forceinline__ void out_long_row(float* __restrict__ g, float* __restrict__ e, int m, const float* __restrict__ p,
                                             const float* __restrict__ qm, int lane) {
  float pr[R];
#pragma unroll
  for (int j = 0; j < R; ++j) pr[j] = p[j];
  for (int k0 = first_column<R>(lane); k0 < m; k0 += 128 * PIECES) {
    float a[PIECES][4];
#pragma unroll
    for (int u = 0; u < PIECES; ++u)
      if (k0 + 128 * u < m) load4<R, false>(e, k0 + 128 * u, m, a[u]);
#pragma unroll
    for (int u = 0; u < PIECES; ++u) {
      if (k0 + 128 * u >= m) continue;
      float q[4][R], o[4];
      load_q4<R>(qm, k0 + 128 * u, m, q);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        o[t] = pr[0] * q[t][0];
#pragma unroll
        for (int j = 1; j < R; ++j) o[t] = fmaf(pr[j], q[t][j], o[t]);
        a[u][t] -= o[t];
      }
      store4<R, true>(g, k0 + 128 * u, m, o);
      store4<R, false>(e, k0 + 128 * u, m, a[u]);
    }
  }
}

template <int R>
__device__ __forceinline__ void out_rows(float* __restrict__ g, float* __restrict__ e, int m, int rows, const float* __restrict__ p,
                                         const float* __restrict__ qm, int lane) {
  float pr[ROWS][R];
#pragma unroll
  for (int u = 0; u < ROWS; ++u)
#pragma unroll
    for (int j = 0; j < R; ++j) pr[u][j] = u < rows ? p[u * R + j] : 0.f;
  for (int k = first_column<R>(lane); k < m; k += 128) {
    float a[ROWS][4];
#pragma unroll
    for (int u = 0; u < ROWS; ++u)
      if (u < rows) load4<R, false>(e + (int64_t)u * m, k, m, a[u]);
    float q[4][R];
    load_q4<R>(qm, k, m, q);
#pragma unroll
    for (int u = 0; u < ROWS; ++u)
      if (u < rows) {
        float o[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          o[t] = pr[u][0] * q[t][0];
#pragma unroll
          for (int j = 1; j < R; ++j) o[t] = fmaf(pr[u][j], q[t][j], o[t]);
          a[u][t] -= o[t];
        }
        store4<R, true>(g + (int64_t)u * m, k, m, o);
        store4<R, false>(e + (int64_t)u * m, k, m, a[u]);
      }
  }
}

// Blocks from row_blocks on carry the 1-D tensors of a single worker: their mean is the gradient itself.
template <int CAP, int R>
__global__ void __launch_bounds__(256) psgd_out_kernel(const __grid_constant__ GradPtrs<CAP> gp, float* __restrict__ e,
                                                       const int64_t* __restrict__ tab, int n_mats,
                                                       const float* __restrict__ p, const float* __restrict__ q, int row_blocks,
                                                       const int64_t* __restrict__ vtab, int n_vecs) {
  if ((int)blockIdx.x >= row_blocks) {
    pdl_wait();
    for (int v = blockIdx.x - row_blocks; v < n_vecs; v += gridDim.x - row_blocks) {
      const int64_t off = vtab[v * VEC_FIELDS], len = vtab[v * VEC_FIELDS + 1];
      const int tensor = (int)vtab[v * VEC_FIELDS + 3];
      const float* src = gp.src(tensor, off);
      float* dst = gp.dst(tensor, off);
      for (int64_t i = threadIdx.x; i < len; i += blockDim.x) { dst[i] = src[i]; e[off + i] = 0.f; }
    }
    return;
  }
  const int lane = threadIdx.x & 31;
  const int mi = find_mat(tab, n_mats, 6, (int64_t)blockIdx.x);
  const Mat mt = load_mat(tab, mi);
  pdl_wait();
  const int rpb = rows_per_block(mt.m), row0 = (int)((int64_t)blockIdx.x - tab[(int64_t)mi * MAT_FIELDS + 6]) * rpb;
  const int row1 = row0 + rpb < mt.n ? row0 + rpb : mt.n;
  const float* qm = q + mt.q_off;
  const int group = rpb < ROWS * 8 ? rpb / 8 : ROWS;
  for (int row = row0 + (threadIdx.x >> 5) * group; row < row1; row += 8 * group) {
    float* g = gp.dst(mt.tensor, mt.off) + (int64_t)row * mt.m;
    float* er = e + mt.off + (int64_t)row * mt.m;
    const float* pr = p + mt.p_off + (int64_t)row * mt.r;
    const int rows = row1 - row < group ? row1 - row : group;
    const bool vec = (((reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(er)) & 15u) == 0) && ((mt.m & 3) == 0) && ((mt.q_off & 3) == 0) && mt.r == R;
    if (vec && group == 1) out_long_row<R>(g, er, mt.m, pr, qm, lane);
    else if (vec) out_rows<R>(g, er, mt.m, rows, pr, qm, lane);
    else
      for (int u = 0; u < rows; ++u, g += mt.m, er += mt.m, pr += mt.r)
        for (int k = lane; k < mt.m; k += 32) {
          float s = 0.f;
          for (int j = 0; j < mt.r; ++j) s = fmaf(pr[j], qm[(int64_t)k * mt.r + j], s);
          g[k] = s;
          er[k] -= s;
        }
  }
}

// 1-D tensors: g[off + i] = alpha * summed[dst + i]; their error memory stays zero.
__global__ void psgd_unpack_vec_kernel(float* __restrict__ g, float* __restrict__ e, const int64_t* __restrict__ vtab,
                                       int n_vecs, const float* __restrict__ summed, float alpha) {
  for (int v = blockIdx.x; v < n_vecs; v += gridDim.x) {
    int64_t off = vtab[v * VEC_FIELDS], len = vtab[v * VEC_FIELDS + 1], dst = vtab[v * VEC_FIELDS + 2];
    for (int64_t i = threadIdx.x; i < len; i += blockDim.x) {
      g[off + i] = alpha * summed[dst + i];
      e[off + i] = 0.f;
    }
  }
}

#define FOR_RANK(rank, CALL) \
  switch (rank) {            \
    case 1: { constexpr int R = 1; CALL; break; } \
    case 2: { constexpr int R = 2; CALL; break; } \
    case 3: { constexpr int R = 3; CALL; break; } \
    case 4: { constexpr int R = 4; CALL; break; } \
    default: return (int)cudaErrorInvalidValue; }

template <int CAP>
int solo(int rank, const SegDesc* d, int n_seg, float* e, const int64_t* tab, int n_mats, int64_t row_blocks, int64_t total_tiles, int max_rows, const int64_t* vtab,
         int n_vecs, float* q, float* p, float* q_parts, int64_t q_total, uint64_t seed, uint32_t stream_id, uint32_t* step, cudaStream_t st) {
  GradPtrs<CAP> gp;
  for (int i = 0; i < n_seg; ++i) { gp.in[i] = d[i].in; gp.out[i] = d[i].out; }
  const int vec_blocks = n_vecs < 64 ? n_vecs : 64;
  if (n_mats > 0) {
    if (step != nullptr) {
      int err = gc_cuda_philox_fill(1, seed, stream_id, 0, step, q_total, q, st);
      if (err) return err;
    }
    // Each kernel is looked up in the tables and waits while its predecessor ends (VGG-16, rank 2: 83.9 -> 73.6 us a call).  Without a
    // draw in front the tables may be the stream's last write: an ordinary launch.
    if (step != nullptr) FOR_RANK(rank, (launch_pdl(psgd_p_kernel<CAP, R>, dim3((unsigned)row_blocks), dim3(256), 0, st, gp, e, tab, n_mats, (const float*)q, p, step)))
    else FOR_RANK(rank, (psgd_p_kernel<CAP, R><<<(unsigned)row_blocks, 256, 0, st>>>(gp, e, tab, n_mats, q, p, step)))
    launch_pdl(psgd_gs_kernel, dim3(n_mats), dim3(GS_THREADS), 0, st, p, tab, 1e-8f);
    const int chunks = gc_cuda_psgd_q_chunks(max_rows);
    float* dst = chunks > 1 ? q_parts : q;
    FOR_RANK(rank, (launch_pdl(psgd_q_kernel<R>, dim3((unsigned)total_tiles), dim3(256), 0, st, (const float*)e, tab, n_mats, (const float*)p, dst, q_total)))
    if (chunks > 1) {
      const int64_t b = (q_total + 255) / 256;
      launch_pdl(psgd_q_sum_kernel, dim3((unsigned)(b < 1024 ? b : 1024)), dim3(256), 0, st, q, (const float*)q_parts, q_total, chunks);
    }
  }
  if (n_mats > 0)
    FOR_RANK(rank, (launch_pdl(psgd_out_kernel<CAP, R>, dim3((unsigned)(row_blocks + vec_blocks)), dim3(256), 0, st, gp, e, tab, n_mats, (const float*)p, (const float*)q,
                               (int)row_blocks, vtab, n_vecs)))
  else if (vec_blocks > 0)
    FOR_RANK(rank, (psgd_out_kernel<CAP, R><<<(unsigned)vec_blocks, 256, 0, st>>>(gp, e, tab, n_mats, p, q, 0, vtab, n_vecs)))
  return (int)cudaGetLastError();
}

}  // namespace

extern "C" {

int gc_cuda_psgd_max_rank() { return RMAX; }

// stage = [P (p_total floats) | packed 1-D tensors]; e <- g + e for the matrices.
int gc_cuda_psgd_p(int rank, const float* g, float* e, const int64_t* tab, int n_mats, int64_t row_blocks, const float* q,
                   float* stage, const int64_t* vtab, int n_vecs, int64_t vec_base, void* cs) {
  cudaStream_t st = (cudaStream_t)cs;
  if (n_mats > 0 && row_blocks > 0) {
    GradPtrs<1> gp;
    gp.in[0] = g;
    gp.out[0] = nullptr;
    FOR_RANK(rank, (psgd_p_kernel<1, R><<<(unsigned)row_blocks, 256, 0, st>>>(gp, e, tab, n_mats, q, stage, nullptr)))
  }
  if (n_vecs > 0) psgd_pack_vec_kernel<<<n_vecs < 256 ? n_vecs : 256, 512, 0, st>>>(g, vtab, n_vecs, stage + vec_base);
  return (int)cudaGetLastError();
}

int gc_cuda_psgd_gs(float* p, const int64_t* tab, int n_mats, float eps, void* cs) {
  if (n_mats > 0) psgd_gs_kernel<<<n_mats, GS_THREADS, 0, (cudaStream_t)cs>>>(p, tab, eps);
  return (int)cudaGetLastError();
}

// Partial sums the Q' kernel leaves for matrices of up to max_rows rows.
int gc_cuda_psgd_q_chunks(int max_rows) {
  const int c = (max_rows + MIN_CHUNK - 1) / MIN_CHUNK;
  return c < MAX_CHUNKS ? c : MAX_CHUNKS;
}

// Blocks the P and output kernels run for an n x m matrix (the table's column 6 counts these).
int64_t gc_cuda_psgd_row_blocks(int n, int m) { return (n + rows_per_block(m) - 1) / rows_per_block(m); }

// Blocks the Q' kernel runs for an n x m matrix: 128-column tiles x row chunks (the table's tile_start column counts these).
int64_t gc_cuda_psgd_q_blocks(int n, int m) { return (int64_t)((m + 127) / 128) * ((n + rows_per_chunk(n) - 1) / rows_per_chunk(n)); }

// qout must hold gc_cuda_psgd_q_chunks(max_rows) * q_total floats, zeroed once; the result ends up in its first q_total.
// total_tiles: sum over matrices of gc_cuda_psgd_q_blocks(n, m), the same count the table's tile_start column accumulates.
int gc_cuda_psgd_q(int rank, const float* e, const int64_t* tab, int n_mats, int64_t total_tiles, const float* p, float* qout,
                   int64_t q_total, int max_rows, void* cs) {
  if (n_mats > 0 && total_tiles > 0) {
    int chunks = gc_cuda_psgd_q_chunks(max_rows);
    FOR_RANK(rank, (psgd_q_kernel<R><<<dim3((unsigned)total_tiles), 256, 0, (cudaStream_t)cs>>>(e, tab, n_mats, p, qout, q_total)))
    if (chunks > 1) {
      int64_t blocks = (q_total + 255) / 256;
      psgd_q_sum_kernel<<<(int)(blocks < 1024 ? blocks : 1024), 256, 0, (cudaStream_t)cs>>>(qout, qout, q_total, chunks);
    }
  }
  return (int)cudaGetLastError();
}

int gc_cuda_psgd_out(int rank, float* g, float* e, const int64_t* tab, int n_mats, int64_t row_blocks, const float* p,
                     const float* q, const int64_t* vtab, int n_vecs, const float* summed_vecs, float alpha, void* cs) {
  cudaStream_t st = (cudaStream_t)cs;
  if (n_mats > 0 && row_blocks > 0) {
    GradPtrs<1> gp;
    gp.in[0] = g;
    gp.out[0] = g;
    FOR_RANK(rank, (psgd_out_kernel<1, R><<<(unsigned)row_blocks, 256, 0, st>>>(gp, e, tab, n_mats, p, q, (int)row_blocks, vtab, 0)))
  }
  if (n_vecs > 0)
    psgd_unpack_vec_kernel<<<n_vecs < 256 ? n_vecs : 256, 512, 0, st>>>(g, e, vtab, n_vecs, summed_vecs, alpha);
  return (int)cudaGetLastError();
}

// The whole step of a single worker on n_seg tensors (one flat segment, or one per tensor).  q: drawn from the seed's stream at
// *step first when `step` is given (the counter is advanced), used as it is otherwise; then the result.  p: p_total floats.
int gc_cuda_psgd_solo(int rank, const void* segs, int n_seg, float* e, const int64_t* tab, int n_mats, int64_t row_blocks, int64_t total_tiles, int max_rows,
                      const int64_t* vtab, int n_vecs, float* q, float* p, float* q_parts, int64_t q_total, uint64_t seed, uint32_t stream_id,
                      uint32_t* step, void* cs) {
  if (n_seg < 1 || n_seg > SEG_CAP_MANY) return (int)cudaErrorInvalidValue;
  const SegDesc* d = (const SegDesc*)segs;
  if (n_seg == 1) return solo<1>(rank, d, n_seg, e, tab, n_mats, row_blocks, total_tiles, max_rows, vtab, n_vecs, q, p, q_parts, q_total, seed, stream_id, step, (cudaStream_t)cs);
  return solo<SEG_CAP_MANY>(rank, d, n_seg, e, tab, n_mats, row_blocks, total_tiles, max_rows, vtab, n_vecs, q, p, q_parts, q_total, seed, stream_id, step, (cudaStream_t)cs);
}

}  // extern "C"
