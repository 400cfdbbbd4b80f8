// Building blocks of the tcgen05 kernels (TF32 GEMMs and implicit-GEMM convolutions): mbarrier / TMA / UMMA
// wrappers, shared-memory descriptors, and the two kernel templates that both the GEMM entry points
// (gc_gemm_tc.cu) and the convolution entry points (gc_conv_tc.cu) instantiate:
//
//   gemm_tf32_persistent_kernel  C[M, N] (=, +=) A[M, K] * B[N, K]^T (+ bias), K-major operands, one CTA per SM.
//                                A comes either from a 2-D map (plain GEMM, 1x1 convolution) or from a 4-D map over
//                                an NHWC activation, one shifted box per filter tap and 32-channel block (implicit
//                                GEMM of an R x S convolution, stride 1 or 2; the zero padding is the TMA's
//                                out-of-range fill).
//   gemm_tn_tf32_kernel          C[Mo, No] += A[P, Mo]^T * B[P, No], MN-major operands, split-K.  B comes either from
//                                a 2-D map or from shifted 4-D boxes of the activation (weight gradient of an R x S
//                                convolution: one filter tap per output tile).
//
// No TMA multicast: every CTA loads its own operands (of a CTA pair: its half of them).  Every mbarrier wait is bounded; when one runs out
// the CTA sets *error_flag, abandons its tile, frees its TMEM and returns.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "gc_device.cuh"

// Measurement knobs shared by every translation unit of the library (set through gc_cuda_gemm_tf32_config /
// gc_cuda_gemm_tn_config): forced tile width (0 = choose), CTAs per SM the split contraction aims at, fewest
// k-blocks (of TBK rows) a split may get.
namespace gctc {
inline int tile_choice = 0;
inline int pair_choice = 0;    // CTA pairs in the persistent kernel: 0 = modelled, 1 = never, 2 = wherever there are two row tiles
inline int tn_ctas_per_sm = 1;
inline int tn_min_kblocks = 8;
inline int wgrad_two_taps = 0;
inline int split_choice = 0;   // contraction splits of the persistent kernel: 0 = modelled, 1 = never, n = n where a product allows it
inline int taps_choice = 0;    // input gradients of 3x3 convolutions with one load of the pixels per filter column: 0 = wherever the shape allows it, 1 = never
inline int tma_mode = 1;   // bit 0: prefetch the tensor maps at kernel start; bit 2: epilogue warps sleep between polls while a tile is being accumulated
}  // namespace gctc

namespace {

constexpr int BM = 128;
constexpr int BK = 32;                       // 32 fp32 = 128 bytes = one swizzle row
constexpr int UMMA_K = 8;                    // tf32
constexpr int TBK = 32;                      // contraction rows per stage of the split-K (MN-major) kernel: 4 KB TMA boxes
constexpr int GEMM_THREADS = 192;           // one-tile-per-CTA kernel: producer warp, MMA warp, four epilogue warps
// The persistent and the split-K kernels have TWO producer warps that take alternate stages of the ring: a warp is through its wait,
// its expect_tx and its copies while the other one waits for the next stage.  With one warp filling every stage (issuing under
// elect.sync all the same) a step of ResNet-50 at batch 128 takes 6438 us instead of 6170, of VGG-16 1233 instead of 1121, an evaluation
// batch of ResNet-50 2933 instead of 2842 (one B200).
constexpr int PRODUCER_WARPS = 2;
constexpr int MMA_WARP = PRODUCER_WARPS;     // warp that allocates TMEM and issues tcgen05.mma
constexpr int FIRST_EPI_WARP = PRODUCER_WARPS + 1;
constexpr unsigned long long WAIT_LIMIT_NS = 2000000000ull;   // a wait gives up after two seconds

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// Bounded wait for the phase with the given parity; false = gave up.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  uint32_t addr = smem_u32(bar);
  unsigned long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((it & 63u) == 63u) {
      if (*abort_flag) return false;
      unsigned long long now;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
      if (t0 == 0) t0 = now;
      else if (now - t0 > WAIT_LIMIT_NS) break;
    }
  }
  *abort_flag = 1;
  return false;
}

// The same wait for a whole converged warp, with one answer for the warp: what follows stays uniform control flow.
// CLUSTER: arrivals may come from the other CTA of a pair.
template <bool CLUSTER = false>
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag) {
  const uint32_t addr = smem_u32(bar);
  unsigned long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t ok;
    if constexpr (CLUSTER)
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(ok)
          : "r"(addr), "r"(parity)
          : "memory");
    else
      asm volatile(
          "{\n\t.reg .pred p;\n\t"
          "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
          "selp.u32 %0, 1, 0, p;\n\t}"
          : "=r"(ok)
          : "r"(addr), "r"(parity)
          : "memory");
    if (__all_sync(0xffffffffu, ok)) return true;
    if ((it & 63u) == 63u) {
      unsigned long long now;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
      if (t0 == 0) t0 = now;
      if (__any_sync(0xffffffffu, *abort_flag != 0 || now - t0 > WAIT_LIMIT_NS)) break;
    }
  }
  *abort_flag = 1;
  return false;
}

// One lane of a converged warp, chosen so that the compiler knows it to be one: TMA and MMA instructions under this predicate
// take their operands from uniform registers.  Under `lane == 0` in a divergent branch each of them first moves its
// descriptors there one by one: four MMAs and a commit took the issuing thread 340 cycles, a stage's TMA loads 400 (clock64,
// B200), and a k-block of every width 590 cycles, whatever its tensor time (128 / 256 / 512 cycles at 64 / 128 / 256 columns).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(p));
  return p != 0;
}

// The same wait for warps that have nothing to do for a long time (the epilogue warps during a tile's main loop): between
// polls they sleep, so that their polling does not take issue slots from the single threads that feed the TMA unit and
// the tensor core on the same SM sub-partitions.
__device__ __forceinline__ bool mbar_wait_idle(uint64_t* bar, uint32_t parity, volatile int* abort_flag, unsigned sleep_ns) {
  uint32_t addr = smem_u32(bar);
  unsigned long long t0 = 0;
  for (uint32_t it = 0;; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
    if (sleep_ns) __nanosleep(sleep_ns);
    if ((it & 15u) == 15u) {
      if (*abort_flag) return false;
      unsigned long long now;
      asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
      if (t0 == 0) t0 = now;
      else if (now - t0 > WAIT_LIMIT_NS) break;
    }
  }
  *abort_flag = 1;
  return false;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

__device__ __forceinline__ void tma_prefetch_map(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}

__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

// The same loads for a CTA of a pair (cta_group::2): the data lands in this CTA's shared memory, the bytes are counted on the
// barrier of the CTA that issues the MMAs (`bar`: a shared::cluster address).
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d_pair(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}
__device__ __forceinline__ void tma_load_5d_pair(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3, int c4, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
      : "memory");
}

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
  return r;
}
// Address of this CTA's shared variable `p` in the CTA of the cluster with the given rank.
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
  return a;
}
// Every thread of both CTAs of a pair.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync_all() {
  cluster_arrive();
  cluster_wait();
}

// Where the rows of an operand come from when it is an NHWC activation [N, H, W, C] read through a 4-D map
// {C, W, H, N} instead of a matrix: output position p = (n, ho, wo) and filter tap (r, s) read the pixel
// (n, ho * stride + r - pad, wo * stride + s - pad); `rows_per_box` consecutive output positions are one box
// (whole output rows of one image, or whole images), taps == 0 means "a plain 2-D matrix".  The map's element
// strides carry the convolution stride, so a box always starts at the first position's pixel.
struct ConvA {
  int taps;        // R * S, 0 = plain matrix
  int fs;          // S (filter width)
  int cblocks;     // C / 32: k-blocks per tap
  int hw_out;      // output positions per image
  int w_out;       // output width
  int stride, pad;
  // B operand given as a matrix W[K rows, taps * ldtap columns] whose N index is the contiguous one (an input gradient
  // reading the forward filter [Cout][R][S][Cin] in place: K = Cout, N = Cin): b_mn = 1.  The A-side tap (fr, fs) then
  // multiplies the filter tap (b_r0 + b_dr * fr, b_s0 + b_ds * fs) -- rotation by 180 degrees for a stride-1 input gradient,
  // every second tap for a parity class of a stride-2 one -- found at column ((r * b_fs + s) * b_ldtap + n).  b_mn = 2: the
  // map is the 3-D view {32 floats, K rows, columns / 32} of the same matrix (b_ldtap a multiple of 32) and one box loads
  // a whole stage of B.
  int b_mn, b_ldtap, b_fs, b_r0, b_dr, b_s0, b_ds;
  // All four parity classes (ph, pw) of a stride-2 input gradient in one launch: taps along an axis of the classes of parity 0 and 1; the
  // filter tap of class (ph, pw) starts at (b_r0 + ph, b_s0 + pw).  0: not used.
  int class_taps0, class_taps1;
};

// The input gradient of a 3x3, stride-1, padding-1 convolution, where the three taps of a filter COLUMN share one copy of dY's pixels.
// The map's dimensions are {C, W, N, H}, so a tile of 128 positions lies in shared memory as rows (h, n, w) of 128 bytes and the pixels one
// image row further down are `step` = W * images * 128 bytes further on: the operand of tap (r, s) is the box of column shift s read
// from a start address moved by r steps (a multiple of 1024 bytes, so the swizzle pattern stays in place).  A stage holds the box
// and the filter's three taps of that column and 32-channel block, read in place (ConvA, b_mn = 2); it is good for 3 k-blocks.  A tile of
// whole images needs no rows from outside: the zeros above and below it are gaps between the stages, written once.  Otherwise the box
// carries one more image row at each end.
// Why: with a box per tap a k-block of a CTA pair fills 16 KB of pixels and BN / 2 rows of filter into shared memory, at some 50 bytes a cycle and
// SM, while its MMAs read the same again; that, not the tensor pipe, took the time.  Pixels are now 5.3 to 8 KB a k-block.  A k-block of a pair at 128
// columns: 200 -> 144 ns (16x16x128, batch 256 against 128), at 64 columns 205 -> 103.  Input gradients back to back, one B200: 32x32x64 at batch 128
// 29.9 -> 21.0 us, 16x16x128 20.5 -> 18.5, 2x2x512 12.1 -> 12.2, 16x16x128 at batch 256 34.7 -> 29.1, at batch 31 12.2 -> 10.9.
// The forward pass keeps a box per tap: this contraction runs through its channel blocks first, and a sum in another order than before moves
// the last bit of an activation, which moves a ResNet-50's logits by up to 1.2 per cent.
struct TapCols {
  int box_bytes;           // pixels of a stage; 0 = off (the kernel variant without it)
  int pitch;               // bytes between the pixels of neighbouring stages
  int first;               // offset of the first stage's pixels = the gap in front of them
  int step;                // one image row further down
  int lead;                // tap (0, s) starts this many bytes in front of the box (whole images: `step`, else 0)
  int h_off;               // image row of the box's first pixel, relative to the tile's
  int stages;
  int b_off;               // filter taps of the first stage
};

// Where the rows of the OUTPUT go when it is not a matrix but a strided sub-grid of an NHWC tensor read through a 4-D map
// {C, W', H', N} (the input gradient of a stride-2 convolution where a parity class of input pixels is a launch of its own; all classes in one: a 5-D map): row
// p = (n, i, j) of the result is stored at coordinates (column, j, i, n).  hw == 0: a plain 2-D matrix.
// nh: the map's dimensions are {C, W', N, H'}, for tiles whose rows run (h, image, w).
struct ConvC {
  int hw;          // rows per image (H' * W'), 0 = plain matrix
  int w;           // W'
  int nh;
};

// Batch-norm statistics finished inside the GEMM that produces the activation: every CTA keeps per-column sums and sums
// of squares of its tiles, adds them to `acc` ([2][N] doubles, zero on entry) with atomics when it is done, and the
// epilogue group that draws the last ticket turns the totals into mean / 1 / sqrt(var + eps) (`stats`, [2N] floats),
// updates the running statistics and leaves `acc` and `ticket` zeroed for the next launch.  Needs every CTA to stay on
// one column tile (the launcher makes the grid a multiple of the number of column tiles).  acc == NULL: off.
struct BnFin {
  double* acc;
  unsigned int* ticket;
  float* stats;
  float* running_mean;     // may be NULL
  float* running_var;
  float momentum, eps;
};

// Batch norm of running statistics in the epilogue (inference): out = act((acc + bias - mean) * rstd * gamma + beta [+ residual]) per
// column, rounded as the apply kernels round it: folded into one multiply-add, the rounding alone moved the logits of a
// ResNet-50 by a per cent (a last bit more or less decides where the next layer's TF32 operands are cut).
// residual: [M, N], row pitch N.
struct Affine {
  const float *gamma, *beta, *mean, *var, *residual;
  float eps;
  int relu;
};

// What the host passes to ask for it: `scratch` holds the ticket (first 256 bytes) and the totals (2 * N doubles), is
// zeroed once when allocated (gc_cuda_bn_fin_scratch_bytes) and is left zeroed by every launch that uses it.
struct BnFinHost {
  void* scratch;
  float* stats;
  float* running_mean;
  float* running_var;
  float momentum, eps;
};

inline BnFin bn_fin_from_host(const void* host_args) {
  BnFin f{};
  if (host_args != nullptr) {
    const BnFinHost* h = static_cast<const BnFinHost*>(host_args);
    if (h->scratch != nullptr) {
      f.ticket = static_cast<unsigned int*>(h->scratch);
      f.acc = reinterpret_cast<double*>(static_cast<uint8_t*>(h->scratch) + 256);
      f.stats = h->stats;
      f.running_mean = h->running_mean;
      f.running_var = h->running_var;
      f.momentum = h->momentum;
      f.eps = h->eps;
    }
  }
  return f;
}

// TMA coordinates {c, w, h, n} of the box that holds output positions p0 .. of filter tap `tap`, channel block `cb`.
__device__ __forceinline__ void conv_box(const ConvA& ca, int64_t p0, int tap, int cb, int (&co)[4]) {
  const int n = (int)(p0 / ca.hw_out);
  const int rem = (int)(p0 - (int64_t)n * ca.hw_out);
  const int h0 = rem / ca.w_out, w0 = rem - h0 * ca.w_out;
  const int r = tap / ca.fs, s = tap - r * ca.fs;
  co[0] = cb * 32;
  co[1] = w0 * ca.stride + s - ca.pad;
  co[2] = h0 * ca.stride + r - ca.pad;
  co[3] = n;
}

// K-major operand tile in the canonical 128-byte-swizzled layout (rows of 128 B, groups of 8 rows = 1024 B).
__device__ __forceinline__ uint64_t make_smem_desc(const void* tile) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_u32(tile) & 0x3FFFF) >> 4);      // start address, bits [0, 14)
  d |= (uint64_t)1 << 16;                                // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;                      // stride byte offset: 8 rows * 128 B
  d |= (uint64_t)1 << 46;                                // descriptor version (sm_100)
  d |= (uint64_t)2 << 61;                                // layout type: SWIZZLE_128B
  return d;
}

// MN-major operand tile: chunks of 32 floats of the M / N dimension x `rows` K rows (128 bytes each), one after the other.
__device__ __forceinline__ uint64_t make_smem_desc_mn_rows(const void* tile, int rows) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_u32(tile) & 0x3FFFF) >> 4);      // start address
  d |= (uint64_t)((rows * 128) >> 4) << 16;              // leading byte offset: next 32-float chunk of the M / N dimension
  d |= (uint64_t)(512 >> 4) << 32;                       // stride byte offset: next group of 4 K rows
  d |= (uint64_t)1 << 46;                                // descriptor version (sm_100)
  d |= (uint64_t)1 << 61;                                // layout type: SWIZZLE_128B_BASE32B
  return d;
}

__device__ __forceinline__ uint64_t make_smem_desc_mn(const void* tile) { return make_smem_desc_mn_rows(tile, TBK); }

// kind::tf32, fp32 accumulate, both operands K-major, M = m (128, or 256 rows of a CTA pair), N = n.
__host__ __device__ constexpr uint32_t make_idesc(int n, int m = BM) {
  return (1u << 4)                 // C format: F32
         | (2u << 7)               // A format: TF32
         | (2u << 10)              // B format: TF32
         | ((uint32_t)(n >> 3) << 17)
         | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void umma_tf32(uint32_t tmem_c, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}"
      ::"r"(tmem_c), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
      : "memory");
}
// 256 rows in two CTAs: rows 0..127 of A and columns 0..n/2 of B in the first CTA's shared memory, the others at the same
// offsets in the second's; each CTA's TMEM receives its 128 rows.  Issued by one thread of the first CTA.
__device__ __forceinline__ void umma_tf32_pair(uint32_t tmem_c, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::tf32 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
      ::"r"(tmem_c), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(0u)
      : "memory");
}
// Arrives on the barrier at this offset in both CTAs of the pair.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16_nowait(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }


// ------------------------------------------------------------------------------------------------
// Persistent variant: one CTA per SM walks a strided list of output tiles.  The accumulator is double
// buffered in TMEM (2 x BN columns), so the MMA warp works on tile i + 1 while the epilogue warps drain
// tile i; the TMA loads run ahead across tile boundaries through the same ring of stages; two groups of
// four epilogue warps take alternate 32-column slabs, each group staging them in its own ring of dedicated
// buffers and waiting for a TMA store only when it needs that store's buffer back.  Tiles are ordered
// with the column tile fastest: CTAs that run at the same time share the rows of A in L2.
template <int BN, bool PAIR, bool TAPS = false>
struct PSmem {
  // Up to 128 columns two staging slabs are enough and the ring gets what they leave (28.7 against 29.7 us at 16x16x128 3x3,
  // 65.5 against 74.9 us at 8x8x512 in pairs); at 256 columns the epilogue has as much to store as the ring to load, and
  // two slabs cost the 1x1 layers 10 % (ResNet-50, batch 128: 900 against 819 us of a step).
  static constexpr int STAGES = PAIR ? ((BN <= 64) ? 9 : ((BN <= 128) ? 7 : 4)) : ((BN <= 64) ? 7 : ((BN <= 128) ? 5 : 3));
  static constexpr int A_BYTES = BM * BK * 4;
  static constexpr int B_COLS = PAIR ? BN / 2 : BN;         // columns of B in this CTA's shared memory
  static constexpr int B_BYTES = B_COLS * BK * 4;           // a multiple of 1024
  static constexpr int NSLAB = BN <= 128 ? 2 : 4;
  static constexpr int SLAB_BYTES = BM * 128;
  static constexpr int TAPS_STAGE_B = 3 * B_BYTES;          // TAPS: the filter's three taps of a column
  static constexpr int MAX_STAGES = 12;
  static constexpr int LIMIT = 232448;                      // shared memory of one CTA
  static constexpr int RING_BYTES = TAPS ? (LIMIT - 1024 - 256 - 4 * BN * 2 * 4 - NSLAB * SLAB_BYTES) / 1024 * 1024 : STAGES * (A_BYTES + B_BYTES);
  static constexpr int STAGING_OFF = RING_BYTES;
  static constexpr int BAR_OFF = STAGING_OFF + NSLAB * SLAB_BYTES;
  static constexpr int COLSUM_OFF = BAR_OFF + 256;
  static constexpr int TOTAL = 1024 /* alignment slack */ + COLSUM_OFF + 4 * BN * 2 * 4;
  static constexpr int TMEM_COLS = 2 * BN;
  static_assert(!TAPS || BN <= 128, "tile widths of the kernel with shared pixels");
  static_assert((2 * MAX_STAGES + 4) * 8 + 4 <= 256 && STAGES <= MAX_STAGES, "barriers");
  static_assert(BN == 64 || BN == 128 || BN == 256, "tile widths of the persistent kernel");
  static_assert(TOTAL <= LIMIT, "shared memory of one CTA");
};

// Named barrier of one epilogue group (ids 1 and 2; 0 is __syncthreads).
__device__ __forceinline__ void group_bar(int grp) {
  if (grp == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
  else asm volatile("bar.sync 2, 128;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_remote(uint32_t cluster_address) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_address) : "memory");
}

constexpr int EPI_GROUPS = 2;
constexpr int PERSISTENT_THREADS = 32 * FIRST_EPI_WARP + 128 * EPI_GROUPS;
constexpr int TN_THREADS = PERSISTENT_THREADS;

// AFFINE: the epilogue of inference (a kernel of its own: its residual registers slowed the training epilogue by 3 %).
//
// PAIR: two CTAs of a cluster work on one tile of 256 rows (cta_group::2).  Each loads its 128 rows of A and HALF of the columns
// of B, so a k-block costs a CTA 128 + BN / 2 rows of shared-memory fill and of operand reads instead of 128 + BN, which is
// what bounds the single-CTA form.  The first CTA of the pair issues the MMAs and holds the barriers they wait for; commits go
// to both.  Work items are the pairs' tiles; everything after the accumulator is each CTA's own.
//
// FORM:
//   PLAIN    one matrix product or convolution
//   SHARED   the input gradient of a 3x3 convolution whose filter columns share a copy of the pixels (TapCols); a stage is 3 k-blocks
//   CLASSES  the input gradient of a stride-2 convolution: four products of different depths (one, two, two and four filter taps for 3x3), one per parity
//            class of input pixels, on the same pixels of dY and the same filter.  Deepest first, and every second round of the workers backwards, so that a
//            worker gets deep and shallow tiles.  The output is a 5-D map {2 C, W / 2, 2, H / 2, N}.  One launch per class left much of
//            the chip idle and could not afford wide tiles: 32x32x128 at batch 128 44.5 -> 28.6 us, 16x16x256 40.5 -> 21.1, 8x8x512 48.1 -> 19.1, at
//            batch 31 32x32x64 -> 128 25.9 -> 8.3, 16x16x128 -> 256 32.9 -> 10.5, 8x8x256 -> 512 45.7 -> 14.2 (back to back).
constexpr int PLAIN = 0, SHARED = 1, CLASSES = 2;

template <int BN, bool AFFINE, bool PAIR, int FORM>
__global__ void __launch_bounds__(PERSISTENT_THREADS, 1)
gemm_tf32_persistent_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                            const __grid_constant__ CUtensorMap tma_c, const ConvA ca, const float* __restrict__ bias, int M, int N, int K,
                            int tiles_m, int tiles_n, int splits, int accumulate, float* __restrict__ col_partials,
                            int* __restrict__ error_flag, int tma_mode, const BnFin fin, const ConvC cc, int cta_sums, const Affine aff,
                            const TapCols tc) {
  constexpr bool TAPS = FORM == SHARED;
  using S = PSmem<BN, PAIR, TAPS>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t stages = TAPS ? (uint32_t)tc.stages : (uint32_t)S::STAGES;
  const int a_pitch = TAPS ? tc.pitch : S::A_BYTES;
  constexpr int B_STAGE = TAPS ? S::TAPS_STAGE_B : S::B_BYTES;
  uint8_t* a_tiles = base + (TAPS ? tc.first : 0);
  uint8_t* b_tiles = base + (TAPS ? tc.b_off : S::STAGES * S::A_BYTES);
  uint8_t* staging = base + S::STAGING_OFF;
  uint64_t* full = reinterpret_cast<uint64_t*>(base + S::BAR_OFF);
  uint64_t* empty = full + S::MAX_STAGES;
  uint64_t* acc_full = empty + S::MAX_STAGES;      // [2] MMA -> epilogue: accumulator complete
  uint64_t* acc_empty = acc_full + 2;          // [2] epilogue -> MMA: accumulator drained
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  float* colsum = reinterpret_cast<float*>(base + S::COLSUM_OFF);      // [4 row quarters][BN columns][2]
  __shared__ int abort_flag;
  __shared__ int epi_go[EPI_GROUPS];

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int num_k = TAPS ? 3 * ca.cblocks : (K + BK - 1) / BK;      // stages of a whole contraction
  // work item = (output tile, split of the contraction); the splits of one tile are neighbours in the list, so they run
  // at the same time on different SMs and add their partial tiles in L2 (the host passes accumulate = 1 and a zeroed C)
  const int per_class = tiles_m * tiles_n;                     // CLASSES: items of a class (no splits); tiles_m: of 128 rows, PAIR: of 256
  const int total_items = FORM == CLASSES ? 4 * per_class : per_class * splits;
  const int kps = (num_k + splits - 1) / splits;
  const int rank = PAIR ? (int)cluster_rank() : 0;
  const int worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x, workers = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  // from a worker's item to its next one; CLASSES: the step after that is 2 * workers - step
  const int first_step = FORM == CLASSES ? 2 * (workers - worker) - 1 : workers;
  auto turn_step = [&](int step) { return FORM == CLASSES ? 2 * workers - step : step; };
  auto class_depth = [&](int ph, int pw) { return (ph ? ca.class_taps1 : ca.class_taps0) * (pw ? ca.class_taps1 : ca.class_taps0) * ca.cblocks; };

  if (threadIdx.x == 32 * FIRST_EPI_WARP && (tma_mode & 1)) { tma_prefetch_map(&tma_a); tma_prefetch_map(&tma_b); tma_prefetch_map(&tma_c); }
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int g = 0; g < EPI_GROUPS; ++g) epi_go[g] = 1;
    for (uint32_t s = 0; s < stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], (PAIR ? 2 : 1) * EPI_GROUPS); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)S::TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)S::TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  if constexpr (TAPS) {
    // the zero rows above and below a tile of whole images: the gap in front of every stage's pixels and behind the last one's
    const int quads = tc.lead >> 4, pitch = tc.pitch;
    for (int i = threadIdx.x; i < quads * (tc.stages + 1); i += PERSISTENT_THREADS) {
      const int gap = i / quads;
      *reinterpret_cast<float4*>(base + gap * pitch + (i - gap * quads) * 16) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (quads != 0) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  tc_fence_before();
  if constexpr (PAIR) cluster_sync_all();      // every thread of both CTAs: the other one's barriers and TMEM are in place, too
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  // everything above (barriers, TMEM) overlapped the tail of the previous kernel of the stream; its results are
  // needed from here on
  gc::pdl_wait();
  gc::pdl_launch_dependents();

  if (warp < PRODUCER_WARPS) {
    // producer warp p fills the stages of k-blocks it == p (mod PRODUCER_WARPS) of the ring
    uint32_t s = 0, phase = 0;                                // stage and its phase of the next k-block, over all tiles
    static_assert(PRODUCER_WARPS == 2, "two warps take turns");
    int turn = 0;                                             // producer warp that fills it
    bool ok = true;
    for (int t = worker, step = first_step; t < total_items && ok; t += step, step = turn_step(step)) {
      const int cls = FORM == CLASSES ? 3 - t / per_class : 0, ph = cls >> 1, pw = cls & 1;
      const int tile = FORM == CLASSES ? t - (3 - cls) * per_class : t / splits, sp = FORM == CLASSES ? 0 : t - tile * splits;
      const int kbeg = sp * kps, kend = FORM == CLASSES ? class_depth(ph, pw) : min(num_k, kbeg + kps);
      const int filter_w = FORM == CLASSES ? (pw ? ca.class_taps1 : ca.class_taps0) : ca.fs;
      const int m0 = (PAIR ? (tile / tiles_n) * 2 + rank : tile / tiles_n) * BM, n0 = (tile % tiles_n) * BN + rank * S::B_COLS;
      int box[4] = {0, 0, 0, 0};
      if (ca.taps != 0) conv_box(ca, (int64_t)m0, 0, 0, box);  // pixel of the tile's first position at tap (0, 0)
      int cb = 0, fr = 0, fs = 0;                             // k-block = (filter tap (fr, fs), 32-channel block cb)
      if constexpr (TAPS) {
        cb = kbeg / 3;                                        // stage = (32-channel block cb, filter column fs)
        fs = kbeg - cb * 3;
      } else if (FORM == PLAIN && ca.taps != 0) {
        const int tap = kbeg / ca.cblocks;
        cb = kbeg - tap * ca.cblocks;
        fr = tap / ca.fs;
        fs = tap - fr * ca.fs;
      }
      for (int k = kbeg; k < kend; ++k) {
        if (turn == warp) {
          if (!mbar_wait_warp(&empty[s], phase ^ 1u, &abort_flag)) { ok = false; break; }
          if constexpr (TAPS) {
            uint8_t *a_dst = a_tiles + s * (uint32_t)a_pitch, *b_dst = b_tiles + s * (uint32_t)B_STAGE;
            const int w0 = fs - 1, h0 = box[2] + ca.pad + tc.h_off;      // pixels {cb * 32, w0, image, h0}: box[2] = row of tap (0, 0)
            if constexpr (PAIR) {
              const uint32_t bar = cluster_addr(&full[s], 0);
              if (elect_one()) {
                if (rank == 0) mbar_expect_tx(&full[s], (uint32_t)(2 * (tc.box_bytes + B_STAGE)));
                tma_load_4d_pair(a_dst, &tma_a, cb * 32, w0, box[3], h0, bar);
                tma_load_5d_pair(b_dst, &tma_b, 0, cb * BK, n0 >> 5, 2 - fs, 0, bar);
              }
            } else if (elect_one()) {
              mbar_expect_tx(&full[s], (uint32_t)(tc.box_bytes + B_STAGE));
              tma_load_4d(a_dst, &tma_a, cb * 32, w0, box[3], h0, &full[s]);
              tma_load_5d(b_dst, &tma_b, 0, cb * BK, n0 >> 5, 2 - fs, 0, &full[s]);
            }
            __syncwarp();
          } else {
          // b_mn: B is the filter read in place (no transposed copy)
          const int tapcol = ca.b_mn == 0 || ca.taps == 0 ? 0 : ((ca.b_r0 + ph + ca.b_dr * fr) * ca.b_fs + (ca.b_s0 + pw + ca.b_ds * fs)) * ca.b_ldtap;
          const int krow = (ca.taps == 0 ? k : cb) * BK;
          uint8_t *a_dst = a_tiles + s * S::A_BYTES, *b_dst = b_tiles + s * S::B_BYTES;
          if constexpr (PAIR) {
            const uint32_t bar = cluster_addr(&full[s], 0);
            if (elect_one()) {
              if (rank == 0) mbar_expect_tx(&full[s], (uint32_t)(2 * (S::A_BYTES + S::B_BYTES)));
              if (ca.taps == 0) tma_load_2d_pair(a_dst, &tma_a, k * BK, m0, bar);
              else tma_load_4d_pair(a_dst, &tma_a, cb * 32, box[1] + fs, box[2] + fr, box[3], bar);
              if (!ca.b_mn) {
                tma_load_2d_pair(b_dst, &tma_b, k * BK, n0, bar);
              } else if (ca.b_mn == 2) {
                tma_load_3d_pair(b_dst, &tma_b, 0, krow, (tapcol + n0) >> 5, bar);
              } else {
#pragma unroll
                for (int c = 0; c < S::B_COLS / 32; ++c) tma_load_2d_pair(b_dst + c * (BK * 128), &tma_b, tapcol + n0 + c * 32, krow, bar);
              }
            }
          } else if (elect_one()) {
            mbar_expect_tx(&full[s], (uint32_t)(S::A_BYTES + S::B_BYTES));
            if (ca.taps == 0) tma_load_2d(a_dst, &tma_a, k * BK, m0, &full[s]);
            else tma_load_4d(a_dst, &tma_a, cb * 32, box[1] + fs, box[2] + fr, box[3], &full[s]);
            if (!ca.b_mn) {
              tma_load_2d(b_dst, &tma_b, k * BK, n0, &full[s]);
            } else if (ca.b_mn == 2) {
              // the matrix seen as {32 floats, K rows, N / 32 chunks}: one box brings all BN / 32 chunks of the stage
              tma_load_3d(b_dst, &tma_b, 0, krow, (tapcol + n0) >> 5, &full[s]);
            } else {
              // BN / 32 boxes of 32 N-floats x 32 K-rows
#pragma unroll
              for (int c = 0; c < S::B_COLS / 32; ++c) tma_load_2d(b_dst + c * (BK * 128), &tma_b, tapcol + n0 + c * 32, krow, &full[s]);
            }
          }
          __syncwarp();
          }
        }
        if (++s == stages) { s = 0; phase ^= 1u; }
        turn ^= 1;
        if constexpr (TAPS) {
          if (++fs == 3) { fs = 0; ++cb; }
        } else if (++cb == ca.cblocks) {                             // (never true for a plain matrix: cblocks == 0)
          cb = 0;
          if (++fs == filter_w) { fs = 0; ++fr; }
        }
      }
    }
    if constexpr (PAIR) {
      // the commits that free the last stages come from the first CTA: see them before this CTA may end.  From the next
      // k-block's stage on, every stage was last filled in phase `phase ^ 1` (passed at once where it never was).
      for (uint32_t j = 0; j < stages && ok; ++j) {
        ok = mbar_wait_warp<true>(&empty[s], phase ^ 1u, &abort_flag);
        if (++s == stages) { s = 0; phase ^= 1u; }
      }
      cluster_arrive();
    }
  } else if (warp == MMA_WARP) {
    constexpr uint32_t idesc = make_idesc(BN, PAIR ? 2 * BM : BM);
    auto mma = [](uint32_t c, uint64_t ad, uint64_t bd, uint32_t id, uint32_t acc) {
      if constexpr (PAIR) umma_tf32_pair(c, ad, bd, id, acc);
      else umma_tf32(c, ad, bd, id, acc);
    };
    auto commit = [](uint64_t* bar) {
      if constexpr (PAIR) umma_commit_pair(bar);
      else umma_commit(bar);
    };
    uint32_t s = 0, phase = 0, lt = 0;                        // stage of the next k-block and its phase, tiles started
    bool ok = true;
    for (int t = worker, step = first_step; rank == 0 && t < total_items && ok; t += step, step = turn_step(step), ++lt) {
      const int sp = t % splits, cls = FORM == CLASSES ? 3 - t / per_class : 0;
      const int nk = FORM == CLASSES ? class_depth(cls >> 1, cls & 1) : min(num_k, (sp + 1) * kps) - sp * kps;
      const uint32_t buf = lt & 1u, aphase = (lt >> 1) & 1u;
      if (!mbar_wait_warp<PAIR>(&acc_empty[buf], aphase ^ 1u, &abort_flag)) break;      // first use of a buffer passes at once
      tc_fence_after();
      const uint32_t tmem_c = tmem_base + buf * (uint32_t)BN;
      for (int k = 0; k < nk; ++k) {
        if (!mbar_wait_warp<PAIR>(&full[s], phase, &abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint64_t adesc = make_smem_desc(a_tiles + s * (uint32_t)a_pitch - (TAPS ? tc.lead : 0));
        if (elect_one()) {
          if constexpr (TAPS) {
            // the three taps of the column: pixels `step` bytes further on each, the filter's rows from the last one back
            const uint64_t down = (uint64_t)(tc.step >> 4);
            const uint64_t bdesc = make_smem_desc_mn_rows(b_tiles + s * (uint32_t)B_STAGE, BK);
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
              for (int kk = 0; kk < BK / UMMA_K; ++kk)
                mma(tmem_c, adesc + (uint64_t)r * down + (uint64_t)(kk * 2), bdesc + (uint64_t)((2 - r) * (S::B_BYTES >> 4) + kk * 64), idesc | (1u << 16),
                    (k | r | kk) != 0 ? 1u : 0u);
          } else if (!ca.b_mn) {
            const uint64_t bdesc = make_smem_desc(b_tiles + s * S::B_BYTES);
#pragma unroll
            for (int kk = 0; kk < BK / UMMA_K; ++kk)
              mma(tmem_c, adesc + (uint64_t)(kk * 2), bdesc + (uint64_t)(kk * 2), idesc, (k | kk) != 0 ? 1u : 0u);
          } else {
            // B is MN-major: 4 KB chunks of 32 N-floats x 32 K-rows; 8 K-rows = 1024 bytes = 64 address units per MMA
            const uint64_t bdesc = make_smem_desc_mn_rows(b_tiles + s * S::B_BYTES, BK);
#pragma unroll
            for (int kk = 0; kk < BK / UMMA_K; ++kk)
              mma(tmem_c, adesc + (uint64_t)(kk * 2), bdesc + (uint64_t)(kk * 64), idesc | (1u << 16), (k | kk) != 0 ? 1u : 0u);
          }
          commit(&empty[s]);
          if (k == nk - 1) commit(&acc_full[buf]);
        }
        __syncwarp();
        if (++s == stages) { s = 0; phase ^= 1u; }
      }
    }
    if constexpr (PAIR) cluster_arrive();
  } else {
    // Two epilogue groups of four warps (TMEM lane quarters warp & 3); group g drains the 32-column slabs
    // g, g + 2, ... of every tile through its own half of the staging ring, with its own named barrier and its
    // own store-issuing thread, so the groups never wait for each other.
    const int ew = warp - FIRST_EPI_WARP;
    const int grp = ew >> 2;
    const int lg = warp & 3;
    const int r = lg * 32 + lane;                              // row of the tile this thread owns
    const int te = (ew & 3) * 32 + lane;                       // 0..127 inside the group
    const bool issuer = te == 0;                               // owns the group's bulk store groups
    constexpr int SLABS = BN / 32;
    constexpr int RING = S::NSLAB / EPI_GROUPS;                // staging buffers per group
    uint8_t* my_staging = staging + grp * (RING * S::SLAB_BYTES);
    float* my_colsum = colsum;                                 // [4 row quarters][BN][2]; a group only touches its slabs' columns
    uint32_t lt = 0, sc = 0;                                   // tiles drained, slabs staged by this group
    const bool fin_on = fin.acc != nullptr;
    const bool want_sums = col_partials != nullptr || fin_on;
    double run_a = 0.0, run_b = 0.0;                           // fin_on, cta_sums: this thread's column, summed over the CTA's tiles
    bool drained_all = true;
    constexpr bool aff_on = AFFINE;
    const bool with_res = AFFINE && aff.residual != nullptr;
    // aff_on: mean, rstd, gamma, beta and bias of the slab's 32 columns, one array of the first four per warp of the group
    float* col_affine = reinterpret_cast<float*>(base + S::COLSUM_OFF) + grp * (5 * 32);
    float cval = 0.f, cbias = 0.f;                             // this thread's of the next slab
    auto load_columns = [&](int col0) {
      const int col = col0 + lane, which = ew & 3;
      const float* from = which == 0 ? aff.mean : which == 1 ? aff.var : which == 2 ? aff.gamma : aff.beta;
      cval = col < N ? from[col] : 0.f;
      if (which == 1) cval = rsqrtf(cval + aff.eps);
      if (which == 0) cbias = col < N && bias != nullptr ? bias[col] : 0.f;
    };
    float4 res[8];                                             // with_res: the next slab's residual, 4 rows of 128 bytes per load of a warp
    auto load_residual = [&](int m0, int col0) {
      const int c = col0 + (te & 7) * 4;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = m0 + (te >> 3) + 16 * i;
        res[i] = row < M && c < N ? __ldcs(reinterpret_cast<const float4*>(aff.residual + (int64_t)row * N + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    for (int t = worker, step = first_step; t < total_items; t += step, step = turn_step(step), ++lt) {
      const int cls = FORM == CLASSES ? 3 - t / per_class : 0;
      const int tile = FORM == CLASSES ? t - (3 - cls) * per_class : t / splits;
      const bool add_bias = bias != nullptr && t == tile * splits;      // the first split of a tile carries the bias
      const int mi = PAIR ? (tile / tiles_n) * 2 + rank : tile / tiles_n;      // row tile of 128; of a pair the second may lie beyond M
      const int m0 = mi * BM, n0 = (tile % tiles_n) * BN;
      const uint32_t buf = lt & 1u, aphase = (lt >> 1) & 1u;
      if (aff_on) load_columns(n0 + grp * 32);
      if (with_res) load_residual(m0, n0 + grp * 32);
      const bool got = (tma_mode & 4) ? mbar_wait_idle(&acc_full[buf], aphase, &abort_flag, 128u) : mbar_wait(&acc_full[buf], aphase, &abort_flag);
      // one thread decides for the group: the TMEM loads are warp-collective and the named barriers below
      // involve all four warps, so either every one of them drains this tile or none does
      if (issuer) epi_go[grp] = (got && abort_flag == 0) ? 1 : 0;
      group_bar(grp);
      if (!epi_go[grp]) { drained_all = false; break; }
      tc_fence_after();
      const uint32_t lane_base = tmem_base + ((uint32_t)(lg * 32) << 16) + buf * (uint32_t)BN;
      const bool full_rows = m0 + BM <= M;
      // The ring's stages are done with once a CTA's last accumulator is complete: that tile's slabs are staged there, each in a
      // place of its own, and none waits for a store to have read the one before (the end of a launch, 2.2 us from the last
      // accumulator to the last store at 128 columns, was mostly that wait).
      const bool last = t + step >= total_items;
      static_assert(SLABS * S::SLAB_BYTES <= S::RING_BYTES, "a tile's slabs in the ring");
#pragma unroll 1
      for (int sl = grp; sl < SLABS; sl += EPI_GROUPS, ++sc) {
        uint8_t* slab = last ? base + sl * S::SLAB_BYTES : my_staging + (sc % RING) * S::SLAB_BYTES;
        if (aff_on) {                                          // the barrier that ended the last slab lets them be overwritten
          col_affine[(ew & 3) * 32 + lane] = cval;
          if ((ew & 3) == 0) col_affine[4 * 32 + lane] = cbias;
          if (sl + EPI_GROUPS < SLABS) load_columns(n0 + (sl + EPI_GROUPS) * 32);
        }
        // the store that last read this buffer was committed RING groups ago
        if (issuer && !last) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(RING - 1) : "memory");
        if (AFFINE || !last) group_bar(grp);
        if (with_res) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int row = (te >> 3) + 16 * i;
            *reinterpret_cast<float4*>(slab + row * 128 + (((te & 7) ^ (row & 7)) << 4)) = res[i];
          }
          if (sl + EPI_GROUPS < SLABS) load_residual(m0, n0 + (sl + EPI_GROUPS) * 32);
          group_bar(grp);
        }
        uint32_t ra[16], rb[16];
        tmem_ld16_nowait(lane_base + (uint32_t)(sl * 32), ra);
        tmem_ld16_nowait(lane_base + (uint32_t)(sl * 32 + 16), rb);
        tmem_ld_wait();
        tc_fence_before();
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint32_t* src = c < 4 ? &ra[c * 4] : &rb[(c - 4) * 4];
          float4 o = make_float4(__uint_as_float(src[0]), __uint_as_float(src[1]), __uint_as_float(src[2]), __uint_as_float(src[3]));
          float4* to = reinterpret_cast<float4*>(slab + r * 128 + ((c ^ (r & 7)) << 4));           // 128-byte swizzle of the store map
          if (aff_on) {
            auto column = [&](int k) { return *reinterpret_cast<const float4*>(col_affine + k * 32 + c * 4); };
            if (bias != nullptr) {
              const float4 b = column(4);
              o.x += b.x; o.y += b.y; o.z += b.z; o.w += b.w;
            }
            const float4 mu = column(0), rs = column(1), gm = column(2), bt = column(3);
            o = make_float4(fmaf((o.x - mu.x) * rs.x, gm.x, bt.x), fmaf((o.y - mu.y) * rs.y, gm.y, bt.y), fmaf((o.z - mu.z) * rs.z, gm.z, bt.z),
                            fmaf((o.w - mu.w) * rs.w, gm.w, bt.w));
            if (with_res) {
              const float4 q = *to;
              o.x += q.x; o.y += q.y; o.z += q.z; o.w += q.w;
            }
            if (aff.relu) { o.x = fmaxf(o.x, 0.f); o.y = fmaxf(o.y, 0.f); o.z = fmaxf(o.z, 0.f); o.w = fmaxf(o.w, 0.f); }
          } else if (add_bias) {
            int col = n0 + sl * 32 + c * 4;
            o.x += col < N ? bias[col] : 0.f; o.y += col + 1 < N ? bias[col + 1] : 0.f;
            o.z += col + 2 < N ? bias[col + 2] : 0.f; o.w += col + 3 < N ? bias[col + 3] : 0.f;
          }
          *to = o;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        group_bar(grp);
        if (issuer) {
          // the group has read its share of the accumulator; nobody waits for that where no later tile uses the buffer (and a
          // signal that nobody waits for could come to a CTA that has ended)
          if (sl + EPI_GROUPS >= SLABS && t + 2 * workers < total_items) {
            if constexpr (PAIR) mbar_arrive_remote(cluster_addr(&acc_empty[buf], 0));
            else mbar_arrive(&acc_empty[buf]);
          }
          if (n0 + sl * 32 < N && (!PAIR || m0 < M)) {
            if constexpr (FORM == CLASSES) {     // rows = pixels (n, i, j) of class (ph, pw)
              const int img = m0 / cc.hw, rem = m0 - img * cc.hw;
              const int i0 = rem / cc.w, j0 = rem - i0 * cc.w;
              if (accumulate)
                asm volatile("cp.reduce.async.bulk.tensor.5d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];"
                             ::"l"(&tma_c), "r"(smem_u32(slab)), "r"((cls & 1) * N + n0 + sl * 32), "r"(j0), "r"(cls >> 1), "r"(i0), "r"(img)
                             : "memory");
              else
                asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];"
                             ::"l"(&tma_c), "r"(smem_u32(slab)), "r"((cls & 1) * N + n0 + sl * 32), "r"(j0), "r"(cls >> 1), "r"(i0), "r"(img)
                             : "memory");
            } else if (cc.hw != 0) {             // rows = pixels (n, i, j) of a strided sub-grid: 4-D store map
              const int img = m0 / cc.hw, rem = m0 - img * cc.hw;
              const int i0 = rem / cc.w, j0 = rem - i0 * cc.w;
              const int c2 = cc.nh ? img : i0, c3 = cc.nh ? i0 : img;
              if (accumulate)
                asm volatile("cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                             ::"l"(&tma_c), "r"(smem_u32(slab)), "r"(n0 + sl * 32), "r"(j0), "r"(c2), "r"(c3)
                             : "memory");
              else
                asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
                             ::"l"(&tma_c), "r"(smem_u32(slab)), "r"(n0 + sl * 32), "r"(j0), "r"(c2), "r"(c3)
                             : "memory");
            } else if (accumulate)               // C += tile: the add happens in L2, C is never read by the SM
              asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
                           ::"l"(&tma_c), "r"(smem_u32(slab)), "r"(n0 + sl * 32), "r"(m0)
                           : "memory");
            else
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
                           ::"l"(&tma_c), "r"(smem_u32(slab)), "r"(n0 + sl * 32), "r"(m0)
                           : "memory");
          }
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");              // one group per slab, empty ones included
        }
        if (want_sums) {
          // sum and sum of squares of 32 rows of one column, read back from the staged slab (a row of a slab is
          // one 128-byte line: conflict free); four independent chains each
          const int col = te & 31, quarter = te >> 5;
          const uint8_t* colbase = slab + (quarter * 32) * 128 + ((col & 3) << 2);
          const int chunk = col >> 2;
          float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f, q0 = 0.f, q1 = 0.f, q2 = 0.f, q3 = 0.f;
          if (full_rows) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              float v0 = *reinterpret_cast<const float*>(colbase + (j + 0) * 128 + ((chunk ^ ((j + 0) & 7)) << 4));
              float v1 = *reinterpret_cast<const float*>(colbase + (j + 1) * 128 + ((chunk ^ ((j + 1) & 7)) << 4));
              float v2 = *reinterpret_cast<const float*>(colbase + (j + 2) * 128 + ((chunk ^ ((j + 2) & 7)) << 4));
              float v3 = *reinterpret_cast<const float*>(colbase + (j + 3) * 128 + ((chunk ^ ((j + 3) & 7)) << 4));
              s0 += v0; s1 += v1; s2 += v2; s3 += v3;
              q0 = fmaf(v0, v0, q0); q1 = fmaf(v1, v1, q1); q2 = fmaf(v2, v2, q2); q3 = fmaf(v3, v3, q3);
            }
          } else {
#pragma unroll 4
            for (int j = 0; j < 32; ++j) {
              float v = *reinterpret_cast<const float*>(colbase + j * 128 + ((chunk ^ (j & 7)) << 4));
              v = (m0 + quarter * 32 + j < M) ? v : 0.f;
              s0 += v;
              q0 = fmaf(v, v, q0);
            }
          }
          my_colsum[(quarter * BN + sl * 32 + col) * 2] = (s0 + s1) + (s2 + s3);
          my_colsum[(quarter * BN + sl * 32 + col) * 2 + 1] = (q0 + q1) + (q2 + q3);
        }
      }
      if (want_sums) {
        group_bar(grp);
        static_assert((SLABS / EPI_GROUPS) * 32 <= 128, "one column per thread and tile");
        for (int idx = te; idx < (SLABS / EPI_GROUPS) * 32; idx += 128) {       // the columns of this group's slabs
          const int c = (grp + EPI_GROUPS * (idx >> 5)) * 32 + (idx & 31);
          const int gc = n0 + c;
          if (gc < N) {
            float a = (my_colsum[c * 2] + my_colsum[(BN + c) * 2]) + (my_colsum[(2 * BN + c) * 2] + my_colsum[(3 * BN + c) * 2]);
            float b = (my_colsum[c * 2 + 1] + my_colsum[(BN + c) * 2 + 1]) + (my_colsum[(2 * BN + c) * 2 + 1] + my_colsum[(3 * BN + c) * 2 + 1]);
            if (fin_on || cta_sums) {
              run_a += (double)a;
              run_b += (double)b;
            } else if (!PAIR || m0 < M) {
              col_partials[((int64_t)mi * 2) * N + gc] = a;
              col_partials[((int64_t)mi * 2 + 1) * N + gc] = b;
            }
          }
        }
      }
    }
    if constexpr (PAIR) cluster_arrive();
    if (cta_sums && drained_all && te < (SLABS / EPI_GROUPS) * 32) {
      // one row of partial sums per CTA that stays on this column tile (instead of one per row tile); where a CTA has several
      // tiles, a second set of rows carries what the first one's rounding left out
      const int gc = (worker % tiles_n) * BN + (grp + EPI_GROUPS * (te >> 5)) * 32 + (te & 31);
      const int64_t row = (int64_t)(PAIR ? (worker / tiles_n) * 2 + rank : worker / tiles_n) * 2;
      if (gc < N) {
        const float hi_a = (float)run_a, hi_b = (float)run_b;
        col_partials[row * N + gc] = hi_a;
        col_partials[(row + 1) * N + gc] = hi_b;
        if (total_items > workers) {
          const int64_t rest = row + (int64_t)(workers / tiles_n) * (PAIR ? 4 : 2);
          col_partials[rest * N + gc] = (float)(run_a - (double)hi_a);
          col_partials[(rest + 1) * N + gc] = (float)(run_b - (double)hi_b);
        }
      }
    }
    if (fin_on && drained_all) {
      // this CTA's column sums -> the global totals; the group that draws the last of gridDim.x * EPI_GROUPS tickets
      // finds every contribution in place and finishes the statistics
      if (te < (SLABS / EPI_GROUPS) * 32) {
        const int c = (grp + EPI_GROUPS * (te >> 5)) * 32 + (te & 31);
        const int gc = (worker % tiles_n) * BN + c;
        if (gc < N) {
          atomicAdd(&fin.acc[gc], run_a);
          atomicAdd(&fin.acc[N + gc], run_b);
        }
      }
      __threadfence();
      group_bar(grp);
      if (issuer) epi_go[grp] = atomicAdd(fin.ticket, 1u) == gridDim.x * (unsigned)EPI_GROUPS - 1u ? 2 : 1;
      group_bar(grp);
      if (epi_go[grp] == 2) {
        __threadfence();
        const double inv_m = 1.0 / (double)M;
        for (int c = te; c < N; c += 128) {
          const double sum = __ldcg(&fin.acc[c]), sq = __ldcg(&fin.acc[N + c]);
          const double mean = sum * inv_m;
          double var = sq * inv_m - mean * mean;
          if (var < 0.0) var = 0.0;
          fin.stats[c] = (float)mean;
          fin.stats[N + c] = (float)(1.0 / sqrt(var + (double)fin.eps));
          if (fin.running_mean != nullptr) {
            const double unbiased = M > 1 ? var * (double)M / (double)(M - 1) : var;
            fin.running_mean[c] = (1.0f - fin.momentum) * fin.running_mean[c] + fin.momentum * (float)mean;
            fin.running_var[c] = (1.0f - fin.momentum) * fin.running_var[c] + fin.momentum * (float)unbiased;
          }
          fin.acc[c] = 0.0;
          fin.acc[N + c] = 0.0;
        }
        if (issuer) *fin.ticket = 0u;
      }
    }
    if (issuer) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // shared memory outlives the stores
  }
  tc_fence_before();
  __syncthreads();
  // Every thread of both CTAs has come to the end of its part (cluster_arrive above; the last statistics and the wait for the stores
  // hide the way there and back): nothing of the other CTA reads or signals this one's shared memory or TMEM any more.
  if constexpr (PAIR) cluster_wait();
  if (warp == MMA_WARP) {
    tc_fence_after();
    if constexpr (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)S::TMEM_COLS) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)S::TMEM_COLS) : "memory");
  }
  if (threadIdx.x == 0 && abort_flag && error_flag != nullptr) atomicExch(error_flag, 1);
}

// ------------------------------------------------------------------------------------------------
// "TN" GEMM for weight gradients:  C[Mo, No] += A[P, Mo]^T * B[P, No], contraction over the rows P (the
// N*H*W positions of a 1x1 convolution: A = dY, B = X, C = dW).  Both operands are MN-major for the tensor
// core (the contraction index is the slow one in memory).  For 32-bit elements that takes the shared-memory
// layout "128-byte swizzle with 32-byte atoms": 32 consecutive output-dimension floats (128 B) of one
// position form a row, 32 positions a 4 KB chunk (one TMA box), and the chunks of a k-block lie one after the
// other.  In descriptor terms: leading byte offset = 4096
// (next 32 floats of the output dimension), stride byte offset = 512 (next group of 4 positions), one MMA
// (K = 8 positions) advances the start address by 1024 bytes.
// Split-K: CTA (tile, split) contracts its slice of positions and adds its 128 x BN partial result onto C
// with TMA reduce stores, so C must hold the value to add to (zeros for a plain product).
//
// PAIR: as in the persistent kernel, two CTAs share a tile of 256 x BN, each with its 128 columns of A and half of B's.
//
// Two groups of epilogue warps, and no staging buffers beside the ring: with one group and two buffers the ring had one or two stages less.
template <int BN, bool PAIR>
struct TnSmem {
  static constexpr int B_COLS = PAIR ? BN / 2 : BN;
  static constexpr int CHUNK_BYTES = TBK * 128;             // one TMA box: 32 floats of the output dimension x TBK rows
  static constexpr int A_BYTES = BM * TBK * 4;
  static constexpr int B_BYTES = B_COLS * TBK * 4;
  static constexpr int STAGES = (232448 - 1024 - 256) / (A_BYTES + B_BYTES);
  static constexpr int RING_BYTES = STAGES * (A_BYTES + B_BYTES);
  static constexpr int SLAB_BYTES = BM * 128;               // the one tile's slabs are staged in the ring, whose stages are done with by then
  static constexpr int BAR_OFF = RING_BYTES;
  static constexpr int TOTAL = 1024 + BAR_OFF + 256;
  static constexpr int TMEM_COLS = BN == 192 ? 256 : BN;    // TMEM is allocated in powers of two
  static_assert(TOTAL <= 232448 && (2 * STAGES + 1) * 8 + 4 <= 256, "shared memory of one CTA");
  static_assert(BN / 32 * SLAB_BYTES <= RING_BYTES, "a tile's slabs in the ring");
};

__host__ __device__ constexpr uint32_t make_idesc_mn(int n, int m = BM) {
  return make_idesc(n, m) | (1u << 15) | (1u << 16);        // A and B are MN-major
}

template <int BN, bool PAIR>
__global__ void __launch_bounds__(TN_THREADS, 1)
gemm_tn_tf32_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                    const __grid_constant__ CUtensorMap tma_c, const ConvA ca, int P, int Mo, int No, int tiles_n, int splits,
                    int kblocks_per_split, int* __restrict__ error_flag, int tma_mode, int box3d, int wait_late) {
  using S = TnSmem<BN, PAIR>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* a_tiles = base;
  uint8_t* b_tiles = base + S::STAGES * S::A_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(base + S::BAR_OFF);
  uint64_t* empty = full + S::STAGES;
  uint64_t* acc_ready = empty + S::STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_ready + 1);
  __shared__ int abort_flag;
  __shared__ int epi_go[EPI_GROUPS];

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const int rank = PAIR ? (int)cluster_rank() : 0, worker = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int split = worker % splits;
  const int tile = worker / splits;
  const int m0 = (PAIR ? (tile / tiles_n) * 2 + rank : tile / tiles_n) * BM, n0 = (tile % tiles_n) * BN;
  const int total_k = (P + TBK - 1) / TBK;
  const int k_begin = split * kblocks_per_split;
  const int k_end = k_begin + kblocks_per_split < total_k ? k_begin + kblocks_per_split : total_k;
  const int num_k = k_end > k_begin ? k_end - k_begin : 0;

  if (threadIdx.x == 32 * FIRST_EPI_WARP && (tma_mode & 1)) { tma_prefetch_map(&tma_a); tma_prefetch_map(&tma_b); tma_prefetch_map(&tma_c); }
  if (threadIdx.x == 0) {
    abort_flag = 0;
    for (int s = 0; s < S::STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_ready, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)S::TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((uint32_t)S::TMEM_COLS) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  if constexpr (PAIR) cluster_sync_all();
  else __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  // wait_late: the kernel in front on the stream is an input-gradient kernel of the same layer, which writes nothing that is read here and let
  // this one start only when the kernels before it were complete.  The two run side by side; this one ends after the other.
  if (!wait_late) gc::pdl_wait();
  gc::pdl_launch_dependents();

  if (num_k > 0) {
    if (warp < PRODUCER_WARPS) {
      // a stage is BM / 32 + BN / 32 boxes of 32 floats x TBK rows; producer warp p fills the stages k == p (mod PRODUCER_WARPS)
      // weight gradient of an R x S convolution: column n of dW[Cout, taps * Cin] belongs to filter tap n / Cin, channel
      // n % Cin; a tile narrower than Cin stays inside one tap, a wider one (Cin = 64) covers several taps side by side.
      // Box c of a stage reads the pixels of its tap, shifted by (fr, fs), for the TBK output positions of the k-block.
      int co[4] = {0, 0, 0, 0};
      int box_ch[S::B_COLS / 32], box_fr[S::B_COLS / 32], box_fs[S::B_COLS / 32];
      const int b0 = n0 + rank * S::B_COLS;                 // first column of B this CTA loads
      if (ca.taps != 0) {
        const int cin = ca.cblocks * 32;
#pragma unroll
        for (int c = 0; c < S::B_COLS / 32; ++c) {
          const int n = b0 + c * 32, tap = n / cin;
          box_ch[c] = n - tap * cin;
          box_fr[c] = tap / ca.fs;
          box_fs[c] = tap - box_fr[c] * ca.fs;
        }
      }
      // boxes that lie wholly beyond the matrix (Mo < 128: the 64-channel layers; No < n0 + BN) are not loaded at all: the
      // rows and columns of the accumulator they feed are never stored
      auto boxes = [](int left, int most) { return left <= 0 ? 0 : (left + 31) / 32 < most ? (left + 31) / 32 : most; };
      const int a_boxes = boxes(Mo - m0, BM / 32), b_boxes = boxes(No - b0, S::B_COLS / 32);
      // box3d bit 0 / 1: the A / B map is the 3-D view {32 floats, rows, chunks} of the matrix and ONE box brings the whole
      // operand of a stage (chunks beyond the matrix arrive as zeros and count as bytes)
      const bool a3 = (box3d & 1) != 0, b3 = (box3d & 2) != 0 && ca.taps == 0;
      // bytes of a stage, of both CTAs of a pair (the second one's rows and columns follow)
      int stage_boxes = (a3 ? BM / 32 : a_boxes) + (b3 ? S::B_COLS / 32 : b_boxes);
      if (PAIR) stage_boxes += (a3 ? BM / 32 : boxes(Mo - m0 - BM, BM / 32)) + (b3 ? S::B_COLS / 32 : boxes(No - b0 - S::B_COLS, S::B_COLS / 32));
      const uint32_t stage_tx = (uint32_t)(stage_boxes * S::CHUNK_BYTES);
      for (int k = warp; k < num_k; k += PRODUCER_WARPS) {
        const int s = k % S::STAGES;
        const uint32_t phase = (uint32_t)(k / S::STAGES) & 1u;
        if (!mbar_wait_warp(&empty[s], phase ^ 1u, &abort_flag)) break;
        const int row0 = (k_begin + k) * TBK;
        if (ca.taps != 0) conv_box(ca, (int64_t)row0, 0, 0, co);           // the k-block's first position at tap (0, 0)
        uint8_t *a_dst = a_tiles + s * S::A_BYTES, *b_dst = b_tiles + s * S::B_BYTES;
        const uint32_t bar = PAIR ? cluster_addr(&full[s], 0) : 0u;
        auto load_2d = [&](uint8_t* dst, const CUtensorMap* map, int x, int y) {
          if constexpr (PAIR) tma_load_2d_pair(dst, map, x, y, bar);
          else tma_load_2d(dst, map, x, y, &full[s]);
        };
        auto load_3d = [&](uint8_t* dst, const CUtensorMap* map, int c0, int c1, int c2) {
          if constexpr (PAIR) tma_load_3d_pair(dst, map, c0, c1, c2, bar);
          else tma_load_3d(dst, map, c0, c1, c2, &full[s]);
        };
        auto load_4d = [&](uint8_t* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3) {
          if constexpr (PAIR) tma_load_4d_pair(dst, map, c0, c1, c2, c3, bar);
          else tma_load_4d(dst, map, c0, c1, c2, c3, &full[s]);
        };
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(&full[s], stage_tx);
          if (a3) {
            load_3d(a_dst, &tma_a, 0, row0, m0 >> 5);
          } else {
#pragma unroll
            for (int c = 0; c < BM / 32; ++c)
              if (c < a_boxes) load_2d(a_dst + c * S::CHUNK_BYTES, &tma_a, m0 + c * 32, row0);
          }
          if (b3) {
            load_3d(b_dst, &tma_b, 0, row0, b0 >> 5);
          } else if (ca.taps == 0) {
#pragma unroll
            for (int c = 0; c < S::B_COLS / 32; ++c)
              if (c < b_boxes) load_2d(b_dst + c * S::CHUNK_BYTES, &tma_b, b0 + c * 32, row0);
          } else {
#pragma unroll
            for (int c = 0; c < S::B_COLS / 32; ++c)
              if (c < b_boxes) load_4d(b_dst + c * S::CHUNK_BYTES, &tma_b, box_ch[c], co[1] + box_fs[c], co[2] + box_fr[c], co[3]);
          }
        }
        __syncwarp();
      }
      if constexpr (PAIR)       // see the commits of the last stages before this CTA may end
        for (int k = (num_k > S::STAGES ? num_k - S::STAGES : 0); k < num_k; ++k)
          if (!mbar_wait_warp<true>(&empty[k % S::STAGES], (uint32_t)(k / S::STAGES) & 1u, &abort_flag)) break;
    } else if (warp == MMA_WARP) {
      constexpr uint32_t idesc = make_idesc_mn(BN, PAIR ? 2 * BM : BM);
      uint32_t s = 0, phase = 0;
      for (int k = 0; rank == 0 && k < num_k; ++k) {
        if (!mbar_wait_warp<PAIR>(&full[s], phase, &abort_flag)) break;
        tc_fence_after();
        const uint64_t adesc = make_smem_desc_mn(a_tiles + s * S::A_BYTES);
        const uint64_t bdesc = make_smem_desc_mn(b_tiles + s * S::B_BYTES);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < TBK / UMMA_K; ++kk)    // 8 positions = 8 rows of 128 bytes = 1024 bytes = 64 address units
          {
            if constexpr (PAIR) umma_tf32_pair(tmem_base, adesc + (uint64_t)(kk * 64), bdesc + (uint64_t)(kk * 64), idesc, (k | kk) != 0 ? 1u : 0u);
            else umma_tf32(tmem_base, adesc + (uint64_t)(kk * 64), bdesc + (uint64_t)(kk * 64), idesc, (k | kk) != 0 ? 1u : 0u);
          }
          if constexpr (PAIR) {
            umma_commit_pair(&empty[s]);
            if (k == num_k - 1) umma_commit_pair(acc_ready);
          } else {
            umma_commit(&empty[s]);
            if (k == num_k - 1) umma_commit(acc_ready);
          }
        }
        __syncwarp();
        if (++s == S::STAGES) { s = 0; phase ^= 1u; }
      }
    } else {
      // two groups of four warps (TMEM lane quarters warp & 3) take alternate slabs
      const int ew = warp - FIRST_EPI_WARP, grp = ew >> 2;
      const int lg = warp & 3;
      const int r = lg * 32 + lane;
      const bool issuer = (ew & 3) == 0 && lane == 0;
      const bool got = (tma_mode & 4) ? mbar_wait_idle(acc_ready, 0u, &abort_flag, 128u) : mbar_wait(acc_ready, 0u, &abort_flag);
      if (issuer) epi_go[grp] = (got && abort_flag == 0) ? 1 : 0;
      group_bar(grp);
      if (epi_go[grp]) {
        tc_fence_after();
        const uint32_t lane_base = tmem_base + ((uint32_t)(lg * 32) << 16);
        constexpr int SLABS = BN / 32;
#pragma unroll 1
        for (int sl = grp; sl < SLABS; sl += EPI_GROUPS) {
          uint8_t* slab = base + sl * S::SLAB_BYTES;
          uint32_t ra[16], rb[16];
          tmem_ld16_nowait(lane_base + (uint32_t)(sl * 32), ra);
          tmem_ld16_nowait(lane_base + (uint32_t)(sl * 32 + 16), rb);
          tmem_ld_wait();
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint32_t* src = c < 4 ? &ra[c * 4] : &rb[(c - 4) * 4];
            *reinterpret_cast<float4*>(slab + r * 128 + ((c ^ (r & 7)) << 4)) =
                make_float4(__uint_as_float(src[0]), __uint_as_float(src[1]), __uint_as_float(src[2]), __uint_as_float(src[3]));
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          group_bar(grp);
          if (issuer) {
            if (n0 + sl * 32 < No && (!PAIR || m0 < Mo))
              asm volatile("cp.reduce.async.bulk.tensor.2d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3}], [%1];"
                           ::"l"(&tma_c), "r"(smem_u32(slab)), "r"(n0 + sl * 32), "r"(m0)
                           : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
      }
    }
  }
  if constexpr (PAIR) cluster_arrive();        // waited for below, behind the stores' reading of shared memory
  if (num_k > 0 && warp >= FIRST_EPI_WARP && ((warp - FIRST_EPI_WARP) & 3) == 0 && lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
  if (wait_late) gc::pdl_wait();
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_wait();
  if (warp == MMA_WARP) {
    tc_fence_after();
    if constexpr (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)S::TMEM_COLS) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)S::TMEM_COLS) : "memory");
  }
  if (threadIdx.x == 0 && abort_flag && error_flag != nullptr) atomicExch(error_flag, 1);
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

int sm_count() {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 148;
  }
  return sms;
}

// 2-D fp32 tensor [rows, cols] with row stride ld (elements); box = box_rows x 32 columns, 128-byte swizzle.
int make_map(CUtensorMap* map, const float* base, int64_t rows, int64_t cols, int64_t ld, int box_rows);

bool tma_store_ok(const float* C, int64_t ldc) { return (reinterpret_cast<uintptr_t>(C) & 15u) == 0 && (ldc & 3) == 0; }

int make_map(CUtensorMap* map, const float* base, int64_t rows, int64_t cols, int64_t ld, int box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return -1;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}



// Row-major [P, D] fp32 matrix as an MN-major operand: box = 32 floats x 32 rows (4 KB), shared-memory layout
// "128-byte swizzle, 32-byte atoms" (the MN-major layout of 32-bit types).
int make_map_mn(CUtensorMap* map, const float* base, int64_t P, int64_t D, int64_t ld, int box_rows = TBK) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return -1;
  cuuint64_t dims[2] = {(cuuint64_t)D, (cuuint64_t)P};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
  cuuint32_t box[2] = {32, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}



// The row-major matrix [K, D] (row stride ld floats, D and ld multiples of 32 for whole chunks) as the 3-D tensor
// {32 floats, K rows, D / 32 chunks}: a box of 32 x box_rows x chunks lands in shared memory chunk after chunk, each chunk
// box_rows rows of 128 bytes -- the MN-major operand layout -- with ONE copy instruction.
int make_map_mn3(CUtensorMap* map, const float* base, int64_t K, int64_t D, int64_t ld, int box_rows, int chunks) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return -1;
  cuuint64_t dims[3] = {32, (cuuint64_t)K, (cuuint64_t)((D + 31) / 32)};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 4, 128};
  cuuint32_t box[3] = {32, (cuuint32_t)box_rows, (cuuint32_t)chunks};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void*)base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -2;
}

// How a product runs on the persistent kernel: tile width, splits of the contraction, CTA pairs (256-row tiles) or single CTAs.
struct Plan {
  int bn, splits;
  bool pair;
  bool taps;                                                 // 3x3 input gradient with shared pixels (TapCols)
  bool classes;                                              // stride-2 input gradient, all parity classes in one launch
  int b_cols() const { return pair ? bn / 2 : bn; }          // columns of B (box rows of its map) one CTA loads
  int rows() const { return pair ? 2 * BM : BM; }
};

// CTA pairs of a kernel that the device runs at once.
inline int pairs_at_once(const void* kernel, int threads, size_t smem) {
  int n = sm_count() / 2, fit = 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * n));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) == cudaSuccess && fit > 0 && fit < n ? fit : n;
}

// CTAs, or CTA pairs, of the persistent kernel that the device runs at once (pairs: half its SMs, unless a GPC has an odd
// number of them); 0 when the kernel cannot be configured.
template <int BN, bool AFFINE, bool PAIR, int FORM>
int persistent_workers() {
  using S = PSmem<BN, PAIR, FORM == SHARED>;
  static int workers = 0;
  if (workers != 0) return workers;
  if (cudaFuncSetAttribute(gemm_tf32_persistent_kernel<BN, AFFINE, PAIR, FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL) != cudaSuccess) return 0;
  int n = sm_count();
  if constexpr (PAIR) n = pairs_at_once((const void*)gemm_tf32_persistent_kernel<BN, AFFINE, PAIR, FORM>, PERSISTENT_THREADS, S::TOTAL);
  return workers = n;
}

// Launch the persistent kernel on ready-made tensor maps (ca.taps == 0: ma is a 2-D map of A[M, K]).
template <int BN, bool AFFINE, bool PAIR, int FORM>
int launch_persistent_maps(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mc, const ConvA& ca, const float* bias,
                           int M, int N, int K, int accumulate, float* col_partials, int* error_flag, cudaStream_t st,
                           const BnFin* fin, const ConvC* cc, int splits, int cta_sums, const Affine* aff, const TapCols* tc) {
  constexpr bool TAPS = FORM == SHARED;
  using S = PSmem<BN, PAIR, TAPS>;
  if ((tc != nullptr && tc->box_bytes != 0) != TAPS || (ca.class_taps0 != 0) != (FORM == CLASSES)) return (int)cudaErrorInvalidValue;
  const int workers_max = persistent_workers<BN, AFFINE, PAIR, FORM>();
  if (workers_max == 0) return (int)cudaGetLastError();
  constexpr int ROWS = PAIR ? 2 * BM : BM;
  int tiles_m = (M + ROWS - 1) / ROWS, tiles_n = (N + BN - 1) / BN;
  if (splits < 1 || splits > (TAPS ? 3 * ca.cblocks : (K + BK - 1) / BK)) return (int)cudaErrorInvalidValue;
  // a split contraction adds partial tiles into C: the caller zeroed C (or wants C += ...), and nothing that needs the
  // finished values (column statistics) can ride along
  if (splits > 1 && (!accumulate || col_partials != nullptr || (fin != nullptr && fin->acc != nullptr) || (cc != nullptr && !cc->nh)))
    return (int)cudaErrorInvalidValue;
  if (FORM == CLASSES && (splits != 1 || bias != nullptr || col_partials != nullptr || fin != nullptr || cc == nullptr || (N & 31))) return (int)cudaErrorInvalidValue;
  int64_t total = (int64_t)tiles_m * tiles_n * (FORM == CLASSES ? 4 : splits);
  int64_t workers = total < workers_max ? total : workers_max;
  BnFin f{};
  if (fin != nullptr && fin->acc != nullptr) {
    if (col_partials != nullptr || tiles_n > workers) return (int)cudaErrorInvalidValue;
    workers = workers / tiles_n * tiles_n;             // every CTA stays on one column tile
    f = *fin;
  }
  if (aff != nullptr && (splits > 1 || accumulate || col_partials != nullptr || fin != nullptr || cc != nullptr)) return (int)cudaErrorInvalidValue;
  if (cta_sums) {
    if (col_partials == nullptr || splits > 1 || tiles_n > workers) return (int)cudaErrorInvalidValue;
    workers = workers / tiles_n * tiles_n;
  }
  gc::launch_cluster(gemm_tf32_persistent_kernel<BN, AFFINE, PAIR, FORM>, PAIR ? 2u : 1u, dim3((unsigned)(PAIR ? 2 * workers : workers)),
                     dim3(PERSISTENT_THREADS), (size_t)S::TOTAL, st, ma, mb, mc, ca, bias, M, N, K, tiles_m, tiles_n, splits, accumulate,
                     col_partials, error_flag, gctc::tma_mode, f, cc != nullptr ? *cc : ConvC{}, cta_sums, aff != nullptr ? *aff : Affine{},
                     tc != nullptr ? *tc : TapCols{});
  return (int)cudaGetLastError();
}

template <bool AFFINE = false>
int launch_plan(const Plan& pl, const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mc, const ConvA& ca, const float* bias,
                int M, int N, int K, int accumulate, float* col_partials, int* error_flag, cudaStream_t st,
                const BnFin* fin = nullptr, const ConvC* cc = nullptr, int cta_sums = 0, const Affine* aff = nullptr, const TapCols* tc = nullptr) {
  auto run = [&](auto launch) {
    return launch(ma, mb, mc, ca, bias, M, N, K, accumulate, col_partials, error_flag, st, fin, cc, pl.splits, cta_sums, aff, tc);
  };
  if (pl.taps) {
    if constexpr (!AFFINE) {
      if (pl.bn == 64) return pl.pair ? run(launch_persistent_maps<64, false, true, SHARED>) : run(launch_persistent_maps<64, false, false, SHARED>);
      if (pl.bn == 128) return pl.pair ? run(launch_persistent_maps<128, false, true, SHARED>) : run(launch_persistent_maps<128, false, false, SHARED>);
    }
    return (int)cudaErrorInvalidValue;
  }
  if (pl.classes) {
    if constexpr (!AFFINE) {
      if (pl.bn == 64) return pl.pair ? run(launch_persistent_maps<64, false, true, CLASSES>) : run(launch_persistent_maps<64, false, false, CLASSES>);
      if (pl.bn == 128) return pl.pair ? run(launch_persistent_maps<128, false, true, CLASSES>) : run(launch_persistent_maps<128, false, false, CLASSES>);
      if (pl.bn == 256) return pl.pair ? run(launch_persistent_maps<256, false, true, CLASSES>) : run(launch_persistent_maps<256, false, false, CLASSES>);
    }
    return (int)cudaErrorInvalidValue;
  }
  switch (pl.bn) {
    case 64: return pl.pair ? run(launch_persistent_maps<64, AFFINE, true, PLAIN>) : run(launch_persistent_maps<64, AFFINE, false, PLAIN>);
    case 128: return pl.pair ? run(launch_persistent_maps<128, AFFINE, true, PLAIN>) : run(launch_persistent_maps<128, AFFINE, false, PLAIN>);
    case 256: return pl.pair ? run(launch_persistent_maps<256, AFFINE, true, PLAIN>) : run(launch_persistent_maps<256, AFFINE, false, PLAIN>);
    default: return (int)cudaErrorInvalidValue;
  }
}

// CTAs or CTA pairs a plan runs at once.
inline int plan_workers(const Plan& pl) {
  if (!pl.pair) return sm_count();
  switch (pl.bn) {
    case 64: return persistent_workers<64, false, true, PLAIN>();
    case 128: return persistent_workers<128, false, true, PLAIN>();
    default: return persistent_workers<256, false, true, PLAIN>();
  }
}

// Rows of partial sums a launch with cta_sums leaves.
inline int cta_sum_rows(int M, int N, const Plan& pl) {
  const int64_t at_once = plan_workers(pl), tiles_n = (N + pl.bn - 1) / pl.bn, total = (int64_t)((M + pl.rows() - 1) / pl.rows()) * tiles_n;
  const int64_t workers = (total < at_once ? total : at_once) / tiles_n * tiles_n;
  return (int)(workers / tiles_n) * (pl.pair ? 2 : 1) * (total > workers ? 2 : 1);
}

// Launch the split-K TN kernel on ready-made tensor maps.  At most tn_ctas_per_sm CTAs per SM over all tiles, at least
// tn_min_kblocks k-blocks each so that the pipeline fills.  One CTA per SM measured 10-25 % faster than two on the
// 131072- and 32768-position weight gradients of ResNet-50 (fewer partial tiles to add, longer pipelines), equal below.
// CTA pairs for the split contraction: two row tiles, and at least 16 k-blocks for every CTA.  A pair loads 128 + BN / 2 columns a
// k-block instead of 128 + BN (at BN = 256 about 0.13 us less) and costs about 1.5 us for meeting at both ends: 16x16 256 -> 256 3x3 at batch 128
// 67.6 -> 53.2 us, 8x8 512 -> 512 64.3 -> 53.2 us; with 8 k-blocks a CTA (8x8 256 -> 1024 1x1 at batch 31) 14.3 -> 16.4 us.
inline bool tn_pair(int P, int Mo, int No, int bn) {
  if ((bn != 128 && bn != 256) || Mo <= BM || gctc::pair_choice == 1) return false;
  const int64_t tiles = (int64_t)((Mo + BM - 1) / BM) * ((No + bn - 1) / bn);
  return gctc::pair_choice == 2 || tiles * ((P + TBK - 1) / TBK) >= (int64_t)16 * sm_count();
}

template <int BN, bool PAIR>
int launch_tn_maps(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mc, const ConvA& ca, int P, int Mo, int No,
                   int* error_flag, cudaStream_t st, int box3d, int wait_late) {
  using S = TnSmem<BN, PAIR>;
  static int at_once = 0;
  if (at_once == 0) {
    cudaError_t e = cudaFuncSetAttribute(gemm_tn_tf32_kernel<BN, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::TOTAL);
    if (e != cudaSuccess) return (int)e;
    at_once = PAIR ? pairs_at_once((const void*)gemm_tn_tf32_kernel<BN, PAIR>, TN_THREADS, S::TOTAL) : sm_count();
  }
  constexpr int ROWS = PAIR ? 2 * BM : BM;
  int tiles_m = (Mo + ROWS - 1) / ROWS, tiles_n = (No + BN - 1) / BN;
  int tiles = tiles_m * tiles_n;
  int total_k = (P + TBK - 1) / TBK;
  // never more CTAs than fit at once (one per SM at this shared-memory size): a second, nearly empty wave would double the
  // kernel's time (measured: 153 CTAs on 148 SMs ran 37 us with the SMs 62 % busy)
  int splits = gctc::tn_ctas_per_sm * at_once / tiles;
  if (splits > (total_k + gctc::tn_min_kblocks - 1) / gctc::tn_min_kblocks) splits = (total_k + gctc::tn_min_kblocks - 1) / gctc::tn_min_kblocks;
  if (splits < 1) splits = 1;
  int per = (total_k + splits - 1) / splits;
  splits = (total_k + per - 1) / per;
  const cudaError_t e = gc::launch_cluster(gemm_tn_tf32_kernel<BN, PAIR>, PAIR ? 2u : 1u, dim3((unsigned)((PAIR ? 2 : 1) * tiles * splits)), dim3(TN_THREADS),
                                           (size_t)S::TOTAL, st, ma, mb, mc, ca, P, Mo, No, tiles_n, splits, per, error_flag, gctc::tma_mode, box3d, wait_late);
  return e != cudaSuccess ? (int)e : (int)cudaGetLastError();
}

inline int launch_tn_plan(int bn, bool pair, const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mc, const ConvA& ca, int P, int Mo, int No,
                          int* error_flag, cudaStream_t st, int box3d, int wait_late) {
  auto run = [&](auto launch) { return launch(ma, mb, mc, ca, P, Mo, No, error_flag, st, box3d, wait_late); };
  switch (bn) {
    case 64: return run(launch_tn_maps<64, false>);
    case 128: return pair ? run(launch_tn_maps<128, true>) : run(launch_tn_maps<128, false>);
    case 192: return run(launch_tn_maps<192, false>);
    case 256: return pair ? run(launch_tn_maps<256, true>) : run(launch_tn_maps<256, false>);
    default: return (int)cudaErrorInvalidValue;
  }
}

// Modelled nanoseconds of a product on the persistent kernel.  A k-block costs a CTA the time its loads and operand reads take
// in shared memory; measured on a B200 with 3x3 convolutions of 72 and 144 k-blocks per tile (16x16x256, 8x8x512, 4x4x512,
// batch 128): 235 / 300 / 490 ns at 64 / 128 / 256 columns for single CTAs, 205 / 260 / 400 ns for pairs.  A tile adds about
// 500 ns of hand-over between the accumulators, a pair's launch about 1500 ns (the two CTAs meet at its start and end).  The product
// cannot be faster than its operands and its result cross DRAM; the two overlap, not quite perfectly.
// `reuse`: how often an element of A is read (filter taps per input pixel of a convolution, 1 for a matrix).
// taps_stage, for the SHARED form, is from 16x16x128 (four waves against two); 11 layers of 32x32x64 to 2x2x512 at batches 24, 31, 64 and 128 give 139 / 171 and
// 97 / 143 ns by least squares with a time per wave beside it.  Over those and eight 1x1 layers the input gradients as planned take 2 % more, added up,
// than the fastest form of each that could be forced.
constexpr double stage_ns[2][3] = {{235.0, 300.0, 490.0}, {205.0, 260.0, 400.0}};
inline double stage_of(const Plan& p) { return stage_ns[p.pair][p.bn == 64 ? 0 : (p.bn == 128 ? 1 : 2)]; }

inline double plan_ns(const Plan& p, int M, int N, int K, double reuse) {
  static constexpr double taps_stage[2][2] = {{157.0, 200.0}, {103.0, 144.0}};
  const int num_k = (K + BK - 1) / BK;
  const int64_t items = (int64_t)((M + p.rows() - 1) / p.rows()) * ((N + p.bn - 1) / p.bn) * p.splits;
  const int64_t workers = p.pair ? sm_count() / 2 : sm_count(), waves = (items + workers - 1) / workers;
  const double sm = (double)waves * ((num_k + p.splits - 1) / p.splits * (p.taps ? taps_stage[p.pair][p.bn == 64 ? 0 : 1] : stage_of(p)) + 500.0);
  const double dram = ((double)M * K / reuse + (double)M * N * (p.splits > 1 ? 2.0 : 1.0) + (double)N * K) * 4.0 / 6500.0;
  return (sm > dram ? sm + 0.15 * dram : dram + 0.15 * sm) + (p.pair ? 1500.0 : 0.0);
}

// Candidates of the plan: widths that do not leave half a tile empty, pairs where there are two row tiles; for the input gradient of a 3x3
// convolution whose filter columns can share their pixels (taps_ok) the kernel that does, which has tiles of up to 128 columns.
template <typename F>
inline void each_plan(int M, int N, bool taps_ok, F&& f) {
  const int cand[3] = {256, 128, 64};
  const bool taps = taps_ok && gctc::taps_choice != 1;
  for (int i = 0; i < 3; ++i) {
    const int bn = cand[i];
    if (gctc::tile_choice ? bn != gctc::tile_choice : ((bn == 256 && N <= 128) || (bn == 128 && N <= 64))) continue;
    for (int pair = 0; pair < 2; ++pair)
      if (pair == 0 ? (gctc::pair_choice != 2 || M <= BM) : (gctc::pair_choice != 1 && M > BM)) f(Plan{bn, 1, pair != 0, taps && bn <= 128, false});
  }
}

// Tile width and pairing of a product that is not split: the candidate with the lowest modelled time.
inline Plan pick_persistent(int M, int N, int K, double reuse = 1.0, bool taps_ok = false) {
  Plan best{64, 1, false, false, false};
  double best_t = 1e30;
  each_plan(M, N, taps_ok, [&](const Plan& p) {
    const double t = plan_ns(p, M, N, K, reuse);
    if (t < best_t) { best_t = t; best = p; }
  });
  return best;
}

// The same for the four parity classes of a stride-2 input gradient in one launch: M pixels and K rows of the filter per class, t0 and t1 taps along
// an axis.  The busiest worker's time, its items dealt out as the kernel does it.
inline Plan pick_classes(int M, int N, int K, int t0, int t1) {
  Plan best{64, 1, false, false, true};
  double best_t = 1e30;
  each_plan(M, N, false, [&](Plan p) {
    const int64_t per_class = (int64_t)((M + p.rows() - 1) / p.rows()) * ((N + p.bn - 1) / p.bn), workers = p.pair ? sm_count() / 2 : sm_count();
    const int64_t first = 4 * per_class < workers ? 4 * per_class : workers;
    const double taps[4] = {(double)t1 * t1, (double)t1 * t0, (double)t0 * t1, (double)t0 * t0}, stage = stage_of(p) * ((K + BK - 1) / BK);
    double worst = 0.0;
    for (int64_t w = 0; w < first; w += 4) {                 // (every fourth worker)
      double t = 0.0;
      for (int64_t i = w, step = 2 * (first - w) - 1; i < 4 * per_class; i += step, step = 2 * first - step) t += taps[i / per_class] * stage + 500.0;
      if (t > worst) worst = t;
    }
    const double all = worst + (p.pair ? 1500.0 : 0.0);
    if (all < best_t) { best_t = all; best = p; best.classes = true; }
  });
  return best;
}

// C[M, N] = 0 in front of a split contraction, which adds its partial tiles.  A kernel of its own instead of a memset node: a programmatic dependent
// itself, and the product behind it can be one, too (it sets up its barriers and TMEM meanwhile):
// ResNet-18's step at batch 31, with 11 of them, 947 -> 942 us, VGG-16's at 128, with 11, 1020 -> 1017, ResNet-50's, with eight, 5804 -> 5808 (no difference).
__global__ void __launch_bounds__(512) zero_kernel(float4* __restrict__ p, int64_t quads) {
  gc::pdl_launch_dependents();
  gc::pdl_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < quads; i += (int64_t)gridDim.x * blockDim.x) p[i] = make_float4(0.f, 0.f, 0.f, 0.f);
}
inline int zero_rows(float* C, int64_t M, int64_t N, int64_t ldc, cudaStream_t st) {
  if (ldc != N || (M * N & 3) || (reinterpret_cast<uintptr_t>(C) & 15u)) return (int)cudaMemset2DAsync(C, (size_t)ldc * 4, 0, (size_t)N * 4, (size_t)M, st);
  const int64_t quads = M * N / 4, blocks = (quads + 2047) / 2048, most = 2 * sm_count();      // four quads a thread where the chip is not full
  return (int)gc::launch_pdl(zero_kernel, dim3((unsigned)(blocks < most ? blocks : most)), dim3(512), 0, st, reinterpret_cast<float4*>(C), quads);
}

// Modelled time of zeroing `elements` floats, and of one more pass over them for column statistics.  zero_kernel in front of the split input gradients of
// 19 layers at batches 24 to 128 takes 1.35 us at 0.5 MB, 2.2 at 4 MB, 2.9 at 8 MB, 4.0 at 17 MB.  Charged is a little more at the small end, where
// plans are close: plan_ns takes split products for faster than they are.  With 1250 ns and 5.3 TB/s here a ResNet-18's inference at batch 77
// went from 372.6 to 378.4 us, VGG-16's at 150 from 375 to 381, ResNet-50's step at batch 77 from 4138 to 4167; no step or inference gained.
inline double zero_ns(int64_t elements) { return 1600.0 + (double)elements * 4.0 / 5700.0; }
inline double stats_pass_ns(int64_t elements) { return 4200.0 + (double)elements * 4.0 / 3800.0; }

// The same for a product whose output may be built from partial tiles (no column statistics wanted, plain 2-D output): the
// contraction is also split where that pays.  extra_split_ns: what a caller pays elsewhere when the product is split
// (zeroing C, a separate pass for the statistics).
inline Plan plan_persistent(int M, int N, int K, double extra_split_ns, double reuse = 1.0, bool taps_ok = false) {
  Plan pl = pick_persistent(M, N, K, reuse, taps_ok);
  if (gctc::split_choice == 1) return pl;
  double best = plan_ns(pl, M, N, K, reuse);
  each_plan(M, N, taps_ok, [&](Plan p) {
    const int num = (K + BK - 1) / BK / (p.taps ? 3 : 1);          // stages of the contraction
    for (int splits = 2; splits <= 16; ++splits) {
      const int per = (num + splits - 1) / splits;
      if (per < (p.taps ? 2 : 6) || (splits - 1) * per >= num) continue;      // every split non-empty and long enough to fill the ring
      if (gctc::split_choice > 1 && splits != gctc::split_choice) continue;
      p.splits = splits;
      const double t = plan_ns(p, M, N, K, reuse) + extra_split_ns;
      if (t < best * 0.93 || (gctc::split_choice > 1 && pl.splits == 1)) { best = t; pl = p; }
    }
  });
  return pl;
}

}  // namespace
