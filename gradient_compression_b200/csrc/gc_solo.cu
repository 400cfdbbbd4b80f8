// Reducers on a single worker: there is no peer to exchange anything with, so a reduce is "norm, then quantise and dequantise"
// straight from the gradient tensors into the gradient tensors.
//
//   solo_maxnorm_kernel  QSGD-MaxNorm and its two-scale variant: one persistent block of 1024 threads per SM.
//   solo_maxnorm_one_kernel  the same of up to 16 K elements, which one block holds.
//   solo_randk_kernel    GlobalRandK-MaxNorm and its two-scale variant.
//   solo_copy_kernel     AllReduce-SGD: the mean over one worker.
//
// What bounds solo_maxnorm.  The vector has to be read before its norm is known and is needed again after, so DRAM moves
// 4 n bytes in and 4 n out, plus whatever part of the second read the chip did not keep.  Kept in two places: the first
// tiles of every block stay in shared memory (KEPT x 16 KB per SM, 22 MB over the chip), and the rest is read again in
// falling order, last tile first, so that what was read most recently comes out of L2 (stores are streaming, so that
// they push out each other and not the tiles still to come).  Both passes load through a ring of
// asynchronous copies, RING tiles (64 KB per SM) ahead.  The second pass is held up by its arithmetic and its stores, which overlap by half: ten
// Philox rounds per quad plus the rounding of four elements, and 4 n bytes out (ResNet-50's arena: 24 of 54 us for the first pass; the second's 29 are 20 without
// Philox, 24 without stores, 12 without both; 64 M floats, of which the chip keeps little: 49 of 145 us, then 96, 87, 62 and 35).  Rounding is therefore written without int <-> float conversions,
// which run at a quarter of the rate of the rest (see round_level), the round keys come with the parameters, what a launch's blocks have in
// common is taken out of the first three rounds, and infinities and NaN, which only a norm of infinity can mean, have a pass of their own.
// 33.5 M floats, instructions of both passes a quad: two scales 309 -> 212, 127 -> 106 us; one scale 154 -> 135, 83.5 -> 80 us.  Two quads side by side in
// a thread spill (50 -> 57 us on VGG-16's tensors), both scales' noise drawn at once, too, took longer (59 us).
#include <cuda_runtime.h>
#include <stdint.h>

#include "gc_comm.cuh"
#include "gc_perm.h"
#include "gc_segs.cuh"
#include "gc_solo.h"

using namespace gc;

namespace {

constexpr int THREADS = SEG_TILE;
constexpr int SLOTS = 13;                  // tiles of shared memory
constexpr int RING = 4;                    // ... of which the copies in flight take these ...
constexpr int KEPT = SLOTS - RING;         // ... when a block has more tiles than slots; the rest stay there between the passes
constexpr int ONE_BLOCK_TILES = 4;         // up to this many tiles run on one block: no grid barrier, an ordinary launch of a kernel of its own

struct SoloParams {
  ArenaHeader* hdr;
  int step_from_device;
  unsigned long long timeout_ns;
  uint32_t rk0[10], rk1[10];               // Philox round keys (they depend on the seed only)
  uint32_t step, stream;
  int s_lo, s_hi;
};

// philox_block (gc_common.h) with the round keys read from the parameters: two wide multiplies and two three-way xors a round.
__device__ __forceinline__ U4 solo_philox(const SoloParams& p, uint64_t block, uint32_t step, uint32_t purpose) {
  uint32_t x = (uint32_t)block, y = (uint32_t)(block >> 32), z = step, w = p.stream | purpose;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t m0 = (uint64_t)0xD2511F53u * x, m1 = (uint64_t)0xCD9E8D57u * z;
    x = (uint32_t)(m1 >> 32) ^ y ^ p.rk0[r];
    z = (uint32_t)(m0 >> 32) ^ w ^ p.rk1[r];
    y = (uint32_t)m1;
    w = (uint32_t)m0;
  }
  return U4{x, y, z, w};
}

// The same for block < 2^32, with what a launch's blocks have in common taken out of the first three rounds (step, purpose and the upper
// half of the block's index, 0, are the same for all of them): 18 multiplies and 19 xors instead of 20 and 20.
struct __align__(16) PhiloxHead { uint32_t a, b, c, d; };

__device__ __forceinline__ PhiloxHead philox_head(const SoloParams& p, uint32_t step, uint32_t purpose) {
  const uint64_t m1 = (uint64_t)0xCD9E8D57u * step;                                   // round 1: z = step, y = 0
  const uint64_t m0 = (uint64_t)0xD2511F53u * ((uint32_t)(m1 >> 32) ^ p.rk0[0]);      // round 2: its x
  return PhiloxHead{(p.stream | purpose) ^ p.rk1[0], (uint32_t)m1 ^ p.rk0[1], (uint32_t)(m0 >> 32) ^ p.rk1[1], (uint32_t)m0 ^ p.rk1[2]};
}

__device__ __forceinline__ U4 solo_philox(const SoloParams& p, const PhiloxHead& h, uint32_t block) {
  uint64_t m0 = (uint64_t)0xD2511F53u * block, m1 = (uint64_t)0xCD9E8D57u * ((uint32_t)(m0 >> 32) ^ h.a);
  uint32_t x = (uint32_t)(m1 >> 32) ^ h.b, z = (uint32_t)m0 ^ h.c, y = (uint32_t)m1, w;
  m0 = (uint64_t)0xD2511F53u * x;
  m1 = (uint64_t)0xCD9E8D57u * z;
  x = (uint32_t)(m1 >> 32) ^ y ^ p.rk0[2];
  z = (uint32_t)(m0 >> 32) ^ h.d;
  y = (uint32_t)m1;
  w = (uint32_t)m0;
#pragma unroll
  for (int r = 3; r < 10; ++r) {
    m0 = (uint64_t)0xD2511F53u * x;
    m1 = (uint64_t)0xCD9E8D57u * z;
    x = (uint32_t)(m1 >> 32) ^ y ^ p.rk0[r];
    z = (uint32_t)(m0 >> 32) ^ w ^ p.rk1[r];
    y = (uint32_t)m1;
    w = (uint32_t)m0;
  }
  return U4{x, y, z, w};
}

__device__ __forceinline__ void copy16_async(float4* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// The counters of the grid barrier as a launch finds them (read by thread 0 of each block before its first arrival).
struct SoloSync {
  uint32_t passed, turn;
  __device__ __forceinline__ explicit SoloSync(const ArenaHeader* h)
      : passed(*((volatile const uint32_t*)&h->solo_passed)), turn(*((volatile const uint32_t*)&h->solo_turn)) {}
};

// Maximum over all threads of all blocks; valid in every thread.  Thread 0 of each block folds its block's maximum into one of
// the header's two slots (the other one is cleared for the next launch) and arrives; the arrival count only ever grows, so
// nothing has to be reset between launches.  A further barrier of the same launch (v = 0) does not carry a maximum.
__device__ __forceinline__ float solo_grid_max(Waiter& w, SoloSync& sync, float v, int nblocks, float* smem) {
  float m = block_max(v, smem);
  if (nblocks > 1) {
    if (threadIdx.x == 0) {
      ArenaHeader* h = w.hdr;
      sync.passed += (uint32_t)nblocks;
      atomicMax(&h->solo_max[sync.turn & 1], __float_as_uint(m));     // bit patterns of non-negative floats order like the floats
      __threadfence();
      atomicAdd(&h->solo_arrived, 1u);
      int it = 0;
      while ((int32_t)(ld_acquire_gpu(&h->solo_arrived) - sync.passed) < 0) {
        if ((++it & 63) == 0) {
          if (w.aborted()) break;
          if (global_ns() > w.deadline) { w.fail(0x90, 0xfffe); break; }
        }
      }
      smem[0] = __uint_as_float(*((volatile uint32_t*)&h->solo_max[sync.turn & 1]));
      ++sync.turn;
      if (blockIdx.x == 0) {               // for the next launch: every block has read the counters of this one
        h->solo_passed = sync.passed;
        h->solo_turn = sync.turn;
        h->solo_max[sync.turn & 1] = 0u;
      }
    }
    __syncthreads();
    m = smem[0];
  }
  return m;
}

// What becomes of one quad, for any input: infinities and NaN (norm = inf), quads beyond 32 bits, a fine scale with no more levels than the
// coarse one, a scale of infinite size (levels / norm overflows: norms below 7.5e-37 at 8 bits, 1.9e-34 at 16; zero times infinity is given the
// last level, without the sign of the zero).
template <bool TWO>
struct AnyValue {
  float s_lo, s_hi, sc_lo, sc_hi, dq_lo, dq_hi;
  __device__ __forceinline__ AnyValue(const SoloParams& p, float norm)
      : s_lo((float)p.s_lo), s_hi((float)p.s_hi), sc_lo(norm > 0.0f ? s_lo / norm : 0.0f), sc_hi(TWO && norm > 0.0f ? s_hi / norm : 0.0f),
        dq_lo(dequant_scale(norm, p.s_lo, 1)), dq_hi(TWO ? dequant_scale(norm, p.s_hi, 1) : 0.0f) {}
  __device__ __forceinline__ float4 operator()(const SoloParams& p, const float4& x, uint64_t quad, uint32_t step) const {
    if (!TWO) {
      const U4 r = solo_philox(p, quad, step, PURPOSE_ROUND);
      return make_float4(signed_value(x.x, round_level(x.x, sc_lo, s_lo, r.x), dq_lo), signed_value(x.y, round_level(x.y, sc_lo, s_lo, r.y), dq_lo),
                         signed_value(x.z, round_level(x.z, sc_lo, s_lo, r.z), dq_lo), signed_value(x.w, round_level(x.w, sc_lo, s_lo, r.w), dq_lo));
    }
    // the fine scale where its level fits the coarse range, else the coarse scale; its noise is only drawn where it is used
    const U4 r = solo_philox(p, quad, step, PURPOSE_ROUND_HI);
    const float h0 = round_level(x.x, sc_hi, s_hi, r.x), h1 = round_level(x.y, sc_hi, s_hi, r.y);
    const float h2 = round_level(x.z, sc_hi, s_hi, r.z), h3 = round_level(x.w, sc_hi, s_hi, r.w);
    float4 y = make_float4(signed_value(x.x, h0, dq_hi), signed_value(x.y, h1, dq_hi), signed_value(x.z, h2, dq_hi), signed_value(x.w, h3, dq_hi));
    if (fmaxf(fmaxf(h0, h1), fmaxf(h2, h3)) > s_lo) {
      const U4 w = solo_philox(p, quad, step, PURPOSE_ROUND);
      if (h0 > s_lo) y.x = signed_value(x.x, round_level(x.x, sc_lo, s_lo, w.x), dq_lo);
      if (h1 > s_lo) y.y = signed_value(x.y, round_level(x.y, sc_lo, s_lo, w.y), dq_lo);
      if (h2 > s_lo) y.z = signed_value(x.z, round_level(x.z, sc_lo, s_lo, w.z), dq_lo);
      if (h3 > s_lo) y.w = signed_value(x.w, round_level(x.w, sc_lo, s_lo, w.w), dq_lo);
    }
    return y;
  }
};

// Pass 2 with it.  Plain loads; a function of its own, as its registers cost the usual path its own.
template <bool TWO, int CAP>
__device__ __noinline__ void pass2_any(const SegTable<CAP>& t, const SoloParams& p, float norm, uint32_t step, uint32_t first, int iters, int kept, const float4* slots) {
  const AnyValue<TWO> value(p, norm);
  SegCursor<CAP, -1> c(t, first + iters - 1);
  for (int it = iters - 1; it >= 0; --it, c.step(t)) {
    if (c.empty(t)) continue;
    const float4 x = it < kept ? slots[it * THREADS + threadIdx.x] : c.load(t);
    c.store(t, value(p, x, c.quad, step));
  }
}

// Up to ONE_BLOCK_TILES tiles: one block, which keeps them in registers.  Such a call is a launch and little more: no ring, no dynamic shared memory,
// no barrier but that of the norm, every load in flight at once.  The kernel below, run with one block, had its ring's prologue and a called function in
// the way (us a call back to back / in a graph; 1024 elements 5.84 / 3.43, before it had that function 5.60 / 3.39, here 4.80 / 2.87, which
// is the host's time; 16384 elements 8.21 / 6.56 -> 7.29 / 5.53, two scales 10.26 / 8.88 -> 10.25 / 8.32).
template <bool TWO, int CAP>
__global__ void __launch_bounds__(THREADS, 1) solo_maxnorm_one_kernel(const __grid_constant__ SegTable<CAP> t, const __grid_constant__ SoloParams p) {
  __shared__ float smem[32];
  const uint32_t epoch = next_epoch(p.hdr);
  const uint32_t step = p.step + (p.step_from_device ? launch_calls(p.hdr) : 0u);
  const int iters = (int)t.tile0[t.n];
  float4 x[ONE_BLOCK_TILES];
  float m = 0.0f;
  {
    SegCursor<CAP, 1> c(t, 0);
#pragma unroll
    for (int u = 0; u < ONE_BLOCK_TILES; ++u) {
      x[u] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (u < iters) { x[u] = c.load(t); c.step(t); }
    }
  }
#pragma unroll
  for (int u = 0; u < ONE_BLOCK_TILES; ++u) m = max_nan(max_nan(max_nan(max_nan(m, x[u].x), x[u].y), x[u].z), x[u].w);
  const float norm = block_max(abs_for_max(m), smem);
  commit_epoch(p.hdr, epoch, 0);
  const AnyValue<TWO> value(p, norm);
  SegCursor<CAP, 1> c(t, 0);
#pragma unroll
  for (int u = 0; u < ONE_BLOCK_TILES; ++u) {
    if (u >= iters) break;
    if (!c.empty(t)) c.store(t, value(p, x[u], c.quad, step));
    c.step(t);
  }
}

template <bool TWO, int CAP>
__global__ void __launch_bounds__(THREADS, 1) solo_maxnorm_kernel(const __grid_constant__ SegTable<CAP> t,
                                                                  const __grid_constant__ SoloParams p) {
  extern __shared__ float4 slots[];        // [SLOTS][THREADS]; a thread only ever touches its own column
  __shared__ float smem[32];
  __shared__ __align__(16) PhiloxHead heads[2];      // two scales: read again for every quad, registers are short there
  Waiter waiter{p.hdr, global_ns() + p.timeout_ns};
  SoloSync sync(p.hdr);
  const uint32_t epoch = next_epoch(p.hdr);
  const uint32_t step = p.step + (p.step_from_device ? launch_calls(p.hdr) : 0u);
  const uint32_t tiles = t.tile0[t.n], nb = gridDim.x;
  const uint32_t per = (tiles + nb - 1) / nb, first = blockIdx.x * per;          // this block's tiles: a contiguous run
  const int iters = first >= tiles ? 0 : (int)(tiles - first < per ? tiles - first : per);
  const int kept = iters <= SLOTS ? iters : KEPT;
  const int q = threadIdx.x;

  auto slot = [&](int it) -> float4& { return slots[it * THREADS + q]; };
  auto ring = [&](int it) -> float4& { return slots[(kept + ((it - kept) & (RING - 1))) * THREADS + q]; };
  auto load = [&](float4& to, const auto& c) {
    if (c.fast_in) copy16_async(&to, c.in);
    else to = c.load(t);
  };

  // pass 1: the norm
  float m = 0.0f;
  auto fold = [&](const float4& x) {
    m = max_nan(max_nan(m, x.x), x.y);
    m = max_nan(max_nan(m, x.z), x.w);
  };
  {
    SegCursor<CAP, 1> ahead(t, first);
#pragma unroll
    for (int it = 0; it < RING; ++it) {
      if (it < iters) { load(it < kept ? slot(it) : ring(it), ahead); ahead.step(t); }
      copy_commit();
    }
    for (int it = 0; it < iters; ++it) {
      // RING tiles at a time where the ring is in step and the next RING loads are whole tiles: nothing but immediate offsets
      while (it >= kept && ((it - kept) & (RING - 1)) == 0 && it + 2 * RING <= iters && ahead.fast_in && ahead.run >= RING) {
        float4* r = &ring(it);
#pragma unroll
        for (int u = 0; u < RING; ++u) {
          copy_wait<RING - 1>();
          fold(r[u * THREADS]);
          copy16_async(r + u * THREADS, ahead.in + u * 4 * SEG_TILE);
          copy_commit();
        }
        ahead.template skip<RING>();
        it += RING;
      }
      copy_wait<RING - 1>();
      fold(it < kept ? slot(it) : ring(it));
      if (it + RING < iters) { load(it + RING < kept ? slot(it + RING) : ring(it + RING), ahead); ahead.step(t); }
      copy_commit();
    }
    copy_wait<0>();
  }
  const float norm = solo_grid_max(waiter, sync, abs_for_max(m), (int)nb, smem);
  commit_epoch(p.hdr, epoch, blockIdx.x);
  const float s_lo = (float)p.s_lo, s_hi = (float)p.s_hi;
  const float sc_lo = norm > 0.0f ? s_lo / norm : 0.0f, dq_lo = dequant_scale(norm, p.s_lo, 1);
  const float sc_hi = TWO && norm > 0.0f ? s_hi / norm : 0.0f, dq_hi = TWO ? dequant_scale(norm, p.s_hi, 1) : 0.0f;

  // From here on: finite numbers and scales, quads of 32-bit index, and a fine scale with more levels than the coarse one.
  PhiloxHead head_one;
  if (TWO) {
    if (threadIdx.x == 0) {
      heads[0] = philox_head(p, step, PURPOSE_ROUND_HI);
      heads[1] = philox_head(p, step, PURPOSE_ROUND);
    }
    __syncthreads();
  } else {
    head_one = philox_head(p, step, PURPOSE_ROUND);
  }
  const float top_lo = ROUND_BASE + s_lo;
  auto coarse = [&](float g, uint32_t rnd) { return signed_value_of_number(g, __fsub_rn(fminf(round_up_base(g, sc_lo, rnd), top_lo), ROUND_BASE), dq_lo); };
  auto value = [&](const float4& x, uint64_t quad) {
    if (!TWO) {
      const U4 r = solo_philox(p, head_one, (uint32_t)quad);
      return make_float4(coarse(x.x, r.x), coarse(x.y, r.y), coarse(x.z, r.z), coarse(x.w, r.w));
    }
    // The fine scale where its level fits the coarse range, else the coarse scale; its noise is only drawn where it is used.  h: ROUND_BASE + fine
    // level (one beyond the fine scale's last is beyond the coarse one's, too, and not used: no clamp).
    const U4 r = solo_philox(p, heads[0], (uint32_t)quad);
    const float4 h = make_float4(round_up_base(x.x, sc_hi, r.x), round_up_base(x.y, sc_hi, r.y), round_up_base(x.z, sc_hi, r.z), round_up_base(x.w, sc_hi, r.w));
    if (fmaxf(fmaxf(h.x, h.y), fmaxf(h.z, h.w)) <= top_lo) {
      auto fine = [&](float g, float level) { return signed_value_of_number(g, __fsub_rn(level, ROUND_BASE), dq_hi); };
      return make_float4(fine(x.x, h.x), fine(x.y, h.y), fine(x.z, h.z), fine(x.w, h.w));
    }
    const U4 w = solo_philox(p, heads[1], (uint32_t)quad);
    auto either = [&](float g, float level, uint32_t rnd) {
      const bool use = level > top_lo;
      const float l = fminf(round_up_base(g, sc_lo, rnd), top_lo);
      return signed_value_of_number(g, __fsub_rn(use ? l : level, ROUND_BASE), use ? dq_lo : dq_hi);
    };
    return make_float4(either(x.x, h.x, w.x), either(x.y, h.y, w.y), either(x.z, h.z, w.z), either(x.w, h.w, w.w));
  };

  // pass 2, last tile first: the ring still holds the last RING tiles
  if (iters == 0) return;
  const float inf = __int_as_float(0x7f800000);
  if (!(norm < inf) || !((TWO ? sc_hi : sc_lo) < inf) || (uint64_t)t.start[t.n] >= (1ull << 34) || (TWO && p.s_hi <= p.s_lo)) {
    pass2_any<TWO, CAP>(t, p, norm, step, first, iters, kept, slots);
    return;
  }
  SegCursor<CAP, -1> c(t, first + iters - 1);
  int it = iters - 1;
  if (iters > kept) {
    SegCursor<CAP, -1> ahead(t, it - RING >= kept ? c.tile - RING : first);
    for (; it >= kept; --it, c.step(t)) {
      while (((it - kept) & (RING - 1)) == RING - 1 && it - 2 * RING + 1 >= kept && c.fast_out && c.run >= RING && ahead.fast_in && ahead.run >= RING) {
        float4* r = &ring(it);
#pragma unroll
        for (int u = 0; u < RING; ++u) {
          copy_wait<RING - 1>();
          const float4 x = r[-u * THREADS];
          copy16_async(r - u * THREADS, ahead.in - u * 4 * SEG_TILE);
          copy_commit();
          __stcs(reinterpret_cast<float4*>(c.out - u * 4 * SEG_TILE), value(x, c.quad - u * SEG_TILE));
        }
        ahead.template skip<RING>();
        c.template skip<RING>();
        it -= RING;
      }
      copy_wait<RING - 1>();
      const float4 x = ring(it);
      if (it - RING >= kept) { load(ring(it - RING), ahead); ahead.step(t); }
      copy_commit();
      if (!c.empty(t)) c.store(t, value(x, c.quad));
    }
  }
  for (; it >= 0; --it, c.step(t))
    if (!c.empty(t)) c.store(t, value(slot(it), c.quad));
}

// This block's share of out = in (or out = 0): four whole tiles in flight.
template <int CAP>
__device__ __forceinline__ void copy_tiles(const SegTable<CAP>& t, bool zero) {
  const uint32_t tiles = t.tile0[t.n], per = (tiles + gridDim.x - 1) / gridDim.x, first = blockIdx.x * per;
  if (first >= tiles) return;
  uint32_t left = tiles - first < per ? tiles - first : per;
  const float4 nothing = make_float4(0.f, 0.f, 0.f, 0.f);
  SegCursor<CAP, 1> c(t, first);
  while (left > 0) {
    if (!zero && c.in == c.out) {            // this tensor stays what it is
      const uint32_t rest = t.tile0[c.s + 1] - c.tile;
      if (rest >= left) return;
      left -= rest;
      c.jump(t, c.tile + rest);
      continue;
    }
    if (left >= 4 && c.run >= 3 && c.fast_out && (zero || c.fast_in)) {
      float4 x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) x[u] = zero ? nothing : __ldcs(reinterpret_cast<const float4*>(c.in) + u * SEG_TILE);
#pragma unroll
      for (int u = 0; u < 4; ++u) __stcs(reinterpret_cast<float4*>(c.out) + u * SEG_TILE, x[u]);
      left -= 4;
      c.template skip<3>();
    } else {
      if (!c.empty(t)) c.store(t, zero ? nothing : c.load(t));
      --left;
    }
    if (left > 0) c.step(t);
  }
}

template <int CAP>
__global__ void __launch_bounds__(THREADS) solo_copy_kernel(const __grid_constant__ SegTable<CAP> t) {
  copy_tiles(t, false);
}

// Rand-K: the selected coordinates are gathered into registers, everything else becomes what it becomes (in or 0), and behind
// the grid barrier that the norm needs anyway the quantised values are put in their places.  Where zeros would overwrite
// coordinates that another block has still to gather (in place), the zeros wait for that barrier and a second one follows.
constexpr int RANDK_PER_THREAD = 4;

struct SoloRandk {
  PermKey perm;
  int64_t start, k;        // the window [start, start + k) of the permutation, cut off at n
  int64_t* window;         // device-resident start (advanced here); NULL: `start`
  int zero, in_place;
};

template <int CAP>
__global__ void __launch_bounds__(THREADS) solo_randk_kernel(const __grid_constant__ SegTable<CAP> t, const __grid_constant__ SoloParams p,
                                                             const __grid_constant__ SoloRandk r) {
  __shared__ float smem[32];
  Waiter waiter{p.hdr, global_ns() + p.timeout_ns};
  SoloSync sync(p.hdr);
  const uint32_t epoch = next_epoch(p.hdr);
  const uint32_t step = p.step + (p.step_from_device ? launch_calls(p.hdr) : 0u);
  const int64_t n = t.start[t.n];
  const int64_t start = r.window != nullptr ? *((volatile const int64_t*)r.window) : r.start;
  const int64_t k = r.k < n - start ? r.k : n - start;
  float x[RANDK_PER_THREAD];
  float* to[RANDK_PER_THREAD];
  float m = 0.0f;
#pragma unroll
  for (int u = 0; u < RANDK_PER_THREAD; ++u) {
    const int64_t i = ((int64_t)u * THREADS + threadIdx.x) * gridDim.x + blockIdx.x;
    to[u] = nullptr;
    x[u] = 0.0f;
    if (i < k) {
      const uint64_t at = perm_eval(r.perm, (uint64_t)(start + i));
      if (GC_INDEX_OK(waiter, at, n)) {
        const int s = seg_of_elem(t, (int64_t)at);
        x[u] = t.in[s][(int64_t)at - t.start[s]];
        to[u] = t.out[s] + ((int64_t)at - t.start[s]);
      }
    }
    m = fmaxf(m, abs_for_max(x[u]));
  }
  const bool late = r.zero && r.in_place;
  if (!late) copy_tiles(t, r.zero != 0);
  const float norm = solo_grid_max(waiter, sync, m, (int)gridDim.x, smem);
  commit_epoch(p.hdr, epoch, blockIdx.x);
  if (r.window != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *r.window = start + k >= n ? 0 : start + k;      // (every block has read it)
  if (late) {
    copy_tiles(t, true);
    __syncthreads();
    solo_grid_max(waiter, sync, 0.0f, (int)gridDim.x, smem);
    __syncthreads();
  }
  const bool two = p.s_hi > 0;
  const float s_lo = (float)p.s_lo, s_hi = (float)p.s_hi;
  const float sc_lo = norm > 0.0f ? s_lo / norm : 0.0f, dq_lo = dequant_scale(norm, p.s_lo, 1);
  const float sc_hi = two && norm > 0.0f ? s_hi / norm : 0.0f, dq_hi = two ? dequant_scale(norm, p.s_hi, 1) : 0.0f;
  auto word = [](const U4& v, int j) { return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w; };
#pragma unroll
  for (int u = 0; u < RANDK_PER_THREAD; ++u) {
    if (to[u] == nullptr) continue;
    const int64_t i = ((int64_t)u * THREADS + threadIdx.x) * gridDim.x + blockIdx.x;
    if (two) {
      const U4 h = solo_philox(p, (uint64_t)(i >> 2), step, PURPOSE_ROUND_HI);
      const float lev = round_level(x[u], sc_hi, s_hi, word(h, (int)(i & 3)));
      if (lev <= s_lo) { *to[u] = signed_value(x[u], lev, dq_hi); continue; }
    }
    const U4 l = solo_philox(p, (uint64_t)(i >> 2), step, PURPOSE_ROUND);
    *to[u] = signed_value(x[u], round_level(x[u], sc_lo, s_lo, word(l, (int)(i & 3))), dq_lo);
  }
}

template <bool TWO, int CAP>
int launch_maxnorm(const SegTable<CAP>& t, const SoloParams& p, int sm_count, int max_blocks, cudaStream_t st) {
  const uint32_t tiles = t.tile0[t.n];
  if (tiles <= ONE_BLOCK_TILES) {
    solo_maxnorm_one_kernel<TWO, CAP><<<1, THREADS, 0, st>>>(t, p);
    return (int)cudaGetLastError();
  }
  auto kernel = solo_maxnorm_kernel<TWO, CAP>;
  static bool ready[64] = {};              // per device: the shared-memory limit has been raised
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return (int)cudaErrorInvalidDevice;
  if (!ready[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SLOTS * THREADS * (int)sizeof(float4));
    if (e != cudaSuccess) return (int)e;
    ready[dev] = true;
  }
  uint32_t blocks = tiles < (uint32_t)sm_count ? tiles : (uint32_t)sm_count;
  if (max_blocks > 0 && blocks > (uint32_t)max_blocks) blocks = (uint32_t)max_blocks;
  const int iters = (int)((tiles + blocks - 1) / blocks);
  void* args[2] = {(void*)&t, (void*)&p};
  const size_t smem = (size_t)(iters < SLOTS ? iters : SLOTS) * THREADS * sizeof(float4);
  if (blocks == 1) return (int)cudaLaunchKernel((const void*)kernel, dim3(1), dim3(THREADS), args, smem, st);
  return (int)cudaLaunchCooperativeKernel((const void*)kernel, dim3(blocks), dim3(THREADS), args, smem, st);
}

template <int CAP>
int maxnorm_segs(CommCtx* c, const SegDesc* segs, int n_seg, int64_t n, int bits_lo, int bits_hi, const SoloParams& p, int max_blocks, cudaStream_t st) {
  SegTable<CAP> t;
  if (!seg_table(t, segs, n_seg, n)) return (int)cudaErrorInvalidValue;
  return bits_hi > 0 ? launch_maxnorm<true, CAP>(t, p, c->sm_count, max_blocks, st) : launch_maxnorm<false, CAP>(t, p, c->sm_count, max_blocks, st);
}

template <int CAP>
int copy_segs(const SegDesc* segs, int n_seg, int64_t n, int sm_count, cudaStream_t st) {
  SegTable<CAP> t;
  if (!seg_table(t, segs, n_seg, n)) return (int)cudaErrorInvalidValue;
  const uint32_t tiles = t.tile0[t.n], most = (uint32_t)sm_count * 2;
  solo_copy_kernel<CAP><<<tiles < most ? tiles : most, THREADS, 0, st>>>(t);
  return (int)cudaGetLastError();
}

SoloParams make_params(CommCtx* c, int bits_lo, int bits_hi, uint64_t seed, uint32_t step, int timeout_ms) {
  SoloParams p;
  p.hdr = (ArenaHeader*)c->local;
  p.step_from_device = c->step_from_device;
  p.timeout_ns = (unsigned long long)(timeout_ms > 0 ? timeout_ms : 30000) * 1000000ull;
  for (int r = 0; r < 10; ++r) {
    p.rk0[r] = (uint32_t)seed + (uint32_t)r * 0x9E3779B9u;
    p.rk1[r] = (uint32_t)(seed >> 32) + (uint32_t)r * 0xBB67AE85u;
  }
  p.step = step;
  p.stream = (uint32_t)c->rank << 8;
  p.s_lo = (1 << bits_lo) - 1;
  p.s_hi = bits_hi > 0 ? (1 << bits_hi) - 1 : 0;
  return p;
}

template <int CAP>
int randk_segs(CommCtx* c, const SegDesc* segs, int n_seg, int64_t n, const SoloParams& p, SoloRandk r, int max_blocks, cudaStream_t st) {
  SegTable<CAP> t;
  if (!seg_table(t, segs, n_seg, n)) return (int)cudaErrorInvalidValue;
  r.in_place = 0;
  bool dense = r.zero != 0;
  for (int i = 0; i < n_seg; ++i) {
    if (segs[i].in == segs[i].out) r.in_place = 1;
    else dense = true;
  }
  // 128 gathers a block keep every one of them in flight at once; a dense pass wants every SM
  int64_t blocks = (r.k + 127) / 128;
  if (dense && blocks < t.tile0[n_seg]) blocks = t.tile0[n_seg];
  if (blocks > c->sm_count) blocks = c->sm_count;
  if (max_blocks > 0 && blocks > max_blocks) blocks = max_blocks;
  if (blocks < 1) blocks = 1;
  if (r.k > blocks * THREADS * RANDK_PER_THREAD) return (int)cudaErrorInvalidValue;
  void* args[3] = {(void*)&t, (void*)&p, (void*)&r};
  const void* kernel = (const void*)solo_randk_kernel<CAP>;
  if (blocks == 1) return (int)cudaLaunchKernel(kernel, dim3(1), dim3(THREADS), args, 0, st);
  return (int)cudaLaunchCooperativeKernel(kernel, dim3((unsigned)blocks), dim3(THREADS), args, 0, st);
}

}  // namespace

extern "C" {

int gc_solo_max_segs() { return SEG_CAP_MANY; }

// One QSGD-MaxNorm reduce of a single worker (bits_hi > 0: two scales) over n_seg tensors of n elements in all.  Tables of one
// entry (a flat vector) get a kernel of their own: its parameters are small and its tiles need no search.
int gc_solo_maxnorm(void* ctx, const void* segs, int n_seg, int64_t n, int bits_lo, int bits_hi, uint64_t seed, uint32_t step, int timeout_ms,
                    int max_blocks, void* cs) {
  CommCtx* c = (CommCtx*)ctx;
  if (c->world != 1 || bits_lo < 1 || bits_lo > 16 || bits_hi < 0 || bits_hi > 16) return (int)cudaErrorInvalidValue;
  if (n <= 0) return 0;
  const SoloParams p = make_params(c, bits_lo, bits_hi, seed, step, timeout_ms);
  const SegDesc* d = (const SegDesc*)segs;
  cudaStream_t st = (cudaStream_t)cs;
  if (n_seg == 1) return maxnorm_segs<1>(c, d, n_seg, n, bits_lo, bits_hi, p, max_blocks, st);
  return maxnorm_segs<SEG_CAP_MANY>(c, d, n_seg, n, bits_lo, bits_hi, p, max_blocks, st);
}

// out = in for every tensor (segments whose two pointers are the same cost nothing when the caller leaves them out).
int gc_solo_copy(void* ctx, const void* segs, int n_seg, int64_t n, void* cs) {
  CommCtx* c = (CommCtx*)ctx;
  if (n <= 0 || n_seg <= 0) return 0;
  const SegDesc* d = (const SegDesc*)segs;
  if (n_seg == 1) return copy_segs<1>(d, n_seg, n, c->sm_count, (cudaStream_t)cs);
  return copy_segs<SEG_CAP_MANY>(d, n_seg, n, c->sm_count, (cudaStream_t)cs);
}

// Most coordinates a single worker's Rand-K takes (they are kept in registers); max_blocks as in the call.
int64_t gc_solo_randk_limit(void* ctx, int max_blocks) {
  const int sms = ((CommCtx*)ctx)->sm_count;
  return (int64_t)(max_blocks > 0 && max_blocks < sms ? max_blocks : sms) * THREADS * RANDK_PER_THREAD;
}

// One Rand-K reduce of a single worker (bits_hi > 0: two scales) on the window [start, start + k) of the keyed permutation of
// [0, n); window (device, may be NULL): the start is read from it and the next one stored.
int gc_solo_randk(void* ctx, const void* segs, int n_seg, int64_t n, uint64_t index_seed, uint32_t npass, int64_t start, int64_t k, int64_t* window,
                  int bits_lo, int bits_hi, int zero, uint32_t step, int timeout_ms, int max_blocks, void* cs) {
  CommCtx* c = (CommCtx*)ctx;
  if (c->world != 1 || bits_lo < 1 || bits_lo > 16 || bits_hi < 0 || bits_hi > 16) return (int)cudaErrorInvalidValue;
  if (n <= 0) return 0;
  const SoloParams p = make_params(c, bits_lo, bits_hi, index_seed, step, timeout_ms);
  SoloRandk r;
  r.perm = make_perm_key((uint64_t)n, index_seed, npass);
  r.start = start;
  r.k = k < n ? k : n;
  r.window = window;
  r.zero = zero;
  const SegDesc* d = (const SegDesc*)segs;
  if (n_seg == 1) return randk_segs<1>(c, d, n_seg, n, p, r, max_blocks, (cudaStream_t)cs);
  return randk_segs<SEG_CAP_MANY>(c, d, n_seg, n, p, r, max_blocks, (cudaStream_t)cs);
}

}  // extern "C"
