// Top-K selection by |value| for many tensors at once (reference: reducer.py:1144-1451, there one torch.topk per tensor), with
// the error feedback folded in: a = g + e; the k largest |a| of every group are selected; e becomes a with the selected
// entries zeroed.  A group is one tensor, or all of them together.
//
//   topk_fold_kernel     a = g + e -> e, and a histogram of the top 13 bits of |a| per group                 (12 bytes an element)
//   topk_pick_kernel     per group: the bin that holds the k-th largest (groups of up to 4096 elements: the whole selection)
//   topk_split_kernel    above that bin: selected.  In it: put on the group's candidate list.  Below: not selected.
//   topk_refine_kernel   per group: exact selection among the candidates by the remaining 18 bits, in two steps of 9, then by index
//
// Two outputs.  LISTS (several workers): index and value of the selected entries, for the exchange.  DENSE (a single
// worker, whose exchange is the identity): the selected entries in an otherwise zero gradient, written by the split
// kernel where it reads, straight into the gradient tensors.
//
// What bounds it: fold reads g and e and writes e, split reads e and writes the gradient: 20 bytes an element against the 16 no
// implementation can avoid.  Thirteen bits (five of the mantissa, so a bin spans three percent in value) make that second
// reading the last one: a bin near the threshold holds about 0.2 % of normally distributed values (some percent once error
// feedback has piled values up below it), few enough for a cluster of blocks per group to finish.  Split walks the tiles backwards: what fold wrote last is read from L2.  Counts and
// candidates are gathered in shared memory and leave it in one atomic per warp and some hundred entries.
// Groups whose bin holds more candidates than their list has room for (one value repeated over much of a tensor) are
// refined by reading the tensor again instead (split then leaves the error memory to refine, which still has to tell the
// selected entries from the candidates).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "gc_device.cuh"
#include "gc_segs.cuh"

using namespace gc;
namespace cg = cooperative_groups;

namespace {

constexpr int THREADS = SEG_TILE;
constexpr int WARPS = THREADS / 32;
constexpr int LOW_BITS = 18, HIGH_BITS = 13;
constexpr int BINS = 1 << HIGH_BITS;
constexpr int SMALL = 4 * THREADS;         // groups of at most this many elements are selected from by one block, in registers
constexpr int WARP_ROOM = 256;             // candidates a warp holds back; a quad per lane adds at most 128
constexpr int SUB_BITS = 9, SUB_BINS = 1 << SUB_BITS;

struct GroupState {        // device resident, all zero between runs except what pick writes
  int32_t bin;             // -1: everything is selected
  int32_t k_rem;           // how many of the bin's entries are selected
  uint32_t in_bin;         // entries in the bin
  uint32_t taken;          // LISTS: slots handed to selected entries
  uint32_t listed;         // candidates on the list
  uint32_t pad[3];
};

struct Cand {
  float a;
  int32_t at;
  __device__ __forceinline__ uint32_t key() const { return __float_as_uint(a) & 0x7fffffffu; }
};

template <int CAP>
struct TopkParams {
  SegTable<CAP> t;
  int k[CAP];              // per group
  int64_t room0[CAP + 1];  // candidate lists: first entry per group
  int64_t slot0[CAP];      // LISTS: first output slot per group
  uint16_t large[CAP];     // groups of more than SMALL elements
  int n_groups, n_large, per_tensor;
  float* e;                // error memory by flat element (nullptr: none, a = g)
  GroupState* state;
  uint32_t* hist;
  Cand* cands;
  int32_t* out_idx;
  float* out_val;
  __device__ __forceinline__ int group(int s) const { return CAP == 1 || per_tensor ? s : 0; }
  __device__ __forceinline__ bool small(int g) const { return per_tensor && t.start[g + 1] - t.start[g] <= SMALL; }
  __device__ __forceinline__ int64_t len(int g) const { return per_tensor ? t.start[g + 1] - t.start[g] : t.start[t.n] - t.start[0]; }
};

__device__ __forceinline__ uint32_t key_of(float a) { return __float_as_uint(a) & 0x7fffffffu; }

template <int CAP>
__device__ __forceinline__ void fold_flush(const TopkParams<CAP>& p, uint32_t* sh, int g) {
  __syncthreads();
  for (int i = threadIdx.x; i < BINS; i += THREADS)
    if (sh[i]) { atomicAdd(&p.hist[(int64_t)g * BINS + i], sh[i]); sh[i] = 0; }
  __syncthreads();
}

// a quad of which only elements [a, b) belong to the tensor
__device__ __forceinline__ void quad_store_part(float* p, const float4& v, int a, int b) {
  if (b - a == 4 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0) { *reinterpret_cast<float4*>(p) = v; return; }
  if (a <= 0 && b > 0) p[0] = v.x;
  if (a <= 1 && b > 1) p[1] = v.y;
  if (a <= 2 && b > 2) p[2] = v.z;
  if (a <= 3 && b > 3) p[3] = v.w;
}
__device__ __forceinline__ float4 quad_load_part(const float* p, int a, int b) {
  if (b - a == 4 && (reinterpret_cast<uintptr_t>(p) & 15u) == 0) return __ldcg(reinterpret_cast<const float4*>(p));
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (a <= 0 && b > 0) v.x = p[0];
  if (a <= 1 && b > 1) v.y = p[1];
  if (a <= 2 && b > 2) v.z = p[2];
  if (a <= 3 && b > 3) v.w = p[3];
  return v;
}

template <int CAP>
__global__ void __launch_bounds__(THREADS, 1) topk_fold_kernel(const __grid_constant__ TopkParams<CAP> p) {
  __shared__ uint32_t sh[BINS];
  const SegTable<CAP>& t = p.t;
  for (int i = threadIdx.x; i < BINS; i += THREADS) sh[i] = 0;
  pdl_launch_dependents();
  __syncthreads();
  const uint32_t tiles = t.tile0[t.n], per = (tiles + gridDim.x - 1) / gridDim.x, first = blockIdx.x * per;
  if (first >= tiles) return;
  uint32_t left = tiles - first < per ? tiles - first : per;
  auto count = [&](const float4& a) {
    atomicAdd(&sh[key_of(a.x) >> LOW_BITS], 1u);
    atomicAdd(&sh[key_of(a.y) >> LOW_BITS], 1u);
    atomicAdd(&sh[key_of(a.z) >> LOW_BITS], 1u);
    atomicAdd(&sh[key_of(a.w) >> LOW_BITS], 1u);
  };
  const bool mem = p.e != nullptr, al_e = (reinterpret_cast<uintptr_t>(p.e) & 15u) == 0;
  SegCursor<CAP, 1> c(t, first);
  int g = p.group(c.s);
  while (left > 0) {
    if (p.group(c.s) != g) { fold_flush(p, sh, g); g = p.group(c.s); }
    const bool counts = p.k[g] < p.len(g) && !p.small(g);          // (everything is selected: no threshold to find)
    if (left >= 4 && c.fast_in && al_e && c.run >= 3) {
      // four whole tiles at a time: 128 KB in flight per SM
      float4 a[4];
      float4* e = reinterpret_cast<float4*>(p.e) + c.quad;
#pragma unroll
      for (int u = 0; u < 4; ++u) a[u] = __ldcs(reinterpret_cast<const float4*>(c.in) + u * SEG_TILE);
      if (mem) {
        float4 b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) b[u] = __ldcg(e + u * SEG_TILE);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          a[u].x += b[u].x; a[u].y += b[u].y; a[u].z += b[u].z; a[u].w += b[u].w;
          e[u * SEG_TILE] = a[u];
        }
      }
      if (counts) {
#pragma unroll
        for (int u = 0; u < 4; ++u) count(a[u]);
      }
      left -= 4;
      c.template skip<3>();
      if (left > 0) c.step(t);
      continue;
    }
    if (!c.empty(t)) {
      const int a0 = c.whole ? 0 : c.first(t), b0 = c.whole ? 4 : c.last(t);
      float4 a = c.load(t);
      if (mem) {
        float* e = p.e + c.quad * 4;
        const float4 b = quad_load_part(e, a0, b0);
        a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
        quad_store_part(e, a, a0, b0);
      }
      if (counts) {
        if (b0 - a0 == 4) count(a);
        else {
          const float v[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j >= a0 && j < b0) atomicAdd(&sh[key_of(v[j]) >> LOW_BITS], 1u);
        }
      }
    }
    --left;
    if (left > 0) c.step(t);
  }
  fold_flush(p, sh, g);
}

// Thread i of the block holds sum; returns the total of the threads before it.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t sum, uint32_t* warp_sums) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t up = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += up;
  }
  __syncthreads();
  if (lane == 31) warp_sums[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    uint32_t w = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0u, s = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t up = __shfl_up_sync(FULL, s, o);
      if (lane >= o) s += up;
    }
    warp_sums[lane] = s - w;
  }
  __syncthreads();
  return warp_sums[wid] + incl - sum;
}

// Appends to the output lists, `n` entries per call of a warp's lanes (n is 0 or 1 per lane).
template <int CAP>
__device__ __forceinline__ void list_take(const TopkParams<CAP>& p, int g, bool take, int64_t at, float a) {
  const unsigned m = __ballot_sync(FULL, take);
  if (m == 0) return;
  const int lane = threadIdx.x & 31;
  uint32_t base = 0;
  if (lane == 0) base = atomicAdd(&p.state[g].taken, (uint32_t)__popc(m));
  base = __shfl_sync(FULL, base, 0);
  if (take) {
    const int64_t slot = p.slot0[g] + base + __popc(m & ((1u << lane) - 1u));
    p.out_idx[slot] = (int32_t)at;
    p.out_val[slot] = a;
  }
}

// A small group, whole: its elements in registers, the threshold found eight bits at a time.
template <int CAP, bool LISTS>
__device__ __forceinline__ void select_small(const TopkParams<CAP>& p, int g, uint32_t* hist, uint32_t* warp_sums, int* found) {
  const SegTable<CAP>& t = p.t;
  const int64_t lo = t.start[g], len = t.start[g + 1] - lo, k = p.k[g];
  float v[4];
  uint32_t key[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int64_t i = threadIdx.x + j * THREADS;
    v[j] = i < len ? (p.e != nullptr ? p.e[lo + i] : t.in[g][i]) : 0.0f;
    key[j] = key_of(v[j]);
  }
  uint32_t prefix = 0;
  int rem = (int)k;
  if (k < len) {
#pragma unroll
    for (int part = 0; part < 4; ++part) {             // 8 + 8 + 8 + 7 bits
      const int shift = part == 3 ? 0 : 23 - 8 * part, bits = part == 3 ? 7 : 8;
      if (threadIdx.x < 256) hist[threadIdx.x] = 0;
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (threadIdx.x + j * THREADS < len && (part == 0 || (key[j] >> (shift + bits)) == prefix)) atomicAdd(&hist[(key[j] >> shift) & ((1u << bits) - 1u)], 1u);
      __syncthreads();
      const uint32_t mine = threadIdx.x < 256 ? hist[255 - threadIdx.x] : 0u;
      const uint32_t above = block_exclusive(mine, warp_sums);
      if (above < (uint32_t)rem && above + mine >= (uint32_t)rem) { found[0] = 255 - threadIdx.x; found[1] = rem - (int)above; }
      __syncthreads();
      prefix = (prefix << bits) | (uint32_t)found[0];
      rem = found[1];
      __syncthreads();
    }
  }
  // of the entries equal to the threshold the first ones are taken
  const bool some = k > 0 && k < len && hist[prefix & 127u] > (uint32_t)rem;
  int before = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int64_t i = threadIdx.x + j * THREADS;
    bool take = i < len && k > 0 && (k >= len || key[j] > prefix);
    bool equal = i < len && k > 0 && k < len && key[j] == prefix;
    if (some) {
      const int order = before + (int)block_exclusive(equal ? 1u : 0u, warp_sums);
      before += __syncthreads_count(equal);
      equal = equal && order < rem;
    }
    take |= equal;
    if (LISTS) list_take(p, g, take, lo + i, v[j]);
    else if (i < len) t.out[g][i] = take ? v[j] : 0.0f;
    if (take && p.e != nullptr) p.e[lo + i] = 0.0f;
  }
}

// One block per group; thread 0 owns the top bins.
template <int CAP, bool LISTS>
__global__ void __launch_bounds__(THREADS) topk_pick_kernel(const __grid_constant__ TopkParams<CAP> p) {
  __shared__ uint32_t warp_sums[32], hist[256];
  __shared__ int found[2];
  const int g = blockIdx.x;
  const int64_t k = p.k[g], len = p.len(g);
  GroupState* st = p.state + g;
  pdl_wait();
  pdl_launch_dependents();
  if (threadIdx.x == 0) { st->taken = 0; st->listed = 0; }
  __syncthreads();
  if (p.small(g)) { select_small<CAP, LISTS>(p, g, hist, warp_sums, found); return; }
  constexpr int PER = BINS / THREADS;
  const int top = BINS - 1 - threadIdx.x * PER;
  uint32_t* h = p.hist + (int64_t)g * BINS + (top - PER + 1);
  uint32_t local[PER], sum = 0;
#pragma unroll
  for (int j = 0; j < PER; j += 4) {
    const uint4 v = *reinterpret_cast<const uint4*>(h + j);
    *reinterpret_cast<uint4*>(h + j) = make_uint4(0, 0, 0, 0);
    local[j] = v.x; local[j + 1] = v.y; local[j + 2] = v.z; local[j + 3] = v.w;
    sum += v.x + v.y + v.z + v.w;
  }
  if (k >= len || k <= 0) {
    if (threadIdx.x == 0) { st->bin = k <= 0 ? BINS : -1; st->k_rem = 0; st->in_bin = 0; }
    return;
  }
  uint32_t run = block_exclusive(sum, warp_sums);
#pragma unroll
  for (int j = PER - 1; j >= 0; --j) {               // local[PER - 1] is this thread's top bin
    if (run < (uint32_t)k && run + local[j] >= (uint32_t)k) {
      st->bin = top - (PER - 1) + j;
      st->k_rem = (int32_t)((uint32_t)k - run);
      st->in_bin = local[j];
    }
    run += local[j];
  }
}

template <int CAP, bool LISTS>
__global__ void __launch_bounds__(THREADS, 1) topk_split_kernel(const __grid_constant__ TopkParams<CAP> p) {
  extern __shared__ Cand held_all[];       // [WARPS][WARP_ROOM]
  __shared__ int held_count[WARPS];
  const SegTable<CAP>& t = p.t;
  const int lane = threadIdx.x & 31;
  Cand* held = held_all + (threadIdx.x >> 5) * WARP_ROOM;
  int* count = held_count + (threadIdx.x >> 5);
  if (lane == 0) *count = 0;
  __syncwarp();
  pdl_wait();
  pdl_launch_dependents();
  const uint32_t tiles = t.tile0[t.n], per = (tiles + gridDim.x - 1) / gridDim.x, first = blockIdx.x * per;
  if (first >= tiles) return;
  uint32_t left = tiles - first < per ? tiles - first : per;
  const bool mem = p.e != nullptr, al_e = (reinterpret_cast<uintptr_t>(p.e) & 15u) == 0;

  auto flush = [&](int g) {
    __syncwarp();
    const int n = *count;
    if (n > 0) {
      uint32_t base = 0;
      if (lane == 0) base = atomicAdd(&p.state[g].listed, (uint32_t)n);
      base = __shfl_sync(FULL, base, 0);
      Cand* list = p.cands + p.room0[g] + base;
      for (int i = lane; i < n; i += 32) list[i] = held[i];          // fits: the bin's count was checked against the room
    }
    __syncwarp();
    if (lane == 0) *count = 0;
    __syncwarp();
  };
  int g = -1;
  uint32_t from = 0, above = 0;              // keys of the bin: [from, above)
  bool listing = false;
  // one quad: a (elements [a0, b0) of it) at flat element `at`; y: what goes into the gradient; true when `a` changed
  auto quad = [&](float4& a, int64_t at, int a0, int b0, float4& y) {
    float* v = &a.x;
    float* o = &y.x;
    uint32_t key[4];
    unsigned cand = 0;
    bool changed = false;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      key[j] = key_of(v[j]);
      const bool mine = j >= a0 && j < b0;
      const bool sure = mine && key[j] >= above;
      if (mine && !sure && key[j] >= from) cand |= 1u << j;
      if (LISTS) list_take(p, g, sure, at + j, v[j]);
      o[j] = sure ? v[j] : 0.0f;
      changed = changed || sure;
    }
    if (changed && listing) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (o[j] != 0.0f) v[j] = 0.0f;       // (a selected zero is a zero either way)
    }
    if (listing && __any_sync(FULL, cand != 0)) {
      if (cand != 0) {
        int to = atomicAdd(count, __popc(cand));
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if ((cand >> j) & 1u) held[to++] = Cand{v[j], (int32_t)(at + j)};
      }
      __syncwarp();
      if (*count > WARP_ROOM - 128) flush(g);
    }
    return changed && listing;
  };

  SegCursor<CAP, -1> c(t, first + left - 1);
  while (left > 0) {
    if (p.group(c.s) != g) {
      if (g >= 0) flush(g);
      g = p.group(c.s);
      if (p.small(g)) {                      // done by the pick kernel
        g = -1;
        if (--left > 0) c.step(t);
        continue;
      }
      const int bin = p.state[g].bin;                                 // -1: everything is above it
      from = bin < 0 ? 0u : (uint32_t)bin << LOW_BITS;
      above = (uint32_t)(bin + 1) << LOW_BITS;
      listing = (int64_t)p.state[g].in_bin <= p.room0[g + 1] - p.room0[g];
    }
    if (left >= 4 && c.fast_in && (LISTS || c.fast_out) && al_e && c.run >= 3) {
      float4 a[4];
      const float4* src = mem ? reinterpret_cast<const float4*>(p.e) + c.quad : reinterpret_cast<const float4*>(c.in);
#pragma unroll
      for (int u = 0; u < 4; ++u) a[u] = __ldcg(src - u * SEG_TILE);
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float4 y;
        const bool changed = quad(a[u], (int64_t)(c.quad - u * SEG_TILE) * 4, 0, 4, y);
        if (mem && changed) *(reinterpret_cast<float4*>(p.e) + c.quad - u * SEG_TILE) = a[u];
        if (!LISTS) __stcs(reinterpret_cast<float4*>(c.out) - u * SEG_TILE, y);
      }
      left -= 4;
      c.template skip<3>();
      if (left > 0) c.step(t);
      continue;
    }
    {
      const int a0 = c.whole ? 0 : c.first(t), b0 = c.whole ? 4 : c.last(t);
      float* e = p.e + c.quad * 4;
      float4 a = mem ? quad_load_part(e, a0, b0) : (a0 < b0 ? c.load(t) : make_float4(0.f, 0.f, 0.f, 0.f));
      float4 y;
      const bool changed = quad(a, (int64_t)c.quad * 4, a0, b0, y);
      if (mem && changed) quad_store_part(e, a, a0, b0);
      if (!LISTS && a0 < b0) c.store(t, y);
    }
    --left;
    if (left > 0) c.step(t);
  }
  if (g >= 0) flush(g);
}

// Of the entries equal to the threshold the first by index are taken, so that the selection does not depend on how blocks run.  Up to
// this many of them (a few of a million random floats share a value) wait in shared memory and are ordered there; among more of them
// the index of the last one taken is found as the threshold was, nine bits at a time: two or three more readings of the candidates.
constexpr int TIES = 128;

// What the blocks of a cluster count together, in rank 0's shared memory.
struct Tally {
  uint4 found;                             // the bin, how many of its entries are wanted, how many it has: one read of another block's memory
  uint32_t hist[SUB_BINS], warp_sums[32];
};

// The bin of the rem-th entry that the blocks have counted, from the highest bin or from the lowest.  rem: how many entries of that bin
// are wanted; same: how many it has.
__device__ __forceinline__ uint32_t settle_bin(Tally& t, bool highest, int& rem, uint32_t& same) {
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned rank = cluster.block_rank();
  cluster.sync();
  if (rank != 0 && threadIdx.x < SUB_BINS && t.hist[threadIdx.x]) atomicAdd(cluster.map_shared_rank(&t.hist[threadIdx.x], 0), t.hist[threadIdx.x]);
  cluster.sync();
  if (rank == 0) {
    const int at = highest ? SUB_BINS - 1 - (int)threadIdx.x : (int)threadIdx.x;
    const uint32_t mine = threadIdx.x < SUB_BINS ? t.hist[at] : 0u;
    const uint32_t before = block_exclusive(mine, t.warp_sums);
    if (before < (uint32_t)rem && before + mine >= (uint32_t)rem) t.found = make_uint4((uint32_t)at, (uint32_t)rem - before, mine, 0u);
  }
  cluster.sync();
  const uint4 found = *cluster.map_shared_rank(&t.found, 0);
  cluster.sync();
  rem = (int)found.y;
  same = found.z;
  return found.x;
}

// One cluster of blocks per group; the blocks share the group's candidates and add their counts up in rank 0's shared memory.  Two blocks
// an SM where there are many groups (the launch counts on them; ResNet-50's reduce 133.6 -> 129.3 us); a single group has 16 at most,
// and is faster with the registers (77.4 against 79.6 us at 16 M elements).
template <int CAP, bool LISTS>
__global__ void __launch_bounds__(THREADS, CAP == 1 ? 1 : 2) topk_refine_kernel(const __grid_constant__ TopkParams<CAP> p) {
  __shared__ Tally tally_of;
  __shared__ uint32_t equal_seen;
  __shared__ Cand ties[TIES];              // rank 0's: entries equal to the threshold
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned rank = cluster.block_rank(), ranks = cluster.num_blocks();
  const SegTable<CAP>& t = p.t;
  const int g = p.large[blockIdx.x / ranks];
  GroupState* st = p.state + g;
  pdl_wait();
  const int k_rem = st->k_rem;
  const uint32_t in_bin = st->in_bin;
  if (k_rem <= 0) return;                  // (the whole cluster)
  const int bin = st->bin;
  const bool listed = (int64_t)in_bin <= p.room0[g + 1] - p.room0[g];
  const int64_t lo = p.per_tensor ? t.start[g] : t.start[0];
  const int64_t count = listed ? (int64_t)in_bin : p.len(g);
  const int64_t from = (int64_t)rank * THREADS, stride = (int64_t)ranks * THREADS;
  const Cand* list = p.cands + p.room0[g];
  auto entry = [&](int64_t i) {
    if (listed) return list[i];
    const int64_t at = lo + i;
    if (p.e != nullptr) return Cand{p.e[at], (int32_t)at};
    const int s = seg_of_elem(t, at);
    return Cand{t.in[s][at - t.start[s]], (int32_t)at};
  };
  auto in_it = [&](const Cand& c) { return listed || (int)(c.key() >> LOW_BITS) == bin; };
  uint32_t prefix = 0, same = 0;           // the threshold's low bits; entries equal to it
  int rem = k_rem;                         // how many of them are taken
  bool by_index = false;
  const bool all = (uint32_t)k_rem >= in_bin;
  if (threadIdx.x == 0) equal_seen = 0;
  if (!all) {
    uint32_t* hist = tally_of.hist;
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      if (threadIdx.x < SUB_BINS) hist[threadIdx.x] = 0;
      __syncthreads();
      auto tally = [&](const Cand& c) {
        const uint32_t low = c.key() & ((1u << LOW_BITS) - 1u);
        if (part == 0) atomicAdd(&hist[low >> SUB_BITS], 1u);
        else if ((low >> SUB_BITS) == prefix) atomicAdd(&hist[low & (SUB_BINS - 1)], 1u);
      };
      int64_t i = from + threadIdx.x;
      if (listed)
        for (; i + 3 * stride < count; i += 4 * stride) {
          const Cand c0 = list[i], c1 = list[i + stride], c2 = list[i + 2 * stride], c3 = list[i + 3 * stride];
          tally(c0); tally(c1); tally(c2); tally(c3);
        }
      for (; i < count; i += stride) {
        const Cand c = entry(i);
        if (in_it(c)) tally(c);
      }
      const uint32_t got = settle_bin(tally_of, true, rem, same);
      prefix = part == 0 ? got : (prefix << SUB_BITS) | got;
    }
    by_index = same > (uint32_t)TIES && same > (uint32_t)rem && (bin != 0 || prefix != 0);          // (zeros are all the same)
  } else {
    cluster.sync();
  }
  uint32_t* equal = cluster.map_shared_rank(&equal_seen, 0);
  Cand* waiting = cluster.map_shared_rank(&ties[0], 0);
  auto place = [&](const Cand& c, bool take, bool taken) {
    if (LISTS) list_take(p, g, take, c.at, c.a);
    if (take && !LISTS) {
      const int s = p.per_tensor ? g : seg_of_elem(t, (int64_t)c.at);
      t.out[s][c.at - t.start[s]] = c.a;
    }
    if ((take || taken) && p.e != nullptr) p.e[c.at] = 0.0f;
  };
  auto settle = [&](const Cand& c, bool there) {
    const bool valid = there && in_it(c), taken = there && !listed && (int)(c.key() >> LOW_BITS) > bin;
    const uint32_t low = c.key() & ((1u << LOW_BITS) - 1u);
    bool take = valid && (all || low > prefix);
    if (valid && !all && low == prefix && !by_index) {
      const uint32_t at = atomicAdd(equal, 1u);
      if (at < (uint32_t)TIES) waiting[at] = c;
      else take = (int)at < rem;           // (all of them are, or they are zeros)
    }
    place(c, take, taken);
  };
  int64_t base = from;
  for (; listed && base + 3 * stride + THREADS <= count; base += 4 * stride) {
    const Cand* l = list + base + threadIdx.x;
    const Cand c0 = l[0], c1 = l[stride], c2 = l[2 * stride], c3 = l[3 * stride];
    settle(c0, true); settle(c1, true); settle(c2, true); settle(c3, true);
  }
  for (; base < count; base += stride) {
    const bool there = base + threadIdx.x < count;
    settle(there ? entry(base + threadIdx.x) : Cand{0.0f, 0}, there);
  }
  cluster.sync();                          // rank 0's shared memory stays until every block is done with it
  if (rank == 0 && threadIdx.x < TIES) {
    const int n = equal_seen < (uint32_t)TIES ? (int)equal_seen : TIES;
    const Cand mine = (int)threadIdx.x < n ? ties[threadIdx.x] : Cand{0.0f, 0};
    int order = 0;
    for (int j = 0; j < n; ++j) order += ties[j].at < mine.at;
    place(mine, (int)threadIdx.x < n && order < rem, false);
  }
  if (!by_index) return;
  // the index of the rem-th of the equal entries, nine bits at a time, and then all of them up to it
  const uint32_t key = (uint32_t)bin << LOW_BITS | prefix;
  uint32_t upper = 0;
  int shift = 0;
  while (p.len(g) >> (shift + SUB_BITS)) shift += SUB_BITS;
#pragma unroll 1
  for (; shift >= 0; shift -= SUB_BITS) {
    if (threadIdx.x < SUB_BINS) tally_of.hist[threadIdx.x] = 0;
    __syncthreads();
#pragma unroll 1
    for (int64_t i = from + threadIdx.x; i < count; i += stride) {
      const Cand c = entry(i);
      const uint32_t at = (uint32_t)(c.at - lo) >> shift;
      if (c.key() == key && (at >> SUB_BITS) == upper) atomicAdd(&tally_of.hist[at & (SUB_BINS - 1)], 1u);
    }
    upper = (upper << SUB_BITS) | settle_bin(tally_of, false, rem, same);
  }
#pragma unroll 1
  for (base = from; base < count; base += stride) {
    const Cand c = base + threadIdx.x < count ? entry(base + threadIdx.x) : Cand{0.0f, 0};
    place(c, base + threadIdx.x < count && c.key() == key && (uint32_t)(c.at - lo) <= upper, false);
  }
}

int64_t list_room(int64_t len) { return len / 8 + 1024; }

template <int CAP>
int run(const SegDesc* segs, int n_seg, int64_t end, const int64_t* k, int per_tensor, float* e, void* state, void* list, int32_t* out_idx, float* out_val,
        cudaStream_t st) {
  TopkParams<CAP> p;
  if (!seg_table(p.t, segs, n_seg, end)) return (int)cudaErrorInvalidValue;
  if (p.t.tile0[n_seg] == 0) return 0;
  p.n_groups = per_tensor ? n_seg : 1;
  p.per_tensor = per_tensor || n_seg == 1;
  p.n_large = 0;
  int64_t room = 0, slot = 0, longest = 0;
  for (int g = 0; g < p.n_groups; ++g) {
    const int64_t len = p.per_tensor ? p.t.start[g + 1] - p.t.start[g] : end - p.t.start[0];
    const int64_t kk = k[g] < len ? k[g] : len;
    p.k[g] = (int)kk;
    p.room0[g] = room;
    p.slot0[g] = slot;
    room += list_room(len);
    longest = len > longest ? len : longest;
    if (!p.per_tensor || len > SMALL) p.large[p.n_large++] = (uint16_t)g;
    slot += kk;
  }
  p.room0[p.n_groups] = room;
  p.e = e;
  p.state = (GroupState*)state;
  p.hist = (uint32_t*)((uint8_t*)state + (int64_t)p.n_groups * sizeof(GroupState));
  p.cands = (Cand*)list;
  p.out_idx = out_idx;
  p.out_val = out_val;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const uint32_t tiles = p.t.tile0[n_seg];
  const unsigned grid = tiles < (uint32_t)sms ? tiles : (unsigned)sms;
  constexpr int held = WARPS * WARP_ROOM * (int)sizeof(Cand);
  const bool lists = out_idx != nullptr;
  const void* split = lists ? (const void*)topk_split_kernel<CAP, true> : (const void*)topk_split_kernel<CAP, false>;
  cudaError_t err = cudaFuncSetAttribute(split, cudaFuncAttributeMaxDynamicSharedMemorySize, held);
  if (err != cudaSuccess) return (int)err;
  topk_fold_kernel<CAP><<<grid, THREADS, 0, st>>>(p);
  // the kernels behind the first one start while their predecessor ends
  err = lists ? launch_pdl(topk_pick_kernel<CAP, true>, dim3(p.n_groups), dim3(THREADS), 0, st, p) : launch_pdl(topk_pick_kernel<CAP, false>, dim3(p.n_groups), dim3(THREADS), 0, st, p);
  if (err != cudaSuccess) return (int)err;
  if (p.n_large == 0) return (int)cudaGetLastError();
  err = lists ? launch_pdl(topk_split_kernel<CAP, true>, dim3(grid), dim3(THREADS), held, st, p) : launch_pdl(topk_split_kernel<CAP, false>, dim3(grid), dim3(THREADS), held, st, p);
  if (err != cudaSuccess) return (int)err;
  // Blocks per group: what the longest group can fill with a few thousand candidates each (with error feedback, values pile up
  // below the threshold and the bin holds some percent of the group), as long as all groups fit on the chip at once, two blocks
  // an SM; clusters of sixteen only for a few groups, as they take whole GPU clusters to place (ResNet-50's 55 groups: 23 us
  // with eight blocks each, 48 us with sixteen; one group of 64 M elements: 210 us with eight, 84 us with sixteen).
  int ranks = 1;
  while (ranks < (p.n_large <= 4 ? 16 : 8) && longest / 32 > (int64_t)ranks * 4 * THREADS && p.n_large * ranks * 2 <= 2 * sms) ranks *= 2;
  if (ranks > 8) {
    const void* refine = lists ? (const void*)topk_refine_kernel<CAP, true> : (const void*)topk_refine_kernel<CAP, false>;
    err = cudaFuncSetAttribute(refine, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (err != cudaSuccess) return (int)err;
  }
  const dim3 blocks((unsigned)(p.n_large * ranks));
  return (int)(lists ? launch_cluster(topk_refine_kernel<CAP, true>, (unsigned)ranks, blocks, dim3(THREADS), 0, st, p)
                     : launch_cluster(topk_refine_kernel<CAP, false>, (unsigned)ranks, blocks, dim3(THREADS), 0, st, p));
}

}  // namespace

extern "C" {

// Tensors one run takes.
int gc_cuda_topk_max_segs() { return SEG_CAP_MANY; }
// Scratch of a run: state is zeroed once after allocation (every run leaves it ready for the next), lists need no initialisation.
int64_t gc_cuda_topk_state_bytes(int n_groups) { return (int64_t)n_groups * ((int64_t)sizeof(GroupState) + BINS * 4); }
int64_t gc_cuda_topk_list_bytes(int64_t len) { return list_room(len) * (int64_t)sizeof(Cand); }

// segs: n_seg SegDesc, consecutive in the flat vector, the last one ending at flat element `end`.  k: one count per group
// (per_tensor: a group per segment, otherwise one group).  e: error memory by flat element (NULL: selection on g itself).
// out_idx / out_val: sum of k entries, group after group; NULL: the selected entries go into the segments' outputs, which
// are zero elsewhere.
int gc_cuda_topk_run(const void* segs, int n_seg, int64_t end, const int64_t* k, int per_tensor, float* e, void* state, void* list, int32_t* out_idx,
                     float* out_val, void* cs) {
  if (n_seg < 1 || n_seg > SEG_CAP_MANY || end > 0x7fffffffll) return (int)cudaErrorInvalidValue;
  if (n_seg == 1) return run<1>((const SegDesc*)segs, 1, end, k, per_tensor, e, state, list, out_idx, out_val, (cudaStream_t)cs);
  return run<SEG_CAP_MANY>((const SegDesc*)segs, n_seg, end, k, per_tensor, e, state, list, out_idx, out_val, (cudaStream_t)cs);
}

}  // extern "C"
