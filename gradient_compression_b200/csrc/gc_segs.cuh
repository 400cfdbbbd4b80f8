// Gradients held in many tensors, addressed as one flat vector.
//
// A reducer is handed a list of tensors.  Kernels that run on a single worker take the list as it is: a table of
// {input pointer, output pointer, flat start} travels by value in the kernel's parameters (no upload, nothing to keep in
// step with the tensors, replayable from a CUDA graph), so neither a concatenation of the inputs nor a scatter of the
// outputs passes over memory.  Tensors that lie back to back in both lists have been merged by the caller: a flat arena is
// one segment.
//
// Work is cut into tiles of SEG_TILE quads.  A quad is four consecutive elements of the FLAT vector starting at a multiple
// of four, because that is the unit the rounding noise is generated in; a quad that straddles two tensors is processed
// once per tensor, each taking its own elements.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace gc {

struct SegDesc {            // host side, as the callers pass it
  const float* in;
  float* out;
  int64_t start;            // first element's index in the flat vector
};

constexpr int SEG_TILE = 1024;      // quads per tile: one per thread of a 1024-thread block

// 24 bytes per tensor: 320 tensors (ResNet-101 has 314) fit well inside the 32 KB of kernel parameters.
template <int CAP>
struct SegTable {
  const float* in[CAP];
  float* out[CAP];
  int64_t start[CAP + 1];
  uint32_t tile0[CAP + 1];
  int n;
};

constexpr int SEG_CAP_MANY = 320;

// First flat element of quad `q` of tile `tile` of segment s.
template <int CAP>
__device__ __forceinline__ int64_t seg_elem(const SegTable<CAP>& t, int s, uint32_t tile, int q) {
  return ((t.start[s] >> 2) + (int64_t)(tile - t.tile0[s]) * SEG_TILE + q) << 2;
}

// Segment that holds a tile (binary search).
template <int CAP>
__device__ __forceinline__ int seg_of_tile(const SegTable<CAP>& t, uint32_t tile) {
  int lo = 0, hi = t.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.tile0[mid] <= tile) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Segment of a flat element (binary search).
template <int CAP>
__device__ __forceinline__ int seg_of_elem(const SegTable<CAP>& t, int64_t e) {
  int lo = 0, hi = CAP == 1 ? 0 : t.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.start[mid] <= e) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// One thread's place in a run of consecutive tiles, walked forwards (DIR = 1) or backwards (-1).  Tiles that lie whole inside a
// tensor are stepped over with a countdown and three additions; everything else is looked up again.
template <int CAP, int DIR>
struct SegCursor {
  const float* in;          // this thread's quad of the tile
  float* out;
  uint64_t quad;            // its index in the flat vector (the block index of its rounding noise)
  uint32_t tile;
  int s;
  int run;                  // how many of the next tiles lie whole inside the same tensor
  bool whole;               // every quad of the tile lies whole inside the tensor
  bool fast_in, fast_out;   // ... and is 16-byte aligned

  __device__ __forceinline__ SegCursor(const SegTable<CAP>& t, uint32_t first) {
    tile = first;
    s = seg_of_tile(t, tile);
    enter(t);
  }
  __device__ __forceinline__ void enter(const SegTable<CAP>& t) {
    const int64_t a = t.start[s], b = t.start[s + 1];
    const int64_t e = seg_elem(t, s, tile, threadIdx.x), e0 = seg_elem(t, s, tile, 0);
    in = t.in[s] + (e - a);
    out = t.out[s] + (e - a);
    quad = (uint64_t)(e >> 2);
    whole = e0 >= a && e0 + 4 * SEG_TILE <= b;
    fast_in = whole && (reinterpret_cast<uintptr_t>(in) & 15u) == 0;
    fast_out = whole && (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
    // only a tensor's first tile (when it starts inside a quad) and its last one are not whole
    const int64_t ahead = DIR > 0 ? (b - (e0 + 4 * SEG_TILE)) / (4 * SEG_TILE) : (e0 - (a + 3) / 4 * 4) / (4 * SEG_TILE);
    run = whole && ahead > 0 ? (int)ahead : 0;
  }
  // any other tile
  __device__ __forceinline__ void jump(const SegTable<CAP>& t, uint32_t to) {
    tile = to;
    s = seg_of_tile(t, tile);
    enter(t);
  }
  // N further tiles at once, all of them whole (N <= run)
  template <int N>
  __device__ __forceinline__ void skip() {
    tile += (uint32_t)(DIR * N);
    run -= N;
    in += DIR * N * 4 * SEG_TILE;
    out += DIR * N * 4 * SEG_TILE;
    quad += (uint64_t)((int64_t)DIR * N * SEG_TILE);
  }
  __device__ __forceinline__ void step(const SegTable<CAP>& t) {
    if (DIR < 0 && tile == 0) return;
    tile += (uint32_t)DIR;
    if (run > 0) {
      --run;
      in += DIR * 4 * SEG_TILE;
      out += DIR * 4 * SEG_TILE;
      quad += (uint64_t)((int64_t)DIR * SEG_TILE);
      return;
    }
    if (tile >= t.tile0[t.n]) return;
    if (DIR > 0) while (tile >= t.tile0[s + 1]) ++s;
    else while (tile < t.tile0[s]) --s;
    enter(t);
  }
  // Elements of this quad that belong to the tensor: [first, last) of 0 .. 4 (empty behind the tensor's end).
  __device__ __forceinline__ int first(const SegTable<CAP>& t) const {
    const int64_t d = t.start[s] - (int64_t)(quad * 4);
    return d > 0 ? (int)d : 0;
  }
  __device__ __forceinline__ int last(const SegTable<CAP>& t) const {
    const int64_t d = t.start[s + 1] - (int64_t)(quad * 4);
    return d > 4 ? 4 : (int)(d < 0 ? 0 : d);
  }
  __device__ __forceinline__ bool empty(const SegTable<CAP>& t) const { return !whole && last(t) == 0; }
  __device__ __forceinline__ float4 load(const SegTable<CAP>& t) const {
    if (fast_in) return __ldcg(reinterpret_cast<const float4*>(in));
    const int a = whole ? 0 : first(t), b = whole ? 4 : last(t);
    if (b - a == 4 && (reinterpret_cast<uintptr_t>(in) & 15u) == 0) return __ldcg(reinterpret_cast<const float4*>(in));
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    if (a <= 0 && b > 0) r.x = in[0];
    if (a <= 1 && b > 1) r.y = in[1];
    if (a <= 2 && b > 2) r.z = in[2];
    if (a <= 3 && b > 3) r.w = in[3];
    return r;
  }
  __device__ __forceinline__ void store(const SegTable<CAP>& t, const float4& r) const {
    if (fast_out) { __stcs(reinterpret_cast<float4*>(out), r); return; }
    const int a = whole ? 0 : first(t), b = whole ? 4 : last(t);
    if (b - a == 4 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) { __stcs(reinterpret_cast<float4*>(out), r); return; }
    if (a <= 0 && b > 0) out[0] = r.x;
    if (a <= 1 && b > 1) out[1] = r.y;
    if (a <= 2 && b > 2) out[2] = r.z;
    if (a <= 3 && b > 3) out[3] = r.w;
  }
};

// Fills a table; false when it cannot hold the segments or the tile count leaves 32 bits.
template <int CAP>
inline bool seg_table(SegTable<CAP>& t, const SegDesc* segs, int n_seg, int64_t n) {
  if (n_seg < 1 || n_seg > CAP) return false;
  int64_t tiles = 0;
  for (int i = 0; i < n_seg; ++i) {
    const int64_t lo = segs[i].start, hi = i + 1 < n_seg ? segs[i + 1].start : n;
    t.in[i] = segs[i].in;
    t.out[i] = segs[i].out;
    t.start[i] = lo;
    t.tile0[i] = (uint32_t)tiles;
    tiles += hi > lo ? ((hi + 3) / 4 - lo / 4 + SEG_TILE - 1) / SEG_TILE : 0;
    if (tiles > 0x7fffffff) return false;
  }
  t.start[n_seg] = n;
  t.tile0[n_seg] = (uint32_t)tiles;
  t.n = n_seg;
  return true;
}

}  // namespace gc
