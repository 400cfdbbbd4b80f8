// Entry points of the single-worker reducers (gc_solo.cu).  `segs`: n_seg SegDesc (gc_segs.cuh) of n elements in all.
#pragma once
#include <stdint.h>

#include "gc_segs.cuh"

extern "C" {
int gc_solo_max_segs();
int gc_solo_maxnorm(void* ctx, const void* segs, int n_seg, int64_t n, int bits_lo, int bits_hi, uint64_t seed, uint32_t step, int timeout_ms,
                    int max_blocks, void* cs);
int64_t gc_solo_randk_limit(void* ctx, int max_blocks);
int gc_solo_randk(void* ctx, const void* segs, int n_seg, int64_t n, uint64_t index_seed, uint32_t npass, int64_t start, int64_t k, int64_t* window,
                  int bits_lo, int bits_hi, int zero, uint32_t step, int timeout_ms, int max_blocks, void* cs);
int gc_solo_copy(void* ctx, const void* segs, int n_seg, int64_t n, void* cs);
}
