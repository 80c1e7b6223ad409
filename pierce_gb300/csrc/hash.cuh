// Pair hash set and small device helpers shared by the join kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"

namespace pgpu {

__device__ __forceinline__ uint64_t fmix64(uint64_t k) {
    k ^= k >> 33;
    k *= 0xff51afd7ed558ccdULL;
    k ^= k >> 33;
    k *= 0xc4ceb9fe1a85ec53ULL;
    k ^= k >> 33;
    return k;
}

__device__ __forceinline__ uint64_t pack_key(int32_t a, int32_t b) {
    return ((uint64_t)(uint32_t)a << 32) | (uint64_t)(uint32_t)b;
}

// Insert; returns slot index or -1 when the probe bound is exhausted.
// `probes` accumulates the slots inspected (for contention statistics).
__device__ __forceinline__ int64_t hash_insert(uint64_t* table, uint64_t mask, uint64_t key, uint32_t* err,
                                               uint32_t& probes) {
    uint64_t h = fmix64(key) & mask;
    for (uint64_t i = 0; i <= mask; ++i) {
        ++probes;
        const uint64_t cur = __ldcg(table + h);
        if (cur == key) return (int64_t)h;
        if (cur == kEmptyKey) {
            const unsigned long long old =
                atomicCAS(reinterpret_cast<unsigned long long*>(table + h), (unsigned long long)kEmptyKey,
                          (unsigned long long)key);
            if (old == kEmptyKey || old == key) return (int64_t)h;
        }
        h = (h + 1) & mask;
    }
    atomicOr(err, ERR_HASH_FULL);
    return -1;
}

// Warp-aggregated counter flush: one atomicAdd per warp.
__device__ __forceinline__ void flush_counter(unsigned long long* dst, unsigned long long v) {
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xFFFFFFFFu, v, off);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(dst, v);
}

__device__ __forceinline__ bool box_overlap(float lx, float hx, float ly, float hy, float lz, float hz,
                                            const float3& lo, const float3& hi) {
    return lx <= hi.x && lo.x <= hx && ly <= hi.y && lo.y <= hy && lz <= hi.z && lo.z <= hz;
}

}  // namespace pgpu
