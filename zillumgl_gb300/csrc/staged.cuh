// staged.cuh — device parts that the staged renderers share (staged.cu: path
// tracer; staged_light.cu: light paths): lists, block-wide append and the sort
// by what a path shades.
#pragma once

#include "path_trace.cuh"
#include "staged.h"
#include "wide.cuh"

namespace zgl {
namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kCountStride = 2;  // per step: paths, shadow rays
constexpr uint32_t kSetAside = 0x80000000u;

// What a launch needs of the pool: the list it reads and the one it writes.
struct StagedLists {
    float4 *org, *dir, *thr, *pos;
    uint2* rng;
    int2* hit;
    float4 *sorg, *sdir, *scon;
};
inline StagedLists staged_list(const StagedPool& p, int i) {
    return StagedLists{p.org[i], p.dir[i], p.thr[i], p.pos[i], p.rng[i], p.hit, p.sorg, p.sdir, p.scon};
}

// Position of this thread's entry in a list that `want` threads of the block
// append to; one atomic per block.  Every thread of the block calls.
template <int BLOCK>
__device__ __forceinline__ uint32_t block_append(bool want, uint32_t* counter, uint32_t* sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned m = __ballot_sync(kAll, want);
    if (lane == 0) sh[w] = (uint32_t)__popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t total = 0;
#pragma unroll
        for (int i = 0; i < BLOCK / 32; i++) {
            const uint32_t c = sh[i];
            sh[i] = total;
            total += c;
        }
        const uint32_t base = total ? atomicAdd(counter, total) : 0u;
#pragma unroll
        for (int i = 0; i < BLOCK / 32; i++) sh[i] += base;
    }
    __syncthreads();
    return sh[w] + (uint32_t)__popc(m & ((1u << lane) - 1u));
}

// What a path's shading runs: nothing but emission (0), the vertex's material
// type + 1, or no path (7).
template <bool FULL>
__device__ __forceinline__ int shade_class(const DeviceScene& sc, int id) {
    if (id < 0 || id >= sc.objPrimCount) return 0;
    const int matTex = __float_as_int(__ldg(reinterpret_cast<const float*>(sc.shade + 5 * (size_t)id + 4) + 2));
    const uint32_t type = loadMaterialType(sc, matTex & 0x0000ffff);
    return 1 + (int)min(type, FULL ? 5u : 1u);
}

// The block's paths in order of class, so that a warp's lanes shade alike:
// thread t takes path perm[t] of the block's window.  A counting sort with one
// ballot per class; every thread of the block calls.
template <int BLOCK>
struct ShadeSort {
    static_assert(BLOCK >= 128, "the scan reads a whole warp's number of counters");
    uint16_t perm[BLOCK];
    uint32_t count[8][BLOCK / 32];
};
template <int BLOCK>
__device__ __forceinline__ int block_sort(int cls, ShadeSort<BLOCK>& sh) {
    constexpr int kWarps = BLOCK / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned mine = 0u;
#pragma unroll
    for (int c = 0; c < 8; c++) {
        const unsigned m = __ballot_sync(kAll, cls == c);
        if (cls == c) mine = m;
        if (lane == c) sh.count[c][w] = (uint32_t)__popc(m);
    }
    __syncthreads();
    if (w == 0) {  // exclusive sums, class-major
        uint32_t v[(8 * kWarps + 31) / 32], total = 0;
        constexpr int kPer = (8 * kWarps + 31) / 32;
        uint32_t* flat = &sh.count[0][0];
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            v[k] = total;
            total += flat[lane * kPer + k];
        }
        uint32_t x = total;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kAll, x, d);
            if (lane >= d) x += y;
        }
#pragma unroll
        for (int k = 0; k < kPer; k++) flat[lane * kPer + k] = x - total + v[k];
    }
    __syncthreads();
    sh.perm[sh.count[cls][w] + (uint32_t)__popc(mine & ((1u << lane) - 1u))] = (uint16_t)threadIdx.x;
    __syncthreads();
    return sh.perm[threadIdx.x];
}

}  // namespace
}  // namespace zgl
