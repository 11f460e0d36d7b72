// accel.h — device-resident MTBVH.
//
// HBM layout (GB300-first; the reference keeps bounds, hit table, indices and
// vertices as separate GL buffer textures, src/core/Scene.cpp:245-250):
//
//   node records  float4[6][M][2]   32-byte record per threaded-table entry,
//                                   in traversal order of its face:
//                                     [0] = pMin.xyz, prim (int bits, -1 = inner)
//                                     [1] = pMax.xyz, miss (int bits)
//                 Each face stores every node in its own visiting order, so the
//                 common step k -> k+1 reads the next 32 bytes (streaming,
//                 sector-aligned, two 16-byte read-only loads).
//   triangles     float4[ntri][3]   a.xyz ab.x | ab.yz ac.xy | ac.z, 0
//                                   (ab = b - a and ac = c - a evaluated on the
//                                   host in float32, exactly the values the
//                                   ray-triangle test forms, intersection.glsl:68-69)
//   dfs nodes     float4[M][2]      one record per node in DFS pre-order:
//                                     [0] = pMin.xyz, subtree size, or
//                                           prim | 0x80000000 at a leaf
//                                     [1] = pMax.xyz, leaves before the node
//                                           | 0x80000000 at odd depths
//   wide tree     uint32[ntri-1][16] two binary levels per 64-byte node: the
//                                   binary inner node of even depth with
//                                   DFS index k is wide node k - (leaves
//                                   before k), so no index has to be
//                                   allocated (odd-depth slots stay unused).
//                                   Children: both of the first binary child
//                                   (slots 0, 1), both of the second (2, 3);
//                                   a binary child that is a leaf sits in the
//                                   first slot of its pair.
//                                     [0..2] grid origin - 2^23 step, xyz
//                                            (floats)
//                                     [3]    float exponents of the grid
//                                            steps (x low byte, y, z) and of
//                                            the largest squared triangle box
//                                            diagonal below, rounded up
//                                     [4..7] child references: wide node,
//                                            ~leaf slot, or 0 (empty)
//                                     [8..13] lo.x hi.x lo.y hi.y lo.z hi.z
//                                            of the children in grid steps
//                                            from the origin, a byte each,
//                                            rounded outwards
//                                     [14]   3 bits per face: bit 0 / 1 the
//                                            first / second pair in reverse
//                                            order, bit 2 the second pair
//                                            first
//   wide tris     float4[ntri][4]   in DFS leaf order: a.xyz ab.x | ab.yz
//                                   ac.xy | ac.z prim box lo.xy | lo.z hi.xyz
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "bvh_build.h"

struct zgl_accel {
    int device = 0;
    int64_t ntri = 0;
    int64_t M = 0;
    zgl::HostBVH host;
    // device-built trees: the one allocation behind the arrays below
    void* d_arena = nullptr;
    float4* d_nodes = nullptr;  // 6*M*2
    float4* d_tris = nullptr;   // ntri*3
    // set when the tree was built on the device: an export makes the
    // PackedBVH from d_dfs and d_nodes, and `host` is empty.  In d_nodes of
    // such a tree the `prim` of an inner node is ~(its DFS number), any
    // negative number to the traversal.  (Hit tables written by the build
    // were 72 of the 300 B a node it wrote: build and release of 2M triangles
    // 5.0 -> 4.7 ms, of 8M 17.3 -> 16.1.)
    bool device_built = false;
    float4* d_dfs = nullptr;  // M*2
    // wide tree (ntri >= 2)
    float4* d_wide = nullptr;   // (ntri-1)*4
    float4* d_wtris = nullptr;  // ntri*4
    // work counter of the persistent trace kernels (reset before each launch;
    // launches of one handle are serialised on its caller's stream)
    unsigned long long* d_counter = nullptr;
    int trace_schedule = 0;  // ZGL_TRACE_*
    // staging for calls made with host arrays
    mutable void* d_stage = nullptr;
    mutable size_t stage_bytes = 0;
};

namespace zgl {

// Lays arrays out in one allocation: a first pass with base = null measures,
// a second one hands out the addresses.  A cudaMalloc costs 30-35 us and a
// cudaFree 15-35 us whatever the size is, on top of 0.7 ms per GB freed.
struct Arena {
    char* base = nullptr;
    size_t bytes = 0;
    template <class T>
    void take(T*& p, size_t n) {
        p = base ? reinterpret_cast<T*>(base + bytes) : nullptr;
        bytes += (n * sizeof(T) + 255) & ~size_t(255);
    }
};

struct DeviceAccel {
    const float4* nodes;
    const float4* tris;
    int32_t M;
    // wide tree; null where there is none (fewer than two triangles)
    const float4* wide = nullptr;
    const float4* wtris = nullptr;
    const float4* dfs = nullptr;
};

inline DeviceAccel device_view(const zgl_accel* a) {
    return DeviceAccel{a->d_nodes, a->d_tris, (int32_t)a->M, a->d_wide, a->d_wtris, a->d_dfs};
}

// Kernel launchers (accel.cu).  All pointers are device pointers.
cudaError_t launch_pack_nodes(const float* bounds, const int32_t* hit, int64_t M, float4* nodes,
                              cudaStream_t s);
// `schedule` is a ZGL_TRACE_* value; ZGL_TRACE_PERSISTENT needs `counter`, a
// device word it resets on the stream.
cudaError_t launch_trace_closest(DeviceAccel a, const float* org, const float* dir, int64_t n,
                                 int32_t* hit_id, float* hit_t, int schedule, unsigned long long* counter,
                                 cudaStream_t s);
cudaError_t launch_trace_any(DeviceAccel a, const float* org, const float* dir, const float* tmax,
                             int64_t n, uint8_t* occluded, int schedule, unsigned long long* counter,
                             cudaStream_t s);
cudaError_t launch_trace_count(DeviceAccel a, const float* org, const float* dir, const float* tmax,
                               int64_t n, int any_hit, int32_t* visits, int32_t* tests,
                               cudaStream_t s);

// Host build + upload (throws zgl::Error) and release of an accelerator.
zgl_accel* accel_create(const float* vertices, const uint32_t* indices, int64_t ntri);
// Device build (bvh_build_gpu.cu); inputs may be device, page-locked or
// pageable host arrays.  `small` = 0 selects the default subtree threshold.
zgl_accel* accel_create_device(const float* vertices, int64_t nv, const uint32_t* indices, int64_t ntri,
                               int small, cudaStream_t s);
// Fills d_nodes, d_tris, d_dfs and the wide tree.  Synchronous on `s`.
void build_bvh_device(const float* v, int64_t nv, const uint32_t* idx, int small, zgl_accel* a, cudaStream_t s);
// Wide tree of an accelerator from its dfs nodes (wide_build.cu) into d_wide
// and d_wtris, unless the device word `err` (may be null) is set.
// Asynchronous on `s`.
void build_wide(zgl_accel* a, const float* l2, const uint32_t* err, cudaStream_t s);
// dfs nodes of a host-built tree from its bounds, sizeIndices and HostWords.
cudaError_t launch_dfs_records(const float* bounds, const int32_t* sizes, const uint32_t* leaves, int64_t M,
                               float4* dfs, cudaStream_t s);
// PackedBVH of a device-built tree into host memory: bounds float[M*6], hit
// table int32[6*M*3].
void export_device_tree(const zgl_accel* a, float* bounds, int32_t* hit_table);
int gpu_build_default_small();
int gpu_build_max_small();
// Device address of p (itself for device/managed memory, the mapped address
// of page-locked host memory) or nullptr for pageable host memory; `host`
// tells whether p is host memory.
void* device_address(const void* p, bool& host);
void accel_free(zgl_accel* a);
int host_threads();

}  // namespace zgl
