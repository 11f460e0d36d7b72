// wide_build.cu — the 4-wide tree of an accelerator (accel.h) from its binary
// tree in DFS order: one thread per binary node writes the wide node of an
// even-depth inner node or the triangle record of a leaf.  Every index follows
// from the DFS records, so there is no allocation of nodes, no second pass and
// no dependence between threads.
//
// Bound by memory: per triangle about 130 B of DFS records and 48 B of
// triangle in, 27 B of wide nodes (64 B per inner node of even depth) and 64 B
// of triangle record out.
#include <algorithm>
#include <cstring>
#include <vector>

#include "accel.h"
#include "zgl_internal.h"

namespace zgl {
namespace {

constexpr uint32_t kTop = 0x80000000u;

struct DfsNode {
    float4 a, b;
};
__device__ __forceinline__ bool is_leaf(const DfsNode& n) { return (__float_as_uint(n.a.w) & kTop) != 0u; }
__device__ __forceinline__ int64_t size_of(const DfsNode& n) { return is_leaf(n) ? 1 : (int64_t)__float_as_uint(n.a.w); }
__device__ __forceinline__ int32_t leaves_before(const DfsNode& n) { return (int32_t)(__float_as_uint(n.b.w) & ~kTop); }
// Reference of node k as a child of a wide node.
__device__ __forceinline__ int32_t child_ref(const DfsNode& n, int64_t k) {
    return is_leaf(n) ? ~leaves_before(n) : (int32_t)(k - leaves_before(n));
}
__device__ __forceinline__ DfsNode load_dfs(const float4* __restrict__ dfs, int64_t k) {
    return DfsNode{__ldg(dfs + 2 * k), __ldg(dfs + 2 * k + 1)};
}

// Bit f: face f visits `r` before `l` (buildHitTable's child order,
// BVH.cpp:298-345: by the centroid of the child boxes).
__device__ __forceinline__ uint32_t right_first(const DfsNode& l, const DfsNode& r) {
    const float lc[3] = {(l.a.x + l.b.x) * 0.5f, (l.a.y + l.b.y) * 0.5f, (l.a.z + l.b.z) * 0.5f};
    const float rc[3] = {(r.a.x + r.b.x) * 0.5f, (r.a.y + r.b.y) * 0.5f, (r.a.z + r.b.z) * 0.5f};
    uint32_t bits = 0u;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        if (!(lc[k] > rc[k])) bits |= 1u << (2 * k);
        if (!(lc[k] < rc[k])) bits |= 2u << (2 * k);
    }
    return bits;
}

// Grid of one axis of a node box: the step is a power of two of at least
// 1/250 of the extent and of 2^-22 of the coordinates, so that indices fit
// in a byte and every grid point, the shifted origin and the sums of the
// traversal's f * s + g are exact in float32.
struct Grid {
    float step, inv;
    float first;  // index of the grid origin, counted from coordinate 0
    uint32_t exponent;

    __device__ __forceinline__ Grid(float lo, float hi) {
        const float need = fmaxf((hi - lo) * (1.0f / 250.0f), fmaxf(fabsf(lo), fabsf(hi)) * 0x1p-22f);
        const int e = (int)(__float_as_uint(need) >> 23) + 1;
        exponent = (uint32_t)max(e, 30);
        step = __uint_as_float(exponent << 23);
        inv = __uint_as_float((254u - exponent) << 23);
        first = floorf(lo * inv);
    }
    __device__ __forceinline__ float origin() const { return (first - 8388608.0f) * step; }
    __device__ __forceinline__ uint32_t below(float x) const { return (uint32_t)(int)(floorf(x * inv) - first); }
    __device__ __forceinline__ uint32_t above(float x) const { return (uint32_t)(int)(ceilf(x * inv) - first); }
};

__global__ void __launch_bounds__(256)
wide_kernel(const float4* __restrict__ dfs, const float* __restrict__ l2, int64_t M,
            const float4* __restrict__ tris, const uint32_t* __restrict__ err, uint4* __restrict__ wide,
            float4* __restrict__ wtris) {
    if (err && *err) return;  // a failed build leaves records unwritten
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= M) return;
    const DfsNode n = load_dfs(dfs, k);
    if (is_leaf(n)) {
        const int64_t prim = (int64_t)(__float_as_uint(n.a.w) & ~kTop);
        const float4 t0 = __ldg(tris + 3 * prim), t1 = __ldg(tris + 3 * prim + 1), t2 = __ldg(tris + 3 * prim + 2);
        float4* o = wtris + 4 * (int64_t)leaves_before(n);
        o[0] = t0;
        o[1] = t1;
        o[2] = make_float4(t2.x, __int_as_float((int32_t)prim), n.a.x, n.a.y);
        o[3] = make_float4(n.a.z, n.b.x, n.b.y, n.b.z);
        return;
    }
    if (__float_as_uint(n.b.w) & kTop) return;  // odd depth: between two wide nodes
    const Grid gx(n.a.x, n.b.x), gy(n.a.y, n.b.y), gz(n.a.z, n.b.z);
    uint32_t plane[6] = {0u, 0u, 0u, 0u, 0u, 0u};
    uint32_t ref[4];
    uint32_t order[3];  // right_first of the pairs and of the two pairs
    DfsNode pair[2];
    int64_t at = k + 1;
#pragma unroll
    for (int g = 0; g < 2; g++) {
        pair[g] = load_dfs(dfs, at);
        DfsNode c[2] = {pair[g], pair[g]};
        const bool leaf = is_leaf(pair[g]);
        order[g] = 0u;
        ref[2 * g] = (uint32_t)child_ref(pair[g], at);
        ref[2 * g + 1] = 0u;
        if (!leaf) {
            c[0] = load_dfs(dfs, at + 1);
            const int64_t second = at + 1 + size_of(c[0]);
            c[1] = load_dfs(dfs, second);
            order[g] = right_first(c[0], c[1]);
            ref[2 * g] = (uint32_t)child_ref(c[0], at + 1);
            ref[2 * g + 1] = (uint32_t)child_ref(c[1], second);
        }
#pragma unroll
        for (int j = 0; j < 2; j++) {  // an empty slot repeats the leaf's box; its reference 0 says empty
            const int shift = 8 * (2 * g + j);
            plane[0] |= gx.below(c[j].a.x) << shift;
            plane[1] |= gx.above(c[j].b.x) << shift;
            plane[2] |= gy.below(c[j].a.y) << shift;
            plane[3] |= gy.above(c[j].b.y) << shift;
            plane[4] |= gz.below(c[j].a.z) << shift;
            plane[5] |= gz.above(c[j].b.z) << shift;
        }
        at += size_of(pair[g]);
    }
    order[2] = right_first(pair[0], pair[1]);
    uint32_t swaps = 0u;
#pragma unroll
    for (int f = 0; f < 6; f++)
        swaps |= ((order[0] >> f & 1u) | (order[1] >> f & 1u) << 1 | (order[2] >> f & 1u) << 2) << (3 * f);
    const uint32_t el = min((__float_as_uint(l2[k]) >> 23) + 1u, 254u);  // rounded up to a power of two
    uint4* o = wide + 4 * (k - leaves_before(n));
    o[0] = make_uint4(__float_as_uint(gx.origin()), __float_as_uint(gy.origin()), __float_as_uint(gz.origin()),
                      gx.exponent | gy.exponent << 8 | gz.exponent << 16 | el << 24);
    o[1] = make_uint4(ref[0], ref[1], ref[2], ref[3]);
    o[2] = make_uint4(plane[0], plane[1], plane[2], plane[3]);
    o[3] = make_uint4(plane[4], plane[5], swaps, 0u);
}

// DFS records of a host-built tree.
__global__ void dfs_records_kernel(const float* __restrict__ bounds, const int32_t* __restrict__ sizes,
                                   const uint32_t* __restrict__ leaves, int64_t M, float4* __restrict__ dfs) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= M) return;
    const float* b = bounds + 6 * i;
    dfs[2 * i] = make_float4(b[0], b[1], b[2], __int_as_float(sizes[i]));
    dfs[2 * i + 1] = make_float4(b[3], b[4], b[5], __uint_as_float(leaves[i]));
}

__global__ void bounds_kernel(const float4* __restrict__ dfs, int64_t first, int64_t n, float* __restrict__ out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 a = dfs[2 * (first + i)], b = dfs[2 * (first + i) + 1];
    float* o = out + 6 * i;
    o[0] = a.x; o[1] = a.y; o[2] = a.z;
    o[3] = b.x; o[4] = b.y; o[5] = b.z;
}

// DFS number of every triangle's leaf.
__global__ void leaf_numbers_kernel(const float4* __restrict__ dfs, int64_t M, int32_t* __restrict__ number) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= M) return;
    const uint32_t w = __float_as_uint(dfs[2 * i].w);
    if (w & kTop) number[w & ~kTop] = (int32_t)i;
}

// Hit table entries (node, prim, miss) [first, first + n) of the six faces.
__global__ void hits_kernel(const float4* __restrict__ nodes, const int32_t* __restrict__ number, int64_t first,
                            int64_t n, int32_t* __restrict__ out) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t prim = __float_as_int(nodes[2 * (first + i)].w);
    out[3 * i + 0] = prim < 0 ? ~prim : number[prim];
    out[3 * i + 1] = prim < 0 ? -1 : prim;
    out[3 * i + 2] = __float_as_int(nodes[2 * (first + i) + 1].w);
}

}  // namespace

void build_wide(zgl_accel* a, const float* l2, const uint32_t* err, cudaStream_t s) {
    wide_kernel<<<(unsigned)((a->M + 255) / 256), 256, 0, s>>>(a->d_dfs, l2, a->M, a->d_tris, err,
                                                               reinterpret_cast<uint4*>(a->d_wide), a->d_wtris);
    ZGL_CUDA(cudaGetLastError());
}

cudaError_t launch_dfs_records(const float* bounds, const int32_t* sizes, const uint32_t* leaves, int64_t M,
                               float4* dfs, cudaStream_t s) {
    dfs_records_kernel<<<(unsigned)((M + 255) / 256), 256, 0, s>>>(bounds, sizes, leaves, M, dfs);
    return cudaGetLastError();
}

namespace {

// Up to this many nodes an export copies the records and rearranges them on
// the host (100 triangles 28 us, with kernels and their memory 37; 1024
// triangles 79 and 40). It is also how a larger tree is exported without
// device memory to spare.
constexpr int64_t kHostExportNodes = 256;

void export_on_host(const zgl_accel* a, float* bounds, int32_t* hit_table) {
    const int64_t M = a->M, total = 6 * M, chunk = std::min<int64_t>(total, 1 << 16);
    std::vector<float4> rec(2 * (size_t)chunk);
    std::vector<int32_t> number((size_t)a->ntri);  // DFS number of every triangle's leaf
    auto bits = [](float f) {
        uint32_t u;
        std::memcpy(&u, &f, 4);
        return u;
    };
    for (int64_t at = 0; at < M; at += chunk) {
        const int64_t n = std::min(chunk, M - at);
        ZGL_CUDA(cudaMemcpy(rec.data(), a->d_dfs + 2 * at, sizeof(float4) * 2 * n, cudaMemcpyDeviceToHost));
        for (int64_t i = 0; i < n; i++) {
            const float4 lo = rec[2 * i], hi = rec[2 * i + 1];
            float* b = bounds + 6 * (at + i);
            b[0] = lo.x; b[1] = lo.y; b[2] = lo.z;
            b[3] = hi.x; b[4] = hi.y; b[5] = hi.z;
            if (bits(lo.w) & kTop) number[bits(lo.w) & ~kTop] = (int32_t)(at + i);
        }
    }
    for (int64_t at = 0; at < total; at += chunk) {
        const int64_t n = std::min(chunk, total - at);
        ZGL_CUDA(cudaMemcpy(rec.data(), a->d_nodes + 2 * at, sizeof(float4) * 2 * n, cudaMemcpyDeviceToHost));
        for (int64_t i = 0; i < n; i++) {
            const int32_t prim = (int32_t)bits(rec[2 * i].w);
            int32_t* h = hit_table + 3 * (at + i);
            h[0] = prim < 0 ? ~prim : number[(size_t)prim];
            h[1] = prim < 0 ? -1 : prim;
            h[2] = (int32_t)bits(rec[2 * i + 1].w);
        }
    }
}

}  // namespace

void export_device_tree(const zgl_accel* a, float* bounds, int32_t* hit_table) {
    if (a->M <= kHostExportNodes) return export_on_host(a, bounds, hit_table);
    // One copy per array where the memory is there: copies of 50 to 100 MB into
    // pages that the caller has not touched run at 1 to 5 GB/s, one of 600 MB
    // at 26 (4M triangles: 484 ms in copies of 48 MB, 31 ms in two).
    const int64_t M = a->M, total = 6 * M;
    int64_t chunk = total;
    auto grid = [](int64_t n) { return (unsigned)((n + 255) / 256); };
    void* p = nullptr;
    float* tmp = nullptr;
    int32_t* number = nullptr;
    Arena arena;
    auto lay = [&] {
        arena.bytes = 0;
        arena.take(tmp, 3 * chunk);
        arena.take(number, a->ntri);
    };
    lay();
    while (cudaMalloc(&p, arena.bytes) != cudaSuccess) {
        cudaGetLastError();
        if (chunk <= 1 << 20) return export_on_host(a, bounds, hit_table);
        chunk = std::max<int64_t>(chunk / 4, 1 << 20);
        lay();
    }
    arena.base = static_cast<char*>(p);
    lay();
    leaf_numbers_kernel<<<grid(M), 256>>>(a->d_dfs, M, number);
    cudaError_t e = cudaGetLastError();
    for (int64_t at = 0; at < M && e == cudaSuccess; at += chunk / 2) {  // half as many: 6 words each
        const int64_t n = std::min(chunk / 2, M - at);
        bounds_kernel<<<grid(n), 256>>>(a->d_dfs, at, n, tmp);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpy(bounds + 6 * at, tmp, sizeof(float) * 6 * n, cudaMemcpyDeviceToHost);
    }
    for (int64_t at = 0; at < total && e == cudaSuccess; at += chunk) {
        const int64_t n = std::min(chunk, total - at);
        int32_t* out = reinterpret_cast<int32_t*>(tmp);
        hits_kernel<<<grid(n), 256>>>(a->d_nodes, number, at, n, out);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpy(hit_table + 3 * at, out, sizeof(int32_t) * 3 * n, cudaMemcpyDeviceToHost);
    }
    cudaFree(p);
    ZGL_CUDA(e);
}

}  // namespace zgl
