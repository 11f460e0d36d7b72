// staged.cu — the MIS path tracer with ray casts and shading in separate
// kernels.
//
// One kernel per path (path_trace.cuh) holds camera, traversal, surface,
// material, light and environment code at once: it is bound by instruction
// fetch (24 stall cycles per issued instruction on the city pass), with 6 to
// 10 of 32 lanes active.  Here every bounce is two launches over dense lists:
//
//   trace   closest hits of the live paths' rays and any hits of the shadow
//           rays that the last shading left, one sequence, on the wide tree
//           with its lane refill (wide.cuh);
//   shade   one step of every path (path_step.cuh): emission and MIS of what
//           the ray hit, Russian roulette, the new vertex's light sample
//           (shadow ray and contribution to a list) and BSDF sample (next
//           ray); paths that go on are appended to the other list.
//
// A path's radiance lives in the output array.  The trace adds a light
// sample's contribution when nothing blocks it, the next shading adds what
// the path's ray hits: the order of the additions, and with it every bit of
// the sum, is that of the one-kernel path tracer.  Lists are appended with one
// atomic per block; their order changes no value.
#include <algorithm>
#include <atomic>

#include "path_step.cuh"
#include "staged.cuh"
#include "zgl_internal.h"

namespace zgl {
namespace {

// Threads of a shading block: its paths are sorted by what they shade, so a
// larger block has more uniform warps (sphere scene, 2M paths: 128 threads 714
// us unsorted, 512 sorted 376 us, 12.6 -> 25.2 lanes and 8.2 -> 1.6
// instruction-fetch stalls per issue).  Scenes with every material type gain
// from 1024 once there are blocks enough (0.75M paths, five bounces: 3.14 ->
// 2.85 ms).  Two blocks of 512: 64 registers; one or three are slower.
constexpr int kShadeBlock = 512;
constexpr int kShadeBlockLarge = 1024;
constexpr int64_t kLargePaths = 512 * 1024;
// Fewer paths than four blocks of 128 per SM are shaded by such blocks, on
// every SM and with 128 registers: a Cornell pass of 65k paths 424 -> 406 us,
// of 9k paths 340 -> 315 us.  64 registers in blocks
// of 256: 409.
constexpr int kShadeBlockSmall = 128;
constexpr int kShadeSmallPerSM = 4;
constexpr int kStartBlock = 256;

// Items of a chunk: paths [q0, q0 + count) of the job, counted over samples
// and 8x4 pixel tiles (a warp's camera rays are neighbours); items outside the
// film are skipped.
struct StagedChunk {
    int64_t q0, count;
    int32_t row0;  // sample of the pool's first Sobol row
    int32_t tilesX;
    int64_t perSample;
    int64_t npix;
    int32_t first, n, counter0;
    float* out;
    int2* hits;
    int32_t castDepth;
    uint32_t* vis;
    const uint32_t* rows;
};

__device__ __forceinline__ void store_path(const StagedLists& l, uint32_t i, const PathState& st, const Sampler& g,
                                           uint32_t path, uint32_t casts) {
    l.org[i] = make_float4(st.ray.ori.x, st.ray.ori.y, st.ray.ori.z, st.bsdfPdf);
    l.dir[i] = make_float4(st.ray.dir.x, st.ray.dir.y, st.ray.dir.z, maxComponent(st.bsdfOverPdf));
    l.thr[i] = make_float4(st.throughput.x, st.throughput.y, st.throughput.z, __uint_as_float(path));
    l.pos[i] = make_float4(st.pos.x, st.pos.y, st.pos.z,
                           __uint_as_float((uint32_t)g.dim | (st.delta ? 0x10000u : 0u) | casts << 17));
    l.rng[i] = make_uint2(g.randSeed, g.sampleSeed);
}

// Sobol rows of the chunk's samples, one block each.
__global__ void staged_rows_kernel(const uint32_t* __restrict__ mats, int32_t row0, uint32_t* __restrict__ rows) {
    const uint32_t off = sample_offset(row0 + (int32_t)blockIdx.x);
    rows[256 * blockIdx.x + threadIdx.x] = sobol_value(mats, off >> 8, threadIdx.x);
}

__global__ void __launch_bounds__(kStartBlock)
staged_start_kernel(const DeviceScene sc, const StagedChunk c, const StagedLists l, uint32_t* counts) {
    __shared__ uint32_t sh[kStartBlock / 32];
    const int64_t k = blockIdx.x * (int64_t)kStartBlock + threadIdx.x;
    const int64_t q = c.q0 + k;
    const int32_t s = (int32_t)(q / c.perSample);
    const int64_t in = q - s * c.perSample;
    const int64_t tile = in >> 5;
    const int px = (int)(tile % c.tilesX) * 8 + ((int)in & 7), py = (int)(tile / c.tilesX) * 4 + (((int)in >> 3) & 3);
    const bool live = k < c.count && px < sc.filmW && py < sc.filmH;
    const uint32_t i = block_append<kStartBlock>(live, counts, sh);
    if (!live) return;
    const int64_t pix = (int64_t)py * sc.filmW + px;
    const uint2 seed = __ldg(&sc.pixelSeeds[pix]);
    Sampler g;
    g.randSeed = seed.x * (uint32_t)(c.first + s + c.counter0) + seed.y;
    g.sampleSeed = seed.x * seed.y;
    g.sampleOffset = sample_offset(c.first + s);
    g.dim = 0;
    g.mode = sc.sampler;
    g.rowCache = c.rows + 256 * (c.first + s - c.row0);
    g.mats = sc.sobol;
    const v2 scr = mk2((float)px, (float)py) / mk2((float)sc.filmW, (float)sc.filmH);
    const float u0 = sample1D(g), u1 = sample1D(g), u2 = sample1D(g), u3 = sample1D(g);
    PathState st;
    st.ray = thinLensCameraSampleRay(sc, scr, u0, u1, u2, u3);
    st.throughput = mk3(1.0f);
    st.pos = mk3(0.0f);
    st.bsdfOverPdf = mk3(0.0f);
    st.bsdfPdf = 0.0f;
    st.delta = false;
    store_path(l, i, st, g, (uint32_t)k, 0u);
    const int64_t path = (int64_t)s * c.npix + pix;
    float* o = c.out + 3 * path;
    o[0] = o[1] = o[2] = 0.0f;
    if (c.vis) c.vis[path] = 0u;
}

// Output index of the path of chunk item k.
__device__ __forceinline__ int64_t path_index(const DeviceScene& sc, const StagedChunk& c, uint32_t k, int32_t& s) {
    const int64_t q = c.q0 + k;
    s = (int32_t)(q / c.perSample);
    const int64_t in = q - s * c.perSample;
    const int64_t tile = in >> 5;
    const int px = (int)(tile % c.tilesX) * 8 + ((int)in & 7), py = (int)(tile / c.tilesX) * 4 + (((int)in >> 3) & 3);
    return (int64_t)s * c.npix + (int64_t)py * sc.filmW + px;
}

// One step of every path of the list: step 0 takes the camera rays' hits.
template <bool FULL, int BLOCK>
__global__ void __launch_bounds__(BLOCK, BLOCK == kShadeBlockSmall ? kShadeSmallPerSM : 1024 / BLOCK)
staged_shade_kernel(const __grid_constant__ DeviceScene sc, const __grid_constant__ StagedChunk c, const PathParams pp,
                    int step, const __grid_constant__ StagedLists in, const __grid_constant__ StagedLists next,
                    uint32_t* counts) {
    __shared__ uint32_t sh[2][BLOCK / 32];
    __shared__ ShadeSort<BLOCK> sort;
    const uint32_t n = counts[kCountStride * step];
    for (uint32_t base = blockIdx.x * BLOCK; base < n; base += gridDim.x * BLOCK) {
        const uint32_t j = base + threadIdx.x;
        const uint32_t i = base + (uint32_t)block_sort(j < n ? shade_class<FULL>(sc, in.hit[j].x) : 7, sort);
        bool on = i < n;
        PathState st;
        Sampler g;
        PendingShadow ps;
        ps.pending = ps.asked = false;
        uint32_t path = 0, casts = 0;
        int64_t slot = 0;
        if (on) {
            const float4 o = in.org[i], d = in.dir[i], t = in.thr[i], p = in.pos[i];
            const uint2 r = in.rng[i];
            const int2 h = in.hit[i];
            path = __float_as_uint(t.w);
            const uint32_t bits = __float_as_uint(p.w);
            int32_t s;
            slot = path_index(sc, c, path, s);
            st.ray = Ray{mk3(o.x, o.y, o.z), mk3(d.x, d.y, d.z)};
            st.bsdfPdf = o.w;
            st.bsdfOverPdf = mk3(d.w);  // only its largest component is used
            st.throughput = mk3(t.x, t.y, t.z);
            st.pos = mk3(p.x, p.y, p.z);
            st.delta = (bits & 0x10000u) != 0u;
            casts = bits >> 17;
            st.bounce = step;
            g.randSeed = r.x;
            g.sampleSeed = r.y;
            g.dim = (int)(bits & 0xffffu);
            g.sampleOffset = sample_offset(c.first + s);
            g.mode = sc.sampler;
            g.rowCache = c.rows + 256 * (c.first + s - c.row0);
            g.mats = sc.sobol;
            if (c.hits && step < c.castDepth)
                c.hits[((int64_t)step * c.n) * c.npix + slot] = h;
            float* out = c.out + 3 * slot;
            st.result = mk3(out[0], out[1], out[2]);
            const v3 before = st.result;
            on = path_step_hit<FULL, true>(sc, pp, g, st, h.x, __int_as_float(h.y), &ps);
            if (!on && !(st.result.x == before.x && st.result.y == before.y && st.result.z == before.z)) {
                out[0] = st.result.x;
                out[1] = st.result.y;
                out[2] = st.result.z;
            }
        }
        const bool shadow = ps.pending;
        const uint32_t at = block_append<BLOCK>(on, &counts[kCountStride * (step + 1)], sh[0]);
        const uint32_t sat = block_append<BLOCK>(shadow, &counts[kCountStride * (step + 1) + 1], sh[1]);
        if (shadow) {
            next.sorg[sat] = make_float4(ps.o.x, ps.o.y, ps.o.z, ps.tmax);
            next.sdir[sat] = make_float4(ps.d.x, ps.d.y, ps.d.z, __uint_as_float(path));
            next.scon[sat] = make_float4(ps.C.x, ps.C.y, ps.C.z, __uint_as_float(casts));
        }
        if (ps.asked && casts < 32u) casts++;
        if (on) store_path(next, at, st, g, path, casts);
    }
}

// The rays of one step: the live paths' first, then the shadow rays.
struct StagedRays {
    static constexpr bool kClosest = true, kAny = true;
    const DeviceScene* sc;
    const StagedChunk* c;
    const StagedLists* l;
    int paths;
    __device__ __forceinline__ bool any(int i) const { return i >= paths; }
    __device__ __forceinline__ float3 origin(int i) const {
        const float4 v = i < paths ? l->org[i] : l->sorg[i - paths];
        return make_float3(v.x, v.y, v.z);
    }
    __device__ __forceinline__ float3 direction(int i) const {
        const float4 v = i < paths ? l->dir[i] : l->sdir[i - paths];
        return make_float3(v.x, v.y, v.z);
    }
    __device__ __forceinline__ float limit(int i) const { return i < paths ? 1e8f : l->sorg[i - paths].w; }
    __device__ __forceinline__ void mark(int i) const {
        if (i < paths) l->hit[i].x = -2;
        else l->scon[i - paths].w = __uint_as_float(__float_as_uint(l->scon[i - paths].w) | kSetAside);
    }
    __device__ __forceinline__ bool marked(int i) const {
        return i < paths ? l->hit[i].x == -2 : (__float_as_uint(l->scon[i - paths].w) & kSetAside) != 0u;
    }
    __device__ __forceinline__ void store(int i, int id, float t) const {
        if (i < paths) {
            l->hit[i] = make_int2(id, __float_as_int(t));
            return;
        }
        const float4 k = l->scon[i - paths];
        int32_t s;
        const int64_t slot = path_index(*sc, *c, __float_as_uint(l->sdir[i - paths].w), s);
        if (id < 0) {  // visible: the light sample counts
            float* out = c->out + 3 * slot;
            out[0] = out[0] + k.x;
            out[1] = out[1] + k.y;
            out[2] = out[2] + k.z;
        } else if (c->vis) {
            const uint32_t n = __float_as_uint(k.w) & ~kSetAside;
            if (n < 32u) c->vis[slot] |= 1u << n;
        }
    }
};

__global__ void __launch_bounds__(kWideBlock, kWideBlocksPerSM)
staged_trace_kernel(const __grid_constant__ DeviceScene sc, const __grid_constant__ StagedChunk c, int step, int sms,
                    const __grid_constant__ StagedLists l, const uint32_t* __restrict__ counts) {
    const int paths = (int)counts[kCountStride * step], shadows = (int)counts[kCountStride * step + 1];
    wide_trace(sc.accel, StagedRays{&sc, &c, &l, paths}, paths + shadows, wide_group(paths + shadows, sms));
}

}  // namespace

int staged_sms() {
    static std::atomic<int> cache[64];
    int dev = 0, k = 0;
    cudaGetDevice(&dev);
    const bool cached = dev >= 0 && dev < 64;
    if (cached) k = cache[dev].load(std::memory_order_relaxed);
    if (k == 0) {
        cudaDeviceGetAttribute(&k, cudaDevAttrMultiProcessorCount, dev);
        if (k <= 0) k = 1;
        if (cached) cache[dev].store(k, std::memory_order_relaxed);
    }
    return k;
}

cudaError_t launch_staged_rows(const StagedPool& pool, const uint32_t* mats, int32_t row0, int32_t n,
                               cudaStream_t st) {
    staged_rows_kernel<<<n, 256, 0, st>>>(mats, row0, pool.rows);
    return cudaGetLastError();
}

bool staged_alloc(StagedPool& pool, int64_t total) {
    const int64_t n = std::max<int64_t>(1, std::min(total, kStagedPaths));
    StagedPool p;
    Arena a;
    for (int pass = 0; pass < 2; pass++) {
        a.bytes = 0;
        for (int i = 0; i < 2; i++) {
            a.take(p.org[i], n);
            a.take(p.dir[i], n);
            a.take(p.thr[i], n);
            a.take(p.pos[i], n);
            a.take(p.rng[i], n);
        }
        a.take(p.hit, n);
        a.take(p.sorg, n);
        a.take(p.sdir, n);
        a.take(p.scon, n);
        a.take(p.counts, kCountStride * (kStagedMaxDepth + 3));
        a.take(p.rows, 256 * kStagedRows);
        if (pass == 0) {
            if (cudaMalloc(&p.arena, a.bytes) != cudaSuccess) {
                cudaGetLastError();
                return false;
            }
            a.base = static_cast<char*>(p.arena);
        }
    }
    p.paths = n;
    p.turns = pool.turns;
    if (!p.turns) {
        p.turns = new StagedTurns();
        if (cudaEventCreateWithFlags(&p.turns->done, cudaEventDisableTiming) != cudaSuccess) {
            cudaGetLastError();
            p.turns->done = nullptr;
            staged_free(p);
            return false;
        }
    }
    staged_release(pool, pool.arena);
    pool = p;
    return true;
}

void staged_release(const StagedPool& p, void* memory) {
    if (!memory) return;
    if (p.turns && p.turns->captured) p.turns->retired.push_back(memory);
    else cudaFree(memory);
}

cudaError_t staged_malloc_beside(StagedPool& p, void** memory, size_t bytes) {
    cudaError_t e = cudaMalloc(memory, bytes);
    if (e != cudaErrorMemoryAllocation || !p.arena) return e;
    cudaGetLastError();
    staged_release(p, p.arena);
    p.arena = nullptr;
    p.paths = 0;
    return cudaMalloc(memory, bytes);
}

void staged_free(StagedPool& p) {
    if (p.arena) cudaFree(p.arena);
    if (p.turns) {
        if (p.turns->done) cudaEventDestroy(p.turns->done);
        for (void* m : p.turns->retired) cudaFree(m);
        delete p.turns;
    }
    p = StagedPool{};
}

StagedTurn::StagedTurn(const StagedPool& pool, cudaStream_t st) : t_(pool.turns), st_(st), lock_(pool.turns->mutex) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &status) != cudaSuccess) cudaGetLastError();  // the launches will say what is wrong
    captured_ = status == cudaStreamCaptureStatusActive;
    t_->captured = t_->captured || captured_;
    ZGL_CUDA(cudaStreamWaitEvent(st, t_->done, captured_ ? cudaEventWaitExternal : cudaEventWaitDefault));
}

StagedTurn::~StagedTurn() {
    cudaEventRecordWithFlags(t_->done, st_, captured_ ? cudaEventRecordExternal : cudaEventRecordDefault);
}

cudaError_t launch_staged(const StagedPool& pool, const StagedJob& job, cudaStream_t st) {
    const PathParams pp{job.maxDepth, job.rr, job.rrStart, job.sampleLight, job.uniformSel, job.portion};
    const int sms = staged_sms();
    StagedChunk c{};
    c.tilesX = (job.sc.filmW + 7) / 8;
    c.perSample = staged_paths(job.sc.filmW, job.sc.filmH, 1);
    c.npix = (int64_t)job.sc.filmW * job.sc.filmH;
    c.first = job.first;
    c.n = job.n;
    c.counter0 = job.counter0;
    c.out = job.out;
    c.hits = job.hits;
    c.castDepth = job.castDepth;
    c.vis = job.vis;
    c.rows = pool.rows;
    const StagedLists lists[2] = {staged_list(pool, 0), staged_list(pool, 1)};
    const int64_t total = c.perSample * job.n;
    for (c.q0 = 0; c.q0 < total; c.q0 += c.count) {
        c.count = std::min(total - c.q0, pool.paths);
        // whole samples up to the Sobol table's rows
        const int64_t s0 = c.q0 / c.perSample;
        c.count = std::min(c.count, (s0 + kStagedRows) * c.perSample - c.q0);
        c.row0 = job.first + (int32_t)s0;
        const int nrows = (int)((c.q0 + c.count - 1) / c.perSample - s0) + 1;
        cudaError_t e = cudaMemsetAsync(pool.counts, 0, sizeof(uint32_t) * kCountStride * (job.maxDepth + 3), st);
        if (e != cudaSuccess) return e;
        if (job.sc.sampler == 1) staged_rows_kernel<<<nrows, 256, 0, st>>>(job.sc.sobol, c.row0, pool.rows);
        staged_start_kernel<<<(unsigned)((c.count + kStartBlock - 1) / kStartBlock), kStartBlock, 0, st>>>(
            job.sc, c, lists[0], pool.counts);
        const bool large = job.full && c.count >= kLargePaths;
        const bool few = c.count <= (int64_t)sms * kShadeSmallPerSM * kShadeBlockSmall;
        const int block = few ? kShadeBlockSmall : large ? kShadeBlockLarge : kShadeBlock;
        // two rounds of resident blocks; each strides over the list
        const unsigned shade =
            (unsigned)std::min<int64_t>((c.count + block - 1) / block, (int64_t)sms * (1024 / block) * 2);
        const auto shading = few ? (job.full ? staged_shade_kernel<true, kShadeBlockSmall>
                                             : staged_shade_kernel<false, kShadeBlockSmall>)
                             : large    ? staged_shade_kernel<true, kShadeBlockLarge>
                             : job.full ? staged_shade_kernel<true, kShadeBlock>
                                        : staged_shade_kernel<false, kShadeBlock>;
        for (int step = 0; step <= job.maxDepth; step++) {
            const StagedLists &in = lists[step & 1], &next = lists[(step & 1) ^ 1];
            staged_trace_kernel<<<wide_blocks(2 * c.count, sms), kWideBlock, 0, st>>>(job.sc, c, step, sms, in,
                                                                                      pool.counts);
            shading<<<shade, block, 0, st>>>(job.sc, c, pp, step, in, next, pool.counts);
        }
        e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace zgl
