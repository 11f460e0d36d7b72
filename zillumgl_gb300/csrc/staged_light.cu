// staged_light.cu — light paths with ray casts and shading in separate
// kernels: the light tracer (lightIntegTrace, light_path_integ.glsl:45-146)
// and the light half of the triple integrator (traceLightPath,
// triple_path_pass_lpt.glsl:58-182), as staged.cu does for camera paths.
//
// A vertex's connection to the camera is shaded first and its visibility ray
// traced with the next step's rays; the film gets the contribution when
// nothing is in the way.  Connections that leave the film or carry nothing
// cast no ray.  200k triangles, depth 8: 49k light paths 1.78 -> 1.03 ms, 312k
// 4.46 -> 1.70 ms; the triple integrator's pass with 98k 4.25 -> 3.06 ms.
#include <algorithm>

#include "staged.cuh"
#include "zgl_internal.h"

namespace zgl {
namespace {

constexpr int kLightStartBlock = 256;
constexpr int kLightShadeBlock = 256;

struct LightChunk {
    uint32_t first, count;  // light paths [first, first + count) of the pass
    uint32_t seed;          // randSeed of path 0
    float scale;            // of a triple connection (uScale)
    float* film;
};

// A connection to the camera: where it lands and what it carries.
struct Splat {
    bool on;
    uint32_t pixel;
    v3 value, from, to;
};
// Film pixel of a camera connection, as accumulateFilm (render_kernels.cuh)
// rounds it; false where that drops it.
__device__ __forceinline__ bool film_pixel(const DeviceScene& sc, v2 uv, uint32_t& pixel) {
    if (!inFilmBound(uv)) return false;
    const int x = zf2i(uv.x * (float)sc.filmW), y = zf2i(uv.y * (float)sc.filmH);
    pixel = (uint32_t)y * (uint32_t)sc.filmW + (uint32_t)x;
    return x < sc.filmW && y < sc.filmH;
}
__device__ __forceinline__ void store_splat(const StagedLists& l, uint32_t i, const Splat& s) {
    // visible (intersection.glsl:429-433)
    const float dist = distance(s.from, s.to) - 2e-5f;
    const v3 wi = normalize(s.to - s.from);
    const v3 o = s.from + wi * 1e-5f;
    l.sorg[i] = make_float4(o.x, o.y, o.z, dist);
    l.sdir[i] = make_float4(wi.x, wi.y, wi.z, __uint_as_float(s.pixel));
    l.scon[i] = make_float4(s.value.x, s.value.y, s.value.z, 0.0f);
}

// A light path between two bounces.
struct LightState {
    Ray ray;
    v3 throughput;
    uint32_t seed;
    // triple: normal and pdf of the vertex left, running MIS ratios
    v3 prevNorm;
    float prevPdfDir, s0t1, s1t1;
};
template <bool TRIPLE>
__device__ __forceinline__ void store_light(const StagedLists& l, uint32_t i, const LightState& st) {
    l.org[i] = make_float4(st.ray.ori.x, st.ray.ori.y, st.ray.ori.z, 0.0f);
    l.dir[i] = make_float4(st.ray.dir.x, st.ray.dir.y, st.ray.dir.z, 0.0f);
    l.thr[i] = make_float4(st.throughput.x, st.throughput.y, st.throughput.z, __uint_as_float(st.seed));
    if (TRIPLE) {
        l.pos[i] = make_float4(st.prevNorm.x, st.prevNorm.y, st.prevNorm.z, st.prevPdfDir);
        l.rng[i] = make_uint2(__float_as_uint(st.s0t1), __float_as_uint(st.s1t1));
    }
}
__device__ __forceinline__ Sampler light_sampler(const DeviceScene& sc, uint32_t seed) {
    Sampler g;
    g.randSeed = seed;
    g.sampleSeed = 0;
    g.sampleOffset = 0;
    g.dim = 0;
    g.mode = 0;
    g.rowCache = nullptr;
    g.mats = sc.sobol;
    return g;
}

// Emission (lightIntegTrace / traceLightPath up to the bounce loop).
template <bool TRIPLE>
__global__ void __launch_bounds__(kLightStartBlock)
light_start_kernel(const __grid_constant__ DeviceScene sc, const LightChunk c, const __grid_constant__ StagedLists l,
                   uint32_t* counts) {
    __shared__ uint32_t sh[kLightStartBlock / 32];
    const uint32_t k = blockIdx.x * kLightStartBlock + threadIdx.x;
    const bool on = k < c.count;
    LightState st;
    Splat sp;
    sp.on = false;
    if (on) {
        Sampler g = light_sampler(sc, c.seed + c.first + k);
        const float a0 = rand01(g), a1 = rand01(g);
        const int light = lightSampleOne(sc, mk2(a0, a1));
        const float pdfSource = lightPdfSampleOne(sc, light);
        const int triId = light + sc.objPrimCount;
        if (TRIPLE) {
            rand01(g);  // the reference samples a point here and never uses it
            rand01(g);
        } else {
            const float b0 = rand01(g), b1 = rand01(g);
            const TriShade t = loadTri(sc, triId);
            const v3 pLit = sampleTriangleUniform(t.a, t.b, t.c, mk2(b0, b1));
            const float c0 = rand01(g), c1 = rand01(g);
            const CameraIiSample ci = thinLensCameraSampleIi(sc, pLit, mk2(c0, c1));
            if (ci.pdf > 0.0f && film_pixel(sc, ci.uv, sp.pixel)) {
                float area;
                lightPowerOf(sc, light, area);
                const float pdfPos = 1.0f / area;
                const v3 Le = lightLe(sc, light, pLit, ci.wi);
                sp.value = Le * ci.Ii / (ci.pdf * pdfPos * pdfSource);
                sp.from = pLit;
                sp.to = pLit + ci.wi * ci.dist;
                sp.on = !isBlack(sp.value);
            }
        }
        const float d0 = rand01(g), d1 = rand01(g), d2 = rand01(g), d3 = rand01(g);
        const LightLeSample le = lightSampleOneLe(sc, light, d0, d1, d2, d3);
        const v3 nl = geomNormal(sc, triId, le.ray.ori);
        const v3 wo = -le.ray.dir;
        st.ray = rayOffseted(le.ray.ori, le.ray.dir);
        st.throughput = le.Le * absDot(nl, -wo) / (pdfSource * le.pdfPos * le.pdfDir);
        if (TRIPLE) {
            st.prevNorm = nl;
            st.prevPdfDir = le.pdfDir;
            st.s0t1 = 1.0f / remap(le.pdfPos * pdfSource);
            st.s1t1 = 1.0f;
        }
        st.seed = g.randSeed;
    }
    const uint32_t at = block_append<kLightStartBlock>(on, counts, sh);
    if (on) store_light<TRIPLE>(l, at, st);
    if (!TRIPLE) {
        __syncthreads();
        const uint32_t sat = block_append<kLightStartBlock>(sp.on, counts + 1, sh);
        if (sp.on) store_splat(l, sat, sp);
    }
}

// One bounce (bounce >= 1) of every path of list `bounce - 1`.
template <bool FULL, bool TRIPLE>
__global__ void __launch_bounds__(kLightShadeBlock, 4)
light_step_kernel(const __grid_constant__ DeviceScene sc, const PathParams pp, const LightChunk c, int bounce,
                  const __grid_constant__ StagedLists in, const __grid_constant__ StagedLists next, uint32_t* counts) {
    __shared__ uint32_t sh[2][kLightShadeBlock / 32];
    __shared__ ShadeSort<kLightShadeBlock> sort;
    const uint32_t n = counts[kCountStride * (bounce - 1)];
    for (uint32_t base = blockIdx.x * kLightShadeBlock; base < n; base += gridDim.x * kLightShadeBlock) {
        const uint32_t j = base + threadIdx.x;
        const uint32_t i = base + (uint32_t)block_sort(j < n ? shade_class<FULL>(sc, in.hit[j].x) : 7, sort);
        bool on = i < n;
        LightState st;
        Splat sp;
        sp.on = false;
        int2 h = make_int2(-1, 0);
        if (on) {
            h = in.hit[i];
            on = h.x != -1 && h.x - sc.objPrimCount < 0;
        }
        if (on) {
            const float4 o = in.org[i], d = in.dir[i], t = in.thr[i];
            const Ray ray{mk3(o.x, o.y, o.z), mk3(d.x, d.y, d.z)};
            const float dist = __int_as_float(h.y);
            st.throughput = mk3(t.x, t.y, t.z);
            const v3 wo = -ray.dir;
            const v3 pos = rayPoint(ray, dist);
            Sampler g = light_sampler(sc, __float_as_uint(t.w));
            Surface surf;
            uint32_t matType;
            BSDFParam mp;
            shadeSurface<FULL>(sc, h.x, pos, wo, surf, matType, mp);
            if (TRIPLE) {
                const float4 p = in.pos[i];
                const uint2 m = in.rng[i];
                st.prevNorm = mk3(p.x, p.y, p.z);
                st.prevPdfDir = p.w;
                st.s0t1 = __uint_as_float(m.x);
                st.s1t1 = __uint_as_float(m.y);
                const float coefToPos = remap(st.prevPdfDir * absDot(surf.ns, wo));
                st.s0t1 /= coefToPos;
                st.s1t1 /= coefToPos / (bounce == 1 ? remap(dist * dist) : 1.0f);
            }
            {
                const float c0 = rand01(g), c1 = rand01(g);
                const CameraIiSample ci = thinLensCameraSampleIi(sc, pos, mk2(c0, c1));
                if (ci.pdf > 0.0f && film_pixel(sc, ci.uv, sp.pixel)) {
                    sp.from = pos;
                    sp.to = pos + ci.wi * ci.dist;
                    const v3 bsdf = materialBSDF<FULL>(matType, mp, wo, ci.wi, surf.ns, kImportance);
                    const float cosWi = satDot(surf.ng, ci.wi) * fabsf(dot(surf.ns, wo) / dot(surf.ng, wo));
                    v3 res = ci.Ii * bsdf * st.throughput * cosWi / ci.pdf;
                    if (TRIPLE) {
                        const float coefToSurf =
                            remap(thinLensCameraPdfIe(sc, Ray{sp.to, -ci.wi}).pdfDir * satDot(surf.ns, ci.wi));
                        const float coefToPrev =
                            remap(materialPdf<FULL>(matType, mp, ci.wi, wo, surf.ns) * absDot(st.prevNorm, wo));
                        const float coefDist = remap(ci.dist * ci.dist);
                        const float coef0 = coefToSurf * coefToPrev / coefDist;
                        const float coef1 = ((bounce == 1) ? 1.0f : coefToPrev) * coefToSurf / coefDist;
                        res = res * weightT1(st.s0t1 * coef0, st.s1t1 * coef1);
                    }
                    sp.on = !hasNan(res) && !zisnan(ci.pdf) && ci.pdf > 1e-8f && !isBlack(res);
                    sp.value = TRIPLE ? res * c.scale : res;
                }
            }
            const float b0 = rand01(g), b1 = rand01(g), b2 = rand01(g);
            const BSDFSample bs = materialSample<FULL>(matType, mp, surf.ns, wo, mk3(b0, b1, b2), g, kImportance);
            const v3 wi = bs.wi;
            const float bsdfPdf = bs.pdf;
            const bool deltaBsdf = (bs.flag == kSpecRefl || bs.flag == kSpecTrans);
            on = !(bsdfPdf < 1e-8f || zisnan(bsdfPdf)) && bounce < pp.maxDepth;
            if (on && pp.rr && bounce >= pp.rrStart) {
                const float continueProb = zmin(maxComponent(bs.bsdf / bsdfPdf), 1.0f);
                if (rand01(g) >= continueProb) on = false;
                else st.throughput = st.throughput / continueProb;
            }
            if (on) {
                if (TRIPLE) {
                    const float coefToPrev =
                        remap(materialPdf<FULL>(matType, mp, wi, wo, surf.ns) * absDot(st.prevNorm, wo));
                    st.s0t1 *= coefToPrev;
                    st.s1t1 *= (bounce == 1) ? 1.0f : coefToPrev;
                    st.prevPdfDir = materialPdf<FULL>(matType, mp, wo, wi, surf.ns);
                    st.prevNorm = surf.ns;
                }
                const float cosWi = deltaBsdf ? 1.0f : fabsf(dot(surf.ng, wi) * dot(surf.ns, wo) / dot(surf.ng, wo));
                st.throughput = st.throughput * (bs.bsdf * cosWi / bsdfPdf);
                st.ray = rayOffseted(pos, wi);
                st.seed = g.randSeed;
            }
        }
        const uint32_t at = block_append<kLightShadeBlock>(on, &counts[kCountStride * bounce], sh[0]);
        const uint32_t sat = block_append<kLightShadeBlock>(sp.on, &counts[kCountStride * bounce + 1], sh[1]);
        if (on) store_light<TRIPLE>(next, at, st);
        if (sp.on) store_splat(next, sat, sp);
    }
}

// The rays of one step: the live paths' first, then the connections'.
struct LightRays {
    static constexpr bool kClosest = true, kAny = true;
    const StagedLists* l;
    float* film;
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
        else l->scon[i - paths].w = __uint_as_float(kSetAside);
    }
    __device__ __forceinline__ bool marked(int i) const {
        return i < paths ? l->hit[i].x == -2 : __float_as_uint(l->scon[i - paths].w) == kSetAside;
    }
    __device__ __forceinline__ void store(int i, int id, float t) const {
        if (i < paths) {
            l->hit[i] = make_int2(id, __float_as_int(t));
        } else if (id < 0) {
            const float4 k = l->scon[i - paths];
            float* p = film + 3 * (size_t)__float_as_uint(l->sdir[i - paths].w);
            atomicAdd(p, k.x);
            atomicAdd(p + 1, k.y);
            atomicAdd(p + 2, k.z);
        }
    }
};

__global__ void __launch_bounds__(kWideBlock, kWideBlocksPerSM)
light_trace_kernel(const __grid_constant__ DeviceAccel a, float* film, int step, int sms,
                   const __grid_constant__ StagedLists l, const uint32_t* __restrict__ counts) {
    const int paths = (int)counts[kCountStride * step], shadows = (int)counts[kCountStride * step + 1];
    wide_trace(a, LightRays{&l, film, paths}, paths + shadows, wide_group(paths + shadows, sms));
}

template <bool FULL, bool TRIPLE>
cudaError_t launch(const StagedPool& pool, const StagedLightJob& job, cudaStream_t st) {
    const PathParams pp{job.maxDepth, job.rr, job.rrStart, 0, 0, 0.0f};
    const StagedLists lists[2] = {staged_list(pool, 0), staged_list(pool, 1)};
    const int sms = staged_sms();
    LightChunk c{0u, 0u, job.seed, job.scale, job.film};
    for (uint32_t at = 0; at < job.paths; at += c.count) {
        c.first = at;
        c.count = (uint32_t)std::min<int64_t>(job.paths - at, pool.paths);
        cudaError_t e = cudaMemsetAsync(pool.counts, 0, sizeof(uint32_t) * kCountStride * (job.maxDepth + 2), st);
        if (e != cudaSuccess) return e;
        light_start_kernel<TRIPLE><<<(c.count + kLightStartBlock - 1) / kLightStartBlock, kLightStartBlock, 0, st>>>(
            job.sc, c, lists[0], pool.counts);
        const unsigned blocks = std::min<unsigned>((c.count + kLightShadeBlock - 1) / kLightShadeBlock, sms * 8u);
        const unsigned rays = wide_blocks(2 * (int64_t)c.count, sms);
        for (int step = 0; step <= job.maxDepth; step++) {
            const StagedLists &in = lists[step & 1], &next = lists[(step & 1) ^ 1];
            // behind the last bounce only its connections are left
            light_trace_kernel<<<rays, kWideBlock, 0, st>>>(job.sc.accel, job.film, step, sms, in, pool.counts);
            if (step < job.maxDepth)
                light_step_kernel<FULL, TRIPLE><<<blocks, kLightShadeBlock, 0, st>>>(job.sc, pp, c, step + 1, in, next,
                                                                                     pool.counts);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace

cudaError_t launch_staged_light(const StagedPool& pool, const StagedLightJob& job, cudaStream_t st) {
    if (job.triple)
        return job.full ? launch<true, true>(pool, job, st) : launch<false, true>(pool, job, st);
    return job.full ? launch<true, false>(pool, job, st) : launch<false, false>(pool, job, st);
}

}  // namespace zgl
