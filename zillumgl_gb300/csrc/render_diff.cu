// render_diff.cu — differentiable path tracing by path replay.
//
// Forward: every (pixel, sample) path of the MIS path tracer
// (pathIntegTrace, path_integ_naive.glsl:35-143, with the plain integrator's
// seeds: sample s uses freeCounter = s + 1) is traced once; its radiance is
// kept per sample and the image is the per-pixel sum over samples in sample
// order divided by spp.
//
// Backward (Path Replay Backpropagation, Vicini, Speierer and Jakob 2021):
// each path is replayed from its seed (no path storage), with sampling
// decisions, pdfs, MIS weights and Russian roulette detached.  The replay
// carries the remaining radiance L_rem = L_total - (contributions already
// met); at a vertex whose sampled BSDF value f enters every later
// contribution, d/dtheta of those contributions is L_rem / f * df/dtheta per
// channel; a light sample at the vertex contributes C / f_light *
// df_light/dtheta; emission contributes C / P * dP for the emitting light
// instance's power P.  BSDF derivatives are analytic (bsdf_grad.cuh).
// Visibility discontinuities are not differentiated.  Gradients are summed
// across each warp in registers, then per block in shared memory, then added
// to the output with one global atomic per parameter per block.
// No counterpart in the reference.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#define ZGL_INLINE_MATH 1
#include "bsdf_grad.cuh"
#include "path_trace.cuh"
#include "scene.h"
#include "staged.h"
#include "zgl_internal.h"

struct zgl_diff {
    zgl_scene* scene = nullptr;
    zgl_integrator_params params{};
    int32_t spp = 0;
    int32_t nmat = 0, ninst = 0, nparams = 0;
    float* d_samples = nullptr;   // spp * npix * 3 per-sample radiance
    // ray casts of the last forward, kept for the replay (null when they
    // would exceed the budget; the replay then traverses again)
    int2* d_hits = nullptr;       // kCastDepth * spp * npix (primitive id, distance bits)
    uint32_t* d_vis = nullptr;    // spp * npix light-sample occlusion bits
    bool castsValid = false;
    zgl::StagedPool pool;         // where forward and backward run staged
    double* d_grad = nullptr;     // gradient sums of the staged backward
    float* d_dimage = nullptr;    // npix * 3, zgl_diff_step_l2's dloss/dimage
    int32_t* d_lightInst = nullptr;  // per light triangle: instance index
    float* d_values = nullptr;       // current parameter values
    std::vector<uint32_t> lightFirst;
    std::vector<float> instPower;  // 3 per instance (current)
    std::vector<float> params_host;
};

namespace zgl {
namespace {

constexpr int kMaxDiffParams = 1024;

struct DiffInfo {
    int32_t nmat;
    int32_t nparams;
    const int32_t* lightInst;
};

// ----------------------------------------------------------------------------
// Ray casts kept between the forward pass and the replay.  The forward
// records, per (sample, pixel) path, the closest hits of its camera ray and
// first kCastDepth - 1 extension rays (primitive id and distance) and the
// occlusion answers of its first 32 light samples; the replay takes them in
// the same order instead of traversing again (casts past the record are
// traced).  Layout: hits[(k * spp + s) * npix + pix], vis[s * npix + pix], so
// that a warp's lanes (neighbouring pixels of one sample) store and load
// consecutive words.  8 bytes per cast: 640 MB for 512^2 pixels x 32 spp.
// ----------------------------------------------------------------------------
constexpr int kCastDepth = 9;
constexpr size_t kCastBudget = (size_t)4 << 30;  // bytes of cast records a renderer may keep

struct CastCursor {
    int nhit, nvis;
    uint32_t vis;
};

struct RecordCast {
    int2* hits;   // this path's first record; record k at hits[k * stride]
    size_t stride;
    CastCursor* cur;
    __device__ __forceinline__ int hit(const DeviceScene& sc, const Ray& r, float& dist) const {
        const int id = bvhHit(sc, r, dist);
        if (cur->nhit < kCastDepth) hits[(size_t)cur->nhit * stride] = make_int2(id, __float_as_int(dist));
        cur->nhit++;
        return id;
    }
    __device__ __forceinline__ bool operator()(const DeviceScene& sc, const Ray& r, float dist) const {
        const bool occ = bvhTest(sc, r, dist);
        if (cur->nvis < 32 && occ) cur->vis |= 1u << cur->nvis;
        cur->nvis++;
        return occ;
    }
};

struct ReplayCast {
    const int2* hits;
    size_t stride;
    CastCursor* cur;
    __device__ __forceinline__ int hit(const DeviceScene& sc, const Ray& r, float& dist) const {
        const int k = cur->nhit++;
        if (k < kCastDepth) {
            const int2 h = __ldg(hits + (size_t)k * stride);
            dist = __int_as_float(h.y);
            return h.x;
        }
        return bvhHit(sc, r, dist);
    }
    __device__ __forceinline__ bool operator()(const DeviceScene& sc, const Ray& r, float dist) const {
        const int k = cur->nvis++;
        if (k < 32) return (cur->vis >> k) & 1u;
        return bvhTest(sc, r, dist);
    }
};

// forward: one thread per (pixel, sample); blockIdx.y = sample.  Both
// kernels run at full occupancy (16 blocks of 128 threads per SM, at most 32
// registers a thread, spills in L1): at 512x512 and 32 spp that measured
// 49.4 -> 28.1 ms for the forward and 91.2 -> 50.5 ms for the replay against
// three to four blocks per SM without spills.
template <bool FULL>
__global__ void __launch_bounds__(kTileX* kTileY, 16)
diff_forward_kernel(DeviceScene sc, PathParams pp, int32_t tilesX, int32_t spp, float* __restrict__ samples,
                    int2* __restrict__ hits, uint32_t* __restrict__ vis) {
    __shared__ uint32_t row[256];
    const int32_t s = blockIdx.y;
    const uint32_t off = sample_offset(s);
    load_sobol_row(sc, off, row);
    const int tile = blockIdx.x;
    const int px = (tile % tilesX) * kTileX + threadIdx.x;
    const int py = (tile / tilesX) * kTileY + threadIdx.y;
    if (px >= sc.filmW || py >= sc.filmH) return;
    const size_t pix = (size_t)py * sc.filmW + px;
    const uint2 seed = __ldg(&sc.pixelSeeds[pix]);
    Sampler g;
    g.randSeed = seed.x * (uint32_t)(s + 1) + seed.y;
    g.sampleSeed = seed.x * seed.y;
    g.sampleOffset = off;
    g.dim = 0;
    g.mode = sc.sampler;
    g.rowCache = row;
    g.mats = sc.sobol;
    v2 scr = mk2((float)px, (float)py) / mk2((float)sc.filmW, (float)sc.filmH);
    float u0 = sample1D(g), u1 = sample1D(g), u2 = sample1D(g), u3 = sample1D(g);
    Ray ray = thinLensCameraSampleRay(sc, scr, u0, u1, u2, u3);
    v3 r;
    if (hits) {
        const size_t npix = (size_t)sc.filmW * sc.filmH, path = (size_t)s * npix + pix;
        CastCursor cur{0, 0, 0u};
        r = pathTraceRC<FULL>(sc, pp, ray, g, RecordCast{hits + path, (size_t)spp * npix, &cur});
        vis[path] = cur.vis;
    } else {
        r = pathTrace<FULL>(sc, pp, ray, g);
    }
    float* o = samples + 3 * ((size_t)s * sc.filmW * sc.filmH + pix);
    o[0] = r.x;
    o[1] = r.y;
    o[2] = r.z;
}

// image = (sum over samples in order, NaN samples dropped) / spp
__global__ void diff_reduce_kernel(const float* __restrict__ samples, int64_t npix, int32_t spp,
                                   float* __restrict__ image) {
    int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (p >= npix) return;
    float r = 0.0f, g = 0.0f, b = 0.0f;
    for (int s = 0; s < spp; s++) {
        const float* x = samples + 3 * ((size_t)s * npix + p);
        if (!(zisnan(x[0]) || zisnan(x[1]) || zisnan(x[2]))) {
            r = r + x[0];
            g = g + x[1];
            b = b + x[2];
        }
    }
    float inv = (float)spp;
    image[3 * p] = r / inv;
    image[3 * p + 1] = g / inv;
    image[3 * p + 2] = b / inv;
}

constexpr unsigned kFullMask = 0xffffffffu;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFullMask, v, o);
    return v;
}

// Adds vals[0..K) of every lane to sg[key + j], summing lanes that share a key
// in registers first: one shared-memory atomic per (distinct key, j) per warp.
// key < 0: the lane adds nothing.  All 32 lanes must call it together.
template <int K>
__device__ __forceinline__ void warp_flush(float* sg, int key, const float* vals) {
    unsigned pending = __ballot_sync(kFullMask, key >= 0);
    unsigned lane;  // the hardware lane id (the block is two-dimensional)
    asm("mov.u32 %0, %%laneid;" : "=r"(lane));
    while (pending) {
        const int leader = __ffs(pending) - 1;
        const int k = __shfl_sync(kFullMask, key, leader);
        const bool mine = key == k;
#pragma unroll
        for (int j = 0; j < K; j++) {
            float v = warp_sum(mine ? vals[j] : 0.0f);
            if (lane == (unsigned)leader && v != 0.0f) atomicAdd(&sg[k + j], v);
        }
        pending &= ~__ballot_sync(kFullMask, mine);
    }
}

// sum_c w_c df[i]_c with w_c = delta_c scale_c / f_c (channels with f_c == 0
// carry no radiance), added to acc[i].
__device__ __forceinline__ float grad_weight(float delta, float scale, float f) {
    float w = f > 1e-30f ? delta * scale / f : 0.0f;
    return isfinite(w) ? w : 0.0f;
}
__device__ __forceinline__ void mat_grad(float* acc, const v3& delta, const v3& scale, const BsdfGrad& bg) {
    const v3 w = mk3(grad_weight(delta.x, scale.x, bg.f.x), grad_weight(delta.y, scale.y, bg.f.y),
                     grad_weight(delta.z, scale.z, bg.f.z));
#pragma unroll
    for (int i = 0; i < kDiffMatParams; i++) acc[i] += w.x * bg.df[i].x + w.y * bg.df[i].y + w.z * bg.df[i].z;
}

// delta_c C_c / P_c for the power P of light triangle lightId's instance;
// returns the slot of the instance's first channel.
__device__ __forceinline__ int power_grad(const DiffInfo& di, const float* params, int lightId, const v3& delta,
                                          const v3& C, float* out) {
    const int inst = __ldg(&di.lightInst[lightId]);
    const int base = kDiffMatParams * di.nmat + 3 * inst;
    const float P[3] = {__ldg(&params[base]), __ldg(&params[base + 1]), __ldg(&params[base + 2])};
    const float c[3] = {C.x, C.y, C.z}, d[3] = {delta.x, delta.y, delta.z};
#pragma unroll
    for (int k = 0; k < 3; k++) out[k] = (P[k] != 0.0f && c[k] != 0.0f) ? d[k] * c[k] / P[k] : 0.0f;
    return base;
}

// A path under replay: the vertex it stands at, what it carries and the
// radiance not yet accounted for.
struct ReplayState {
    int id;
    v3 pos, wo, throughput, Lrem;
};
// One bounce's gradient contributions: one material, up to two light
// instances (keys below 0: none).
struct ReplayGrad {
    int mkey, nkey, hkey;
    float mg[kDiffMatParams], npw[3], hpw[3];
    __device__ __forceinline__ void clear() {
        mkey = nkey = hkey = -1;
#pragma unroll
        for (int i = 0; i < kDiffMatParams; i++) mg[i] = 0.0f;
    }
    // Every lane of the warp calls.
    __device__ __forceinline__ void flush(float* sg) {
        warp_flush<kDiffMatParams>(sg, mkey, mg);
        warp_flush<3>(sg, nkey, npw);
        warp_flush<3>(sg, hkey, hpw);
    }
};

// One bounce of a path's replay (pathIntegTrace, path_integ_naive.glsl:35-143):
// the light sample and the BSDF sample of the vertex and what the next ray
// meets, with their gradient contributions.  Returns whether the path goes on.
// `g` is the sampler, `Ltot` the sample's radiance and `delta`
// dL/d(radiance) of the sample; the ray casts come from `rc` (traversal, or
// the results recorded by the forward pass).
template <bool FULL, class RC>
__device__ __forceinline__ bool replayStep(const DeviceScene& sc, const PathParams& pp, const DiffInfo& di,
                                           const float* __restrict__ params, int bounce, ReplayState& st, Sampler& g,
                                           v3 Ltot, v3 delta, const RC& rc, ReplayGrad& gr) {
    int& id = st.id;
    v3 &pos = st.pos, &wo = st.wo, &throughput = st.throughput, &Lrem = st.Lrem;
    int &mkey = gr.mkey, &nkey = gr.nkey, &hkey = gr.hkey;
    float *mg = gr.mg, *npw = gr.npw, *hpw = gr.hpw;
    bool alive = true, textured = false;
    TriShade tri = loadTri(sc, id);
    Surface surf = surfaceInfo(tri, pos);
    const int matId = tri.matTex & 0x0000ffff;
    const uint32_t matType = loadMaterialType(sc, matId);
    if (matType != kDielectric && matType != kThinDielectric && dot(surf.ns, wo) < 0.0f) {
        surf.ns = -surf.ns;
        surf.ng = -surf.ng;
    }
    const BSDFParam mp = loadMaterial<FULL>(sc, matType, tri.matTex, id, surf);
    // metal-workflow and dielectric materials have no differentiable
    // parameters; their vertices only carry the paths
    const bool diffMat = !FULL || matType == kLambertian || matType == kPrincipled;
    mkey = diffMat ? kDiffMatParams * matId : -1;
    // a textured triangle's base colour is the texture's, not a parameter
    textured = FULL && (tri.matTex >> 16) != -1;
    if (pp.sampleLight) {
        const float ud = sample1D(g);
        const float u0 = sample1D(g), u1 = sample1D(g), u2 = sample1D(g), u3 = sample1D(g);
        float pdfSampleLight = 0.0f;  // the light pick of sampleLightAndEnv
        if (sc.nLight > 0) pdfSampleLight = pdfSampleLightSel(sc, pp.uniformSel, pp.portion);
        const int lid = ud < pdfSampleLight ? lightSampleOne(sc, mk2(u0, u1)) : -1;
        const LiSample ls = sampleLightAndEnvV(sc, pp, pos, ud, u0, u1, u2, u3, rc);
        if (ls.pdf > 0.0f) {
            BsdfGrad bg;
            if (diffMat) bg = bsdfGrad(matType, mp, wo, ls.wi, surf.ns);
            const v3 f = diffMat ? bg.f : materialBSDF<FULL>(matType, mp, wo, ls.wi, surf.ns);
            const float fpdf = materialPdf<FULL>(matType, mp, wo, ls.wi, surf.ns);
            const float weight = biHeuristic(ls.pdf, fpdf);
            const v3 C = f * throughput * satDot(surf.ns, ls.wi) * ls.coef * weight;
            if (diffMat) mat_grad(mg, delta, C, bg);
            if (lid >= 0) nkey = power_grad(di, params, lid, delta, C, npw);
            // what is left below the rounding of the total is no radiance
            Lrem = Lrem - C;
            Lrem.x = Lrem.x > 1e-6f * Ltot.x ? Lrem.x : 0.0f;
            Lrem.y = Lrem.y > 1e-6f * Ltot.y ? Lrem.y : 0.0f;
            Lrem.z = Lrem.z > 1e-6f * Ltot.z ? Lrem.z : 0.0f;
        }
    }
    const float b0 = sample1D(g), b1 = sample1D(g), b2 = sample1D(g);
    const BSDFSample bs = materialSample<FULL>(matType, mp, surf.ns, wo, mk3(b0, b1, b2), g);
    const v3 wi = bs.wi;
    const float bsdfPdf = bs.pdf;
    const bool deltaBsdf = (bs.flag == kSpecRefl || bs.flag == kSpecTrans);
    if (bsdfPdf < 1e-8f) {
        alive = false;
    } else {
        // every later contribution carries this vertex's sampled BSDF value
        if (diffMat) mat_grad(mg, delta, Lrem, bsdfGrad(matType, mp, wo, wi, surf.ns));
        throughput = throughput * (bs.bsdf / bsdfPdf * (deltaBsdf ? 1.0f : absDot(surf.ns, wi)));
        const Ray ray = rayOffseted(pos, wi);
        float dist;
        const int nextId = rc.hit(sc, ray, dist);
        const int lightId = nextId - sc.objPrimCount;
        const v3 nextPos = rayPoint(ray, dist);
        if (nextId == -1) {
            alive = false;  // environment emission: no parameter
        } else if (lightId >= 0) {
            const v3 radiance = lightLe(sc, lightId, nextPos, -wi);
            float weight = 1.0f;
            if (pp.sampleLight && !deltaBsdf) {
                const float lightPdf = lightPdfLi(sc, lightId, pos, nextPos) * pdfSelectLight(sc, pp, lightId);
                weight = (lightPdf <= 0.0f) ? 0.0f : biHeuristic(bsdfPdf, lightPdf);
            }
            hkey = power_grad(di, params, lightId, delta, radiance * throughput * weight, hpw);
            alive = false;
        } else {
            if (pp.rr && bounce >= pp.rrStart) {
                const float continueProb = zmin(maxComponent(bs.bsdf / bsdfPdf), 0.95f);
                if (sample1D(g) >= continueProb) alive = false;
                throughput = throughput / continueProb;
            }
            id = nextId;
            pos = nextPos;
            wo = -wi;
        }
    }
    if (textured) mg[0] = mg[1] = mg[2] = 0.0f;
    return alive && bounce < pp.maxDepth;
}

// The camera ray's hit: a light's emission (its gradient to `pkey`, `pw`) or
// the first vertex.  Returns whether there is a vertex.
template <class RC>
__device__ __forceinline__ bool replayFirst(const DeviceScene& sc, const DiffInfo& di, const float* __restrict__ params,
                                            const Ray& ray, v3 L, v3 delta, const RC& rc, ReplayState& st, int& pkey,
                                            float* pw) {
    float primDist;
    st.id = rc.hit(sc, ray, primDist);
    st.pos = rayPoint(ray, primDist);
    st.wo = -ray.dir;
    st.throughput = mk3(1.0f);
    st.Lrem = L;
    if (st.id == -1) return false;  // environment: no differentiable parameter
    if (st.id - sc.objPrimCount >= 0) {
        const int lightId = st.id - sc.objPrimCount;
        pkey = power_grad(di, params, lightId, delta, lightLe(sc, lightId, st.pos, -ray.dir), pw);
        return false;
    }
    return true;
}

// The replay of one path with its gradient contributions, in warp lockstep:
// one bounce per iteration of a warp-uniform loop, so that each iteration's
// gradients are reduced across the warp before the shared-memory atomics.  All
// 32 lanes of the warp call it together; a lane with alive == false only takes
// part in the reductions.  `g` is the sample's sampler right after its four
// camera dimensions, `ray` its camera ray, `L` its radiance.
template <bool FULL, class RC>
__device__ __forceinline__ void replayPath(const DeviceScene& sc, const PathParams& pp, const DiffInfo& di,
                                           const float* __restrict__ params, float* sg, bool alive, Sampler& g,
                                           Ray ray, v3 L, v3 delta, const RC& rc) {
    ReplayState st;
    float pw[3];
    int pkey = -1;
    if (alive) alive = replayFirst(sc, di, params, ray, L, delta, rc, st, pkey, pw);
    warp_flush<3>(sg, pkey, pw);
    // the first vertex is shaded whatever the depth, as the forward loop's
    // bound is checked behind a bounce
    for (int bounce = 1; __any_sync(kFullMask, alive); bounce++) {
        ReplayGrad gr;
        gr.clear();
        if (alive) alive = replayStep<FULL>(sc, pp, di, params, bounce, st, g, L, delta, rc, gr);
        gr.flush(sg);
    }
}

// ----------------------------------------------------------------------------
// The staged backward: the replay of the recorded casts one bounce a launch,
// over lists without the ended paths, each block's paths in order of material.
// The one-kernel replay is bound by instruction fetch, and its warp reductions
// run once per distinct material among 32 neighbours; here a warp's lanes
// mostly share one.  512x512, 32 spp, depth 6, 8 materials: 26.1 -> 10.6 ms.
// ----------------------------------------------------------------------------
struct ReplayList {
    float4 *pos, *wo, *thr, *rem;
    uint2* rng;
};
struct ReplayJob {
    DiffInfo di;
    const float* params;
    int32_t tilesX;
    int64_t perSample, npix;
    int32_t spp;
    int64_t q0, count;
    int32_t row0;
    const float *samples, *dimage;
    const int2* hits;
    const uint32_t* vis;
    const uint32_t* rows;
    double* grad;
};

// Recorded casts only (a path no longer than the record).
struct KeptCast {
    const int2* hits;  // the next closest hit
    uint32_t vis;
    int* nvis;
    __device__ __forceinline__ int hit(const DeviceScene&, const Ray&, float& dist) const {
        const int2 h = __ldg(hits);
        dist = __int_as_float(h.y);
        return h.x;
    }
    __device__ __forceinline__ bool operator()(const DeviceScene&, const Ray&, float) const {
        return (vis >> (*nvis)++) & 1u;
    }
};

constexpr int kReplayBlock = 256;
constexpr int kReplayBlocksPerSM = 4;  // 64 registers: 10.6 ms of 512x512x32; 2, 5, 6 blocks 11.2, 11.4, 12.1
constexpr int kReplayBins = 32;  // the last: no path

struct ReplaySort {
    uint16_t perm[kReplayBlock];
    uint32_t count[kReplayBins][kReplayBlock / 32];
};
// This thread's path of the block's window when ordered by bin.
__device__ __forceinline__ int replay_sort(int bin, ReplaySort& sh) {
    constexpr int kWarps = kReplayBlock / 32, kPer = kReplayBins * kWarps / 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    sh.count[lane][w] = 0u;
    __syncwarp();
    const unsigned m = __match_any_sync(kFullMask, bin);
    const int rank = __popc(m & ((1u << lane) - 1u));
    if (rank == 0) sh.count[bin][w] = (uint32_t)__popc(m);
    __syncthreads();
    if (w == 0) {
        uint32_t v[kPer], total = 0;
        uint32_t* flat = &sh.count[0][0];
#pragma unroll
        for (int k = 0; k < kPer; k++) {
            v[k] = total;
            total += flat[lane * kPer + k];
        }
        uint32_t x = total;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kFullMask, x, d);
            if (lane >= d) x += y;
        }
#pragma unroll
        for (int k = 0; k < kPer; k++) flat[lane * kPer + k] = x - total + v[k];
    }
    __syncthreads();
    sh.perm[sh.count[bin][w] + rank] = (uint16_t)threadIdx.x;
    __syncthreads();
    return sh.perm[threadIdx.x];
}
__device__ __forceinline__ int replay_bin(const DeviceScene& sc, int id) {
    const int matTex = __float_as_int(__ldg(reinterpret_cast<const float*>(sc.shade + 5 * (size_t)id + 4) + 2));
    return (int)((uint32_t)(matTex & 0x0000ffff) % (kReplayBins - 1));
}

// Appends this thread's path to a list, one atomic per block.
__device__ __forceinline__ uint32_t replay_append(bool want, uint32_t* counter, uint32_t* sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned m = __ballot_sync(kFullMask, want);
    if (lane == 0) sh[w] = (uint32_t)__popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t total = 0;
        for (int i = 0; i < kReplayBlock / 32; i++) {
            const uint32_t c = sh[i];
            sh[i] = total;
            total += c;
        }
        const uint32_t base = total ? atomicAdd(counter, total) : 0u;
        for (int i = 0; i < kReplayBlock / 32; i++) sh[i] += base;
    }
    __syncthreads();
    return sh[w] + (uint32_t)__popc(m & ((1u << lane) - 1u));
}
__device__ __forceinline__ void replay_store(const ReplayList& l, uint32_t i, const ReplayState& st, const Sampler& g,
                                             uint32_t path, int nvis) {
    l.pos[i] = make_float4(st.pos.x, st.pos.y, st.pos.z, __int_as_float(st.id));
    l.wo[i] = make_float4(st.wo.x, st.wo.y, st.wo.z, __uint_as_float((uint32_t)g.dim | (uint32_t)nvis << 16));
    l.thr[i] = make_float4(st.throughput.x, st.throughput.y, st.throughput.z, __uint_as_float(path));
    l.rem[i] = make_float4(st.Lrem.x, st.Lrem.y, st.Lrem.z, 0.0f);
    l.rng[i] = make_uint2(g.randSeed, g.sampleSeed);
}
// Sample and pixel of chunk item k (8x4 pixel tiles per sample); false outside
// the film.
__device__ __forceinline__ bool replay_item(const DeviceScene& sc, const ReplayJob& job, int64_t k, int32_t& s, int& px,
                                            int& py) {
    const int64_t q = job.q0 + k;
    s = (int32_t)(q / job.perSample);
    const int64_t in = q - s * job.perSample, tile = in >> 5;
    px = (int)(tile % job.tilesX) * 8 + ((int)in & 7);
    py = (int)(tile / job.tilesX) * 4 + (((int)in >> 3) & 3);
    return px < sc.filmW && py < sc.filmH;
}
__device__ __forceinline__ v3 sample_radiance(const ReplayJob& job, int64_t path) {
    const float* p = job.samples + 3 * path;
    return mk3(p[0], p[1], p[2]);
}
__device__ __forceinline__ v3 sample_adjoint(const ReplayJob& job, int64_t pix) {
    const float inv = 1.0f / (float)job.spp;
    const float* p = job.dimage + 3 * pix;
    return mk3(p[0] * inv, p[1] * inv, p[2] * inv);
}
// A block's gradient: a window's sums in float32, the windows' in 64 bits
// (thousands of windows in one float32 sum lost a digit against one sum per
// 128 paths).
struct BlockGrad {
    float window[kMaxDiffParams];
    double total[kMaxDiffParams];
    __device__ __forceinline__ void clear(int n) {
        for (int i = threadIdx.x; i < n; i += kReplayBlock) {
            window[i] = 0.0f;
            total[i] = 0.0;
        }
        __syncthreads();
    }
    // After the window's last flush and a barrier; before the next flush.
    __device__ __forceinline__ void close(int n) {
        for (int i = threadIdx.x; i < n; i += kReplayBlock) {
            total[i] += (double)window[i];
            window[i] = 0.0f;
        }
        __syncthreads();
    }
    __device__ __forceinline__ void add(int n, double* grad) {
        for (int i = threadIdx.x; i < n; i += kReplayBlock)
            if (total[i] != 0.0) atomicAdd(&grad[i], total[i]);
    }
};

__global__ void __launch_bounds__(kReplayBlock)
replay_start_kernel(const __grid_constant__ DeviceScene sc, const __grid_constant__ ReplayJob job,
                    const __grid_constant__ ReplayList next, uint32_t* counts) {
    __shared__ uint32_t sh[kReplayBlock / 32];
    __shared__ BlockGrad bg;
    bg.clear(job.di.nparams);
    for (int64_t base = blockIdx.x * (int64_t)kReplayBlock; base < job.count; base += (int64_t)gridDim.x * kReplayBlock) {
        const int64_t k = base + threadIdx.x;
        int32_t s = 0;
        int px = 0, py = 0;
        bool alive = k < job.count && replay_item(sc, job, k, s, px, py);
        const int64_t pix = (int64_t)py * sc.filmW + px, path = (int64_t)s * job.npix + pix;
        v3 L = mk3(0.0f), delta = mk3(0.0f);
        if (alive) {
            L = sample_radiance(job, path);
            delta = sample_adjoint(job, pix);
            // NaN samples are left out of the image; zero adjoints need no replay
            alive = !hasNan(L) && (delta.x != 0.0f || delta.y != 0.0f || delta.z != 0.0f);
        }
        ReplayState st;
        Sampler g;
        float pw[3];
        int pkey = -1;
        if (alive) {
            const uint2 seed = __ldg(&sc.pixelSeeds[pix]);
            g.randSeed = seed.x * (uint32_t)(s + 1) + seed.y;
            g.sampleSeed = seed.x * seed.y;
            g.sampleOffset = sample_offset(s);
            g.dim = 0;
            g.mode = sc.sampler;
            g.rowCache = job.rows + 256 * (s - job.row0);
            g.mats = sc.sobol;
            const v2 scr = mk2((float)px, (float)py) / mk2((float)sc.filmW, (float)sc.filmH);
            const float u0 = sample1D(g), u1 = sample1D(g), u2 = sample1D(g), u3 = sample1D(g);
            const Ray ray = thinLensCameraSampleRay(sc, scr, u0, u1, u2, u3);
            int nvis = 0;
            alive = replayFirst(sc, job.di, job.params, ray, L, delta, KeptCast{job.hits + path, 0u, &nvis}, st, pkey,
                                pw);
        }
        warp_flush<3>(bg.window, pkey, pw);
        const uint32_t at = replay_append(alive, counts, sh);  // its barriers end the flush
        bg.close(job.di.nparams);
        if (alive) replay_store(next, at, st, g, (uint32_t)k, 0);
    }
    bg.add(job.di.nparams, job.grad);
}

template <bool FULL>
__global__ void __launch_bounds__(kReplayBlock, kReplayBlocksPerSM)
replay_step_kernel(const __grid_constant__ DeviceScene sc, const PathParams pp, const __grid_constant__ ReplayJob job,
                   int bounce, const __grid_constant__ ReplayList in, const __grid_constant__ ReplayList next,
                   uint32_t* counts) {
    __shared__ uint32_t sh[kReplayBlock / 32];
    __shared__ ReplaySort sort;
    __shared__ BlockGrad bg;
    const uint32_t n = counts[bounce - 1];
    if (blockIdx.x * kReplayBlock >= n) return;
    bg.clear(job.di.nparams);
    for (uint32_t base = blockIdx.x * kReplayBlock; base < n; base += gridDim.x * kReplayBlock) {
        const uint32_t j = base + threadIdx.x;
        const int bin = j < n ? replay_bin(sc, __float_as_int(in.pos[j].w)) : kReplayBins - 1;
        const uint32_t i = base + (uint32_t)replay_sort(bin, sort);
        bool alive = i < n;
        ReplayState st;
        Sampler g;
        ReplayGrad gr;
        gr.clear();
        uint32_t k = 0;
        int nvis = 0;
        if (alive) {
            const float4 p = in.pos[i], w = in.wo[i], t = in.thr[i], m = in.rem[i];
            const uint2 r = in.rng[i];
            st.pos = mk3(p.x, p.y, p.z);
            st.id = __float_as_int(p.w);
            st.wo = mk3(w.x, w.y, w.z);
            st.throughput = mk3(t.x, t.y, t.z);
            st.Lrem = mk3(m.x, m.y, m.z);
            k = __float_as_uint(t.w);
            int32_t s;
            int px, py;
            replay_item(sc, job, k, s, px, py);
            const int64_t pix = (int64_t)py * sc.filmW + px, path = (int64_t)s * job.npix + pix;
            g.randSeed = r.x;
            g.sampleSeed = r.y;
            g.dim = (int)(__float_as_uint(w.w) & 0xffffu);
            nvis = (int)(__float_as_uint(w.w) >> 16);
            g.sampleOffset = sample_offset(s);
            g.mode = sc.sampler;
            g.rowCache = job.rows + 256 * (s - job.row0);
            g.mats = sc.sobol;
            const KeptCast kept{job.hits + (int64_t)bounce * job.spp * job.npix + path, __ldg(job.vis + path), &nvis};
            alive = replayStep<FULL>(sc, pp, job.di, job.params, bounce, st, g, sample_radiance(job, path),
                                     sample_adjoint(job, pix), kept, gr);
        }
        gr.flush(bg.window);
        const uint32_t at = replay_append(alive, &counts[bounce], sh);  // its barriers end the flush
        bg.close(job.di.nparams);
        if (alive) replay_store(next, at, st, g, k, nvis);
    }
    bg.add(job.di.nparams, job.grad);
}

__global__ void replay_grad_kernel(const double* __restrict__ sum, int n, float* __restrict__ grad) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) grad[i] = (float)sum[i];
}

cudaError_t launch_replay(const StagedPool& pool, const DeviceScene& sc, const PathParams& pp, bool full, ReplayJob job,
                          float* grad, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(job.grad, 0, sizeof(double) * (size_t)job.di.nparams, st);
    if (e != cudaSuccess) return e;
    ReplayList lists[2];
    for (int i = 0; i < 2; i++) lists[i] = ReplayList{pool.org[i], pool.dir[i], pool.thr[i], pool.pos[i], pool.rng[i]};
    job.tilesX = (sc.filmW + 7) / 8;
    job.perSample = staged_paths(sc.filmW, sc.filmH, 1);
    job.npix = (int64_t)sc.filmW * sc.filmH;
    job.rows = pool.rows;
    const int64_t total = job.perSample * job.spp;
    const int sms = staged_sms();
    for (job.q0 = 0; job.q0 < total; job.q0 += job.count) {
        const int64_t s0 = job.q0 / job.perSample;
        job.count = std::min(std::min(total - job.q0, pool.paths), (s0 + kStagedRows) * job.perSample - job.q0);
        job.row0 = (int32_t)s0;
        const int nrows = (int)((job.q0 + job.count - 1) / job.perSample - s0) + 1;
        e = cudaMemsetAsync(pool.counts, 0, sizeof(uint32_t) * (pp.maxDepth + 2), st);
        if (e != cudaSuccess) return e;
        if (sc.sampler == 1 && (e = launch_staged_rows(pool, sc.sobol, job.row0, nrows, st)) != cudaSuccess) return e;
        const unsigned blocks = (unsigned)std::min<int64_t>((job.count + kReplayBlock - 1) / kReplayBlock,
                                                            (int64_t)sms * kReplayBlocksPerSM * 2);
        replay_start_kernel<<<blocks, kReplayBlock, 0, st>>>(sc, job, lists[0], pool.counts);
        for (int bounce = 1; bounce <= pp.maxDepth; bounce++) {
            const ReplayList &in = lists[(bounce - 1) & 1], &next = lists[bounce & 1];
            if (full)
                replay_step_kernel<true><<<blocks, kReplayBlock, 0, st>>>(sc, pp, job, bounce, in, next, pool.counts);
            else
                replay_step_kernel<false><<<blocks, kReplayBlock, 0, st>>>(sc, pp, job, bounce, in, next, pool.counts);
        }
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    replay_grad_kernel<<<(unsigned)((job.di.nparams + 255) / 256), 256, 0, st>>>(job.grad, job.di.nparams, grad);
    return cudaGetLastError();
}

// Backward: one thread per (pixel, sample), blockIdx.y = sample; the replay
// takes the ray casts the forward recorded (`hits` / `vis`), or traverses the
// accelerator again when there is no record.
template <bool FULL>
__global__ void __launch_bounds__(kTileX* kTileY, 16)
diff_backward_kernel(DeviceScene sc, PathParams pp, DiffInfo di, const float* __restrict__ params, int32_t tilesX,
                     int32_t spp, const float* __restrict__ samples, const float* __restrict__ dimage,
                     const int2* __restrict__ hits, const uint32_t* __restrict__ vis, float* __restrict__ grad) {
    __shared__ uint32_t row[256];
    __shared__ float sg[kMaxDiffParams];
    for (int i = threadIdx.y * kTileX + threadIdx.x; i < di.nparams; i += kTileX * kTileY) sg[i] = 0.0f;
    const int32_t s = blockIdx.y;
    const uint32_t off = sample_offset(s);
    load_sobol_row(sc, off, row);  // includes the barrier that publishes sg
    const int tile = blockIdx.x;
    const int px = (tile % tilesX) * kTileX + threadIdx.x;
    const int py = (tile / tilesX) * kTileY + threadIdx.y;

    bool alive = px < sc.filmW && py < sc.filmH;
    v3 L = mk3(0.0f), delta = mk3(0.0f);
    size_t pix = 0;
    if (alive) {
        const size_t npix = (size_t)sc.filmW * sc.filmH;
        pix = (size_t)py * sc.filmW + px;
        const float* Ls = samples + 3 * ((size_t)s * npix + pix);
        L = mk3(Ls[0], Ls[1], Ls[2]);
        const float inv = 1.0f / (float)spp;
        delta = mk3(dimage[3 * pix] * inv, dimage[3 * pix + 1] * inv, dimage[3 * pix + 2] * inv);
        // NaN samples are left out of the image; zero adjoints need no replay
        alive = !hasNan(L) && (delta.x != 0.0f || delta.y != 0.0f || delta.z != 0.0f);
    }
    Sampler g;
    Ray ray;
    if (alive) {
        const uint2 seed = __ldg(&sc.pixelSeeds[pix]);
        g.randSeed = seed.x * (uint32_t)(s + 1) + seed.y;
        g.sampleSeed = seed.x * seed.y;
        g.sampleOffset = off;
        g.dim = 0;
        g.mode = sc.sampler;
        g.rowCache = row;
        g.mats = sc.sobol;
        v2 scr = mk2((float)px, (float)py) / mk2((float)sc.filmW, (float)sc.filmH);
        float u0 = sample1D(g), u1 = sample1D(g), u2 = sample1D(g), u3 = sample1D(g);
        ray = thinLensCameraSampleRay(sc, scr, u0, u1, u2, u3);
    }
    if (hits) {
        const size_t npix = (size_t)sc.filmW * sc.filmH, path = (size_t)s * npix + pix;
        CastCursor cur{0, 0, alive ? __ldg(vis + path) : 0u};
        replayPath<FULL>(sc, pp, di, params, sg, alive, g, ray, L, delta,
                         ReplayCast{hits + path, (size_t)spp * npix, &cur});
    } else {
        replayPath<FULL>(sc, pp, di, params, sg, alive, g, ray, L, delta, DirectCast{});
    }
    __syncthreads();
    for (int i = threadIdx.y * kTileX + threadIdx.x; i < di.nparams; i += kTileX * kTileY)
        if (sg[i] != 0.0f) atomicAdd(&grad[i], sg[i]);
}

// dloss/dimage = 2 s (image - target) and the loss s * sum (image - target)^2
// of zgl_diff_step_l2; one atomic per block for the loss.
__global__ void diff_l2_kernel(const float* __restrict__ image, const float* __restrict__ target, int64_t n,
                               float scale, float* __restrict__ dimage, float* __restrict__ loss) {
    __shared__ float part[8];
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    float l = 0.0f;
    if (i < n) {
        const float diff = image[i] - target[i];
        dimage[i] = diff * (2.0f * scale);
        l = diff * diff * scale;
    }
    l = warp_sum(l);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += part[w];
        if (t != 0.0f) atomicAdd(loss, t);
    }
}

}  // namespace

}  // namespace zgl

using namespace zgl;

namespace {

PathParams path_params(const zgl_integrator_params& p) {
    return PathParams{p.max_depth, p.russian_roulette, p.rr_start_depth, p.sample_light, p.light_env_uniform_sample,
                      p.light_portion};
}

bool device_ptr(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

}  // namespace

extern "C" {

zgl_status zgl_diff_create(zgl_scene* scene, const zgl_integrator_params* params, int32_t spp, zgl_diff** out) {
    ZGL_API_BEGIN
    if (!scene || !out) fail(ZGL_ERR_INVALID_ARG, "zgl_diff_create: NULL argument");
    *out = nullptr;
    if (scene->host_only) fail(ZGL_ERR_STATE, "zgl_diff_create: scene was created host-only");
    if (spp < 1 || spp > 4096) fail(ZGL_ERR_INVALID_ARG, "zgl_diff_create: spp %d out of range", spp);
    auto* d = new zgl_diff();
    try {
        d->scene = scene;
        zgl_integrator_params_default(&d->params);
        if (params) d->params = *params;
        d->spp = spp;
        d->nmat = (int32_t)(scene->materials.size() / 16);
        d->lightFirst = scene->lightFirst;
        d->instPower = scene->lightInstPower;
        d->ninst = (int32_t)(d->instPower.size() / 3);
        d->nparams = kDiffMatParams * d->nmat + 3 * d->ninst;
        if (d->nparams > kMaxDiffParams) fail(ZGL_ERR_INVALID_ARG, "zgl_diff_create: %d parameters exceed %d", d->nparams, kMaxDiffParams);
        size_t npix = (size_t)scene->filmW * scene->filmH;
        ZGL_CUDA(cudaMalloc(&d->d_samples, sizeof(float) * 3 * npix * (size_t)spp));
        const size_t paths = npix * (size_t)spp;
        if ((sizeof(int2) * kCastDepth + sizeof(uint32_t)) * paths <= kCastBudget) {
            ZGL_CUDA(cudaMalloc(&d->d_hits, sizeof(int2) * kCastDepth * paths));
            ZGL_CUDA(cudaMalloc(&d->d_vis, sizeof(uint32_t) * paths));
        }
        std::vector<int32_t> inst((size_t)std::max(scene->nLight, 1), 0);
        for (int k = 0; k < d->ninst; k++)
            for (uint32_t t = d->lightFirst[(size_t)k]; t < d->lightFirst[(size_t)k + 1]; t++) inst[t] = k;
        ZGL_CUDA(cudaMalloc(&d->d_lightInst, sizeof(int32_t) * inst.size()));
        ZGL_CUDA(cudaMemcpy(d->d_lightInst, inst.data(), sizeof(int32_t) * inst.size(), cudaMemcpyHostToDevice));
        // current parameter values
        d->params_host.assign((size_t)d->nparams, 0.0f);
        for (int m = 0; m < d->nmat; m++) {
            const float* r = &scene->materials[16 * (size_t)m];
            float v[6] = {r[0], r[1], r[2], r[3], r[5], r[6]};
            std::memcpy(&d->params_host[(size_t)kDiffMatParams * m], v, sizeof(v));
        }
        for (int k = 0; k < 3 * d->ninst; k++) d->params_host[(size_t)kDiffMatParams * d->nmat + k] = d->instPower[(size_t)k];
        ZGL_CUDA(cudaMalloc(&d->d_values, sizeof(float) * (size_t)std::max(d->nparams, 1)));
        ZGL_CUDA(cudaMemcpy(d->d_values, d->params_host.data(), sizeof(float) * (size_t)d->nparams, cudaMemcpyHostToDevice));
        // last, so that it takes no memory from what has to be there; without
        // it the one-kernel forward and replay run
        if (staged_covers(scene->view(), d->params.max_depth) && staged_diff_pays((int64_t)paths) &&
            staged_alloc(d->pool, staged_paths(scene->filmW, scene->filmH, spp)) &&
            cudaMalloc(&d->d_grad, sizeof(double) * (size_t)std::max(d->nparams, 1)) != cudaSuccess) {
            cudaGetLastError();
            d->d_grad = nullptr;
            staged_free(d->pool);
        }
    } catch (...) {
        if (d->d_samples) cudaFree(d->d_samples);
        if (d->d_hits) cudaFree(d->d_hits);
        if (d->d_vis) cudaFree(d->d_vis);
        if (d->d_lightInst) cudaFree(d->d_lightInst);
        if (d->d_values) cudaFree(d->d_values);
        if (d->d_grad) cudaFree(d->d_grad);
        staged_free(d->pool);
        delete d;
        throw;
    }
    *out = d;
    ZGL_API_END
}

zgl_status zgl_diff_param_count(const zgl_diff* d, int32_t* n) {
    ZGL_API_BEGIN
    if (!d || !n) fail(ZGL_ERR_INVALID_ARG, "zgl_diff_param_count: NULL");
    *n = d->nparams;
    ZGL_API_END
}

zgl_status zgl_diff_get_params(const zgl_diff* d, float* out) {
    ZGL_API_BEGIN
    if (!d || !out) fail(ZGL_ERR_INVALID_ARG, "zgl_diff_get_params: NULL");
    std::memcpy(out, d->params_host.data(), sizeof(float) * d->params_host.size());
    ZGL_API_END
}

zgl_status zgl_diff_set_params(zgl_diff* d, const float* params) {
    ZGL_API_BEGIN
    if (!d || !params) fail(ZGL_ERR_INVALID_ARG, "zgl_diff_set_params: NULL");
    // work queued on any stream may still read the scene or write `params`
    ZGL_CUDA(cudaDeviceSynchronize());
    std::vector<float> p((size_t)d->nparams);
    if (device_ptr(params)) ZGL_CUDA(cudaMemcpy(p.data(), params, sizeof(float) * p.size(), cudaMemcpyDeviceToHost));
    else std::memcpy(p.data(), params, sizeof(float) * p.size());
    for (float v : p)
        if (!std::isfinite(v)) fail(ZGL_ERR_INVALID_ARG, "zgl_diff_set_params: non-finite parameter");
    scene_set_diff_params(d->scene, p.data(), d->nmat, d->instPower);
    // new roughness or metallic values move the sampled directions: the kept casts no longer apply
    d->castsValid = false;
    d->params_host = p;
    ZGL_CUDA(cudaMemcpy(d->d_values, p.data(), sizeof(float) * p.size(), cudaMemcpyHostToDevice));
    ZGL_API_END
}

zgl_status zgl_diff_forward(zgl_diff* d, float* image, void* stream) {
    ZGL_API_BEGIN
    ZGL_RANGE("zgl_diff_forward");
    if (!d || !image) fail(ZGL_ERR_INVALID_ARG, "zgl_diff_forward: NULL");
    if (!device_ptr(image)) fail(ZGL_ERR_INVALID_ARG, "zgl_diff_forward: image must be device memory");
    const zgl_scene* s = d->scene;
    cudaStream_t st = (cudaStream_t)stream;
    int tilesX = (s->filmW + kTileX - 1) / kTileX, tilesY = (s->filmH + kTileY - 1) / kTileY;
    dim3 grid((unsigned)(tilesX * tilesY), (unsigned)d->spp);
    if (d->pool.arena) {
        const zgl_integrator_params& p = d->params;
        StagedJob job{};
        job.sc = s->view();
        job.maxDepth = p.max_depth;
        job.rr = p.russian_roulette;
        job.rrStart = p.rr_start_depth;
        job.sampleLight = p.sample_light;
        job.uniformSel = p.light_env_uniform_sample;
        job.portion = p.light_portion;
        job.full = s->fullMaterials;
        job.first = 0;
        job.n = d->spp;
        job.counter0 = 1;
        job.out = d->d_samples;
        job.hits = d->d_hits;
        job.castDepth = kCastDepth;
        job.vis = d->d_vis;
        const StagedTurn turn(d->pool, st);
        ZGL_CUDA(launch_staged(d->pool, job, st));
    } else if (s->fullMaterials)
        diff_forward_kernel<true><<<grid, dim3(kTileX, kTileY), 0, st>>>(s->view(), path_params(d->params), tilesX,
                                                                         d->spp, d->d_samples, d->d_hits, d->d_vis);
    else
        diff_forward_kernel<false><<<grid, dim3(kTileX, kTileY), 0, st>>>(s->view(), path_params(d->params), tilesX,
                                                                          d->spp, d->d_samples, d->d_hits, d->d_vis);
    d->castsValid = d->d_hits != nullptr;
    ZGL_CUDA(cudaGetLastError());
    int64_t npix = (int64_t)s->filmW * s->filmH;
    diff_reduce_kernel<<<(unsigned)((npix + 255) / 256), 256, 0, st>>>(d->d_samples, npix, d->spp, image);
    ZGL_CUDA(cudaGetLastError());
    ZGL_API_END
}

zgl_status zgl_diff_backward(zgl_diff* d, const float* d_image, float* d_params, void* stream) {
    ZGL_API_BEGIN
    ZGL_RANGE("zgl_diff_backward");
    if (!d || !d_image || !d_params) fail(ZGL_ERR_INVALID_ARG, "zgl_diff_backward: NULL");
    if (!device_ptr(d_image) || !device_ptr(d_params))
        fail(ZGL_ERR_INVALID_ARG, "zgl_diff_backward: arrays must be device memory");
    const zgl_scene* s = d->scene;
    cudaStream_t st = (cudaStream_t)stream;
    ZGL_CUDA(cudaMemsetAsync(d_params, 0, sizeof(float) * (size_t)d->nparams, st));
    DiffInfo di{d->nmat, d->nparams, d->d_lightInst};
    int tilesX = (s->filmW + kTileX - 1) / kTileX, tilesY = (s->filmH + kTileY - 1) / kTileY;
    dim3 grid((unsigned)(tilesX * tilesY), (unsigned)d->spp);
    const int2* hits = d->castsValid ? d->d_hits : nullptr;
    const uint32_t* vis = d->castsValid ? d->d_vis : nullptr;
    // a path of maxDepth bounces takes maxDepth + 1 recorded hits
    if (hits && d->pool.arena && d->params.max_depth >= 1 && d->params.max_depth < kCastDepth) {
        ReplayJob job{};
        job.di = di;
        job.params = d->d_values;
        job.spp = d->spp;
        job.samples = d->d_samples;
        job.dimage = d_image;
        job.hits = hits;
        job.vis = vis;
        job.grad = d->d_grad;
        const StagedTurn turn(d->pool, st);
        ZGL_CUDA(launch_replay(d->pool, s->view(), path_params(d->params), s->fullMaterials, job, d_params, st));
    } else if (s->fullMaterials)
        diff_backward_kernel<true><<<grid, dim3(kTileX, kTileY), 0, st>>>(s->view(), path_params(d->params), di,
                                                                          d->d_values, tilesX, d->spp, d->d_samples,
                                                                          d_image, hits, vis, d_params);
    else
        diff_backward_kernel<false><<<grid, dim3(kTileX, kTileY), 0, st>>>(s->view(), path_params(d->params), di,
                                                                           d->d_values, tilesX, d->spp, d->d_samples,
                                                                           d_image, hits, vis, d_params);
    ZGL_CUDA(cudaGetLastError());
    ZGL_API_END
}

zgl_status zgl_diff_step_l2(zgl_diff* d, const float* target, float loss_scale, float* image, float* d_params,
                            float* loss, void* stream) {
    ZGL_API_BEGIN
    ZGL_RANGE("zgl_diff_step_l2");
    if (!d || !target || !image || !d_params || !loss) fail(ZGL_ERR_INVALID_ARG, "zgl_diff_step_l2: NULL");
    if (!device_ptr(target) || !device_ptr(image) || !device_ptr(d_params) || !device_ptr(loss))
        fail(ZGL_ERR_INVALID_ARG, "zgl_diff_step_l2: arrays must be device memory");
    if (!std::isfinite(loss_scale)) fail(ZGL_ERR_INVALID_ARG, "zgl_diff_step_l2: non-finite loss scale");
    const zgl_scene* s = d->scene;
    cudaStream_t st = (cudaStream_t)stream;
    const int64_t n = (int64_t)s->filmW * s->filmH * 3;
    if (!d->d_dimage) ZGL_CUDA(staged_malloc_beside(d->pool, (void**)&d->d_dimage, sizeof(float) * (size_t)n));
    zgl_status r = zgl_diff_forward(d, image, stream);
    if (r != ZGL_OK) return r;
    ZGL_CUDA(cudaMemsetAsync(loss, 0, sizeof(float), st));
    diff_l2_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(image, target, n, loss_scale, d->d_dimage, loss);
    ZGL_CUDA(cudaGetLastError());
    return zgl_diff_backward(d, d->d_dimage, d_params, stream);
    ZGL_API_END
}

zgl_status zgl_diff_destroy(zgl_diff* d) {
    ZGL_API_BEGIN
    if (!d) return ZGL_OK;
    if (d->d_samples) cudaFree(d->d_samples);
    if (d->d_hits) cudaFree(d->d_hits);
    if (d->d_vis) cudaFree(d->d_vis);
    if (d->d_dimage) cudaFree(d->d_dimage);
    if (d->d_lightInst) cudaFree(d->d_lightInst);
    if (d->d_values) cudaFree(d->d_values);
    if (d->d_grad) cudaFree(d->d_grad);
    staged_free(d->pool);
    delete d;
    ZGL_API_END
}

}  // extern "C"
