// path_step.cuh — the MIS path tracer (pathIntegTrace,
// path_integ_naive.glsl:35-143) as a state machine of one bounce per step, for
// schedules that trace rays apart from shading: the batched renderer's
// persistent and queue schedules (render_batch.cu) and the staged path tracer
// (staged.cu).
#pragma once

#include "path_trace.cuh"

namespace zgl {
namespace {

struct PathState {
    Ray ray;        // pending ray
    v3 result, throughput;
    v3 wo, pos;     // vertex being left (valid after the first bounce)
    v3 bsdfOverPdf; // bsdf / pdf of the last sample (Russian roulette)
    float bsdfPdf;
    int32_t bounce; // 0 = camera ray pending
    bool delta;
};

// The light sample of a vertex whose occlusion test is left to a later
// trace: the shadow ray and the contribution the sample makes if nothing
// blocks it.
struct PendingShadow {
    v3 o, d, C;
    float tmax;
    bool pending;
    bool asked;  // the sample came as far as its occlusion test
};

// Visibility source that records the shadow ray instead of tracing it and
// answers "not occluded"; the contribution is added after the trace.
struct DeferVis {
    PendingShadow* ps;
    __device__ __forceinline__ bool operator()(const DeviceScene&, const Ray& r, float dist) const {
        ps->o = r.ori;
        ps->d = r.dir;
        ps->tmax = dist;
        ps->asked = true;
        return false;
    }
};

// One step of pathIntegTrace after the pending ray has been traced (closest
// hit `id` at `dist`): account for what it hits and, if the path continues,
// shade the new vertex (light sample + BSDF sample) to produce the next
// pending ray.  Returns false when the path ends.  DEFER: the light sample's
// occlusion test is recorded in `ps` for a later trace instead of run here.
template <bool FULL, bool DEFER>
__device__ __forceinline__ bool path_step_hit(const DeviceScene& sc, const PathParams& pp, Sampler& g, PathState& st, int id, float dist,
                                              PendingShadow* ps) {
    v3 hitPos = rayPoint(st.ray, dist);
    if (st.bounce == 0) {
        // primary hit (path_integ_naive.glsl:37-44)
        if (id == -1) {
            st.result = envLe(sc, st.ray.dir);
            return false;
        }
        if (id - sc.objPrimCount >= 0) {
            st.result = lightLe(sc, id - sc.objPrimCount, hitPos, -st.ray.dir);
            return false;
        }
        st.wo = -st.ray.dir;
    } else {
        // extension hit of bounce st.bounce (path_integ_naive.glsl:97-133)
        v3 wi = st.ray.dir;
        int lightId = id - sc.objPrimCount;
        if (id == -1) {
            v3 radiance = envLe(sc, wi);
            float weight = 1.0f;
            if (pp.sampleLight && !st.delta) {
                float envPdf = envPdfLi(sc, wi) * (pp.uniformSel ? (1.0f - pp.portion)
                                                                 : sc.envSum / (sc.lightSum + sc.envSum));
                weight = (envPdf <= 0.0f) ? 0.0f : biHeuristic(st.bsdfPdf, envPdf);
            }
            st.result = st.result + radiance * st.throughput * weight;
            return false;
        }
        if (lightId >= 0) {
            v3 radiance = lightLe(sc, lightId, hitPos, -wi);
            float weight = 1.0f;
            if (pp.sampleLight && !st.delta) {
                float snd = pp.uniformSel ? pp.portion : sc.lightSum / (sc.lightSum + sc.envSum);
                float lightPdf = lightPdfLi(sc, lightId, st.pos, hitPos) * (lightPdfSampleOne(sc, lightId) * snd);
                weight = (lightPdf <= 0.0f) ? 0.0f : biHeuristic(st.bsdfPdf, lightPdf);
            }
            st.result = st.result + radiance * st.throughput * weight;
            return false;
        }
        if (pp.rr && st.bounce >= pp.rrStart) {
            float continueProb = zmin(maxComponent(st.bsdfOverPdf), 0.95f);
            if (sample1D(g) >= continueProb) return false;
            st.throughput = st.throughput / continueProb;
        }
        st.wo = -wi;
    }
    // next bounce at the new vertex
    st.bounce++;
    if (st.bounce > pp.maxDepth) return false;
    st.pos = hitPos;
    TriShade tri = loadTri(sc, id);
    Surface surf = surfaceInfo(tri, hitPos);
    int matId = tri.matTex & 0x0000ffff;
    uint32_t matType = loadMaterialType(sc, matId);
    if (matType != kDielectric && matType != kThinDielectric && dot(surf.ns, st.wo) < 0.0f) {
        surf.ns = -surf.ns;
        surf.ng = -surf.ng;
    }
    BSDFParam mp = loadMaterial<FULL>(sc, matType, tri.matTex, id, surf);
    if (pp.sampleLight) {
        float ud = sample1D(g);
        float u0 = sample1D(g), u1 = sample1D(g), u2 = sample1D(g),
              u3 = sample1D(g);
        LiSample ls;
        if (DEFER) ls = sampleLightAndEnvV(sc, pp, hitPos, ud, u0, u1, u2, u3, DeferVis{ps});
        else ls = sampleLightAndEnvV(sc, pp, hitPos, ud, u0, u1, u2, u3, TraceVis{});
        if (ls.pdf > 0.0f) {
            v3 f = materialBSDF<FULL>(matType, mp, st.wo, ls.wi, surf.ns);
            float fpdf = materialPdf<FULL>(matType, mp, st.wo, ls.wi, surf.ns);
            float weight = biHeuristic(ls.pdf, fpdf);
            const v3 C = f * st.throughput * satDot(surf.ns, ls.wi) * ls.coef * weight;
            if (DEFER) {
                ps->C = C;
                ps->pending = true;
            } else {
                st.result = st.result + C;
            }
        }
    }
    float b0 = sample1D(g), b1 = sample1D(g), b2 = sample1D(g);
    BSDFSample bs = materialSample<FULL>(matType, mp, surf.ns, st.wo, mk3(b0, b1, b2), g);
    st.delta = (bs.flag == kSpecRefl || bs.flag == kSpecTrans);
    if (bs.pdf < 1e-8f) return false;
    st.throughput = st.throughput * (bs.bsdf / bs.pdf * (st.delta ? 1.0f : absDot(surf.ns, bs.wi)));
    st.bsdfPdf = bs.pdf;
    st.bsdfOverPdf = bs.bsdf / bs.pdf;
    st.ray = rayOffseted(hitPos, bs.wi);
    return true;
}

}  // namespace
}  // namespace zgl
