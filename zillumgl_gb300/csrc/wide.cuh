// wide.cuh — device-side traversal of the 4-wide tree (accel.h: DeviceAccel
// wide / wtris), the trace kernels' and integrators' closest-hit and any-hit
// path.
//
// The reference's threaded loop (traverse.cuh: traverse_m) visits about 160
// binary table entries per ray, one dependent 32-byte load each.  Here one
// node holds the four grandchildren of a binary node: a ray visits a quarter
// as many nodes, from one table that serves all six faces (64 B per two
// binary levels, against six tables of 32 B per binary node).  Hit ids and
// distances are the reference's, bit for bit:
//
//  * Order.  A node's children are visited in the order of the ray's face
//    table (three swap bits per face), so leaves come in the reference's
//    order and strict `t < dist` resolves ties the same way.
//  * Superset.  Child boxes are stored in 8 bits per plane, rounded outwards
//    to a grid of whole float32 numbers.  A child is entered when
//    max(tmin, 0) <= min(tmax, dist) with boxHit's float32 slab formula on the
//    larger box.  Subtracting the origin and multiplying by a fixed reciprocal
//    are monotone in float32, so everything boxHit accepts passes; distances
//    only shrink between the test of a child and the reference's visit of it.
//  * Acceptance.  A triangle counts only if boxHit accepts its leaf box and
//    !(tmin > dist) there, both evaluated as the reference does on the exact
//    box.  Of its ancestors the reference also asks boxHit and !(tmin > dist).
//    By the same monotony a box inside another never has the smaller tmin or
//    the larger tmax: the ancestors' distance tests and slab overlaps follow
//    from the leaf's.  Not monotone are the three conditions of the general branch
//    (dy + dz > fz - ny and its rotations: fy > nz up to rounding).  In exact
//    arithmetic the ancestors' slack is at least the leaf's; the rounding of
//    one condition is below 5 u (Y + Z), u = 2^-24, where Y and Z bound the
//    slab values on the two axes, for which the root's values serve.  A leaf
//    slack above 8 u (Y + Z) therefore settles all ancestors.  Otherwise
//    (1 accept in 10^4 to 10^5 on the soups and the city) chain_accepts
//    evaluates boxHit on every ancestor.
//
// Rays with one near-zero component (MODE 4 with one flag).  boxHit ignores
// that axis (say x), so the reference enters every box along the whole line
// in x: tens of thousands.  Such a box cannot hold a hit unless it is near
// the ray in x.  Let L bound the distance from the origin to any point of the
// tree and l = max(|ab|, |ac|) of a triangle; all components of d are below
// 1.  Counting roundings (u = 2^-24), tri_test's u and v are within 13 u L l
// of their exact values and det within 12 u l^2; so for l^2 < 0.7, where det
// passing 1e-6 means an exact det above 0.5e-6, the line meets the triangle's
// plane within 78 u L l^2 / 0.5e-6 < 10 L l^2 of the triangle.  Up to there x
// moves by at most 1e-6 times the ray parameter, which is below 16 L because
// another component is at least 1/2.  So a child farther from the origin in x
// than P = 3e-5 (L + |ox|) + 12 L l^2 holds no triangle that tri_test
// accepts, and is skipped (l^2 is the largest squared triangle box diagonal
// in the node's subtree; from 0.7 on nothing is skipped).  Rays of modes 0-2
// (axis-dominant) use the same code with P = 0: boxHit itself asks the origin
// to lie inside the box on the other two axes.
//
// All other rays (two near-zero components but none dominant, NaN, very far
// origins) and trees too deep for the stack keep the reference loop.
#pragma once

#include "traverse.cuh"

namespace zgl {

constexpr int kWideStack = 64;            // entries per thread (local memory)
constexpr int kWideDone = (int)0x80000000;  // bottom of the stack
// Nodes a ray of the rarer modes visits on its lane before its warp takes it
// over on the face table: on meshes of small triangles, where P binds, such a
// ray needs a few hundred; with large ones, tens of thousands.  1M camera rays
// with a column of 1100 such rays, 1M triangles: 6.4 ms at 256 nodes, 0.99,
// 0.99, 0.98 at 1024, 4096, 16384; 16M shadow rays 12.8, 6.42, 6.36, 6.39.
// Trees whose root says that P cannot bind everywhere (a triangle with a
// squared box diagonal of 0.7 or more) get kLongRayBudget.
constexpr int kPadBudget = 4096;

// Result of one wide traversal: `ok` false when the stack ran out or a ray of
// the rarer modes outran kPadBudget nodes (triangles too large for P to
// bind); the caller starts over with the reference loop.
struct WideHit {
    int id;
    float dist;
    bool ok;
};

__device__ __forceinline__ float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// Slab values of one plane of the four children: byte j of `q` is child j's
// grid index, its plane is f * s + g with f = 2^23 + index (exact, so is the
// plane), the slab value (plane - o) * inv with two roundings, as boxHit has.
__device__ __forceinline__ float4 slab4(unsigned q, float s, float g, float no, float inv) {
    const unsigned f0 = __byte_perm(q, 0x4b000000u, 0x7540), f1 = __byte_perm(q, 0x4b000000u, 0x7541);
    const unsigned f2 = __byte_perm(q, 0x4b000000u, 0x7542), f3 = __byte_perm(q, 0x4b000000u, 0x7543);
    float4 r;
    asm("{\n\t.reg .b64 a, b, s, g, o, i;\n\t"
        "mov.b64 a, {%4, %5};\n\tmov.b64 b, {%6, %7};\n\tmov.b64 s, {%8, %8};\n\tmov.b64 g, {%9, %9};\n\t"
        "mov.b64 o, {%10, %10};\n\tmov.b64 i, {%11, %11};\n\t"
        "fma.rn.f32x2 a, a, s, g;\n\tfma.rn.f32x2 b, b, s, g;\n\t"
        "add.rn.f32x2 a, a, o;\n\tadd.rn.f32x2 b, b, o;\n\t"
        "mul.rn.f32x2 a, a, i;\n\tmul.rn.f32x2 b, b, i;\n\t"
        "mov.b64 {%0, %1}, a;\n\tmov.b64 {%2, %3}, b;\n\t}"
        : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
        : "r"(f0), "r"(f1), "r"(f2), "r"(f3), "f"(s), "f"(g), "f"(no), "f"(inv));
    return r;
}
// 32 bytes in one load: the L1 serves a gather one lane at a time whatever its
// width, so wide loads are what a divergent traversal saves it by.
__device__ __forceinline__ void load32(const void* p, unsigned (&v)[8]) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
        : "l"(p));
}

// Whether the wide traversal covers a ray (see the head of this file).
__device__ __forceinline__ bool wide_covers(const TraceRay& r) {
    const float far = 1e12f;
    if (!(fabsf(r.o.x) < far && fabsf(r.o.y) < far && fabsf(r.o.z) < far)) return false;
    const float ax = fabsf(r.d.x), ay = fabsf(r.d.y), az = fabsf(r.d.z);
    if (r.mode == 3) return ax >= 1e-6f && ay >= 1e-6f && az >= 1e-6f;  // false for NaN
    if (r.mode == 4) return (int)r.sx + (int)r.sy + (int)r.sz == 1 && (ax >= 0.5f || ay >= 0.5f || az >= 0.5f) &&
                            ax + ay + az < 4.0f;
    return ax + ay + az < 1e30f;
}

// boxHit on every ancestor of the triangle in leaf slot `slot` (the leaf
// itself excluded), from the root down.
static __device__ __noinline__ bool chain_accepts(const float4* dfs, int slot, float3 o, float3 d) {
    const TraceRay r = make_trace_ray(o, d);
    int64_t k = 0;
    float4 lo = __ldg(dfs), hi = __ldg(dfs + 1);
    while (!(__float_as_uint(lo.w) & 0x80000000u)) {
        float tmin;
        if (!box_hit(lo, hi, r, tmin)) return false;
        k++;
        lo = __ldg(dfs + 2 * k);
        hi = __ldg(dfs + 2 * k + 1);
        // the second child when the slot is beyond the first one's leaves
        const unsigned w = __float_as_uint(lo.w);
        const int64_t size = (w & 0x80000000u) ? 1 : (int64_t)w;
        if ((int64_t)(__float_as_uint(hi.w) & 0x7fffffffu) + (size + 1) / 2 <= slot) {
            k += size;
            lo = __ldg(dfs + 2 * k);
            hi = __ldg(dfs + 2 * k + 1);
        }
    }
    return true;
}

// Whether a leaf's slack settles the ancestors' conditions (head of this
// file); lo / hi is the leaf box, the root's box comes from entry 0 of the
// first face table.
__device__ __forceinline__ bool leaf_settles(const DeviceAccel& a, const float4 lo, const float4 hi,
                                             const TraceRay& r) {
    const float4 rl = __ldg(a.nodes), rh = __ldg(a.nodes + 1);
    const float3 o = r.o, i = r.dinv;
    const float ax = (lo.x - o.x) * i.x, bx = (hi.x - o.x) * i.x;
    const float ay = (lo.y - o.y) * i.y, by = (hi.y - o.y) * i.y;
    const float az = (lo.z - o.z) * i.z, bz = (hi.z - o.z) * i.z;
    const float X = fmaxf(fabsf((rl.x - o.x) * i.x), fabsf((rh.x - o.x) * i.x));
    const float Y = fmaxf(fabsf((rl.y - o.y) * i.y), fabsf((rh.y - o.y) * i.y));
    const float Z = fmaxf(fabsf((rl.z - o.z) * i.z), fabsf((rh.z - o.z) * i.z));
    const float e = 4.76837158203125e-7f;  // 8 u
    const bool yz = fmaxf(ay, by) - fminf(az, bz) > e * (Y + Z);
    const bool zx = fmaxf(az, bz) - fminf(ax, bx) > e * (Z + X);
    const bool xy = fmaxf(ax, bx) - fminf(ay, by) > e * (X + Y);
    if (r.mode == 4) return r.sx ? yz : r.sy ? zx : xy;
    return r.mode < 3 || (yz && zx && xy);
}

// What the wide traversal of a ray beyond mode 3 needs beside the ray.
struct WidePad {
    float ix, iy, iz;  // reciprocal per axis
    float padA, padB;
    bool px, py, pz;

    __device__ __forceinline__ void set(const DeviceAccel& a, const TraceRay& r) {
        // an axis boxHit does not measure along becomes an inside test: any
        // difference times infinity is decisive, however small, and the NaN
        // of a zero difference is dropped by max and min (the child is then
        // entered, a superset)
        const float pass = __int_as_float(0x7f800000);
        px = r.mode == 4 ? r.sx : r.mode != 0;
        py = r.mode == 4 ? r.sy : r.mode != 1;
        pz = r.mode == 4 ? r.sz : r.mode != 2;
        ix = px ? pass : r.dinv.x;
        iy = py ? pass : r.dinv.y;
        iz = pz ? pass : r.dinv.z;
        padA = padB = 0.0f;
        if (r.mode == 4) {
            const float4 rl = __ldg(a.nodes), rh = __ldg(a.nodes + 1);
            const float3 o = r.o;
            const float L = fmaxf(fabsf(rl.x - o.x), fabsf(rh.x - o.x)) + fmaxf(fabsf(rl.y - o.y), fabsf(rh.y - o.y)) +
                            fmaxf(fabsf(rl.z - o.z), fabsf(rh.z - o.z));
            padA = 3e-5f * (L + fabsf(r.sx ? o.x : r.sy ? o.y : o.z));
            padB = 12.0f * L;
        }
    }
};

// One node: tests its four children and replaces the reference on top of the
// stack (`cur`, an inner node; the rest in `stack`, `sp` entries) by those
// entered, in visiting order.  PAD = false: rays of mode 3; PAD = true: every
// other ray that wide_covers admits.
template <bool PAD>
__device__ __forceinline__ void wide_node(const float4* wide, const float3 o, const float3 inv, int face,
                                          const WidePad& w, float dist, int* stack, int& sp, int& cur) {
    const float4* const n = wide + (size_t)(unsigned)cur * 4;
    unsigned u[8], v[8];
    load32(n, u);
    load32(n + 2, v);
    const float gx = __uint_as_float(u[0]), gy = __uint_as_float(u[1]), gz = __uint_as_float(u[2]);
    const float sx = __uint_as_float((u[3] << 23) & 0x7f800000u);
    const float sy = __uint_as_float((u[3] << 15) & 0x7f800000u);
    const float sz = __uint_as_float((u[3] << 7) & 0x7f800000u);
    // one axis after the other, so that eight running bounds are live instead
    // of 24 slab values (48 registers a thread)
    float4 tn, tf;
    {
        const float inx = PAD ? w.ix : inv.x, iny = PAD ? w.iy : inv.y, inz = PAD ? w.iz : inv.z;
        float pad = 0.0f;
        if (PAD) {
            const float l2 = __uint_as_float((u[3] >> 1) & 0x7f800000u);
            pad = l2 < 0.7f ? w.padA + w.padB * l2 : 1e30f;
        }
        const bool bx = inx < 0.0f, by = iny < 0.0f, bz = inz < 0.0f;
        const float xn = PAD && w.px ? -(o.x + pad) : -o.x, xf = PAD && w.px ? -(o.x - pad) : -o.x;
        tn = slab4(bx ? v[1] : v[0], sx, gx, xn, inx);
        tf = slab4(bx ? v[0] : v[1], sx, gx, xf, inx);
        const float yn = PAD && w.py ? -(o.y + pad) : -o.y, yf = PAD && w.py ? -(o.y - pad) : -o.y;
        float4 q = slab4(by ? v[3] : v[2], sy, gy, yn, iny);
        tn = make_float4(fmaxf(tn.x, q.x), fmaxf(tn.y, q.y), fmaxf(tn.z, q.z), fmaxf(tn.w, q.w));
        q = slab4(by ? v[2] : v[3], sy, gy, yf, iny);
        tf = make_float4(fminf(tf.x, q.x), fminf(tf.y, q.y), fminf(tf.z, q.z), fminf(tf.w, q.w));
        const float zn = PAD && w.pz ? -(o.z + pad) : -o.z, zf = PAD && w.pz ? -(o.z - pad) : -o.z;
        q = slab4(bz ? v[5] : v[4], sz, gz, zn, inz);
        tn = make_float4(max3f(tn.x, q.x, 0.0f), max3f(tn.y, q.y, 0.0f), max3f(tn.z, q.z, 0.0f), max3f(tn.w, q.w, 0.0f));
        q = slab4(bz ? v[4] : v[5], sz, gz, zf, inz);
        tf = make_float4(min3f(tf.x, q.x, dist), min3f(tf.y, q.y, dist), min3f(tf.z, q.z, dist), min3f(tf.w, q.w, dist));
    }
    // child reference, 0 (the root, never a child; also an empty slot) where missed
    int r0 = tn.x <= tf.x ? (int)u[4] : 0;
    int r1 = tn.y <= tf.y ? (int)u[5] : 0;
    int r2 = tn.z <= tf.z ? (int)u[6] : 0;
    int r3 = tn.w <= tf.w ? (int)u[7] : 0;
    // visiting order of the ray's face
    const unsigned swaps = v[6] >> (3 * face);
    const int q0 = (swaps & 1u) ? r1 : r0, q1 = (swaps & 1u) ? r0 : r1;
    const int q2 = (swaps & 2u) ? r3 : r2, q3 = (swaps & 2u) ? r2 : r3;
    r0 = (swaps & 4u) ? q2 : q0;
    r1 = (swaps & 4u) ? q3 : q1;
    r2 = (swaps & 4u) ? q0 : q2;
    r3 = (swaps & 4u) ? q1 : q3;
    cur = stack[--sp];
    if (r3) { stack[sp++] = cur; cur = r3; }
    if (r2) { stack[sp++] = cur; cur = r2; }
    if (r1) { stack[sp++] = cur; cur = r1; }
    if (r0) { stack[sp++] = cur; cur = r0; }
}

// One triangle (rays of mode 3) against the reference: 0 not taken, 1 taken at
// distance t, 2 taken if the ancestors' conditions hold, which the leaf's
// slack leaves open.
__device__ __forceinline__ int wide_leaf(const DeviceAccel& a, const float3 o, const float3 inv, const float3 d, int ref,
                                         float dist, float& t, int& prim) {
    const float4* const tr = a.wtris + (size_t)(unsigned)~ref * 4;
    unsigned u[8], v[8];
    load32(tr, u);
    load32(tr + 2, v);
    const auto f = [](unsigned x) { return __uint_as_float(x); };
    prim = (int)v[1];
    if (!tri_test(make_float4(f(u[0]), f(u[1]), f(u[2]), f(u[3])), make_float4(f(u[4]), f(u[5]), f(u[6]), f(u[7])),
                  make_float4(f(v[0]), 0.0f, 0.0f, 0.0f), o, d, t) ||
        !(t < dist))
        return 0;
    TraceRay r;
    r.o = o;
    r.dinv = inv;
    r.mode = 3;
    const float4 lo = make_float4(f(v[2]), f(v[3]), f(v[4]), 0.0f);
    const float4 hi = make_float4(f(v[5]), f(v[6]), f(v[7]), 0.0f);
    float tmin;
    if (!box_hit_m<3>(lo, hi, r, tmin) || tmin > dist) return 0;
    return leaf_settles(a, lo, hi, r) ? 1 : 2;
}

// The same for any ray that wide_covers admits, the ancestors included.
__device__ __forceinline__ bool wide_leaf_any_mode(const DeviceAccel& a, const TraceRay& r, int ref, float dist,
                                                   float& t, int& prim) {
    const int slot = ~ref;
    const float4* const tr = a.wtris + (size_t)(unsigned)slot * 4;
    const float4 t2 = __ldg(tr + 2), t3 = __ldg(tr + 3);
    prim = __float_as_int(t2.y);
    if (!tri_test(__ldg(tr), __ldg(tr + 1), t2, r.o, r.d, t) || !(t < dist)) return false;
    const float4 lo = make_float4(t2.z, t2.w, t3.x, 0.0f), hi = make_float4(t3.y, t3.z, t3.w, 0.0f);
    float tmin;
    return box_hit(lo, hi, r, tmin) && !(tmin > dist) &&
           (leaf_settles(a, lo, hi, r) || chain_accepts(a.dfs, slot, r.o, r.d));
}

// Closest hit (ANY = false) or any hit closer than `dist` of one ray.
template <bool ANY, bool PAD>
__device__ __forceinline__ WideHit traverse_wide(const DeviceAccel& a, const TraceRay& r, float dist) {
    int stack[kWideStack];
    WidePad w;
    if (PAD) w.set(a, r);
    int closest = -1, sp = 1, cur = 0, nodes = 0, budget = kPadBudget;
    if (PAD && ((__float_as_uint(__ldg(reinterpret_cast<const float*>(a.wide) + 3)) >> 1) & 0x7f800000u) >=
                   __float_as_uint(1.0f))
        budget = kLongRayBudget;  // the root's l^2 passes 0.7
    stack[0] = kWideDone;
    for (;;) {
        while (cur >= 0) {
            if (sp > kWideStack - 4 || (PAD && ++nodes > budget)) return WideHit{-1, dist, false};
            wide_node<PAD>(a.wide, r.o, r.dinv, r.face, w, dist, stack, sp, cur);
        }
        if (cur == kWideDone) break;
        float t;
        int prim;
        if (wide_leaf_any_mode(a, r, cur, dist, t, prim)) {
            closest = prim;
            dist = t;
            if (ANY) break;
        }
        cur = stack[--sp];
    }
    return WideHit{closest, dist, true};
}

// Rays that the wide tree's loop leaves out, marked by `want`: one per lane on
// the wide tree, those it does not cover on the face table; those that outrun
// kPadBudget nodes or kLongRayBudget entries there, or the stack, on the face
// table with the whole warp.  Every lane calls.
template <bool ANY>
__device__ __forceinline__ bool lane_walk(const DeviceAccel& a, const TraceRay& r, float& dist, int& k, int& closest,
                                          int budget) {
    return budget > 0 && traverse_lane_m<ANY, false, 0>(a, r, dist, k, closest, budget);
}
template <class Io>
static __device__ __noinline__ void wide_rest(DeviceAccel a, Io io, int i, bool want) {
    const bool any = want && io.any(i);
    const TraceRay r = make_trace_ray(want ? io.origin(i) : make_float3(0.0f, 0.0f, 0.0f),
                                      want ? io.direction(i) : make_float3(0.0f, 0.0f, 1.0f));
    float dist = want ? io.limit(i) : 0.0f;
    int closest = -1;
    bool done = !want;
    int budget = kLongRayBudget;
    if (want && wide_covers(r)) {
        budget = 0;  // what stays unfinished here goes to the warp at once
        WideHit h;
        if (r.mode == 3) h = any ? traverse_wide<true, false>(a, r, dist) : traverse_wide<false, false>(a, r, dist);
        else h = any ? traverse_wide<true, true>(a, r, dist) : traverse_wide<false, true>(a, r, dist);
        if (h.ok) {
            closest = h.id;
            dist = h.dist;
            done = true;
        }
    }
    if (!__all_sync(0xffffffffu, done)) {
        int k = 0, k2 = 0;
        bool done1 = done || any, done2 = done || !any;
        if (Io::kClosest) {
            done1 = done1 || lane_walk<false>(a, r, dist, k, closest, budget);
            finish_long_rays<false>(a, r, dist, k, closest, done1);
        }
        if (Io::kAny) {
            done2 = done2 || lane_walk<true>(a, r, dist, k2, closest, budget);
            finish_long_rays<true>(a, r, dist, k2, closest, done2);
        }
    }
    if (want) io.store(i, closest, dist);
}

// Closest or any hit of n rays, one grid.  Io says what ray i is and takes its
// result:
//   kClosest, kAny    which queries occur
//   any(i)            whether ray i asks for any hit
//   origin, direction, limit(i)  the ray (limit: 1e8 or the any-hit distance)
//   store(i, id, t)   id -1: nothing hit
//   mark(i), marked(i)  sets ray i aside: a value its result never has
//
// Divergence is what this loop fights.  Rays of one warp visit between a few
// and 400 nodes (mean 31 on the 4M soup's bounce rays, 4 triangles); one ray
// per thread to the end kept 5.5 lanes busy and ran at 740 Mrays/s.  So
//  * the grid is one wave of resident warps, each taking every nwarps-th group
//    of 32 rays; lanes without a ray are refilled from the sequence once
//    kRefill of them are idle (no counter in memory, so launches on other
//    streams and in graphs stay independent).  256 consecutive rays per warp
//    instead: 1083 Mrays/s against 1268 (its tails come once a launch);
//  * a lane that reaches a triangle sets it aside and goes on with the nodes
//    behind it (a later, larger distance only adds nodes; triangles are still
//    tested in order).  The warp turns to the waiting triangles when fewer
//    than kInner lanes have a node left, counted every second node (4M bounce
//    rays: 12 lanes 2.83, 16 2.65, 20 2.55 ms, counting every node; every
//    second 2.55 at 16, 2.54 at 20, 2.49 at 22 with refills from 6 idle lanes;
//    24 lanes is faster on the large soup only).  With fewer rays the number
//    goes down with them: 65k rays on 4096 triangles 98 -> 93 us, a
//    256x256 Cornell pass (six launches) 453 -> 424 us.
// 64-byte nodes in two 32-byte loads: with 128-byte nodes of full floats in
// eight 16-byte loads the L1 was 70% busy (a gather takes a cycle a lane) and
// the same loop ran at 760 Mrays/s.  No call in the loop: 1268 -> 1601 Mrays/s
// (see its end).  48 registers (20 blocks of 64 threads per SM) hide more
// latency than 56 (1485) and 40 (1447).  4M soup, 4M bounce rays: 2.49 ms,
// 7.35 before on the threaded tables; at 2.62 ms issue slots 61% and L1 66% busy, 19 of
// 32 lanes active.
constexpr int kWideBlock = 64;
constexpr int kWideBlocksPerSM = 20;
constexpr int64_t kWideMaxRays = int64_t(1) << 30;  // of one grid
constexpr int kInner = 22;
constexpr int kRefill = 6;

// Rays per warp and round: 32, fewer when n does not give 32 to kThinWarps
// warps per SM (see wide_blocks).
constexpr int kThinWarps = 16;
__host__ __device__ __forceinline__ int wide_group(int64_t n, int sms) {
    const int64_t g = (n + (int64_t)sms * kThinWarps - 1) / ((int64_t)sms * kThinWarps);
    return (int)(g < 1 ? 1 : g > 32 ? 32 : g);
}
// Blocks of kWideBlock threads for up to n rays (a kernel that gets a smaller
// number from the device takes wide_group of that): one wave of resident
// warps, and never fewer warps than wide_group counts on.  Rays
// too few for 16 warps of 32 per SM are spread thinner over 16 warps per SM,
// so that they do not wait for each other's branches (997 rays on 2048
// triangles 76 -> 55 us, 5000 on 1M 237 -> 198 us with the whole launch, at
// eight warps).  With 8, 16, 24 and 40 warps per SM, us: 20000 rays on 4096
// triangles 74, 64, 72, 81, on 4M 866, 699, 651, 653; 65536 rays 95, 87, 103,
// 124 and 1113, 1088, 1032, 1231: full warps share their loads.
inline unsigned wide_blocks(int64_t n, int sms) {
    const int64_t warps = (int64_t)sms * kWideBlocksPerSM * (kWideBlock / 32);
    const int64_t full = (n + 31) / 32 > (int64_t)sms * kThinWarps ? (n + 31) / 32 : (int64_t)sms * kThinWarps;
    int64_t used = full < warps ? full : warps;
    used = n < used ? n : used;
    return (unsigned)((used + kWideBlock / 32 - 1) / (kWideBlock / 32));
}

//
// Every round of the loop makes progress: it takes new rays, steps a node, or
// tests a triangle.  The node loop is left before
// a step only for a waiting triangle, or when kRefill lanes are free or about
// to be, which the next round refills.
template <class Io>
__device__ __forceinline__ void wide_trace(const DeviceAccel& a, const Io& io, int n, int group) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    // ray p of this warp's sequence is ray ((p / 32) * nwarps + warp) * 32 +
    // p % 32; with fewer rays than that takes, the warp has `group` of them
    const int warp = (int)(blockIdx.x * (kWideBlock / 32) + (threadIdx.x >> 5));
    const int stride = (int)(gridDim.x * kWideBlock);
    int taken = 0;
    bool more = warp * group < n;
    int stack[kWideStack];
    stack[0] = kWideDone;
    int ray = 0;
    float3 o = make_float3(0.0f, 0.0f, 0.0f), inv = o;
    const WidePad none{};
    float dist = 0.0f;
    int face = 0, closest = -1, sp = 1, cur = kWideDone, leaf = 0;
    bool live = false, rest = false;  // rest: this lane set a ray aside
    for (;;) {
        // refill the lanes without a ray
        const unsigned idle = __ballot_sync(full, !live);
        if (idle == full && !more) break;
        if (more && __popc(idle) >= kRefill) {
            const int p = taken + __popc(idle & lt);
            int mine;
            if (group == 32) {
                mine = (p >> 5) * stride + warp * 32 + (p & 31);
                taken += __popc(idle);
                more = (taken >> 5) * stride + warp * 32 + (taken & 31) < n;
            } else {
                mine = p < group ? warp * group + p : n;
                more = false;
            }
            if (!live && mine < n) {
                ray = mine;
                const TraceRay r = make_trace_ray(io.origin(ray), io.direction(ray));
                if (r.d.x == 0.0f && r.d.y == 0.0f && r.d.z == 0.0f) {
                    // det is 0 for every triangle: nothing is hit (a BSDF
                    // sample below the horizon leaves such a ray)
                    io.store(ray, -1, io.limit(ray));
                } else if (r.mode == 3 && wide_covers(r)) {
                    o = r.o;
                    inv = r.dinv;
                    face = r.face;
                    dist = io.limit(ray);
                    closest = -1;
                    sp = 1;
                    cur = 0;
                    live = true;
                } else {
                    io.mark(ray);
                    rest = true;
                }
            }
        }
        // of the lanes with a ray: few have any in a small launch, and at the end
        const int few = min(kInner, 27 * __popc(__ballot_sync(full, live)) >> 5);
        // nodes, until few lanes have one and some wait with a triangle or
        // could be refilled
        for (;;) {
            const unsigned inner = __ballot_sync(full, cur >= 0);
            if (inner == 0u) break;
            if (__popc(inner) < few &&
                (__any_sync(full, leaf != 0) || (more && __popc(__ballot_sync(full, cur == kWideDone)) >= kRefill)))
                break;
#pragma unroll
            for (int twice = 0; twice < 2; twice++) {
                if (cur < 0) continue;
                if (sp > kWideStack - 4) {
                    io.mark(ray);
                    rest = true;
                    live = false;
                    cur = kWideDone;
                    leaf = 0;
                } else {
                    wide_node<false>(a.wide, o, inv, face, none, dist, stack, sp, cur);
                    if (cur < 0 && cur != kWideDone && leaf == 0) {
                        leaf = cur;
                        cur = stack[--sp];
                    }
                }
            }
        }
        // the waiting triangles
        if (leaf != 0) {
            float t;
            int prim;
            const int take = wide_leaf(a, o, inv, io.direction(ray), leaf, dist, t, prim);
            leaf = 0;
            if (take == 1) {
                closest = prim;
                dist = t;
                if (io.any(ray)) cur = kWideDone;
            } else if (take == 2) {
                io.mark(ray);
                rest = true;
                live = false;
                cur = kWideDone;
            }
            if (cur < 0 && cur != kWideDone) {
                leaf = cur;
                cur = stack[--sp];
            }
        }
        if (live && cur == kWideDone && leaf == 0) {
            io.store(ray, closest, dist);
            live = false;
        }
    }
    // the rays set aside.  A call inside the loop made the compiler keep eight
    // of its values in local memory (58 million reloads in a 1.1 billion
    // instruction launch); here nothing is live across it.
    if (!__any_sync(full, rest)) return;
    __syncwarp();  // the marks are other lanes' stores
    for (int at = 0;; at++) {
        const int i = group == 32 ? at * stride + warp * 32 + lane : at == 0 && lane < group ? warp * group + lane : n;
        if (!__any_sync(full, i < n)) break;
        const bool want = i < n && io.marked(i);
        if (__any_sync(full, want)) wide_rest(a, io, i, want);
    }
}

}  // namespace zgl
