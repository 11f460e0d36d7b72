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

// Result of one wide traversal: `ok` false when the stack ran out (the caller
// starts over with the reference loop).
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
static __device__ __noinline__ bool chain_accepts(const float4* dfs, int slot, TraceRay r) {
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
        // difference times 1e30 is below 0 or beyond every distance
        px = r.mode == 4 ? r.sx : r.mode != 0;
        py = r.mode == 4 ? r.sy : r.mode != 1;
        pz = r.mode == 4 ? r.sz : r.mode != 2;
        ix = px ? 1e30f : r.dinv.x;
        iy = py ? 1e30f : r.dinv.y;
        iz = pz ? 1e30f : r.dinv.z;
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
__device__ __forceinline__ void wide_node(const float4* wide, const TraceRay& r, const WidePad& w, float dist,
                                          int* stack, int& sp, int& cur) {
    const float4* const n = wide + (size_t)(unsigned)cur * 4;
    unsigned u[8], v[8];
    load32(n, u);
    load32(n + 2, v);
    const float gx = __uint_as_float(u[0]), gy = __uint_as_float(u[1]), gz = __uint_as_float(u[2]);
    const float sx = __uint_as_float((u[3] << 23) & 0x7f800000u);
    const float sy = __uint_as_float((u[3] << 15) & 0x7f800000u);
    const float sz = __uint_as_float((u[3] << 7) & 0x7f800000u);
    float4 nx, ny, nz, fx, fy, fz;
    if (PAD) {
        const float l2 = __uint_as_float((u[3] >> 1) & 0x7f800000u);
        const float pad = l2 < 0.7f ? w.padA + w.padB * l2 : 1e30f;
        const bool bx = w.ix < 0.0f, by = w.iy < 0.0f, bz = w.iz < 0.0f;
        nx = slab4(bx ? v[1] : v[0], sx, gx, w.px ? -(r.o.x + pad) : -r.o.x, w.ix);
        fx = slab4(bx ? v[0] : v[1], sx, gx, w.px ? -(r.o.x - pad) : -r.o.x, w.ix);
        ny = slab4(by ? v[3] : v[2], sy, gy, w.py ? -(r.o.y + pad) : -r.o.y, w.iy);
        fy = slab4(by ? v[2] : v[3], sy, gy, w.py ? -(r.o.y - pad) : -r.o.y, w.iy);
        nz = slab4(bz ? v[5] : v[4], sz, gz, w.pz ? -(r.o.z + pad) : -r.o.z, w.iz);
        fz = slab4(bz ? v[4] : v[5], sz, gz, w.pz ? -(r.o.z - pad) : -r.o.z, w.iz);
    } else {
        const bool bx = r.dinv.x < 0.0f, by = r.dinv.y < 0.0f, bz = r.dinv.z < 0.0f;
        nx = slab4(bx ? v[1] : v[0], sx, gx, -r.o.x, r.dinv.x);
        fx = slab4(bx ? v[0] : v[1], sx, gx, -r.o.x, r.dinv.x);
        ny = slab4(by ? v[3] : v[2], sy, gy, -r.o.y, r.dinv.y);
        fy = slab4(by ? v[2] : v[3], sy, gy, -r.o.y, r.dinv.y);
        nz = slab4(bz ? v[5] : v[4], sz, gz, -r.o.z, r.dinv.z);
        fz = slab4(bz ? v[4] : v[5], sz, gz, -r.o.z, r.dinv.z);
    }
    // child reference, 0 (the root, never a child; also an empty slot) where missed
    int r0 = fmaxf(max3f(nx.x, ny.x, nz.x), 0.0f) <= fminf(min3f(fx.x, fy.x, fz.x), dist) ? (int)u[4] : 0;
    int r1 = fmaxf(max3f(nx.y, ny.y, nz.y), 0.0f) <= fminf(min3f(fx.y, fy.y, fz.y), dist) ? (int)u[5] : 0;
    int r2 = fmaxf(max3f(nx.z, ny.z, nz.z), 0.0f) <= fminf(min3f(fx.z, fy.z, fz.z), dist) ? (int)u[6] : 0;
    int r3 = fmaxf(max3f(nx.w, ny.w, nz.w), 0.0f) <= fminf(min3f(fx.w, fy.w, fz.w), dist) ? (int)u[7] : 0;
    // visiting order of the ray's face
    const unsigned swaps = v[6] >> (3 * r.face);
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

// One triangle: whether the reference would take it at distance `dist`.
template <bool PAD>
__device__ __forceinline__ bool wide_leaf(const DeviceAccel& a, const TraceRay& r, int ref, float dist, float& t,
                                          int& prim) {
    const int slot = ~ref;
    const float4* const tr = a.wtris + (size_t)(unsigned)slot * 4;
    unsigned u[8], v[8];
    load32(tr, u);
    load32(tr + 2, v);
    const auto f = [](unsigned x) { return __uint_as_float(x); };
    prim = (int)v[1];
    if (!tri_test(make_float4(f(u[0]), f(u[1]), f(u[2]), f(u[3])), make_float4(f(u[4]), f(u[5]), f(u[6]), f(u[7])),
                  make_float4(f(v[0]), 0.0f, 0.0f, 0.0f), r, t) ||
        !(t < dist))
        return false;
    const float4 lo = make_float4(f(v[2]), f(v[3]), f(v[4]), 0.0f);
    const float4 hi = make_float4(f(v[5]), f(v[6]), f(v[7]), 0.0f);
    float tmin;
    return (PAD ? box_hit(lo, hi, r, tmin) : box_hit_m<3>(lo, hi, r, tmin)) && !(tmin > dist) &&
           (leaf_settles(a, lo, hi, r) || chain_accepts(a.dfs, slot, r));
}

// Closest hit (ANY = false) or any hit closer than `dist` of one ray.
template <bool ANY, bool PAD>
__device__ __forceinline__ WideHit traverse_wide(const DeviceAccel& a, const TraceRay& r, float dist) {
    int stack[kWideStack];
    WidePad w;
    if (PAD) w.set(a, r);
    int closest = -1, sp = 1, cur = 0;
    stack[0] = kWideDone;
    for (;;) {
        while (cur >= 0) {
            if (sp > kWideStack - 4) return WideHit{-1, dist, false};
            wide_node<PAD>(a.wide, r, w, dist, stack, sp, cur);
        }
        if (cur == kWideDone) break;
        float t;
        int prim;
        if (wide_leaf<PAD>(a, r, cur, dist, t, prim)) {
            closest = prim;
            dist = t;
            if (ANY) break;
        }
        cur = stack[--sp];
    }
    return WideHit{closest, dist, true};
}

}  // namespace zgl
