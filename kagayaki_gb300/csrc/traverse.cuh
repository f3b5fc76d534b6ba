// traverse.cuh - closest-hit and occlusion traversal of the 8-wide
// compressed BVH with watertight FP32 ray/triangle intersection.
// Replaces willIntersectWithTriangle_nonRecursive (ConstructBVH.cuh:286-368)
// and Triangle::intersectTest (struct_Triangle.cuh:30-79) on the device.
//
// Semantics kept from the reference: a hit needs t >= 1e-5 (double compare,
// struct_Triangle.cuh:57), the result is the closest hit, and the reported
// distance is computed by the reference's own expression (ref_distance).  Where the
// reference resolves equal distances by its traversal order, this resolves
// them to the smaller triangle id, independent of the tree.
// Differences by design: the test is watertight (Woop, Benthin, Wald 2013)
// instead of Cramer's rule, and node culling uses the ray's [tmin, tmax]
// interval (closest-hit pruning) instead of the whole line.
#pragma once

#include "kgk_device.cuh"
#include "kgk_internal.h"

namespace kgk {

constexpr int kTravStack = 32;
// Node visits a resumable traversal step may make before it tests triangles
// (the closest-hit rays of k_extend and the batch queries; the shadow passes).
constexpr int kNodesPerStep = 2;
constexpr int kNodesPerStepShadow = 2;
// Conservative slack of box planes relative to the node's offset (64 units of
// 2^-24, see node_intersect), and widening of the search limit.
constexpr float kBoxSlack = 0x1p-18f;
constexpr float kBoxWiden = 1.0000012f;

struct RayPre {
    float3 o, d, inv;
    float sx, sy, sz;
    int kx, ky, kz;
    unsigned oct;  // octant_masks
};

__device__ __forceinline__ float safe_inv(float d) {
    // |d| < 1e-20 -> +-1e20 so that scale * inv never forms 0 * inf
    float a = fabsf(d) < 1e-20f ? copysignf(1e-20f, d) : d;
    return 1.0f / a;
}

// A node's children are visited by slot XOR (7 - octant), nearest first.  The
// three masks of the delta swaps that permute eight slot bits this way (swap
// neighbours, pairs, nibbles), a byte each; the bits themselves are those of
// 7 - octant (bit 0, 9 and 18).
__device__ __forceinline__ unsigned octant_masks(float3 d) {
    return (d.z < 0.0f ? 0u : 0x55u) | (d.y < 0.0f ? 0u : 0x3300u) | (d.x < 0.0f ? 0u : 0x0f0000u);
}
__device__ __forceinline__ unsigned octant_xor(unsigned m) { return (m & 1u) | ((m >> 8) & 2u) | ((m >> 14) & 4u); }
__device__ __forceinline__ unsigned octant_permute(unsigned x, unsigned m) {
    unsigned t = ((x >> 1) ^ x) & m;  // x has eight bits: the other masks meet zeros
    x ^= t ^ (t << 1);
    t = ((x >> 2) ^ x) & (m >> 8);
    x ^= t ^ (t << 2);
    t = ((x >> 4) ^ x) & (m >> 16);
    return x ^ t ^ (t << 4);
}

__device__ __forceinline__ RayPre make_ray(float3 o, float3 d) {
    RayPre r;
    r.o = o;
    r.d = d;
    r.inv = f3(safe_inv(d.x), safe_inv(d.y), safe_inv(d.z));
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    int kz = ax > ay ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    int kx = kz == 2 ? 0 : kz + 1;
    int ky = kx == 2 ? 0 : kx + 1;
    if (comp(d, kz) < 0.0f) { int t = kx; kx = ky; ky = t; }
    r.kx = kx;
    r.ky = ky;
    r.kz = kz;
    const float dz = comp(d, kz);
    r.sx = comp(d, kx) / dz;
    r.sy = comp(d, ky) / dz;
    r.sz = fabsf(dz) < 1e-20f ? 1.0f / dz : comp(r.inv, kz);
    r.oct = octant_masks(d);
    return r;
}

// Watertight test.  On a hit returns true with t, b1 (weight of v1) and b2
// (weight of v2).  The 2D edge functions are formed with explicit
// round-to-nearest multiplies and subtractions (no FMA contraction), so the
// two triangles sharing an edge compute exactly negated values.
__device__ __forceinline__ bool tri_intersect(const RayPre &r, float4 a4, float4 b4, float4 c4,
                                              float *t, float *b1, float *b2) {
    const float3 A = f3(a4) - r.o, B = f3(b4) - r.o, C = f3(c4) - r.o;
    const float Akz = comp(A, r.kz), Bkz = comp(B, r.kz), Ckz = comp(C, r.kz);
    const float Ax = comp(A, r.kx) - r.sx * Akz, Ay = comp(A, r.ky) - r.sy * Akz;
    const float Bx = comp(B, r.kx) - r.sx * Bkz, By = comp(B, r.ky) - r.sy * Bkz;
    const float Cx = comp(C, r.kx) - r.sx * Ckz, Cy = comp(C, r.ky) - r.sy * Ckz;
    const float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
    const float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
    const float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    const float det = U + V + W;
    if (det == 0.0f) return false;
    const float T = U * (r.sz * Akz) + V * (r.sz * Bkz) + W * (r.sz * Ckz);
    const float tt = T / det;
    if (!(tt >= kTMin)) return false;  // also rejects NaN
    *t = tt;
    *b1 = V / det;
    *b2 = W / det;
    return true;
}

// Distance and barycentrics of an accepted hit by the reference's own
// expressions (struct_Triangle.cuh:46-49), every operation rounded
// separately like the reference's host build: the reported t is the
// reference's t bit for bit.  u = weight of v1, v = weight of v2.
__device__ __forceinline__ float3 rn_sub(float3 a, float3 b) {
    return f3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z));
}
__device__ __forceinline__ float3 rn_cross(float3 a, float3 b) {
    return f3(__fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y)),
              __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z)),
              __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float rn_dot(float3 a, float3 b) {
    return __fadd_rn(__fadd_rn(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y)), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ void ref_distance(const RayPre &r, float4 a4, float4 b4, float4 c4, float *t, float *u,
                                             float *v) {
    const float3 v0 = f3(a4), e1 = rn_sub(f3(b4), v0), e2 = rn_sub(f3(c4), v0), so = rn_sub(r.o, v0);
    const float3 de2 = rn_cross(r.d, e2), se1 = rn_cross(so, e1);
    const float term1 = __fdiv_rn(1.0f, rn_dot(de2, e1));
    *t = __fmul_rn(term1, rn_dot(se1, e2));
    *u = __fmul_rn(term1, rn_dot(de2, so));
    *v = __fmul_rn(term1, rn_dot(se1, r.d));
}

// 2^15 + (byte i of x) as a float, exactly, in one byte permute: the byte
// becomes mantissa bits 8..15 under the exponent of 2^15 (bits 0x47000000).
// The box test folds the bias into its per-node plane offsets, so a plane
// costs one permute and half of a paired multiply-add (no integer-to-float
// conversion and no subtraction).
__device__ __forceinline__ float byte_biased(unsigned x, int i) {
    return __uint_as_float(__byte_perm(x, 0x4700u, 0x5404u | ((unsigned)i << 4)));
}
// (a0, a1) * b + (c0, c1) in one instruction (two FP32 multiply-adds, each
// rounded as fmaf): a child's near and far plane of one axis.
__device__ __forceinline__ float2 fma2(float a0, float a1, float b, float c0, float c1) {
    float2 r;
    asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmov.b64 c, {%5, %6};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a0), "f"(a1), "f"(b), "f"(c0), "f"(c1));
    return r;
}

// Hit mask of one compressed node: bits 24..31 = inner children
// (octant-permuted slots), bits 0..23 = triangles of hit leaf children (bits
// of the node's leaf field).
__device__ __forceinline__ unsigned node_intersect(float3 o, float3 inv, unsigned oct, float tmax, const float4 n0,
                                                   const float4 n1, const float4 n2, const float4 n3,
                                                   const float4 n4) {
    const unsigned e = __float_as_uint(n0.w);
    const float adx = __uint_as_float((e & 0xffu) << 23) * inv.x;
    const float ady = __uint_as_float(((e >> 8) & 0xffu) << 23) * inv.y;
    const float adz = __uint_as_float(((e >> 16) & 0xffu) << 23) * inv.z;
    // Plane b of an axis lies at t = (2^15 + b) * ad + (o - 2^15 * ad),
    // formed as one multiply-add with an exact product.  With u = 2^-24, o
    // carries 3 u |o| (origin offset, product, inverse); the offset is
    // rounded twice (o - 2^15 ad, then -/+ the slack), each time by at most
    // u (|o| + 2^15 |ad|); the multiply-add by u (|o| + 255 |ad|); b ad carries
    // 255 u |ad| of the inverse: together 6 u |o| + 2^-8 (1 + 2^-5) |ad|.  A
    // slack of 64 u |o| + |ad| / 64 (per axis: |ad| is huge on an axis the ray
    // nearly parallels) moves near planes down and far planes up; what is left
    // of it covers the rounding of the hit distances themselves.
    const float ox = (n0.x - o.x) * inv.x;
    const float oy = (n0.y - o.y) * inv.y;
    const float oz = (n0.z - o.z) * inv.z;
    const float bx = fmaf(-32768.0f, adx, ox), by = fmaf(-32768.0f, ady, oy), bz = fmaf(-32768.0f, adz, oz);
    const float sx = fmaf(fabsf(ox), kBoxSlack, fabsf(adx) * 0.015625f);
    const float sy = fmaf(fabsf(oy), kBoxSlack, fabsf(ady) * 0.015625f);
    const float sz = fmaf(fabsf(oz), kBoxSlack, fabsf(adz) * 0.015625f);
    const float oxn = bx - sx, oyn = by - sy, ozn = bz - sz;
    const float oxf = bx + sx, oyf = by + sy, ozf = bz + sz;
    const float tm = tmax * kBoxWiden;
    unsigned miss = 0;  // slot 7 first, so that slot s ends at bit s
#pragma unroll
    for (int half = 1; half >= 0; --half) {
        const unsigned qlx = __float_as_uint(half ? n2.y : n2.x), qhx = __float_as_uint(half ? n2.w : n2.z);
        const unsigned qly = __float_as_uint(half ? n3.y : n3.x), qhy = __float_as_uint(half ? n3.w : n3.z);
        const unsigned qlz = __float_as_uint(half ? n4.y : n4.x), qhz = __float_as_uint(half ? n4.w : n4.z);
        const unsigned xn = inv.x < 0.0f ? qhx : qlx, xf = inv.x < 0.0f ? qlx : qhx;
        const unsigned yn = inv.y < 0.0f ? qhy : qly, yf = inv.y < 0.0f ? qly : qhy;
        const unsigned zn = inv.z < 0.0f ? qhz : qlz, zf = inv.z < 0.0f ? qlz : qhz;
#pragma unroll
        for (int j = 3; j >= 0; --j) {
            const float2 tx = fma2(byte_biased(xn, j), byte_biased(xf, j), adx, oxn, oxf);
            const float2 ty = fma2(byte_biased(yn, j), byte_biased(yf, j), ady, oyn, oyf);
            const float2 tz = fma2(byte_biased(zn, j), byte_biased(zf, j), adz, ozn, ozf);
            const float lo = fmaxf(fmaxf(tx.x, ty.x), fmaxf(tz.x, 0.0f));
            const float hi = fminf(fminf(tx.y, ty.y), fminf(tz.y, tm));
            // the sign of hi - lo shifted in: one multiply-add-pipe instruction
            // and one shift a slot, where a compare and the slot's own bits
            // took five
            miss = __funnelshift_l(__float_as_uint(hi - lo), miss, 1);
        }
    }
    const unsigned hit = ~miss & 0xffu, field = __float_as_uint(n1.z);
    return (hit * 0x010101u & field & 0xffffffu) | octant_permute(hit & (field >> 24), oct) << 24;
}

struct TravStats {
    unsigned nodes, tris, overflow;
};

// Closest hit.  best_t in: search limit (exclusive of farther hits); out: hit
// distance.  Returns the BVH-order triangle index of the hit or -1.
// Both traversals check every node and triangle index against the buffer
// sizes; a bad index sets st.overflow = 2 and ends the traversal instead of
// reading out of range.
template <bool kCount>
__device__ __forceinline__ int trace_closest(const WideNode *__restrict__ nodes, unsigned n_nodes,
                                             const float4 *__restrict__ tri, unsigned n_tris,
                                             const RayPre &r, float &best_t, int &best_id, float &bu,
                                             float &bv, TravStats &st) {
    uint2 stack[kTravStack];
    int sp = 0;
    int hit_slot = -1;
    const unsigned oct = octant_xor(r.oct);
    uint2 group = make_uint2(0u, 0x80000000u);
    while (true) {
        uint2 tg = make_uint2(0u, 0u);
        unsigned leaves = 0u;
        if (group.y & 0xff000000u) {
            const unsigned hits_imask = group.y;
            const int child_bit = 31 - __clz(hits_imask & 0xff000000u);
            const unsigned base = group.x;
            group.y &= ~(1u << child_bit);
            if (group.y & 0xff000000u) {
                if (sp < kTravStack) stack[sp++] = group;
                else st.overflow = 1;
            }
            const unsigned slot = (unsigned)(child_bit - 24) ^ oct;
            const unsigned rel = __popc(hits_imask & ~(0xffffffffu << slot));
            if (base + rel >= n_nodes) { st.overflow = 2; break; }
            const WideNode *nd = nodes + base + rel;
            const float4 n0 = __ldg(&nd->n0), n1 = __ldg(&nd->n1), n2 = __ldg(&nd->n2),
                         n3 = __ldg(&nd->n3), n4 = __ldg(&nd->n4);
            if (kCount) ++st.nodes;
            const unsigned hm = node_intersect(r.o, r.inv, r.oct, best_t, n0, n1, n2, n3, n4);
            const unsigned imask = __float_as_uint(n1.z) >> 24;
            leaves = __float_as_uint(n1.z);
            group = make_uint2(__float_as_uint(n1.x), (hm & 0xff000000u) | imask);
            tg = make_uint2(__float_as_uint(n1.y), hm & 0x00ffffffu);
        }
        while (tg.y != 0u) {
            const int k = __ffs(tg.y) - 1;
            tg.y &= tg.y - 1u;
            const int ti = (int)tg.x + __popc(leaves & ((1u << k) - 1u));
            if ((unsigned)ti >= n_tris) { st.overflow = 2; tg.y = 0u; group = make_uint2(0u, 0u); sp = 0; break; }
            const float4 a = __ldg(&tri[3 * ti]), b = __ldg(&tri[3 * ti + 1]), c = __ldg(&tri[3 * ti + 2]);
            if (kCount) ++st.tris;
            float t, u, v;
            if (tri_intersect(r, a, b, c, &t, &u, &v)) {
                ref_distance(r, a, b, c, &t, &u, &v);
                if (!(t >= kTMin)) continue;
                const int id = __float_as_int(a.w);
                if (t < best_t || (t == best_t && id < best_id)) {
                    best_t = t;
                    best_id = id;
                    bu = u;
                    bv = v;
                    hit_slot = ti;
                }
            }
        }
        if ((group.y & 0xff000000u) == 0u) {
            if (sp == 0) break;
            group = stack[--sp];
        }
    }
    return hit_slot;
}

// Occlusion: true when any triangle lies at kTMin <= t < tmax.
template <bool kCount>
__device__ __forceinline__ bool trace_any(const WideNode *__restrict__ nodes, unsigned n_nodes,
                                          const float4 *__restrict__ tri, unsigned n_tris,
                                          const RayPre &r, float tmax, TravStats &st) {
    uint2 stack[kTravStack];
    int sp = 0;
    const unsigned oct = octant_xor(r.oct);
    uint2 group = make_uint2(0u, 0x80000000u);
    while (true) {
        uint2 tg = make_uint2(0u, 0u);
        unsigned leaves = 0u;
        if (group.y & 0xff000000u) {
            const unsigned hits_imask = group.y;
            const int child_bit = 31 - __clz(hits_imask & 0xff000000u);
            const unsigned base = group.x;
            group.y &= ~(1u << child_bit);
            if (group.y & 0xff000000u) {
                if (sp < kTravStack) stack[sp++] = group;
                else st.overflow = 1;
            }
            const unsigned slot = (unsigned)(child_bit - 24) ^ oct;
            const unsigned rel = __popc(hits_imask & ~(0xffffffffu << slot));
            if (base + rel >= n_nodes) { st.overflow = 2; break; }
            const WideNode *nd = nodes + base + rel;
            const float4 n0 = __ldg(&nd->n0), n1 = __ldg(&nd->n1), n2 = __ldg(&nd->n2),
                         n3 = __ldg(&nd->n3), n4 = __ldg(&nd->n4);
            if (kCount) ++st.nodes;
            const unsigned hm = node_intersect(r.o, r.inv, r.oct, tmax, n0, n1, n2, n3, n4);
            const unsigned imask = __float_as_uint(n1.z) >> 24;
            leaves = __float_as_uint(n1.z);
            group = make_uint2(__float_as_uint(n1.x), (hm & 0xff000000u) | imask);
            tg = make_uint2(__float_as_uint(n1.y), hm & 0x00ffffffu);
        }
        while (tg.y != 0u) {
            const int k = __ffs(tg.y) - 1;
            tg.y &= tg.y - 1u;
            const int ti = (int)tg.x + __popc(leaves & ((1u << k) - 1u));
            if ((unsigned)ti >= n_tris) { st.overflow = 2; tg.y = 0u; group = make_uint2(0u, 0u); sp = 0; break; }
            const float4 a = __ldg(&tri[3 * ti]), b = __ldg(&tri[3 * ti + 1]), c = __ldg(&tri[3 * ti + 2]);
            if (kCount) ++st.tris;
            float t, u, v;
            if (tri_intersect(r, a, b, c, &t, &u, &v)) {
                ref_distance(r, a, b, c, &t, &u, &v);
                if (t >= kTMin && t < tmax) return true;
            }
        }
        if ((group.y & 0xff000000u) == 0u) {
            if (sp == 0) break;
            group = stack[--sp];
        }
    }
    return false;
}

// ---------------------------------------------------------------------------
// Warp traversal: resumable, a few node visits per call, for kernels that
// refill finished lanes with new rays (dynamic ray fetch) instead of letting a
// warp wait for its longest ray.  Same node order, culling and hit rules as
// trace_closest / trace_any, so the results are the same.
//
// Node visits run a ray per lane.  Triangle tests do not: a node yields none
// on most lanes and several on a few, so a loop over each lane's own triangles
// runs as long as the warp's longest list with a handful of lanes active.
// Here the lanes list their (ray, triangle) pairs in shared memory and the
// warp tests 32 pairs at a time, whichever rays they belong to, from a shared
// copy of the rays; a ray's closest hit is kept in shared memory too, so the
// lane's registers hold only what node visits need.
// Instruction issue bounds it (68 to 72 % of slots on incoherent rays, the ALU
// pipe at 53 %, DRAM below 10 %).  On the 5.2M-triangle frame a step's own-triangle loop ran 2.6 times
// at 6.9 lanes; pairs run 1.3 times at 14.2.  With the leaf field and the
// paired multiply-adds of node_intersect, closest-hit batches (2^22 rays, 1.3M
// triangles) 524 -> 479 us, the 64-sample 1080p frame 93.3 -> 89.6 ms, two
// 1-sample orbit frames 6.73 -> 6.49 ms.  Measured and left out: keeping fewer
// than 32 pairs for the next step (frame 88.1 ms, but orbit 6.58 ms), three
// nodes a step (frame 90.2, batches 508 us), three-input min / max (batches
// 490 us), seven blocks per SM without spills (frame 92.0 ms), 96-byte nodes
// or 64-byte triangle records read by 32-byte loads (batches + 1.5 %).
// ---------------------------------------------------------------------------
constexpr int kPairsPerLane = 3;  // triangles a lane lists at a time (two ballots give its place)

struct WarpRays {  // one warp's part of shared memory
    float4 o[32];          // origin, shear x
    float4 d[32];          // direction, shear y
    float2 z[32];          // shear z; axes kx | ky << 2 | kz << 4, bit 8: occlusion
    unsigned t[32];        // closest hit: distance bits (the search limit before any hit),
    int id[32], slot[32];  // triangle, 2 * BVH-order index + material class (-1: no hit),
    float2 uv[32];         // barycentrics
    int2 pair[32 * kPairsPerLane];  // BVH-order triangle, owning lane
};

// What a lane keeps of its ray between steps.
struct Lane {
    float3 o, inv;
    unsigned oct;       // octant_masks
    uint2 group;
    int sp;
    float best_t;
};
// The stack lives in a separate local array so that the scalar state stays in
// registers.
struct TravStack {
    uint2 e[kTravStack];
};

__device__ __forceinline__ void lane_init(WarpRays &w, Lane &c, float3 o, float3 d, float tmax, bool any_mode) {
    const int lane = threadIdx.x & 31;
    const RayPre r = make_ray(o, d);
    c.o = o;
    c.inv = r.inv;
    c.oct = r.oct;
    c.group = make_uint2(0u, 0x80000000u);
    c.sp = 0;
    c.best_t = tmax;
    w.o[lane] = make_float4(o.x, o.y, o.z, r.sx);
    w.d[lane] = make_float4(d.x, d.y, d.z, r.sy);
    w.z[lane] = make_float2(r.sz, __int_as_float(r.kx | r.ky << 2 | r.kz << 4 | (any_mode ? 256 : 0)));
    w.t[lane] = __float_as_uint(tmax);
    w.id[lane] = 0x7fffffff;
    w.slot[lane] = -1;
}

// One step of the warp: active lanes visit nodes until one has hit leaf
// triangles (at most kVisits nodes), then the warp tests all of them.
// Returns true on a lane whose ray is finished: w.slot is -1 (no hit) or
// names the hit; an occlusion ray ends at its first triangle with
// kTMin <= t < its limit.  All 32 lanes must call it.
template <bool kCount, int kVisits = kNodesPerStep>
__device__ __forceinline__ bool warp_step(const WideNode *__restrict__ nodes, unsigned n_nodes,
                                          const float4 *__restrict__ tri, unsigned n_tris, WarpRays &w, Lane &c,
                                          TravStack &stk, bool active, bool any_mode, TravStats &st) {
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    uint2 tg = make_uint2(0u, 0u);
    unsigned leaves = 0u;
    bool dead = false;
    if (active) {
#pragma unroll 1
        for (int visit = 0; visit < kVisits && tg.y == 0u; ++visit) {
            if ((c.group.y & 0xff000000u) == 0u) {
                if (c.sp == 0) break;
                c.group = stk.e[--c.sp];
            }
            const unsigned hits_imask = c.group.y;
            const int child_bit = 31 - __clz(hits_imask & 0xff000000u);
            const unsigned base = c.group.x;
            c.group.y &= ~(1u << child_bit);
            if (c.group.y & 0xff000000u) {
                if (c.sp < kTravStack) stk.e[c.sp++] = c.group;
                else st.overflow = 1;
            }
            const unsigned slot = (unsigned)(child_bit - 24) ^ octant_xor(c.oct);
            const unsigned rel = __popc(hits_imask & ~(0xffffffffu << slot));
            if (base + rel >= n_nodes) { st.overflow = 2; dead = true; break; }
            const WideNode *nd = nodes + base + rel;
            const float4 n0 = __ldg(&nd->n0), n1 = __ldg(&nd->n1), n2 = __ldg(&nd->n2), n3 = __ldg(&nd->n3),
                         n4 = __ldg(&nd->n4);
            if (kCount) ++st.nodes;
            const unsigned hm = node_intersect(c.o, c.inv, c.oct, c.best_t, n0, n1, n2, n3, n4);
            leaves = __float_as_uint(n1.z);
            const unsigned imask = leaves >> 24;
            c.group = make_uint2(__float_as_uint(n1.x), (hm & 0xff000000u) | imask);
            tg = make_uint2(__float_as_uint(n1.y), hm & 0x00ffffffu);
        }
    }
    bool any_hit = false;
    while (true) {
        const int n = min(__popc(tg.y), kPairsPerLane);
        const unsigned b0 = __ballot_sync(~0u, n & 1), b1 = __ballot_sync(~0u, n & 2);
        if ((b0 | b1) == 0u) break;
        const int total = __popc(b0) + 2 * __popc(b1);
        int at = __popc(b0 & lt) + 2 * __popc(b1 & lt);
#pragma unroll
        for (int i = 0; i < kPairsPerLane; ++i)
            if (i < n) {
                w.pair[at + i] = make_int2((int)tg.x + __popc(leaves & ((tg.y & (0u - tg.y)) - 1u)), lane);
                tg.y &= tg.y - 1u;
            }
        __syncwarp();
        for (int p0 = 0; p0 < total; p0 += 32) {
            bool hit = false;
            int own = 0, ti = 0, id = 0, cls = 0;
            float t = 0.0f, u = 0.0f, v = 0.0f, old = 0.0f;
            if (p0 + lane < total) {
                const int2 pr = w.pair[p0 + lane];
                ti = pr.x;
                own = pr.y;
                if ((unsigned)ti >= n_tris) {
                    st.overflow = 2;
                } else {
                    const float4 a = __ldg(&tri[3 * ti]), b = __ldg(&tri[3 * ti + 1]), cc = __ldg(&tri[3 * ti + 2]);
                    const float4 ro = w.o[own], rd = w.d[own];
                    const float2 rz = w.z[own];
                    const int ax = __float_as_int(rz.y);
                    RayPre r;
                    r.o = f3(ro);
                    r.d = f3(rd);
                    r.sx = ro.w;
                    r.sy = rd.w;
                    r.sz = rz.x;
                    r.kx = ax & 3;
                    r.ky = (ax >> 2) & 3;
                    r.kz = (ax >> 4) & 3;
                    if (kCount) ++st.tris;
                    if (tri_intersect(r, a, b, cc, &t, &u, &v)) {
                        ref_distance(r, a, b, cc, &t, &u, &v);
                        old = __uint_as_float(w.t[own]);
                        id = __float_as_int(a.w);
                        cls = __float_as_int(b.w);
                        // a tie goes to the smaller id below; an occlusion ray's limit is exclusive
                        hit = t >= kTMin && ((ax & 256) ? t < old : t <= old);
                    }
                }
            }
            if (!__any_sync(~0u, hit)) continue;
            any_hit = true;
            // distances are positive: their bits order like the values
            if (hit) atomicMin(&w.t[own], __float_as_uint(t));
            __syncwarp();
            hit = hit && __float_as_uint(t) == w.t[own];
            if (hit && t < old) w.id[own] = 0x7fffffff;
            __syncwarp();
            if (hit) atomicMin(&w.id[own], id);
            __syncwarp();
            if (hit && w.id[own] == id) {
                w.slot[own] = 2 * ti + cls;
                w.uv[own] = make_float2(u, v);
            }
        }
        __syncwarp();
    }
    if (!active) return false;
    if (any_hit) c.best_t = __uint_as_float(w.t[lane]);
    if (dead || (any_mode && any_hit && w.slot[lane] >= 0)) return true;
    if ((c.group.y & 0xff000000u) == 0u) {
        if (c.sp == 0) return true;
        c.group = stk.e[--c.sp];
    }
    return false;
}

// The same step with each lane testing the triangles of its own visit, an occluded
// ray none after its first hit.  In closed rooms nearly every ray has its hit in
// the first node it meets, and listing all of that node's triangles in shared
// memory is what the pairs cost there.  Same nodes, culling and hit rules.
struct OwnRay {
    RayPre r;
    uint2 group;
    int sp;
    float best_t;
    int best_id;  // kNoHit: none yet
};
constexpr int kNoHit = 0x7fffffff;

__device__ __forceinline__ void own_init(OwnRay &c, float3 o, float3 d, float tmax) {
    c.r = make_ray(o, d);
    c.group = make_uint2(0u, 0x80000000u);
    c.sp = 0;
    c.best_t = tmax;
    c.best_id = kNoHit;
}

// Returns true when the lane's ray is finished.
template <bool kAny, bool kCount>
__device__ __forceinline__ bool own_step(const WideNode *__restrict__ nodes, unsigned n_nodes,
                                         const float4 *__restrict__ tri, unsigned n_tris, OwnRay &c, TravStack &stk,
                                         TravStats &st) {
    uint2 tg = make_uint2(0u, 0u);
    unsigned leaves = 0u;
#pragma unroll 1
    for (int visit = 0; visit < kNodesPerStep && tg.y == 0u; ++visit) {
        if ((c.group.y & 0xff000000u) == 0u) {
            if (c.sp == 0) break;
            c.group = stk.e[--c.sp];
        }
        const unsigned hits_imask = c.group.y;
        const int child_bit = 31 - __clz(hits_imask & 0xff000000u);
        const unsigned base = c.group.x;
        c.group.y &= ~(1u << child_bit);
        if (c.group.y & 0xff000000u) {
            if (c.sp < kTravStack) stk.e[c.sp++] = c.group;
            else st.overflow = 1;
        }
        const unsigned slot = (unsigned)(child_bit - 24) ^ octant_xor(c.r.oct);
        const unsigned rel = __popc(hits_imask & ~(0xffffffffu << slot));
        if (base + rel >= n_nodes) { st.overflow = 2; return true; }
        const WideNode *nd = nodes + base + rel;
        const float4 n0 = __ldg(&nd->n0), n1 = __ldg(&nd->n1), n2 = __ldg(&nd->n2), n3 = __ldg(&nd->n3),
                     n4 = __ldg(&nd->n4);
        if (kCount) ++st.nodes;
        const unsigned hm = node_intersect(c.r.o, c.r.inv, c.r.oct, c.best_t, n0, n1, n2, n3, n4);
        leaves = __float_as_uint(n1.z);
        c.group = make_uint2(__float_as_uint(n1.x), (hm & 0xff000000u) | leaves >> 24);
        tg = make_uint2(__float_as_uint(n1.y), hm & 0x00ffffffu);
    }
    while (tg.y != 0u) {
        const int k = __ffs(tg.y) - 1;
        tg.y &= tg.y - 1u;
        const int ti = (int)tg.x + __popc(leaves & ((1u << k) - 1u));
        if ((unsigned)ti >= n_tris) { st.overflow = 2; return true; }
        const float4 a = __ldg(&tri[3 * ti]), b = __ldg(&tri[3 * ti + 1]), cc = __ldg(&tri[3 * ti + 2]);
        if (kCount) ++st.tris;
        float t, u, v;
        if (!tri_intersect(c.r, a, b, cc, &t, &u, &v)) continue;
        ref_distance(c.r, a, b, cc, &t, &u, &v);
        if (!(t >= kTMin)) continue;
        const int id = __float_as_int(a.w);
        if (kAny) {
            if (t < c.best_t) {
                c.best_id = id;
                return true;
            }
        } else if (t < c.best_t || (t == c.best_t && id < c.best_id)) {
            c.best_t = t;
            c.best_id = id;
        }
    }
    if ((c.group.y & 0xff000000u) == 0u) {
        if (c.sp == 0) return true;
        c.group = stk.e[--c.sp];
    }
    return false;
}

}  // namespace kgk
