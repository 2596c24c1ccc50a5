// Closest hit of scenes of at most kFlatTris triangles without a tree: every
// lane of a warp tests every triangle in the same order, so the lanes never
// part, where the tree's traversal of a few dozen triangles keeps 11-12 of
// 32 lanes busy.
//
// 1. A conservative test of all triangles from precomputed per-triangle
//    vectors (22 multiply-adds, no division): with m = o x d,
//      det = d . (e2 x e1)          T = v0 . (e2 x e1) - o . (e2 x e1)
//      U = e2 . m - d . (e2 x v0)   V = d . (e1 x v0) - e1 . m
//    are the numerators of the triangle test (t = T / det, b1 = U / det,
//    b2 = V / det) up to rounding. A triangle stays a candidate unless one of
//    det, T, U, V, det - U - V is negative by more than its error margin.
//    With u = 2^-24, |.| 1-norms, E the longest edge and S = |o| + max |v0|,
//    the roundings here and in the triangle test together stay below 32 u
//    times |d| E E for det, E E S for T and |d| E S for U and V; 2e-6 is
//    that factor.
// 2. The triangle test itself (intersect_triangle_e's operations) on each
//    lane's candidates, usually one to three.
// 3. The nearest accepted triangle is closest_hit's answer when the choice
//    does not hang on rounding: its numerators clear their margins (so the
//    ray really passes through the triangle and through every box above it,
//    which the slab test, exact to a few ulp of t, then cannot cull), it lies
//    clear of tmin and tmax, and no other accepted triangle is as near. With
//    no accepted triangle there is no hit. Otherwise (about one ray in 10^4)
//    the tree is traversed, whose order decides. Hits are thus closest_hit's
//    bit for bit.
//
// For batches of unordered rays (the trace kernels). Measured on the Cornell
// box (36 triangles), 1M random rays + 1M shadow queries in one pass: 249 us
// over the tree in shared memory, 201 with the records in global memory, one
// triangle at a time (load pipe 82% busy), 155 as here. The renderer's
// camera and shadow rays run 5-8% slower this way (256 x 256 frame 613 ->
// 657 us, 16 views 10.3 -> 11.4 ms): neighbouring paths take the tree
// together, and its boxes cull most of the triangles.
#pragma once
#include "bvh.cuh"

namespace crt {

constexpr int kFlatTris = 64;  // candidates in two 32-bit words

// float4 words of a scene's records and scales.
__host__ __device__ inline int flat_float4s(int n) { return 8 * ((n + 1) / 2) + 1; }

#ifdef __CUDACC__

template <bool kEarlyExit>
static __device__ __noinline__ void flat_tree(const BvhView &bvh, V3 o, V3 d, float tmin, float tmax, float t_exit,
                                              Hit &hit) {
    hit = closest_hit<kEarlyExit>(bvh, o, d, tmin, tmax, t_exit);
}

// Copies a scene's records into the block's shared memory (the caller
// synchronises the block afterwards).
constexpr int kFlatWords = 8 * (kFlatTris / 2) + 1;
__device__ __forceinline__ void flat_fill(float4 *rec, const BvhView &bvh) {
    const int words = flat_float4s(bvh.num_tris);
    for (int k = threadIdx.x; k < words; k += blockDim.x) rec[k] = __ldg(bvh.flat + k);
}

// rec: the records in shared memory, two triangles interleaved:
// 8 float4 per pair, component j of triangle 2p and of 2p + 1 in consecutive
// floats; the scales after the last pair.
template <bool kEarlyExit>
__device__ __forceinline__ Hit closest_hit_flat(const float4 *rec, const BvhView &bvh, V3 o, V3 d, float tmin,
                                                float tmax, float t_exit = 0.f) {
    const int n = bvh.num_tris, pairs = (n + 1) >> 1;
    const float4 sc = rec[8 * pairs];  // E, max |v0|, in the ranges k_flat keeps them in
    const float d1 = fabsf(d.x) + fabsf(d.y) + fabsf(d.z);
    const float s1n = fabsf(o.x) + fabsf(o.y) + fabsf(o.z) + sc.y;
    const float sd = s1n * d1;
    const float md = 2e-6f * d1 * sc.x * sc.x, mt = 2e-6f * s1n * sc.x * sc.x, mu = 2e-6f * sc.x * sd;
    const float mw = 2.f * (mu + md);
    // Products beyond the floats, or so small that their roundings are not
    // relative (huge, tiny or non-finite rays; k_flat keeps 1e-10 <= E <= 1e10
    // and S >= 1e-12, so no margin falls below 1e-40): the tree decides.
    bool odd = !(md + mt + mu + sd < 1e30f) || !(d1 > 1e-12f);
    const float mx = o.y * d.z - o.z * d.y, my = o.z * d.x - o.x * d.z, mz = o.x * d.y - o.y * d.x;
    const F2 dx = f2(d.x, d.x), dy = f2(d.y, d.y), dz = f2(d.z, d.z);
    const F2 ox = f2(-o.x, -o.x), oy = f2(-o.y, -o.y), oz = f2(-o.z, -o.z);
    const F2 cx = f2(mx, mx), cy = f2(my, my), cz = f2(mz, mz), minus = f2(-1.f, -1.f);
    unsigned cand[2] = {0u, 0u};
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        const int end = min(pairs - 16 * w, 16);
#pragma unroll 2
        for (int k = 0; k < end; ++k) {
            const ulonglong2 *r = reinterpret_cast<const ulonglong2 *>(rec + 8 * (16 * w + k));
            const ulonglong2 a = r[0], b = r[1], c = r[2], e = r[3], f = r[4], g = r[5], h = r[6], q = r[7];
            const F2 det = f2fma(F2{a.x}, dx, f2fma(F2{a.y}, dy, f2mul(F2{b.x}, dz)));
            const F2 T = f2fma(F2{a.x}, ox, f2fma(F2{a.y}, oy, f2fma(F2{b.x}, oz, F2{b.y})));
            const F2 uf = f2fma(F2{e.y}, dx, f2fma(F2{g.y}, dy, f2mul(F2{q.y}, dz)));
            const F2 ue = f2fma(F2{c.x}, cx, f2fma(F2{c.y}, cy, f2mul(F2{e.x}, cz)));
            const F2 ve = f2fma(F2{f.x}, cx, f2fma(F2{f.y}, cy, f2mul(F2{g.x}, cz)));
            const F2 U = f2fma(uf, minus, ue);
            const F2 V = f2fma(F2{h.x}, dx, f2fma(F2{h.y}, dy, f2fma(F2{q.x}, dz, f2mul(ve, minus))));
            const F2 W = f2fma(V, minus, f2fma(U, minus, det));
            const float2 D2 = f2get(det), T2 = f2get(T), U2 = f2get(U), V2 = f2get(V), W2 = f2get(W);
            if (D2.x >= -md && T2.x >= -mt && U2.x >= -mu && V2.x >= -mu && W2.x >= -mw) cand[w] |= 1u << (2 * k);
            if (D2.y >= -md && T2.y >= -mt && U2.y >= -mu && V2.y >= -mu && W2.y >= -mw) cand[w] |= 2u << (2 * k);
        }
    }
    Hit hit;
    hit.t = tmax;
    hit.slot = -1;
    hit.b1 = hit.b2 = 0.f;
    float best = INFINITY, second = INFINITY, inv_b = 1.f;
    bool clear = false;
    while (cand[0] | cand[1]) {
        int slot;
        if (cand[0]) {
            slot = __ffs(cand[0]) - 1;
            cand[0] &= cand[0] - 1;
        } else {
            slot = 31 + __ffs(cand[1]);
            cand[1] &= cand[1] - 1;
        }
        // intersect_triangle_e's operations, without its bound on t
        const float4 *tp = bvh.tris + 3 * slot;
        const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
        const V3 v0 = v3(a.x, a.y, a.z), e1 = vsub(v3(b.x, b.y, b.z), v0), e2 = vsub(v3(c.x, c.y, c.z), v0);
        const V3 s = vsub(o, v0), p1 = vcross(d, e2), p2 = vcross(s, e1);
        const float det = vdot(e1, p1);
        if (det == 0.f || det < 0.f) continue;
        const float inv = rrcp(det);
        const float T = vdot(p2, e2), U = vdot(p1, s), V = vdot(p2, d);
        const float t = rmul(inv, T);
        const float b1 = rmul(inv, U);
        if (b1 < 0.f || b1 > 1.f) continue;
        const float b2 = rmul(inv, V);
        if (b2 < 0.f || radd(b1, b2) > 1.f) continue;
        if (t < 0.f || t > kTriTMax) continue;
        if (!(t >= 0.f)) odd = true;  // NaN
        if (t < best) {
            second = best;
            best = t;
            inv_b = inv;
            hit.slot = slot;
            hit.b1 = b1;
            hit.b2 = b2;
            clear = T > mt && U > mu && V > mu && det - U - V > mw;
        } else {
            second = fminf(second, t);
        }
    }
    if (hit.slot >= 0) {
        // rounding of t = T / det in the triangle test: T's and det's, 8 u of
        // their scales with the edges' own (the margins are 32 u), and more
        // than the quotient's and the slabs' few ulp
        const float gap = 0.25f * (mt + md * best) * inv_b + 2e-6f * best;
        if (best > tmax + gap) {  // beyond the caller's bound, clearly: no hit
            hit.slot = -1;
            hit.b1 = hit.b2 = 0.f;
        } else {
            hit.t = best;
            odd = odd || !clear || !(best < tmax - gap) || !(best > tmin + gap) || !(second > best + gap);
        }
    }
    if (odd) flat_tree<kEarlyExit>(bvh, o, d, tmin, tmax, t_exit, hit);
    return hit;
}

#endif  // __CUDACC__

}  // namespace crt
