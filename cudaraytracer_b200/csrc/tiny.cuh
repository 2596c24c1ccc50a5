// Closest hit over a small scene's tree held in shared memory: interior
// nodes (4 float4 each) and triangles (3 float4 each: v0 with the primitive
// index, e1 = v1 - v0, e2 = v2 - v0 rounded to nearest as the triangle test
// forms them), with closest_hit's order, tests and bounds checks, so the
// same hits. Used by the trace kernels (trace.cu) and the path kernel
// (path_loop.cuh).
#pragma once
#include "bvh.cuh"

namespace crt {

constexpr int kTinyBytes = 32 * 1024;        // largest tree the trace kernels keep in shared memory
constexpr int kTinyDefaultBytes = 8 * 1024;  // largest that they do by default

inline int64_t tiny_bytes(const BvhView &bvh) {
    return ((int64_t)4 * bvh.num_nodes + (int64_t)3 * bvh.num_tris) * (int64_t)sizeof(float4);
}

#ifdef __CUDACC__

template <bool kEarlyExit, class Stack>
__device__ __forceinline__ Hit closest_hit_tiny(const float4 *sn, const float4 *se, const BvhView &bvh, Stack &st,
                                                V3 o, V3 d, float tmin, float tmax, float t_exit) {
    Hit hit;
    hit.t = tmax;
    hit.slot = -1;
    hit.b1 = hit.b2 = 0.f;
    const V3 inv = v3(rrcp(d.x), rrcp(d.y), rrcp(d.z));
    unsigned lm[Stack::kLocal];
    st.reset();
    int link = 0;
    while (link != kSentinel) {
        while (link >= 0) {
            if (link >= bvh.num_nodes) {
                report_traversal_bounds(bvh);
                return hit;
            }
            const float4 *nd = sn + 4 * link;
            const float4 n0 = nd[0], n1 = nd[1], n2 = nd[2];
            const int4 n3 = reinterpret_cast<const int4 *>(nd)[3];
            float t0, t1;
            const bool h0 = slab(n0.x, n0.y, n0.z, n0.w, n2.x, n2.y, o, inv, tmin, hit.t, t0);
            const bool h1 = slab(n1.x, n1.y, n1.z, n1.w, n2.z, n2.w, o, inv, tmin, hit.t, t1);
            if (h0 && h1) {
                int near = n3.x, far = n3.y;
                if (t1 < t0) {
                    near = n3.y;
                    far = n3.x;
                }
                if (st.sp >= kStackSize) {
                    report_traversal_bounds(bvh);
                    return hit;
                }
                st.push((unsigned)far, lm);
                link = near;
            } else if (h0) {
                link = n3.x;
            } else if (h1) {
                link = n3.y;
            } else {
                link = st.empty() ? kSentinel : (int)st.pop(lm);
            }
        }
        if (link == kSentinel) break;
        const int code = ~link;
        const int first = code >> 4, count = code & 15;
        if (first + count > bvh.num_tris) {
            report_traversal_bounds(bvh);
            return hit;
        }
        for (int k = 0; k < count; ++k) {
            const int slot = first + k;
            const float4 *tp = se + 3 * slot;
            const float4 a = tp[0], b = tp[1], c = tp[2];
            const bool acc = intersect_triangle_e<true>(o, d, v3(a.x, a.y, a.z), v3(b.x, b.y, b.z), v3(c.x, c.y, c.z),
                                                        slot, hit);
            if (kEarlyExit && acc && hit.t < t_exit) return hit;
        }
        link = st.empty() ? kSentinel : (int)st.pop(lm);
    }
    return hit;
}

// Copies the interior nodes and the triangles as (v0, e1, e2) records into
// s_tree (the caller synchronises the block afterwards).
__device__ __forceinline__ void tiny_fill(float4 *s_tree, const BvhView &bvh) {
    const int nn = 4 * bvh.num_nodes;
    for (int k = threadIdx.x; k < nn; k += blockDim.x) s_tree[k] = __ldg(bvh.nodes + k);
    for (int k = threadIdx.x; k < bvh.num_tris; k += blockDim.x) {
        const float4 a = __ldg(bvh.tris + 3 * k), b = __ldg(bvh.tris + 3 * k + 1), c = __ldg(bvh.tris + 3 * k + 2);
        s_tree[nn + 3 * k] = a;
        s_tree[nn + 3 * k + 1] = make_float4(rsub(b.x, a.x), rsub(b.y, a.y), rsub(b.z, a.z), 0.f);
        s_tree[nn + 3 * k + 2] = make_float4(rsub(c.x, a.x), rsub(c.y, a.y), rsub(c.z, a.z), 0.f);
    }
}

#endif  // __CUDACC__

}  // namespace crt
