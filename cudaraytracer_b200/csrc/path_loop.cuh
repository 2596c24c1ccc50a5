// A whole path per lane: extend, shade and shadow of bounce after bounce in
// one kernel, from a queue of path states to the pixels, without the stage
// kernels' queues, records and launches in between.
//
// A lane whose path ended takes the next path of the queue (one atomic per
// warp and turn), so the warps stay full while paths last. Per path the
// arithmetic is the stage kernels': the same functions on the same values,
// which pass through memory there and through opaque registers here
// (path_opaque), so that the compiler contracts the same multiplies and adds.
#pragma once
#include "path.cuh"

namespace crt {

#ifdef __CUDACC__

// Values the compiler may not trace through.
__device__ __forceinline__ void opaque(float &x) { asm volatile("" : "+f"(x)); }
__device__ __forceinline__ void opaque(V3 &v) {
    opaque(v.x);
    opaque(v.y);
    opaque(v.z);
}
__device__ __forceinline__ void path_opaque(PathState &s) {
    opaque(s.o);
    opaque(s.d);
    opaque(s.w);
    opaque(s.dc);
    opaque(s.ic);
    opaque(s.pdf);
}

// Src supplies, for this lane's path (per-path scene and request in the
// server, one scene elsewhere):
//   bool load(int i, PathState &ps, int &max_bounces)
//   const SceneView &scene(); StepParams params();
//   Hit closest(V3 o, V3 d); bool visible(const NeeRecord &nee);
//   void add(const PathState &ps)    a finished path into its pixel
//   kTraceLast   whether the shadow ray of a path that the bounce limit
//                drops is traced (and counted) all the same
// n paths starting at bounce b0; `next` counts the paths handed out (0 at
// the start). Returns the extend and shadow rays this lane traced.
template <class Src>
__device__ __forceinline__ uint2 path_loop(Src &src, int n, int b0, int *next) {
    const unsigned full = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
    // With fewer paths than lanes, every warp takes a share: a warp's lanes
    // wait for its longest traversal, so fewer lanes per warp finish sooner.
    const int warps = (int)((gridDim.x * blockDim.x) >> 5);
    const int cap = min(32, max(1, (n + warps - 1) / warps));
    uint2 rays = make_uint2(0, 0);
    PathState ps;
    bool alive = false, left = true;
    int bounce = 0, max_bounces = 0;
    while (true) {
        const unsigned idle = __ballot_sync(full, !alive && (int)lane < cap);
        if (idle && left) {
            int base = 0;
            if (lane == 0) base = atomicAdd(next, __popc(idle));
            base = __shfl_sync(full, base, 0);
            const int i = base + __popc(idle & lt);
            if ((idle >> lane & 1u) && i < n) {
                alive = src.load(i, ps, max_bounces);
                bounce = b0;
            }
            left = base + __popc(idle) < n;
        }
        if (!__any_sync(full, alive)) break;
        Hit h;
        h.slot = -1;
        if (alive) {
            ++rays.x;
            h = src.closest(ps.o, ps.d);
            opaque(h.t);
            opaque(h.b1);
            opaque(h.b2);
        }
        __syncwarp();
        NeeRecord nee;
        nee.valid = false;
        bool end = false, hit = alive && h.slot >= 0;
        if (alive && !hit) {
            // miss (IntersectionKernel, Src/Core/renderer.cuh:139-157)
            const SceneView &s = src.scene();
            if (s.env_light >= 0) {
                const V3 bg = env_emission(s.env, ps.d);
                if (ps.first)
                    ps.dc = ps.dc + mul(ps.w, bg);
                else
                    ps.ic = ps.ic + mul(ps.w, bg);
            }
            end = true;
        }
        __syncwarp();
        if (hit) {
            StepParams sp = src.params();
            sp.bounce = bounce;
            end = path_step(src.scene(), sp, ps, h, nee) == kTerminate;
            path_opaque(ps);
            opaque(nee.C);
            ++bounce;
        }
        __syncwarp();
        const bool drop = hit && !end && bounce >= max_bounces;
        if (hit && nee.valid && (Src::kTraceLast || !drop)) {
            ++rays.y;
            if (src.visible(nee)) {
                if (nee.direct)
                    ps.dc = vadd(ps.dc, nee.C);
                else
                    ps.ic = vadd(ps.ic, nee.C);
            }
        }
        __syncwarp();
        if (alive && end) src.add(ps);
        if (end || drop) alive = false;
    }
    return rays;
}

#endif  // __CUDACC__

}  // namespace crt
