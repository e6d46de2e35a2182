// pe_walk.cuh — the queues' ray/scene queries over the 4-wide tree: a warp walks 32 rays, one per
// lane, in one converged loop.
//
// What bounds a ray query here is instruction issue under divergence.  A loop that descends to a
// leaf, tests the whole leaf and pops lets every lane wait for the warp's longest descent, then for
// its longest leaf, then for its longest run of skipped entries: a warp instruction had 6.2 of 32
// lanes active (8.0 for any hit).  Here each turn of the loop moves every lane on by one unit of
// work: a lane on an interior node tests its four children, then a lane on a leaf tests ONE
// primitive of it, then a lane left without a reference pops.  Lanes whose rays have ended take the
// queue's next ones as soon as kRefill of them wait, so the warp stays full until the queue is empty:
// 11.9 of 32 lanes active and 217 against 506 warp instructions per ray on the second bounce of the
// 960x540 torus knot; closest hits of its 1920x1080 x 4-spp wave 7.07 -> 5.12 ms, any hits 3.72 -> 2.82 ms.
// Four lanes per ray (child k of a node to lane k, ballots and shuffles in place of the loop over
// children; built two ways) measured 13.4 and 10.5 ms for those closest hits.
//
// A ray's own sequence of node visits and primitive tests is the one-lane walk's
// (walkClosestWide), so hits are the same bit for bit whatever shares the warp.
#pragma once

#include "pe_trace.cuh"

namespace pe {

// References that are neither node nor leaf (a leaf's first record is below 2^23, so ~(first << 8 |
// count - 1) takes neither value): nothing is left; the instance's walk is over.
constexpr int kRayDone = static_cast<int>(0x80000000u);
constexpr int kLeaveInstance = static_cast<int>(0x80000001u);
constexpr unsigned kWarp = 0xffffffffu;
// Lanes without a ray at which a warp takes new ones: 7.66 / 7.27 / 7.23 / 7.28 ms of traversal per
// 1920x1080 x 4-spp knot wave at 4 / 8 / 12 / 16, Cornell 2.91 / 2.68 / 2.59 / 2.55, room 14.6 / 14.0 / 13.7 / 13.7.
constexpr int kRefill = 12;
// A walk's stack: with instances a top-level walk's, an instance's above it and the two entries between.
constexpr int walkStack(bool instances) { return instances ? 2 * kWideStack + 2 : kWideStack; }

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
// slab() from tMin = 0 for a ray whose reciprocal direction is finite: no operand is a NaN then, so
// the hardware's min and max give the same intervals as std::min / std::max and the swap.
__device__ __forceinline__ bool slabFinite(const float4 a, const float4 b, V3 o, V3 inv, float tMax, float& tNear) {
    const float ax = (a.x - o.x) * inv.x, bx = (a.w - o.x) * inv.x;
    const float ay = (a.y - o.y) * inv.y, by = (b.x - o.y) * inv.y;
    const float az = (a.z - o.z) * inv.z, bz = (b.y - o.z) * inv.z;
    const float t0 = max3f(fminf(ax, bx), fminf(ay, by), fmaxf(fminf(az, bz), 0.0f));
    const float t1 = min3f(fmaxf(ax, bx), fmaxf(ay, by), fminf(fmaxf(az, bz), tMax)) * 1.0000004f;
    tNear = t0;
    return t0 <= t1;
}

// The ray carried into instance `inst`'s space at shutter time `time` (MeshInstance::intersect).
struct LocalRay {
    V3 o, d;
};
static __device__ __noinline__ LocalRay instanceRay(const SceneGPU& S, int inst, float time, V3 o, V3 d) {
    float4 buf[8];
    const float4 *l2w, *w2l;
    float uvScale;
    instancePose(S, S.instances[inst], time, buf, l2w, w2l, uvScale);
    LocalRay r;
    r.o = xfPointD(w2l, o);
    r.d = xfVectorD(w2l, d);
    return r;
}

// One lane's ray and the state of its walk.
struct RayWalk {
    V3 o, d, inv;
    float tMax;
    uint32_t mask;
    int prim;        // closest hit: the primitive (instanceHitCode inside an instance), -1 none; any hit: 1 blocked
    int cur;         // the reference in hand, or kRayDone
    int sp;
    int inst;        // the instance the ray is in, -1 at the top level
    bool finite;     // inv is finite
    bool any;        // WALK_MIXED: this ray asks for any hit

    __device__ __forceinline__ void setRay(V3 o_, V3 d_) {
        o = o_;
        d = d_;
        inv = mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
        finite = isFinite3(inv);
    }
    __device__ __forceinline__ void start(const SceneGPU& S, int root, V3 o_, V3 d_, uint32_t mask_, float tMax_, int noHit) {
        setRay(o_, d_);
        mask = mask_;
        tMax = tMax_;
        prim = noHit;
        sp = 0;
        inst = -1;
        float tn;
        cur = S.nTris != 0 && slab(S.rootMin[0], S.rootMax[0], S.rootMin[1], S.rootMax[1], S.rootMin[2], S.rootMax[2], o,
                                   inv, 0.0f, tMax, tn)
                  ? root
                  : kRayDone;
    }
};

// What a warp's rays ask for: the closest hit, any hit, or (RayWalk::any) some the one and some the other.
enum WalkKind { WALK_CLOSEST, WALK_ANY, WALK_MIXED };

// One turn of the walk for every lane of the warp that has a reference.  T: uint2 (reference, entry
// distance), or for any hit uint32_t (reference).
// world(o, d, mask) gives the lane's ray back when it leaves an instance, time() its shutter time;
// found(t, u, v, prim, meta) takes a closest hit nearer than (or as near as) those before it.
// INSTANCES: the scene has mesh instances.
template <WalkKind KIND, bool COUNT, bool INSTANCES, typename T, typename World, typename Time, typename Found>
__device__ __forceinline__ void walkTurn(const SceneGPU& S, RayWalk& w, T* stack, uint32_t& nodeVisits, uint32_t& triTests,
                                         World world, Time time, Found found) {
    auto entry = [](int ref, float t) {
        if constexpr (sizeof(T) == 8) return make_uint2(static_cast<uint32_t>(ref), __float_as_uint(t));
        else return static_cast<uint32_t>(ref);
    };
    bool pop = false;
    // the turn's loads, issued together whichever unit the lane is at: a node's eight float4, or
    // the three of a leaf's next primitive
    const bool isNode = w.cur >= 0, isLeaf = !isNode && w.cur != kRayDone;
    int pi, more;
    leafRange(w.cur, pi, more);
    --more;
    const float4* at = isNode ? S.wide + 8 * static_cast<size_t>(w.cur) : S.tris + 3 * static_cast<size_t>(pi);
    WideNode n;
    if (isNode || isLeaf) {
        n.a[0] = __ldg(at);
        n.a[1] = __ldg(at + 1);
        n.a[2] = __ldg(at + 2);
    }
    if (isNode) {
        n.a[3] = __ldg(at + 3);
#pragma unroll
        for (int k = 0; k < 4; ++k) n.b[k] = __ldg(at + 4 + k);
    }
    if (isNode) {
        if (COUNT) ++nodeVisits;
        float t[4];
        bool hit[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            hit[k] = w.finite ? slabFinite(n.a[k], n.b[k], w.o, w.inv, w.tMax, t[k])
                              : slab(n.a[k].x, n.a[k].w, n.a[k].y, n.b[k].x, n.a[k].z, n.b[k].y, w.o, w.inv, 0.0f, w.tMax, t[k]);
            if (k >= 2) hit[k] = hit[k] && __float_as_int(n.b[k].w) != 0; // two children at least
        }
        const int count = (hit[0] ? 1 : 0) + (hit[1] ? 1 : 0) + (hit[2] ? 1 : 0) + (hit[3] ? 1 : 0);
        if constexpr (KIND == WALK_ANY) {
            // the first child hit is next, the others wait on the stack
            bool have = false;
            int next = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (hit[k]) {
                    if (have) stack[w.sp++] = entry(wideRef(n.b[k]), 0.0f);
                    else next = wideRef(n.b[k]);
                    have = true;
                }
            if (have) w.cur = next;
            else pop = true;
        } else {
            // nearest first, ties by child order; the farther ones wait, pushed farthest first
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (!hit[k]) t[k] = kInf;
            const int p01 = t[1] < t[0], p02 = t[2] < t[0], p03 = t[3] < t[0], p12 = t[2] < t[1], p13 = t[3] < t[1],
                      p23 = t[3] < t[2];
            const int rank[4] = {p01 + p02 + p03, 1 - p01 + p12 + p13, 2 - p02 - p12 + p23, 3 - p03 - p13 - p23};
            const int top = w.sp + count - 1;
            int next = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (rank[k] == 0) next = wideRef(n.b[k]);
                else if (hit[k]) stack[top - rank[k]] = entry(wideRef(n.b[k]), t[k]);
            }
            if (count > 0) {
                w.sp = top;
                w.cur = next;
            } else {
                pop = true;
            }
        }
    }
    if (isLeaf) {
        const float4 a = n.a[0], b = n.a[1];
        const uint32_t meta = __float_as_uint(b.w);
        bool enter = false;
        if ((meta & w.mask) != 0u) {
            enter = INSTANCES && (meta & PRIM_INSTANCE);
            if (!enter) {
                if (COUNT) ++triTests;
                float t, u = 0.0f, v = 0.0f;
                const bool in = (meta & PRIM_SPHERE)
                                    ? sphereLean(a, w.o, w.d, 0.0f, w.tMax, t)
                                    : triLean(a, b, n.a[2], w.o, w.d, 0.0f, w.tMax, t, u, v);
                if (in) {
                    if (KIND == WALK_ANY || (KIND == WALK_MIXED && w.any)) {
                        w.prim = 1;
                        w.sp = 0;
                        more = 0;
                    } else {
                        w.tMax = t;
                        w.prim = !INSTANCES || w.inst < 0 ? pi : instanceHitCode(w.inst, pi - S.instances[w.inst].recBase);
                        found(t, u, v, w.prim, meta);
                    }
                }
            }
        }
        if (INSTANCES && enter) {
            // the rest of the leaf and the way out wait on the stack
            const int id = __float_as_int(a.x);
            if (more > 0) stack[w.sp++] = entry(w.cur - 255, 0.0f);
            stack[w.sp++] = entry(kLeaveInstance, 0.0f);
            const LocalRay lr = instanceRay(S, id, time(), w.o, w.d);
            w.setRay(lr.o, lr.d);
            w.mask = VIS_ALL;
            w.inst = id;
            w.cur = S.instances[id].rootWide;
        } else if (more > 0) {
            w.cur -= 255; // the leaf's next primitive: first + 1, count - 1
        } else {
            pop = true;
        }
    }
    while (pop) {
        // entries farther than the current hit are skipped
        pop = false;
        if (w.sp == 0) {
            w.cur = kRayDone;
        } else {
            const T e = stack[--w.sp];
            if constexpr (sizeof(T) == 8) {
                w.cur = static_cast<int>(e.x);
                pop = __uint_as_float(e.y) > w.tMax;
            } else {
                w.cur = static_cast<int>(e);
            }
            if (INSTANCES && w.cur == kLeaveInstance) {
                V3 o, d;
                world(o, d, w.mask);
                w.setRay(o, d);
                w.inst = -1;
                pop = true;
            }
        }
    }
}

} // namespace pe
