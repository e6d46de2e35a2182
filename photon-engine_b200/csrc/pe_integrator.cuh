// pe_integrator.cuh — the wavefront form of PathTracer::Li (src/integrators/path_tracer.cpp:321-890).
//
// One path slot per (pixel, sample) of a wave.  A slot's state lives in HBM as SoA float4
// columns; each bounce runs persistent kernels over compacted queues:
//   trace   (queue of live rays, shadow records of the bounce before) → hit records; visible NEE terms
//           added to the slots' L
//   bin     (the queue) → a bin per shading key
//   shade   (the bins) → next-ray queue + shadow records (warp-aggregated appends)
// and the last paths of a wave run to their ends in a tail kernel.
// The state machine below is Li's loop body split at its two scene queries.  Radiance terms are
// added to L in the reference's order (emission of vertex k, NEE of vertex k, emission of
// vertex k+1, ...), and each slot draws Sobol dimensions in the reference's order.
#pragma once

#include "photon_cuda.h"
#include "pe_bsdf.h"
#include "pe_guide.cuh"
#include "pe_light.h"
#include "pe_medium.h"
#include "pe_trace.cuh"
#include "pe_walk.cuh"
#include "pe_wave.h"

namespace pe {

// Persistent-warp work distribution: lane 0 claims the next `items` items for its warp.
__device__ __forceinline__ int warpFetch(uint32_t* cursor, int items = 32) {
    int base = 0;
    if ((threadIdx.x & 31) == 0) base = static_cast<int>(atomicAdd(cursor, static_cast<uint32_t>(items)));
    return __shfl_sync(0xffffffffu, base, 0);
}

__device__ __forceinline__ uint32_t packCounters(int depth, int diffuse, int pass, int skips) {
    return static_cast<uint32_t>(depth) | (static_cast<uint32_t>(diffuse) << 8) | (static_cast<uint32_t>(pass) << 16) |
           (static_cast<uint32_t>(skips) << 24);
}

// Warp-aggregated queue append: one atomicAdd per warp (ballot + popc).
__device__ __forceinline__ void queuePush(int32_t* queue, uint32_t* counter, bool want, int32_t value) {
    const unsigned mask = __ballot_sync(__activemask(), want);
    if (!want) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    const int rank = __popc(mask & ((1u << lane) - 1u));
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counter, static_cast<uint32_t>(__popc(mask)));
    base = __shfl_sync(mask, base, leader);
    queue[base + rank] = value;
}

// ---- generate: camera rays ------------------------------------------------------------------
// Wave path `path` (its segment, sample and pixel) starts in `slot`.
// ---- render passes (path_tracer.cpp:373-395) ---------------------------------------------------
__device__ __forceinline__ float4* passBlock(const Paths& P, int path) {
    return P.pass + static_cast<size_t>(path) * static_cast<size_t>(P.passStride);
}
__device__ __forceinline__ void passAdd(float4* q, V3 c) {
    float4 v = *q;
    v.x += c.x;
    v.y += c.y;
    v.z += c.z;
    *q = v;
}
// Shares of f's diffuse, glossy and transmission groups, per channel; 1, 0, 0 where the groups
// sum to zero (path_tracer.cpp:683-690, 803-811).
__device__ __forceinline__ void lobeShares(const LobeSplit3& sp, V3 out[3]) {
    const V3 sum = sp.diffuse + sp.glossy + sp.transmission;
    const V3* parts[3] = {&sp.diffuse, &sp.glossy, &sp.transmission};
    for (int k = 0; k < 3; ++k) {
        out[k].x = sum.x > 0.0f ? parts[k]->x / sum.x : (k == 0 ? 1.0f : 0.0f);
        out[k].y = sum.y > 0.0f ? parts[k]->y / sum.y : (k == 0 ? 1.0f : 0.0f);
        out[k].z = sum.z > 0.0f ? parts[k]->z / sum.z : (k == 0 ? 1.0f : 0.0f);
    }
}
// creditGroup: a term of light group `group` (ids outside the groups count for group 0).
static __device__ __noinline__ void creditGroup(const SceneGPU& S, const Paths& P, int path, int group, V3 added) {
    if (S.nLightGroups <= 0 || isBlack(added)) return;
    const int g = (group >= 0 && group < S.nLightGroups) ? group : 0;
    if (g < PE_MAX_LIGHT_GROUPS) passAdd(passBlock(P, path) + PASS_GROUPS + g, added);
}
// creditPath: light reaching the path past its first surface, split by that surface's lobe
// shares into the direct (found by the first bounce) or indirect passes.
static __device__ __noinline__ void creditPath(const Paths& P, int path, V3 added, bool direct) {
    float4* b = passBlock(P, path);
    for (int k = 0; k < 3; ++k) {
        const float4 share = b[PASS_LOBES + k];
        passAdd(b + 2 * k + (direct ? 0 : 1), added * mk(share.x, share.y, share.z));
    }
}
__device__ __forceinline__ int lightGroupOf(const SceneGPU& S, int light) {
    return light < 0 ? S.envGroup : (S.lightGroup ? S.lightGroup[light] : -1);
}
// A NEE term's passes: its light's group, and the direct passes by the vertex's own lobe shares
// at the first surface (shares non-null), else the first surface's shares as indirect light.
static __device__ __noinline__ void creditNee(const SceneGPU& S, const Paths& P, int path, int light, V3 added,
                                       const float4* shares) {
    if (isBlack(added)) return;
    creditGroup(S, P, path, lightGroupOf(S, light), added);
    if (shares) {
        float4* b = passBlock(P, path);
        for (int k = 0; k < 3; ++k) passAdd(b + 2 * k, added * mk(shares[k].x, shares[k].y, shares[k].z));
    } else {
        creditPath(P, path, added, false);
    }
}

// ---- closest hit over a queue -----------------------------------------------------------------
// Closest hit for every queued ray; kBin then bins the rays by shading key (miss or the hit
// material's type) so that the shading kernels run warps of one material kind.  Traversals of
// pe_tuning::closest_traversal: 0 the binary tree in the reference's order, one lane per ray; 1-9 the
// 4-wide tree in the converged walk of pe_walk.cuh (one kernel for all these numbers).
enum TraceMode { TRACE_BINARY = 0, TRACE_DEFAULT = 6, TRACE_MODES = 10 };

// The shading key of a closest hit by its primitive.
__device__ __forceinline__ int shadeKeyOfPrim(const SceneGPU& S, uint32_t rayMask, int prim) {
    if (rayMask & RAY_WALK) return kShadeKeys - 1;
    if (isMiss(prim)) return 0;
    if (isInstanceHit(prim)) return 1 + S.materials[S.instances[instanceOfHit(prim)].material].type;
    return 1 + static_cast<int>((__float_as_uint(__ldg(&S.tris[3 * prim + 1]).w) >> 8) & 0xFFu);
}

// The shading key of a hit by the record of its triangle or sphere.
__device__ __forceinline__ uint8_t shadeKeyOfMeta(uint32_t rayMask, uint32_t meta) {
    return static_cast<uint8_t>((rayMask & RAY_WALK) ? kShadeKeys - 1 : 1 + ((meta >> 8) & 0xFFu));
}

// The binary tree, a ray per lane.
template <bool COUNT>
__global__ void __launch_bounds__(128) kIntersectBinary(const __grid_constant__ SceneGPU S, const __grid_constant__ Paths P, const int32_t* queue,
                                                        unsigned long long* stats) {
    const int n = static_cast<int>(P.now[BC_QUEUE]);
    uint32_t nodes = 0, tris = 0;
    for (;;) {
        const int base = warpFetch(&P.now[BC_WORK_ISECT]);
        if (base >= n) break;
        const int i = base + (threadIdx.x & 31);
        if (i >= n) continue;
        const int slot = queue[i];
        const float4 ro = P.rayO[slot];
        const float4 rd = P.rayD[slot];
        const Hit h = traceClosest<COUNT>(S, mk(ro.x, ro.y, ro.z), mk(rd.x, rd.y, rd.z), __float_as_uint(ro.w), 0.0f, 1e30f,
                                          nodes, tris, pathTime(S, P, slot));
        P.hit[slot] = make_float4(h.t, h.u, h.v, __int_as_float(h.prim));
        P.key[slot] = kKeyOfPrim;
    }
    if (COUNT) {
        atomicAdd(&stats[0], static_cast<unsigned long long>(nodes));
        atomicAdd(&stats[1], static_cast<unsigned long long>(tris));
    }
}

// Surface coverage of a hit for a ray that may pass through cutouts (DisneyMaterial::opacity,
// disney.cpp:505-509: the opacity times the opacity map's red channel, a level-0 lookup).
static __device__ __noinline__ float mappedOpacity(const SceneGPU& S, const MatGPU& m, const Isect& is) {
    ShadePoint sp;
    sp.uv = is.uv;
    sp.p = is.point;
    sp.n = is.normal;
    sp.ng = is.ng;
    const V2 uv = textureCoord(m, sp);
    return m.opacity * sclamp(texBilinear(S.textures[m.texOpacity], uv.x, uv.y, 0).x, 0.0f, 1.0f);
}
__device__ __forceinline__ float surfaceOpacity(const SceneGPU& S, const MatGPU& m, const Isect& is) {
    if (m.type != PE_MAT_DISNEY) return 1.0f;
    return m.texOpacity >= 0 ? mappedOpacity(S, m, is) : m.opacity;
}

// passesCutout (path_tracer.cpp:161-167): true = the ray goes on through this hit.
__device__ __forceinline__ bool passesCutout(const SceneGPU& S, const MatGPU& m, const Isect& is, Sobol& sb) {
    const float alpha = surfaceOpacity(S, m, is);
    if (alpha >= 1.0f) return false;
    if (alpha <= 0.0f) return true;
    return get1D(sb) >= alpha;
}

// russianRoulette (path_tracer.cpp:131-137): false ends the path.
__device__ __forceinline__ bool russianRoulette(V3& thr, Sobol& sb) {
    const float m = smax3(thr.x, thr.y, thr.z);
    if (m >= 1.0f) return true;
    if (!(m > 0.0f) || get1D(sb) >= m) return false;
    thr /= m;
    return true;
}

enum SegmentOutcome { SEG_SURFACE = 0, SEG_SCATTERED = 1, SEG_END = 2 };

// Absorption and scattering over the segment a path just travelled inside the medium of the
// innermost volume boundary it entered (path_tracer.cpp:456-479).  SEG_SCATTERED sets up the
// next ray (origin newO, direction newD).
static __device__ __noinline__ int mediumSegment(const TablesGPU* T, const MatGPU& mm, V3 segStart, V3 dir, bool hit, V3 hitPoint,
                                          Sobol& sb, V3& thr, uint32_t& volCtr, V3& newO, V3& newD) {
    const float dirLen = length(dir);
    const float segment = hit ? length(hitPoint - segStart) : kFltMax;
    const V3 sA = m3f(mm.sigmaA), sS = m3f(mm.sigmaS);
    if (mm.flags & MF_MEDIUM_SCATTERS) {
        const float uc = get1D(sb);
        const float u = get1D(sb);
        float t = 0.0f;
        if (sampleFreeFlight(sA + sS, sS, segment, hit, thr, uc, u, thr, t)) {
            const uint32_t events = (volCtr & 0xFFFFu) + 1u;
            volCtr = (volCtr & 0xFFFF0000u) | events;
            if (events > static_cast<uint32_t>(kMaxMediumEvents) || !isFinite3(thr)) return SEG_END;
            const V3 d = dir / dirLen;
            newO = segStart + d * t;
            newD = sampleHG(d, mm.mediumG, get2D(T, sb));
            if (events > 8u && !russianRoulette(thr, sb)) return SEG_END;
            return SEG_SCATTERED;
        }
    } else if (hit) {
        thr *= expNeg(sA, segment);
    } else if (!isBlack(sA)) {
        return SEG_END; // open mesh: an infinitely long absorbing segment
    }
    if (isBlack(thr) || !isFinite3(thr)) return SEG_END;
    return SEG_SURFACE;
}

// The next segment of a path that scatters before the hit its current ray has in P.hit: a step
// of a random subsurface walk (shadeSlot's PF_WALK state, path_tracer.cpp:263-303) or an event in the
// medium the ray is in (mediumSegment).  True: the path's state has moved on to the segment `next`.
// False, and nothing is changed: the ray's end is shadeSlot's to handle, which draws the same numbers.
struct ScatterRay {
    V3 o, d;
    uint32_t mask;
};
static __device__ __noinline__ bool scatterOn(const SceneGPU& S, const Paths& P, const Wave& W, int slot, ScatterRay& next) {
    const float4 hr = P.hit[slot];
    const float t = hr.x, u = hr.y, v = hr.z;
    const int prim = __float_as_int(hr.w);
    const float4 ro = P.rayO[slot];
    const uint32_t mask = __float_as_uint(ro.w);
    const bool walk = (mask & RAY_WALK) != 0;
    float4 md = P.med[slot];
    int top = -1;
    if (!walk) {
        MediaStack media;
        media.lo = __float_as_uint(md.x);
        media.hi = __float_as_uint(md.y);
        media.n = __float_as_int(md.w);
        top = media.top();
        if (top < 0 || !(S.materials[top].flags & MF_HAS_MEDIUM) || !(S.materials[top].flags & MF_MEDIUM_SCATTERS)) return false;
    }
    const TablesGPU* T = S.tables;
    const bool hit = !isMiss(prim);
    const float4 rd = P.rayD[slot], pp = P.pickP[slot];
    float4 th = P.thr[slot], ln = P.lastN[slot], lp = P.lastP[slot];
    const V3 o = mk(ro.x, ro.y, ro.z), dir = mk(rd.x, rd.y, rd.z);
    const int path = pathOfSlot(P, slot);
    const WaveSeg& A = W.segs[segOfSlot(W, path)];
    Sobol sb;
    sb.pixelHash = __float_as_uint(pp.w);
    sb.revIndex = rev32(static_cast<uint32_t>(A.sampleFirst + sampleOfPath(A, path)));
    sb.dim = __float_as_uint(lp.w);
    V3 thr = mk(th.x, th.y, th.z);
    uint32_t volCtr = __float_as_uint(md.z);
    uint32_t flags = __float_as_uint(ln.w);
    if (walk) {
        const V3 sigT = mk(lp.x, lp.y, lp.z), alb = mk(ln.x, ln.y, ln.z);
        uint32_t step = volCtr >> 16;
        const float uc = get1D(sb);
        const float uf = get1D(sb);
        float ts = 0.0f;
        if (!sampleFreeFlight(sigT, alb * sigT, hit ? t : kFltMax, hit, thr * alb, uc, uf, thr, ts)) return false;
        if (!isFinite3(thr) || isBlack(thr)) return false;
        next.o = o + dir * ts;
        next.d = sampleHG(dir, pp.x, get2D(T, sb));
        next.mask = mask;
        if ((step >= 8u && !russianRoulette(thr, sb)) || ++step >= static_cast<uint32_t>(kMaxWalkSteps)) return false;
        volCtr = (volCtr & 0xFFFFu) | (step << 16);
    } else {
        if (flags & PF_FIRST_SEGMENT) return false;
        V3 point = mk(0.0f);
        if (hit) {
            Hit h;
            h.t = t;
            h.u = u;
            h.v = v;
            h.prim = prim;
            Isect is;
            fillHit(S, h, o, dir, is, pathTime(S, P, slot));
            // surfaces the ray may pass through before the medium is asked
            const MatGPU& m = S.materials[is.material];
            if ((flags & PF_CAMERA_RAY) && (S.shapes[is.shape].flags & SF_CAMERA_INVISIBLE)) return false;
            if (m.type == PE_MAT_DISNEY && (m.opacity < 1.0f || m.texOpacity >= 0)) return false;
            point = is.point;
        }
        if (mediumSegment(T, S.materials[top], o, dir, hit, point, sb, thr, volCtr, next.o, next.d) != SEG_SCATTERED) return false;
        next.mask = VIS_DIFFUSE;
        flags = (flags | PF_SPECULAR_BOUNCE) & ~PF_CAMERA_RAY;
        if (S.hasMips && P.cone) P.cone[slot] = make_float2(0.0f, 0.0f);
    }
    P.rayO[slot] = make_float4(next.o.x, next.o.y, next.o.z, __uint_as_float(next.mask));
    P.rayD[slot] = make_float4(next.d.x, next.d.y, next.d.z, rd.w);
    P.thr[slot] = make_float4(thr.x, thr.y, thr.z, th.w);
    ln.w = __uint_as_float(flags);
    P.lastN[slot] = ln;
    lp.w = __uint_as_float(sb.dim);
    P.lastP[slot] = lp;
    md.z = __uint_as_float(volCtr);
    P.med[slot] = md;
    return true;
}

// A warp's share of a queue: it takes 32 entries at a time from the global cursor and hands them to
// lanes that ask.  All 32 lanes call next(); a lane that wants an entry gets its number, or -1.
struct WarpFeed {
    uint32_t* cursor;
    int n;
    int at = 0, end = 0;
    __device__ __forceinline__ int next(bool want) {
        const unsigned lanes = __ballot_sync(kWarp, want);
        const int rank = __popc(lanes & ((1u << (threadIdx.x & 31)) - 1u));
        const int wanted = __popc(lanes);
        const int had = end - at, from = at;
        if (had < wanted && end >= 0) {
            const int base = warpFetch(cursor);
            at = base + wanted - had;
            if (base >= n) {
                end = -1; // the queue is empty
                at = -1;
                return want && rank < had ? from + rank : -1;
            }
            end = min(base + 32, n);
            const int i = rank < had ? from + rank : base + rank - had;
            if (at > end) at = end;
            return want && (rank < had || i < end) ? i : -1;
        }
        if (end < 0) return -1;
        at += wanted;
        return want ? from + rank : -1;
    }
    __device__ __forceinline__ bool dry() const { return end < 0; }
};

// Material::shadowTransmittance: thin-walled glass passes (1 − R_thin)·tint, a cutout Disney
// surface 1 − opacity, every other surface nothing.
__device__ __forceinline__ V3 surfaceShadowTransmittance(const SceneGPU& S, const MatGPU& m, const Isect& is, V3 dir) {
    if (m.type == PE_MAT_DIELECTRIC) return glassShadowTransmittance(m, is.ng, is.normal, dir);
    if (m.type == PE_MAT_DISNEY) return mk(1.0f - surfaceOpacity(S, m, is));
    return mk(0.0f);
}

// Scene::hasShadowLinkFor: light `light` (explicit, else -1) lets some blockers through.
__device__ __forceinline__ bool shadowLinkFor(const SceneGPU& S, int light) {
    return S.hasShadowLinks && light >= 0 && S.links[light].shadowMode != 0;
}

// shadowTransmittance (path_tracer.cpp:172-202).  Without shadow-transmitting materials or a
// shadow link for the light it is the any-hit test; otherwise the shadow ray walks from surface
// to surface (at most 64), passing the blockers the light's shadow link leaves out and
// multiplying the transmittance of thin-walled glass and cutouts, and stops black at any other
// surface.
template <bool COUNT>
__device__ V3 shadowVisibility(const SceneGPU& S, V3 o, V3 d, float tMax, int light, uint32_t& nodes, uint32_t& tris,
                              float time) {
    const bool link = shadowLinkFor(S, light);
    if (!S.hasShadowTransmitters && !link)
        return traceAnyWide<COUNT>(S, o, d, VIS_SHADOW, 0.0f, tMax, nodes, tris, time) ? mk(0.0f) : mk(1.0f);
    V3 T = mk(1.0f);
    V3 origin = o;
    float remaining = tMax;
    for (int i = 0; i < 64; ++i) {
        const Hit h = traceClosestWide<COUNT>(S, origin, d, VIS_SHADOW, 0.0f, remaining, nodes, tris, time);
        if (isMiss(h.prim)) return T;
        Isect is;
        fillHit(S, h, origin, d, is, time);
        if (link && !linkAllows(S.links[light].shadowMode, S.links[light].shadowMask, S.shapes[is.shape].linkNode)) {
            origin = offsetRayOrigin(is.point, is.pError, len2(is.ng) > 0.0f ? is.ng : is.normal, d);
            remaining -= h.t;
            if (remaining <= 0.0f) return T;
            continue;
        }
        const MatGPU& m = S.materials[is.material];
        if (!(m.flags & MF_TRANSMITS_SHADOWS)) return mk(0.0f);
        T *= surfaceShadowTransmittance(S, m, is, d);
        if (isBlack(T)) return T;
        origin = offsetRayOrigin(is.point, is.pError, len2(is.ng) > 0.0f ? is.ng : is.normal, d);
        remaining -= h.t;
        if (remaining <= 0.0f) return T;
    }
    return mk(0.0f);
}

// A NEE sample's term: throughput × f·Li·vis·(cos·w / (lightPdf·n)), clamped when indirect
// (path_tracer.cpp:683-690).
__device__ __forceinline__ V3 neeTerm(V3 fLi, V3 vis, float scalar, V3 thr, bool indirect, float clampIndirect) {
    const V3 neeLocal = (fLi * vis) * scalar;
    V3 c = thr * neeLocal;
    if (indirect && clampIndirect > 0.0f) {
        const float m = smax3(c.x, c.y, c.z);
        if (m > clampIndirect) c = c * (clampIndirect / m);
    }
    return c;
}

// ---- any hit over the shadow queue ------------------------------------------------------------
// Shadow record i's visibility, found, into its path's radiance.
__device__ __forceinline__ void addShadowTerm(const SceneGPU& S, const Paths& P, int i, int slot, float scalar, V3 vis) {
    float4* const at = slot >= 0 ? P.L + slot : P.Lout + ~slot; // ~path: the path has ended (Paths::direct)
    const float4 sc = P.shC[i];
    const float4 st = P.shT[i];
    const V3 c = neeTerm(mk(sc.x, sc.y, sc.z), vis, scalar, mk(st.x, st.y, st.z), (__float_as_uint(sc.w) & 1u) != 0, st.w);
    if (!isFinite3(c)) return;
    float4 L = *at;
    L.x += c.x;
    L.y += c.y;
    L.z += c.z;
    *at = L;
    if (P.pass) {
        const int light = static_cast<int>(__float_as_uint(sc.w) >> 1) - 1;
        const float4* shares = P.shPass + 3 * static_cast<size_t>(i);
        creditNee(S, P, pathOfSlot(P, slot), light, c, shares[0].w != 0.0f ? shares : nullptr);
    }
}

// Scenes with shadow-transmitting surfaces or shadow links: a ray per lane, the transmittance walk.
template <bool COUNT>
__global__ void __launch_bounds__(128) kShadow(const __grid_constant__ SceneGPU S, const __grid_constant__ Paths P, unsigned long long* stats) {
    const int n = static_cast<int>(P.now[BC_SHADOW]);
    uint32_t nodes = 0, tris = 0;
    for (;;) {
        const int base = warpFetch(&P.now[BC_WORK_SHADOW]);
        if (base >= n) break;
        const int i = base + (threadIdx.x & 31);
        if (i >= n) continue;
        const int slot = P.shadowQ[i];
        const float4 so = P.shO[i];
        const float4 sd = P.shD[i];
        const int light = static_cast<int>(__float_as_uint(P.shC[i].w) >> 1) - 1;
        const V3 vis = shadowVisibility<COUNT>(S, mk(so.x, so.y, so.z), mk(sd.x, sd.y, sd.z), so.w, light, nodes, tris,
                                               pathTime(S, P, slot));
        if (!isBlack(vis)) addShadowTerm(S, P, i, slot, sd.w, vis);
    }
    if (COUNT) {
        atomicAdd(&stats[2], static_cast<unsigned long long>(nodes));
        atomicAdd(&stats[3], static_cast<unsigned long long>(tris));
    }
}

// The closest hits of a queue over the 4-wide tree, a ray per lane (walkTurn); all 32 lanes call it.
// A ray that scatters before its hit (a step of a subsurface walk, an event in a medium) goes on from
// there at once (scatterOn): such chains, up to hundreds of segments long, would otherwise take a
// bounce of the whole wave per segment.  `segments` counts their further rays.  At most kScatterChain
// segments a bounce: the bounce lasts as long as its longest chain (1280x720 x 4-spp media wave, rays
// and shading and tail together: 19.8 ms at 2 and at 4, 20.7 at 8, 21.5 at 16, 30 unbounded, 21.7 at 0).
constexpr int kScatterChain = 4;
template <bool COUNT, bool SCATTER, bool INSTANCES>
__device__ __forceinline__ void traceQueue(const SceneGPU& S, const Paths& P, const Wave& W, const int32_t* queue,
                                           uint2* stack, int root, uint32_t& nodes, uint32_t& tris, uint32_t& segments) {
    WarpFeed feed{&P.now[BC_WORK_ISECT], static_cast<int>(P.now[BC_QUEUE])};
    int slot = -1, chain = 0;
    RayWalk w;
    w.cur = kRayDone;
    for (;;) {
        const unsigned idle = __ballot_sync(kWarp, w.cur == kRayDone);
        if (idle == kWarp || (!feed.dry() && __popc(idle) >= kRefill)) {
            // ended rays (a hit is in P.hit already); then the queue's next rays
            if (w.cur == kRayDone && slot >= 0) {
                ScatterRay next;
                if (w.prim == -1) {
                    P.hit[slot] = make_float4(w.tMax, 0.0f, 0.0f, __int_as_float(-1));
                    P.key[slot] = static_cast<uint8_t>((w.mask & RAY_WALK) ? kShadeKeys - 1 : 0);
                }
                if (SCATTER && chain < kScatterChain && scatterOn(S, P, W, slot, next)) {
                    w.start(S, root, next.o, next.d, next.mask, 1e30f, -1);
                    ++segments;
                    ++chain;
                } else {
                    slot = -1;
                }
            }
            const int i = feed.next(slot < 0);
            if (i >= 0) {
                slot = queue[i];
                chain = 0;
                const float4 ro = P.rayO[slot];
                const float4 rd = P.rayD[slot];
                w.start(S, root, mk(ro.x, ro.y, ro.z), mk(rd.x, rd.y, rd.z), __float_as_uint(ro.w), 1e30f, -1);
            }
            if (__all_sync(kWarp, slot < 0)) break;
            continue;
        }
        walkTurn<WALK_CLOSEST, COUNT, INSTANCES>(
            S, w, stack, nodes, tris,
            [&](V3& o, V3& d, uint32_t& mask) {
                const float4 ro = P.rayO[slot], rd = P.rayD[slot];
                o = mk(ro.x, ro.y, ro.z);
                d = mk(rd.x, rd.y, rd.z);
                mask = __float_as_uint(ro.w);
            },
            [&]() { return pathTime(S, P, slot); },
            [&](float t, float u, float v, int prim, uint32_t meta) {
                P.hit[slot] = make_float4(t, u, v, __int_as_float(prim));
                P.key[slot] = INSTANCES && w.inst >= 0 ? kKeyOfPrim : shadeKeyOfMeta(w.mask, meta);
            });
        __syncwarp();
    }
}

// The plain any-hit queries of the shadow records, a ray per lane.
template <bool COUNT, bool INSTANCES>
__device__ __forceinline__ void traceShadows(const SceneGPU& S, const Paths& P, uint32_t* stack, int root, uint32_t& nodes,
                                             uint32_t& tris) {
    WarpFeed feed{&P.now[BC_WORK_SHADOW], static_cast<int>(P.now[BC_SHADOW])};
    int rec = -1;
    RayWalk w;
    w.cur = kRayDone;
    for (;;) {
        const unsigned idle = __ballot_sync(kWarp, w.cur == kRayDone);
        if (idle == kWarp || (!feed.dry() && __popc(idle) >= kRefill)) {
            if (w.cur == kRayDone && rec >= 0) {
                if (w.prim == 0) addShadowTerm(S, P, rec, P.shadowQ[rec], P.shD[rec].w, mk(1.0f));
                rec = -1;
            }
            __syncwarp();
            const int i = feed.next(w.cur == kRayDone);
            if (i >= 0) {
                rec = i;
                const float4 so = P.shO[i];
                const float4 sd = P.shD[i];
                w.start(S, root, mk(so.x, so.y, so.z), mk(sd.x, sd.y, sd.z), VIS_SHADOW, so.w, 0);
            }
            if (__all_sync(kWarp, rec < 0)) break;
            continue;
        }
        walkTurn<WALK_ANY, COUNT, INSTANCES>(
            S, w, stack, nodes, tris,
            [&](V3& o, V3& d, uint32_t& mask) {
                const float4 so = P.shO[rec], sd = P.shD[rec];
                o = mk(so.x, so.y, so.z);
                d = mk(sd.x, sd.y, sd.z);
                mask = VIS_SHADOW;
            },
            [&]() { return pathTime(S, P, P.shadowQ[rec]); }, [](float, float, float, int, uint32_t) {});
        __syncwarp();
    }
}

// A bounce's ray queries in one launch: the closest hits of its queue, then (`shadows`) the shadow
// rays the bounce before left.  The two do not depend on each other (shadow rays only add to the
// radiance that the next shading reads), and a launch's time for a short queue is that of its longest
// ray; warps that run out of closest hits go on with shadow rays while the long ones finish.
// SCATTER: the scene has media or subsurface walks (scatterOn's call costs the others 6 %).
template <bool COUNT, bool SCATTER, bool INSTANCES>
__global__ void __launch_bounds__(128, 8) kTrace(const __grid_constant__ SceneGPU S, const __grid_constant__ Paths P,
                                                 const __grid_constant__ Wave W, const int32_t* queue, int shadows,
                                                 unsigned long long* stats) {
    uint2 stack[walkStack(INSTANCES)];
    const int root = rootRef(S);
    uint32_t nodes = 0, tris = 0, shNodes = 0, shTris = 0, segments = 0;
    traceQueue<COUNT, SCATTER, INSTANCES>(S, P, W, queue, stack, root, nodes, tris, segments);
    if (segments) atomicAdd(&stats[8], static_cast<unsigned long long>(segments));
    if (shadows) traceShadows<COUNT, INSTANCES>(S, P, reinterpret_cast<uint32_t*>(stack), root, shNodes, shTris);
    if (COUNT) {
        atomicAdd(&stats[0], static_cast<unsigned long long>(nodes));
        atomicAdd(&stats[1], static_cast<unsigned long long>(tris));
        atomicAdd(&stats[2], static_cast<unsigned long long>(shNodes));
        atomicAdd(&stats[3], static_cast<unsigned long long>(shTris));
    }
}

// The shadow rays alone (waves whose radiance is needed before the next closest hits).
template <bool COUNT>
__global__ void __launch_bounds__(128, 8) kShadowAny(const __grid_constant__ SceneGPU S, const __grid_constant__ Paths P,
                                                     unsigned long long* stats) {
    uint32_t stack[walkStack(true)];
    uint32_t nodes = 0, tris = 0;
    traceShadows<COUNT, true>(S, P, stack, rootRef(S), nodes, tris);
    if (COUNT) {
        atomicAdd(&stats[2], static_cast<unsigned long long>(nodes));
        atomicAdd(&stats[3], static_cast<unsigned long long>(tris));
    }
}

// accumulate(): adds a finite term and returns it; a non-finite one is skipped and counts as
// black (path_tracer.cpp:355-359).
__device__ __forceinline__ V3 addL(float4& L, V3 c) {
    if (!isFinite3(c)) return mk(0.0f);
    L.x += c.x;
    L.y += c.y;
    L.z += c.z;
    return c;
}

// ---- learned proposal in the shading step ------------------------------------------------------
// Vertices the proposal may serve: non-delta surfaces that are neither volume boundaries nor
// shadow transmitters (the reference's useGuiding condition, path_tracer.cpp:623-626).
__device__ __forceinline__ bool guidable(const MatGPU& m) {
    return (m.flags & (MF_DELTA | MF_VOLUME_BOUNDARY | MF_TRANSMITS_SHADOWS)) == 0;
}

__device__ __forceinline__ const float4* slotMixture(const Paths& P, int slot) {
    return P.guideOut + static_cast<size_t>(slot) * kSlotMixture;
}

static __device__ __noinline__ float guidePdf(const Paths& P, int slot, V3 w) { return mixturePdf(slotMixture(P, slot), w); }

// Training record of a path's first guidable vertex; its radiance along wi is what the path adds
// from here on (kGuideCollect).  False when the path has one already.
static __device__ __noinline__ bool guideRecord(const Paths& P, int slot, V3 p, V3 n, V3 wo, V3 wi, V3 thrBefore) {
    float4* rec = P.guideRec + static_cast<size_t>(slot) * 6;
    if (rec[4].w != 0.0f) return false;
    rec[0] = make_float4(p.x, p.y, p.z, 0.0f);
    rec[1] = make_float4(n.x, n.y, n.z, 0.0f);
    rec[2] = make_float4(wo.x, wo.y, wo.z, 0.0f);
    rec[3] = make_float4(wi.x, wi.y, wi.z, 0.0f);
    rec[4] = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
    rec[5] = make_float4(thrBefore.x, thrBefore.y, thrBefore.z, 0.0f);
    return true;
}

// One-sample MIS of the proposal and the BSDF, 50/50 (path_tracer.cpp:703-735 with the
// learned mixture in place of the SD-tree): the branch number picks the strategy, the
// proposal draws a lobe from the rest of it and a direction from one get2D.
static __device__ __noinline__ bool guidedSample(const TablesGPU* T, const MatGPU& mat, V3 wo, const ShadePoint& sp, const Paths& P,
                                          int slot, const DisneyVertex* dv, Sobol& sb, BsdfSample& bs) {
    const float4* mix = slotMixture(P, slot);
    const float uBranch = get1D(sb);
    if (uBranch < 0.5f) {
        const V3 gwi = mixtureSample(mix, uBranch * 2.0f, get2D(T, sb));
        const float gPdf = mixturePdf(mix, gwi);
        if (!(gPdf > 0.0f)) return false;
        float bPdf = 0.0f;
        const V3 f = bsdfEvalPdfT<-1>(T, mat, wo, gwi, sp, dv, bPdf, nullptr);
        const float mixPdf = 0.5f * gPdf + 0.5f * bPdf;
        if (isBlack(f) || !(mixPdf > 0.0f)) return false;
        bs.wi = gwi;
        bs.f = f;
        bs.pdf = mixPdf;
        bs.delta = false;
        bs.passThrough = false;
        bs.subsurface = false;
        bs.weight = mk(0.0f);
        return true;
    }
    const float uc = get1D(sb);
    const V2 u2 = get2D(T, sb);
    if (!bsdfSampleT<-1>(T, mat, wo, sp, dv, uc, u2, bs)) return false;
    if (bs.subsurface) bs.weight = bs.weight * 2.0f;
    else if (bs.delta || bs.passThrough) bs.pdf *= 0.5f;
    else if (bs.pdf > 0.0f) bs.pdf = 0.5f * bs.pdf + 0.5f * mixturePdf(mix, bs.wi);
    return true;
}

// The same one-sample MIS with the SD-tree's sampling quadtree rooted at `root`
// (path_tracer.cpp:703-735): a direction from one get2D on the guide branch, the BSDF's
// get1D + get2D on the other.
static __device__ __noinline__ bool sdGuidedSample(const TablesGPU* T, const MatGPU& mat, V3 wo, const ShadePoint& sp,
                                            const SdQuad* tree, int root, const DisneyVertex* dv, Sobol& sb,
                                            BsdfSample& bs) {
    const float uBranch = get1D(sb);
    if (uBranch < 0.5f) {
        float gPdf = 0.0f;
        const V3 gwi = sdTreeSample(tree, root, get2D(T, sb), gPdf);
        if (!(gPdf > 0.0f)) return false;
        float bPdf = 0.0f;
        const V3 f = bsdfEvalPdfT<-1>(T, mat, wo, gwi, sp, dv, bPdf, nullptr);
        const float mixPdf = 0.5f * gPdf + 0.5f * bPdf;
        if (isBlack(f) || !(mixPdf > 0.0f)) return false;
        bs.wi = gwi;
        bs.f = f;
        bs.pdf = mixPdf;
        bs.delta = false;
        bs.passThrough = false;
        bs.subsurface = false;
        bs.weight = mk(0.0f);
        return true;
    }
    const float uc = get1D(sb);
    const V2 u2 = get2D(T, sb);
    if (!bsdfSampleT<-1>(T, mat, wo, sp, dv, uc, u2, bs)) return false;
    if (bs.subsurface) bs.weight = bs.weight * 2.0f;
    else if (bs.delta || bs.passThrough) bs.pdf *= 0.5f;
    else if (bs.pdf > 0.0f) bs.pdf = 0.5f * bs.pdf + 0.5f * sdTreePdf(tree, root, bs.wi);
    return true;
}

// ---- surface effects of Li that cast rays of their own ------------------------------------------
// Contact ambient occlusion (approxAo, path_tracer.cpp:27-45): `samples` cosine rays of at most
// 0.35 over the shading normal; the path's throughput is scaled by lerp(1, visibility, strength).
static __device__ __noinline__ float approxAo(const SceneGPU& S, const Isect& is, Sobol& sb, float strength, int samples,
                                       float time) {
    if (strength <= 0.0f || samples <= 0) return 1.0f;
    const TablesGPU* T = S.tables;
    const Frame frame = frameFromNormal(is.normal);
    float occ = 0.0f;
    uint32_t n0 = 0, n1 = 0;
    for (int i = 0; i < samples; ++i) {
        const V3 local = sampleCosineHemisphere(get2D(T, sb));
        const V3 dir = normalize(toWorld(frame, local));
        if (traceAnyWide<false>(S, spawnOrigin(is, dir), dir, VIS_SHADOW, 0.0f, 0.35f, n0, n1, time)) occ += 1.0f;
    }
    const float visibility = 1.0f - (occ / static_cast<float>(samples));
    return lerpf(1.0f, visibility, strength);
}

// Rounded edges (roundedEdgeNormal, path_tracer.cpp:209-255): six points on a disk of `radius`
// around the hit, each probed along one of the frame's axes (normal ½, tangents ¼ each) from both
// sides with rays of 2·radius; the outward normals of hits on the same shape within 1.5·radius,
// weighted by their projection on the probe axis, average with a quarter of the own normal.
static __device__ __noinline__ V3 roundedEdgeNormal(const SceneGPU& S, const Isect& is, float radius, Sobol& sb, float time) {
    const TablesGPU* T = S.tables;
    const V3 N = is.normal;
    const Frame f = frameFromNormal(N);
    V3 sum = N * 0.25f;
    uint32_t n0 = 0, n1 = 0;
    for (int i = 0; i < 6; ++i) {
        const float ua = get1D(sb);
        const V2 dd = sampleDiskConcentric(get2D(T, sb));
        const V2 d = mk2(dd.x * radius, dd.y * radius);
        V3 axis, s, t;
        if (ua < 0.5f) {
            axis = f.n; s = f.s; t = f.t;
        } else if (ua < 0.75f) {
            axis = f.s; s = f.t; t = f.n;
        } else {
            axis = f.t; s = f.n; t = f.s;
        }
        for (int k = 0; k < 2; ++k) {
            const float sign = k == 0 ? 1.0f : -1.0f;
            const V3 origin = is.point + s * d.x + t * d.y + axis * (sign * radius);
            const V3 rdir = axis * -sign;
            const Hit h = traceClosestWide<false>(S, origin, rdir, VIS_ALL, 0.0f, 2.0f * radius, n0, n1, time);
            if (isMiss(h.prim)) continue;
            Isect hit;
            fillHit(S, h, origin, rdir, hit, time);
            if (hit.shape != is.shape) continue;
            if (len2(hit.point - is.point) > 2.25f * radius * radius) continue;
            const V3 outward = hit.frontFace ? hit.normal : -hit.normal;
            sum += outward * fabsf(dot(outward, axis));
        }
    }
    V3 n = normalize(sum);
    const V3 outwardN = is.frontFace ? N : -N;
    if (dot(n, outwardN) < 0.0f) n = -n;
    return is.frontFace ? n : -n;
}

// Shadow catcher (path_tracer.cpp:515-563): a camera ray that hits the catcher sees the
// background `bg` times the share `ratio` of the direct light, over 4 × shadowSamples NEE
// samples, that reaches the hit point.
static __device__ __noinline__ V3 shadowCatcher(const SceneGPU& S, const Isect& is, V3 dir, int shadowSamples, Sobol& sb,
                                         float& ratioOut, float time) {
    const TablesGPU* T = S.tables;
    V3 bg = mk(0.0f);
    if (S.bgMode == PE_BG_COLOR) bg = m3f(S.bgColor);
    else if (S.bgMode == PE_BG_ENVIRONMENT && S.env.present) bg = envEval(S.env, dir);
    float visible = 0.0f, total = 0.0f;
    if (S.lightCount > 0) {
        LightCtx picker;
        lightPrepare(S, is.point, is.normal, picker);
        const int n = 4 * shadowSamples;
        uint32_t n0 = 0, n1 = 0;
        for (int k = 0; k < n; ++k) {
            float pmf = 0.0f;
            const int li = lightCtxSample(S, picker, get1D(sb), pmf);
            if (li < 0 || !(pmf > 0.0f)) {
                (void)get2D(T, sb);
                continue;
            }
            if (li < S.nLights && S.hasLightLinks &&
                !linkAllows(S.links[li].mode, S.links[li].mask, S.shapes[is.shape].linkNode)) {
                (void)get2D(T, sb);
                continue;
            }
            const V2 u = get2D(T, sb);
            const LightSample ls = li < S.nLights ? sampleLight(S.lights[li], is.point, u) : envSampleFull(S.env, S.envFull, u);
            const float cosT = dot(ls.wi, is.normal);
            if (!lsValid(ls) || cosT <= 0.0f) continue;
            const float c = luminance(ls.Li) * cosT / (pmf * ls.pdf);
            if (!(c > 0.0f) || !pe::finitef(c)) continue;
            total += c;
            V3 so, sd;
            float stMax;
            if (makeShadowRay(is, ls.wi, ls.distance, so, sd, stMax))
                visible += c * luminance(shadowVisibility<false>(S, so, sd, stMax, li < S.nLights ? li : -1, n0, n1, time));
        }
    }
    ratioOut = total > 0.0f ? sclamp(visible / total, 0.0f, 1.0f) : 1.0f;
    return bg;
}

// ---- shade: Li's loop body between two closest-hit queries ------------------------------------
// One path's step: reads the slot's state and hit record, adds the radiance found to L and
// writes back the state for its next closest-hit query.  A path is in one of three states at
// each query: an ordinary ray (medium segment, then the surface or the sky), a step of a random
// subsurface walk (PF_WALK), whose exit point is shaded at once as the walk's white-Lambert exit
// vertex, or a ray scattered inside a medium (an ordinary ray with specularBounce set).  NEE
// shadow rays go to the any-hit queue or to the caller, or with SHADOW_INLINE are traced here and their terms
// added to L at once, in the same order.  Returns whether the path goes on.
//
// FEAT: the features the instantiation carries, at least those its waves' scene and settings need
// (SceneGPU::features, waveFeatures); the others are compiled out, so that the code fits in registers.
// KEY >= 0 also fixes the shading key (0 a miss, 1 + material type a surface hit), -1 leaves it to the hit.
// What shadeSlot does with the shadow ray of a NEE sample: appends it to the any-hit queue, traces it
// at once, or hands it to the caller (one per vertex: waves with one shadow sample).
enum ShadowMode { SHADOW_QUEUE, SHADOW_INLINE, SHADOW_HAND };
// A shadow record: origin, tMax | direction, scalar (cos·w/(pdf·n)) | f·Li, flags (bit 0 indirect, bits
// 1.. the light index + 1, 0 the environment) | throughput, clamp.
struct ShadowRec {
    float4 o, d, c, t;
};

template <ShadowMode SHADOW, bool COUNT, bool OUT, int FEAT = FEAT_ALL, int KEY = -1>
__device__ __forceinline__ bool shadeSlot(const SceneGPU& S, const Paths& P, const WaveSeg& A, int slot, int path,
                                          uint32_t& shNodes, uint32_t& shTris, uint32_t& shRays,
                                          ShadowRec* hand = nullptr, bool* handed = nullptr) {
    constexpr bool MEDIA = (FEAT & FEAT_MEDIA) != 0, GUIDE = (FEAT & FEAT_GUIDE) != 0, REST = (FEAT & FEAT_REST) != 0;
    constexpr int MT = KEY >= 1 ? KEY - 1 : -1; // the material type a surface key fixes
    const TablesGPU* T = S.tables;
    const bool volumetric = MEDIA && (S.hasVolumes | S.hasSubsurface) != 0;
    bool cont = false;
    float4 ro = P.rayO[slot];
    float4 rd = P.rayD[slot];
    float4 th = P.thr[slot];
    float4 L = P.L[slot];
    float4 ln = P.lastN[slot];
    float4 lp = P.lastP[slot];
    float4 pp = P.pickP[slot];
    float4 pn = P.pickN[slot];
    const float4 hr = P.hit[slot];
    float4 md = volumetric ? P.med[slot] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    MediaStack media;
    media.lo = __float_as_uint(md.x);
    media.hi = __float_as_uint(md.y);
    media.n = __float_as_int(md.w);
    uint32_t volCtr = __float_as_uint(md.z);
    float lambda = th.w; // 0 = RGB path; > 0 = single-wavelength path after a dispersive hit
    uint32_t flags = __float_as_uint(ln.w);
    if (GUIDE && (flags & PF_GUIDE_SNAP)) {
        // radiance so far, the previous vertex's NEE included: the training record's baseline
        if (P.sdMode & SD_RECORD) {
            const uint32_t n = P.sdCount[slot];
            if (n > 0)
                P.sdRec[(static_cast<size_t>(slot) * kSdRecords + n - 1) * 4 + 3] = make_float4(L.x, L.y, L.z, 2.0f);
        } else {
            P.guideRec[static_cast<size_t>(slot) * 6 + 4] = make_float4(L.x, L.y, L.z, 2.0f);
        }
        flags &= ~PF_GUIDE_SNAP;
    }
    uint32_t ctr = __float_as_uint(pn.w);
    int depth = ctr & 0xFF, diffuseBounces = (ctr >> 8) & 0xFF, passThroughs = (ctr >> 16) & 0xFF,
        skips = (ctr >> 24) & 0xFF;
    Sobol sb;
    sb.pixelHash = __float_as_uint(pp.w);
    sb.revIndex = rev32(static_cast<uint32_t>(A.sampleFirst + sampleOfPath(A, path)));
    sb.dim = __float_as_uint(lp.w);
    V3 thr = mk(th.x, th.y, th.z);
    const V3 dir = mk(rd.x, rd.y, rd.z);
    const V3 rayO = mk(ro.x, ro.y, ro.z);
    const float lastBsdfPdf = rd.w;
    const bool specularBounce = flags & PF_SPECULAR_BOUNCE;
    bool cameraRay = flags & PF_CAMERA_RAY;
    const int shadowSamples = A.shadowSamples;
    const int explicitLights = S.nLights;
    const int prim = __float_as_int(hr.w);
    const bool hit = KEY == 0 ? false : (KEY > 0 ? true : !isMiss(prim));
    const float time = pathTime(S, P, slot);
    // ray cone (path_tracer.cpp:428-454, 777-783, 853-857): only scenes with mipmapped textures
    const bool cones = REST && S.hasMips && P.cone;
    float2 cone = cones ? P.cone[slot] : make_float2(0.0f, 0.0f);
    Isect is;
    bool done = false;
    bool vertex = false; // a surface vertex to shade (NEE + BSDF sampling) below
    bool exitVertex = false; // ... the exit vertex of a subsurface walk
    int shadowRec = -1;      // this vertex's record in the shadow queue
    V3 wo = -dir;
    if (MEDIA && (flags & PF_WALK)) {
        // one step of the random walk (path_tracer.cpp:263-303)
        const V3 sigT = mk(lp.x, lp.y, lp.z), alb = mk(ln.x, ln.y, ln.z);
        const V3 sigS = alb * sigT;
        uint32_t step = volCtr >> 16;
        const float uc = get1D(sb);
        const float uf = get1D(sb);
        float t = 0.0f;
        const bool scattered = sampleFreeFlight(sigT, sigS, hit ? hr.x : kFltMax, hit, thr * alb, uc, uf, thr, t);
        if (!isFinite3(thr) || isBlack(thr)) {
            done = true;
        } else if (!scattered) {
            if (!hit) {
                done = true; // escaped through open geometry
            } else {
                Hit h;
                h.t = hr.x;
                h.u = hr.y;
                h.v = hr.z;
                h.prim = prim;
                fillHit(S, h, rayO, dir, is, time);
                // exit vertex: outward normal, white Lambert; the depth does not grow
                is.normal = -is.normal;
                is.material = S.exitMaterial;
                flags &= ~PF_WALK;
                wo = is.normal;
                exitVertex = true;
                if (depth >= A.maxDepth) done = true;
                else vertex = true;
            }
        } else {
            const V3 no = rayO + dir * t;
            const V3 nd = sampleHG(dir, pp.x, get2D(T, sb));
            if ((step >= 8u && !russianRoulette(thr, sb)) || ++step >= static_cast<uint32_t>(kMaxWalkSteps)) {
                done = true;
            } else {
                ro = make_float4(no.x, no.y, no.z, ro.w);
                rd = make_float4(nd.x, nd.y, nd.z, rd.w);
                volCtr = (volCtr & 0xFFFFu) | (step << 16);
                cont = true;
            }
        }
    } else {
        if (hit) {
            Hit h;
            h.t = hr.x;
            h.u = hr.y;
            h.v = hr.z;
            h.prim = prim;
            fillHit(S, h, rayO, dir, is, time);
            // Camera-invisible light quads (for camera rays) and cutouts are passed through;
            // the vertex does not count (path_tracer.cpp:426-439).
            if (skips < 64 && ((cameraRay && (S.shapes[is.shape].flags & SF_CAMERA_INVISIBLE)) ||
                               (REST && passesCutout(S, S.materials[is.material], is, sb)))) {
                const V3 no = offsetRayOrigin(is.point, is.pError, is.ng, dir);
                ro = make_float4(no.x, no.y, no.z, ro.w);
                if (cones) cone.x = cone.x + cone.y * smax(0.0f, is.t);
                ++skips;
                cont = true;
                done = true;
            }
        }
        if (!done) {
            // AOVs of the camera path's first surface past the skipped ones (path_tracer.cpp:440-443;
            // tracePixel, renderer.cpp:177-203): albedo, normal and coverage, or the background
            // data passes of the first hit (tracePixel, renderer.cpp:162-176)
            if ((flags & PF_FIRST_SEGMENT) && (OUT && P.pass) && hit) {
                float4* b = passBlock(P, path);
                const float4 o = b[PASS_HIT];
                b[PASS_HIT] = make_float4(is.point.x, is.point.y, is.point.z, length(is.point - mk(o.x, o.y, o.z)));
                const float4 oc = S.idColor[is.shape];
                b[PASS_OBJECT] = make_float4(oc.x, oc.y, oc.z, 1.0f);
                b[PASS_MATERIAL] = S.idColor[S.nShapes + is.material];
                // Cryptomatte ids ride in the w of the id colours (renderer.cpp:170-175)
                b[PASS_CRYPTO] = make_float4(oc.w, b[PASS_MATERIAL].w, 0.0f, 0.0f);
            }
            if ((flags & PF_FIRST_SEGMENT) && OUT && P.aovA) {
                const int path = pathOfSlot(P, slot);
                if (hit) {
                    const V3 a = clamp3(m3f(S.materials[is.material].base), 0.0f, 1.0f);
                    P.aovA[path] = make_float4(a.x, a.y, a.z, 1.0f);
                    P.aovN[path] = make_float4(is.normal.x, is.normal.y, is.normal.z, 0.0f);
                } else {
                    V3 a = mk(0.0f);
                    if (S.bgMode == PE_BG_COLOR) a = m3f(S.bgColor);
                    else if (S.env.present) a = envEval(S.env, dir);
                    a = clamp3(a, 0.0f, 1.0f);
                    P.aovA[path] = make_float4(a.x, a.y, a.z, 0.0f);
                    P.aovN[path] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                }
            }
            flags &= ~PF_FIRST_SEGMENT;
            // inside an object: absorption and, when the medium scatters, free flight
            const int top = volumetric ? media.top() : -1;
            if (top >= 0 && (S.materials[top].flags & MF_HAS_MEDIUM)) {
                V3 no, nd;
                const int r = mediumSegment(T, S.materials[top], rayO, dir, hit, is.point, sb, thr, volCtr, no, nd);
                if (r == SEG_END) {
                    done = true;
                } else if (r == SEG_SCATTERED) {
                    // the next query starts at the scattering point; no NEE inside, so
                    // emission found next takes full weight
                    ro = make_float4(no.x, no.y, no.z, __uint_as_float(VIS_DIFFUSE));
                    rd = make_float4(nd.x, nd.y, nd.z, rd.w);
                    flags = (flags | PF_SPECULAR_BOUNCE) & ~PF_CAMERA_RAY;
                    if (cones) cone = make_float2(0.0f, 0.0f); // a new ray without a cone (path_tracer.cpp:465)
                    cont = true;
                    done = true;
                }
            }
        }
        if (!done) {
            if (!hit) {
                // environment / background (path_tracer.cpp:482-514)
                if (depth == 0 && S.bgMode != PE_BG_ENVIRONMENT) {
                    if (S.bgMode == PE_BG_COLOR) {
                        const V3 added = addL(L, thr * m3f(S.bgColor));
                        if ((OUT && P.pass)) {
                            passAdd(passBlock(P, path) + PASS_BACKGROUND, added);
                            creditGroup(S, P, path, S.envGroup, added);
                        }
                    } else if (passThroughs > 0 && OUT && P.aovA) {
                        // straight through thin glass to a transparent background: coverage is
                        // what the glass held back
                        P.aovA[pathOfSlot(P, slot)].w = smax(0.0f, 1.0f - luminance(thr));
                    }
                } else if (S.env.present) {
                    const V3 Le = envEval(S.env, dir);
                    float weight = 1.0f;
                    if (!specularBounce) {
                        float pmf = 0.0f;
                        if (flags & PF_PICKER_VALID) {
                            LightCtx c;
                            lightPrepare(S, mk(pp.x, pp.y, pp.z), mk(pn.x, pn.y, pn.z), c);
                            pmf = lightCtxPmf(S, c, explicitLights);
                        }
                        const float lightPdf = pmf * envPdf(S.env, dir);
                        weight = powerHeuristic(1, lastBsdfPdf, shadowSamples, lightPdf);
                    }
                    V3 c = thr * (Le * weight);
                    if (diffuseBounces >= 2 && A.clampIndirect > 0.0f) {
                        const float m = smax3(c.x, c.y, c.z);
                        if (m > A.clampIndirect) c = c * (A.clampIndirect / m);
                    }
                    const V3 added = addL(L, c);
                    if ((OUT && P.pass)) {
                        if (depth == 0) passAdd(passBlock(P, path) + PASS_BACKGROUND, added);
                        else creditPath(P, path, added, depth == 1);
                        creditGroup(S, P, path, S.envGroup, added);
                    }
                }
                done = true;
            } else if (REST && cameraRay && is.shape == S.catcherShape) {
                // the shadow catcher ends the camera path with the shadowed background
                float ratio = 1.0f;
                const V3 bg = shadowCatcher(S, is, dir, shadowSamples, sb, ratio, time);
                const V3 added = addL(L, thr * bg * ratio);
                if ((OUT && P.pass)) {
                    passAdd(passBlock(P, path) + PASS_BACKGROUND, added);
                    creditGroup(S, P, path, S.envGroup, added);
                }
                if (depth == 0 && OUT && P.aovA) {
                    // the catcher's AOVs: the background it shows, its shadow as coverage
                    const V3 a = clamp3(bg, 0.0f, 1.0f);
                    P.aovA[pathOfSlot(P, slot)] =
                        make_float4(a.x, a.y, a.z, S.bgMode == PE_BG_TRANSPARENT ? 1.0f - ratio : 1.0f);
                }
                done = true;
            } else {
                const MatGPU& mat = S.materials[is.material];
                // emission with MIS against the previous vertex's NEE (path_tracer.cpp:565-593)
                if (mat.flags & MF_EMISSIVE) {
                    const ShapeInfo& sh = S.shapes[is.shape];
                    int li = -1;
                    if (sh.emitter >= 0)
                        li = (sh.flags & SF_AREA_TRIANGLE) ? sh.emitter : sh.emitter + (is.tri - static_cast<int>(sh.firstTri));
                    // Light linking: the previous receiver must be linked to this light
                    // (path_tracer.cpp:571-572; camera rays always see it)
                    const bool linked = depth == 0 || li < 0 || !REST || !S.hasLightLinks ||
                                        linkAllows(S.links[li].mode, S.links[li].mask,
                                                   static_cast<int>((flags >> kPrevNodeShift) & 0xFFu));
                    float weight = 1.0f;
                    if (linked && !specularBounce) {
                        float lightPdf = 0.0f;
                        if (li >= 0) {
                            float pmf = 0.0f;
                            if (flags & PF_PICKER_VALID) {
                                LightCtx c;
                                lightPrepare(S, mk(pp.x, pp.y, pp.z), mk(pn.x, pn.y, pn.z), c);
                                pmf = lightCtxPmf(S, c, li);
                            }
                            lightPdf = pmf * lightPdfHit(S.lights[li], mk(lp.x, lp.y, lp.z), is.point);
                        }
                        if (lightPdf > 0.0f && lastBsdfPdf > 0.0f)
                            weight = powerHeuristic(1, lastBsdfPdf, shadowSamples, lightPdf);
                    }
                    if (linked) {
                        V3 c = thr * (m3f(mat.emission) * weight);
                        if (diffuseBounces >= 2 && A.clampIndirect > 0.0f) {
                            const float m = smax3(c.x, c.y, c.z);
                            if (m > A.clampIndirect) c = c * (A.clampIndirect / m);
                        }
                        const V3 added = addL(L, c);
                        if ((OUT && P.pass)) {
                            if (depth == 0) passAdd(passBlock(P, path) + PASS_EMISSION, added);
                            else creditPath(P, path, added, depth == 1);
                            creditGroup(S, P, path, li >= 0 ? lightGroupOf(S, li) : 0, added);
                        }
                    }
                }
                if (depth >= A.maxDepth) done = true;
                else vertex = true;
            }
        }
    }
    if (vertex) {
        const MatGPU& mat = S.materials[is.material];
        // dispersion: the first wavelength-dependent surface fixes one λ for the path
        if (MEDIA && lambda == 0.0f && (mat.flags & MF_DISPERSIVE)) {
            V3 w;
            lambda = sampleWavelength(T, get1D(sb), w);
            thr *= w;
        }
        // rounded edges on the first three vertices (not a walk's exit vertex), then contact AO at
        // the camera hit (path_tracer.cpp:612-621)
        if (REST && depth <= 2 && mat.roundEdge > 0.0f && !exitVertex) {
            const V3 n = roundedEdgeNormal(S, is, mat.roundEdge, sb, time);
            if (dot(n, wo) > 0.02f) is.normal = n;
        }
        if (REST && A.aoStrength > 0.0f && depth == 0) thr *= approxAo(S, is, sb, A.aoStrength, shadowSamples, time);
        ShadePoint sp;
        sp.uv = is.uv;
        sp.textures = S.textures;
        sp.uvDensity = is.uvDensity;
        sp.footprint = 0.0f;
        if (cones && !exitVertex && (cone.x > 0.0f || cone.y > 0.0f)) {
            const V3 nGeom = len2(is.ng) > 0.0f ? is.ng : is.normal;
            const float cosInc = smax(0.15f, fabsf(dot(-dir, nGeom)));
            sp.footprint = (cone.x + cone.y * smax(0.0f, is.t)) / cosInc;
        }
        sp.p = is.point;
        sp.n = is.normal;
        sp.ng = is.ng;
        sp.tangent = is.tangent;
        sp.frontFace = is.frontFace;
        sp.wavelength = lambda;
        const bool isSpecular = (mat.flags & MF_DELTA) != 0;
        DisneyVertex disney;
        const DisneyVertex* dv = &disney;
        if (MT == kDisneyType || (MT < 0 && mat.type == kDisneyType)) disneyVertex(T, mat, wo, sp, disney);
        // this bounce's proposal, when the inference kernel left one for the slot
        const bool useGuide = GUIDE && P.guiding == 2 && guidable(mat) && P.guideMark[slot] != 0u;
        if (useGuide) P.guideMark[slot] = 0u;
        // or the SD-tree's sampling quadtree of the vertex's spatial leaf (path_tracer.cpp:627-629)
        int sdRoot = -1;
        if (GUIDE && (P.sdMode & SD_SAMPLE) && !useGuide && guidable(mat)) {
            const int leaf = sdLeafWithData(P.sd, is.point);
            if (leaf >= 0) sdRoot = P.sd.leaves[leaf].sampRoot;
        }
        // next-event estimation (path_tracer.cpp:631-698)
        if (S.lightCount > 0 && !isSpecular) {
            LightCtx picker;
            lightPrepare(S, is.point, is.normal, picker);
            flags |= PF_PICKER_VALID;
            pp = make_float4(is.point.x, is.point.y, is.point.z, pp.w);
            pn.x = is.normal.x;
            pn.y = is.normal.y;
            pn.z = is.normal.z;
            for (int s = 0; s < shadowSamples; ++s) {
                float lightPmf = 0.0f;
                const int lightIndex = lightCtxSample(S, picker, get1D(sb), lightPmf);
                if (lightIndex < 0 || !(lightPmf > 0.0f)) {
                    (void)get2D(T, sb);
                    continue;
                }
                const bool fromEnv = lightIndex >= explicitLights;
                if (REST && !fromEnv && S.hasLightLinks &&
                    !linkAllows(S.links[lightIndex].mode, S.links[lightIndex].mask, S.shapes[is.shape].linkNode)) {
                    (void)get2D(T, sb);
                    continue;
                }
                const V2 ul = get2D(T, sb);
                const LightSample ls = fromEnv ? envSample(S.env, ul) : sampleLight(S.lights[lightIndex], is.point, ul);
                if (!lsValid(ls)) continue;
                V3 so, sd;
                float stMax;
                if (!makeShadowRay(is, ls.wi, ls.distance, so, sd, stMax)) continue;
                float bsdfPdf = 0.0f;
                LobeSplit3 split;
                const bool firstShares = (OUT && P.pass) && depth == 0;
                const V3 f = bsdfEvalPdfT<MT>(T, mat, wo, ls.wi, sp, dv, bsdfPdf, firstShares ? &split : nullptr);
                const float cosTheta = fabsf(dot(ls.wi, is.normal));
                if (isBlack(f) || !(cosTheta > 0.0f)) continue;
                const float lightPdf = lightPmf * ls.pdf;
                const float contPdf = useGuide     ? 0.5f * bsdfPdf + 0.5f * guidePdf(P, slot, ls.wi)
                                      : sdRoot >= 0 ? 0.5f * bsdfPdf + 0.5f * sdTreePdf(P.sd.samp, sdRoot, ls.wi)
                                                    : bsdfPdf;
                const float weight = powerHeuristic(shadowSamples, lightPdf, 1, contPdf);
                const float scalar = cosTheta * weight / (lightPdf * static_cast<float>(shadowSamples));
                const V3 fLi = f * ls.Li;
                if (SHADOW == SHADOW_INLINE) {
                    // the any-hit query now; its term follows this vertex's emission in L
                    ++shRays;
                    const V3 vis = shadowVisibility<COUNT>(S, so, sd, stMax, fromEnv ? -1 : lightIndex, shNodes, shTris, time);
                    if (!isBlack(vis)) {
                        const V3 c = neeTerm(fLi, vis, scalar, thr, diffuseBounces >= 1, A.clampIndirect);
                        if (isFinite3(c)) {
                            L.x += c.x;
                            L.y += c.y;
                            L.z += c.z;
                            if ((OUT && P.pass)) {
                                float4 shares[3];
                                if (firstShares) {
                                    V3 sh[3];
                                    lobeShares(split, sh);
                                    for (int k = 0; k < 3; ++k) shares[k] = make_float4(sh[k].x, sh[k].y, sh[k].z, 1.0f);
                                }
                                creditNee(S, P, path, fromEnv ? -1 : lightIndex, c, firstShares ? shares : nullptr);
                            }
                        }
                    }
                } else if (SHADOW == SHADOW_HAND) {
                    const uint32_t lightBits = static_cast<uint32_t>(fromEnv ? 0 : lightIndex + 1) << 1;
                    hand->o = make_float4(so.x, so.y, so.z, stMax);
                    hand->d = make_float4(sd.x, sd.y, sd.z, scalar);
                    hand->c = make_float4(fLi.x, fLi.y, fLi.z, __uint_as_float((diffuseBounces >= 1 ? 1u : 0u) | lightBits));
                    hand->t = make_float4(thr.x, thr.y, thr.z, A.clampIndirect);
                    *handed = true;
                } else {
                    // shadow queue append (waves with one shadow sample per vertex), one atomic per
                    // group of lanes that are here together
                    const unsigned here = __activemask();
                    const int lane = threadIdx.x & 31, leader = __ffs(here) - 1;
                    uint32_t pos = 0;
                    if (lane == leader) pos = atomicAdd(&P.next[BC_SHADOW], static_cast<uint32_t>(__popc(here)));
                    pos = __shfl_sync(here, pos, leader) + __popc(here & ((1u << lane) - 1u));
                    shadowRec = static_cast<int>(pos);
                    P.shO[pos] = make_float4(so.x, so.y, so.z, stMax);
                    P.shD[pos] = make_float4(sd.x, sd.y, sd.z, scalar);
                    // flags: bit 0 indirect, bits 1.. the light index + 1 (0: the environment)
                    const uint32_t lightBits = static_cast<uint32_t>(fromEnv ? 0 : lightIndex + 1) << 1;
                    P.shC[pos] = make_float4(fLi.x, fLi.y, fLi.z, __uint_as_float((diffuseBounces >= 1 ? 1u : 0u) | lightBits));
                    P.shT[pos] = make_float4(thr.x, thr.y, thr.z, A.clampIndirect);
                    if ((OUT && P.pass)) {
                        float4* q = P.shPass + 3 * static_cast<size_t>(pos);
                        if (firstShares) {
                            V3 sh[3];
                            lobeShares(split, sh);
                            for (int k = 0; k < 3; ++k) q[k] = make_float4(sh[k].x, sh[k].y, sh[k].z, 1.0f);
                        } else {
                            q[0] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        }
                    }
                }
            }
        }
        // BSDF (and proposal) sampling (path_tracer.cpp:700-743)
        BsdfSample bs;
        bool sampled;
        if (useGuide) {
            sampled = guidedSample(T, mat, wo, sp, P, slot, dv, sb, bs);
        } else if (sdRoot >= 0) {
            sampled = sdGuidedSample(T, mat, wo, sp, P.sd.samp, sdRoot, dv, sb, bs);
        } else {
            const float uc = get1D(sb);
            const V2 u2 = get2D(T, sb);
            sampled = bsdfSampleT<MT>(T, mat, wo, sp, dv, uc, u2, bs);
        }
        if (!sampled) {
            done = true;
        } else if (MEDIA && bs.subsurface) {
            // random-walk entry (path_tracer.cpp:745-761): the walk's coefficients ride
            // in the columns it does not need (lastP, lastN, pickP.x)
            V3 sigT, alb;
            float g = 0.0f;
            if (!disneySubsurfaceCoeffs(mat, dv->p, sigT, alb, g)) {
                done = true;
            } else {
                thr *= bs.weight;
                const V3 d = normalize(bs.wi);
                const V3 no = spawnOrigin(is, d);
                ro = make_float4(no.x, no.y, no.z, __uint_as_float(VIS_ALL | RAY_WALK));
                rd = make_float4(d.x, d.y, d.z, rd.w);
                lp = make_float4(sigT.x, sigT.y, sigT.z, 0.0f);
                ln = make_float4(alb.x, alb.y, alb.z, 0.0f);
                pp.x = g;
                volCtr &= 0xFFFFu; // walk step 0
                flags = (flags | PF_WALK) & ~PF_CAMERA_RAY;
                cont = true;
            }
        } else if (bs.pdf <= 0.0f || isBlack(bs.f)) {
            done = true;
        } else if (bs.passThrough) {
            thr *= bs.f * (fabsf(dot(bs.wi, is.normal)) / bs.pdf);
            if (!isFinite3(thr) || ++passThroughs > 64) {
                done = true;
            } else {
                const V3 no = spawnOrigin(is, bs.wi);
                ro = make_float4(no.x, no.y, no.z, ro.w);
                rd = make_float4(bs.wi.x, bs.wi.y, bs.wi.z, rd.w);
                if (cones) cone.x = cone.x + cone.y * smax(0.0f, is.t);
                skips = 0;
                cont = true;
            }
        } else {
            const V3 wi = bs.wi;
            const bool refracted = dot(wo, is.ng) * dot(wi, is.ng) < 0.0f;
            if ((OUT && P.pass) && depth == 0) {
                // the first surface's lobe shares: all later light splits by them (path_tracer.cpp:797-812)
                V3 sh[3];
                if (bs.delta) {
                    sh[0] = mk(0.0f);
                    sh[1] = mk(refracted ? 0.0f : 1.0f);
                    sh[2] = mk(refracted ? 1.0f : 0.0f);
                } else {
                    LobeSplit3 split;
                    float unusedPdf = 0.0f;
                    (void)bsdfEvalPdfT<MT>(T, mat, wo, wi, sp, dv, unusedPdf, &split);
                    lobeShares(split, sh);
                }
                float4* b = passBlock(P, path);
                for (int k = 0; k < 3; ++k) b[PASS_LOBES + k] = make_float4(sh[k].x, sh[k].y, sh[k].z, 0.0f);
            }
            const float cosTheta = fabsf(dot(wi, is.normal));
            const V3 thrBefore = thr;
            thr *= bs.f * (cosTheta / bs.pdf);
            if (GUIDE && P.guiding && !bs.delta && guidable(mat) && isFinite3(thr) &&
                trainOrder(A, path) % P.guideStride == 0 &&
                guideRecord(P, slot, is.point, is.normal, wo, wi, thrBefore))
                flags |= PF_GUIDE_SNAP;
            if (!isFinite3(thr)) {
                done = true;
            } else {
                flags = bs.delta ? (flags | PF_SPECULAR_BOUNCE) : (flags & ~PF_SPECULAR_BOUNCE);
                // this vertex is the next emission hit's receiver (path_tracer.cpp:832)
                flags = (flags & ~kPrevNodeMask) | (static_cast<uint32_t>(S.shapes[is.shape].linkNode) << kPrevNodeShift);
                if (!bs.delta) ++diffuseBounces;
                cameraRay = cameraRay && bs.delta && dot(wi, is.normal) < 0.0f;
                flags = cameraRay ? (flags | PF_CAMERA_RAY) : (flags & ~PF_CAMERA_RAY);
                // crossing a volume boundary: enter the object's medium from outside,
                // leave it from inside
                if (MEDIA && (mat.flags & MF_VOLUME_BOUNDARY)) {
                    const float a = dot(wo, is.ng), b = dot(wi, is.ng);
                    if (a * b < 0.0f) {
                        if (a > 0.0f) media.enter(is.material);
                        else media.leave(is.material);
                    }
                }
                const uint32_t nextMask = refracted ? VIS_TRANSMISSION : (bs.delta ? VIS_GLOSSY : VIS_DIFFUSE);
                if (cones) {
                    cone.x = cone.x + cone.y * smax(0.0f, is.t);
                    cone.y = cone.y + (bs.delta ? 0.0f : 0.12f);
                }
                ln = make_float4(is.normal.x, is.normal.y, is.normal.z, 0.0f);
                lp = make_float4(is.point.x, is.point.y, is.point.z, 0.0f);
                const V3 no = spawnOrigin(is, wi);
                ro = make_float4(no.x, no.y, no.z, __uint_as_float(nextMask));
                rd = make_float4(wi.x, wi.y, wi.z, bs.pdf);
                ++depth;
                skips = 0;
                cont = true;
                if (depth > A.rrDepth && !russianRoulette(thr, sb)) {
                    cont = false;
                    done = true;
                }
                // SD-tree training vertex (path_tracer.cpp:823-827, recordable ones only): its
                // incident radiance is what L gains from here on over the throughput after the
                // bounce and the roulette
                if (GUIDE && cont && (P.sdMode & SD_RECORD) && !bs.delta && !(mat.flags & MF_VOLUME_BOUNDARY)) {
                    const uint32_t n = P.sdCount[slot];
                    if (n < static_cast<uint32_t>(kSdRecords)) {
                        float4* rec = P.sdRec + (static_cast<size_t>(slot) * kSdRecords + n) * 4;
                        rec[0] = make_float4(is.point.x, is.point.y, is.point.z, bs.pdf);
                        rec[1] = make_float4(wi.x, wi.y, wi.z, 0.0f);
                        rec[2] = make_float4(thr.x, thr.y, thr.z, 0.0f);
                        rec[3] = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
                        P.sdCount[slot] = n + 1;
                        flags |= PF_GUIDE_SNAP;
                    }
                }
            }
        }
    }
    // write back
    if (P.direct && !cont) P.Lout[path] = L;
    else P.L[slot] = L;
    if (SHADOW == SHADOW_QUEUE && shadowRec >= 0) P.shadowQ[shadowRec] = P.direct && !cont ? ~path : slot;
    if (cont) {
        if (cones) P.cone[slot] = cone;
        P.rayO[slot] = ro;
        P.rayD[slot] = rd;
        P.thr[slot] = make_float4(thr.x, thr.y, thr.z, lambda);
        P.lastN[slot] = make_float4(ln.x, ln.y, ln.z, __uint_as_float(flags));
        P.lastP[slot] = make_float4(lp.x, lp.y, lp.z, __uint_as_float(sb.dim));
        P.pickP[slot] = pp;
        P.pickN[slot] = make_float4(pn.x, pn.y, pn.z, __uint_as_float(packCounters(depth, diffuseBounces, passThroughs, skips)));
        if (volumetric)
            P.med[slot] = make_float4(__uint_as_float(media.lo), __uint_as_float(media.hi), __uint_as_float(volCtr),
                                      __int_as_float(media.n));
    }
    return cont;
}

// Consumes the rays binned by shading key (segment by segment, so a warp mostly shades one
// material kind) and appends the continuing paths to nextQueue.
// OUT: the wave records AOVs or render passes (their code is compiled out of the plain kernel).
// INLINE: NEE shadow rays are traced here, each sample's term added in the sample loop's order
// (waves with shadowQuality > 1, whose several records per vertex the shadow queue does not hold).
template <int FEAT, bool OUT, bool INLINE = false>
__global__ void __launch_bounds__(128, 6) kShade(const __grid_constant__ SceneGPU S, const __grid_constant__ Paths P, const __grid_constant__ Wave W, int32_t* nextQueue) {
    uint32_t seg[kShadeKeys];
    int n = 0;
    for (int k = 0; k < kShadeKeys; ++k) {
        seg[k] = P.now[BC_KEYS + k];
        n += static_cast<int>(seg[k]);
    }
    const int lane = threadIdx.x & 31;
    uint32_t unused0 = 0, unused1 = 0, unused2 = 0;
    for (;;) {
        const int base = warpFetch(&P.now[BC_WORK_SHADE]);
        if (base >= n) break;
        const int i = base + lane;
        bool cont = false, sweepable = false;
        int slot = -1;
        if (i < n) {
            int k = 0;
            uint32_t j = static_cast<uint32_t>(i);
            while (k < kShadeKeys - 1 && j >= seg[k]) {
                j -= seg[k];
                ++k;
            }
            slot = P.sortQ[static_cast<size_t>(k) * P.capacity + j];
            const int path = pathOfSlot(P, slot);
            const WaveSeg& A = W.segs[segOfSlot(W, path)];
            cont = shadeSlot<INLINE ? SHADOW_INLINE : SHADOW_QUEUE, false, OUT, FEAT>(S, P, A, slot, path, unused0, unused1, unused2);
            sweepable = (A.flags & SEG_SWEEP) != 0;
        }
        // a continuous wave sweeps its interactive paths that have lived sweepAge bounces into a
        // tail launch, so that their requests do not wait on one bounce per wavefront step
        const bool old = P.sweepAge > 0 && cont && sweepable && P.iter - P.born[slot] >= P.sweepAge;
        queuePush(nextQueue, &P.next[BC_QUEUE], cont && !old, slot);
        if (P.sweepAge > 0) queuePush(P.sweepQ, &P.counters[CNT_SWEEP], old, slot);
        // a regenerating wave refills the slots of ended paths
        if (P.pathOf) queuePush(P.freeQ, &P.counters[CNT_FREE], !cont && slot >= 0, slot);
    }
}

// Lean shading of one shading key's bin by the shadeSlot instantiation that carries the code of that
// key alone; all 32 lanes call it.
template <bool OUT, int KEY>
__device__ __forceinline__ void shadeBin(const SceneGPU& S, const Paths& P, const Wave& W, int32_t* nextQueue) {
    const int n = static_cast<int>(P.now[BC_KEYS + KEY]);
    const int32_t* bin = P.sortQ + static_cast<size_t>(KEY) * P.capacity;
    const int lane = threadIdx.x & 31;
    uint32_t unused0 = 0, unused1 = 0, unused2 = 0;
    while (n > 0) {
        const int base = warpFetch(&P.now[BC_WORK_KEYS + KEY]);
        if (base >= n) break;
        const int i = base + lane;
        bool cont = false, sweepable = false;
        int slot = -1;
        if (i < n) {
            slot = bin[i];
            const int path = pathOfSlot(P, slot);
            const WaveSeg& A = W.segs[segOfSlot(W, path)];
            cont = shadeSlot<SHADOW_QUEUE, false, OUT, 0, KEY>(S, P, A, slot, path, unused0, unused1, unused2);
            sweepable = (A.flags & SEG_SWEEP) != 0;
        }
        if (KEY != 0) {
            // continuous waves sweep interactive paths that have lived sweepAge bounces, as kShade does
            const bool old = P.sweepAge > 0 && cont && sweepable && P.iter - P.born[slot] >= P.sweepAge;
            queuePush(nextQueue, &P.next[BC_QUEUE], cont && !old, slot);
            if (P.sweepAge > 0) queuePush(P.sweepQ, &P.counters[CNT_SWEEP], old, slot);
        }
        if (P.pathOf) queuePush(P.freeQ, &P.counters[CNT_FREE], !cont && slot >= 0, slot);
    }
}

// The lean shading kernels (waves of lean-shading scenes without guiding), one per shading key.  They
// wait for memory and instructions more than they issue, so blocks on the SM count for more than
// registers: at least MINB 128-thread blocks per SM (96 registers for Lambert, 80 for Disney) — shading
// of the 1920x1080 x 4-spp knot wave 9.5 / 7.1 / 6.7 / 6.4 / 6.3 ms at 2 / 4 / 5 / 6 / 8 blocks, of the
// Cornell wave 4.20 / 2.85 / 2.70 / 2.82 / 3.24 ms.  All surface kinds in one launch
// measured slower: the compiler keeps what the kinds share in registers across them and spills 1.2 KB
// a thread (Cornell, Lambert alone: 3.11 against 2.84 ms of shading per 4.2M-path wave).
template <bool OUT, int KEY, int MINB>
__global__ void __launch_bounds__(128, MINB) kShadeKey(const __grid_constant__ SceneGPU S, const __grid_constant__ Paths P,
                                                       const __grid_constant__ Wave W, int32_t* nextQueue) {
    shadeBin<OUT, KEY>(S, P, W, nextQueue);
}

// ---- tail: the last paths of a wave, each run to its end by one thread -------------------------
// Once few paths of a wave are left (defaultTailPaths), per-bounce launches cost more than they
// save.  Here each thread takes a path from the queue, alternates closest-hit queries with shadeSlot
// (shadow rays inline) until the path ends, then takes the next (`traced`: the queue's paths have
// their first hits).  The arithmetic and the order of
// L's terms are the wavefront's, so the film is the same bit for bit.  This one-warp-per-block
// form serves the counting pass and waves with pass outputs or inline AOVs; other waves and the
// request server's sweeps and drains use kTailWarps and kTailLockstep below.
constexpr int kTailBlock = 32;

template <bool COUNT, bool OUT>
__global__ void __launch_bounds__(kTailBlock) kTail(const __grid_constant__ SceneGPU S, const __grid_constant__ Paths P, const __grid_constant__ Wave W, const int32_t* queue, const uint32_t* count,
                                             uint32_t* cursor, int traced, unsigned long long* stats) {
    const int n = static_cast<int>(*count);
    uint32_t nodes = 0, tris = 0, shNodes = 0, shTris = 0, rays = 0, shRays = 0;
    for (;;) {
        const int i = static_cast<int>(atomicAdd(cursor, 1u));
        if (i >= n) break;
        const int slot = queue[i];
        const int path = pathOfSlot(P, slot);
        const WaveSeg& A = W.segs[segOfSlot(W, path)];
        for (int q = 0;; ++q) {
            if (q >= kMaxPathQueries) {
                atomicAdd(&stats[7], 1ull);
                break;
            }
            if (q > 0 || !traced) {
                const float4 ro = P.rayO[slot];
                const float4 rd = P.rayD[slot];
                const Hit h = traceClosestWide<COUNT>(S, mk(ro.x, ro.y, ro.z), mk(rd.x, rd.y, rd.z), __float_as_uint(ro.w),
                                                      0.0f, 1e30f, nodes, tris, pathTime(S, P, slot));
                ++rays;
                P.hit[slot] = make_float4(h.t, h.u, h.v, __int_as_float(h.prim));
            }
            if (!shadeSlot<SHADOW_INLINE, COUNT, OUT>(S, P, A, slot, path, shNodes, shTris, shRays)) break;
        }
    }
    if (COUNT) {
        atomicAdd(&stats[0], static_cast<unsigned long long>(nodes));
        atomicAdd(&stats[1], static_cast<unsigned long long>(tris));
        atomicAdd(&stats[2], static_cast<unsigned long long>(shNodes));
        atomicAdd(&stats[3], static_cast<unsigned long long>(shTris));
    }
    atomicAdd(&stats[5], static_cast<unsigned long long>(rays));
    atomicAdd(&stats[6], static_cast<unsigned long long>(shRays));
}

// The tail of waves whose shadow rays are traced inline (several shadow samples per vertex, shadow
// transmitters or links), in lockstep: the same per-path work as kTail<false, false>, but the four warps of a 128-thread block meet at a barrier between each bounce's closest-hit query and
// its shading, so the warps sharing an SM run the same phase's code at once.  The loop body
// (traversal, every lean material's shading, the inline shadow ray) is far larger than an SM
// sub-partition's instruction cache; warps of 32-thread blocks, each at its own point of the
// loop, spend most of their stalls fetching instructions.  Threads whose paths have ended take
// the queue's next path at the top of the loop; the block leaves when none of its threads holds
// one.  Each path's queries and terms are kTail's, so the film is the same bit for bit.
constexpr int kTailLockstepBlock = 128;
template <bool OUT>
__global__ void __launch_bounds__(kTailLockstepBlock) kTailLockstep(const __grid_constant__ SceneGPU S, const __grid_constant__ Paths P, const __grid_constant__ Wave W, const int32_t* queue,
                                                                  const uint32_t* count, uint32_t* cursor, int traced,
                                                                  unsigned long long* stats) {
    const int n = static_cast<int>(*count);
    uint32_t nodes = 0, tris = 0, shNodes = 0, shTris = 0, rays = 0, shRays = 0;
    int slot = -1, path = 0, q = 0;
    const WaveSeg* A = nullptr;
    bool exhausted = false; // this thread found the queue taken
    for (;;) {
        if (slot < 0 && !exhausted) {
            const int i = static_cast<int>(atomicAdd(cursor, 1u));
            if (i < n) {
                slot = queue[i];
                path = pathOfSlot(P, slot);
                A = &W.segs[segOfSlot(W, path)];
                q = 0;
            } else {
                exhausted = true;
            }
        }
        if (!__syncthreads_or(slot >= 0)) break;
        if (slot >= 0 && (q > 0 || !traced)) {
            const float4 ro = P.rayO[slot];
            const float4 rd = P.rayD[slot];
            const Hit h = traceClosestWide<false>(S, mk(ro.x, ro.y, ro.z), mk(rd.x, rd.y, rd.z), __float_as_uint(ro.w), 0.0f,
                                              1e30f, nodes, tris, pathTime(S, P, slot));
            ++rays;
            P.hit[slot] = make_float4(h.t, h.u, h.v, __int_as_float(h.prim));
        }
        __syncthreads();
        if (slot >= 0) {
            if (!shadeSlot<SHADOW_INLINE, false, OUT>(S, P, *A, slot, path, shNodes, shTris, shRays)) {
                slot = -1;
            } else if (++q >= kMaxPathQueries) {
                // as kTail: a path past the per-path query bound is ended and reported
                atomicAdd(&stats[7], 1ull);
                slot = -1;
            }
        }
    }
    atomicAdd(&stats[5], static_cast<unsigned long long>(rays));
    atomicAdd(&stats[6], static_cast<unsigned long long>(shRays));
}

// The tail of every other wave: a warp carries up to `perWarp` paths and alternates between shading
// them, a path per lane, and tracing all the rays they left — each path's next closest hit and the
// shadow ray of the vertex just shaded, which do not depend on each other — a ray per lane in one
// converged loop.  A path's bounce then takes the longer of its two rays instead of their sum.  Few
// paths are spread thinly over the resident warps, because the rays of a warp wait for its longest
// one.  The block's warps shade between barriers (one phase's code at a time, as kTailLockstep).
// Each path's queries and terms are kTail's, so the film is the same bit for bit.
// Shading a vertex is what bounds it: about 70k cycles of dependent instructions, half of them waiting
// to be fetched (a warp's turn of the walk: 2k).  The kinds a warp's lanes hold follow each other, so the block first
// sorts its paths by shading key: each kind has warps of its own while there are as many warps as kinds.
// Torus knot, 64x64 tile of one sample 1.17 -> 1.09 ms, 333x217 x 5 spp 5.46 -> 5.16 ms; with 128 threads
// a block 5.24 ms, but 128 is better where the kernel holds all shading code (media 1280x720 x 4 spp, 17.6 / 17.8 ms).
constexpr int tailWarpsBlock(int features) { return features == 0 ? 256 : 128; }
template <int FEAT, bool OUT>
__global__ void __launch_bounds__(tailWarpsBlock(FEAT)) kTailWarps(const __grid_constant__ SceneGPU S,
                                                                   const __grid_constant__ Paths P,
                                                                   const __grid_constant__ Wave W, const int32_t* queue,
                                                                   const uint32_t* count, uint32_t* cursor, int traced,
                                                                   int perWarp, unsigned long long* stats) {
    constexpr int kBlock = tailWarpsBlock(FEAT), kWarps = kBlock / 32;
    __shared__ ShadowRec recs[kBlock];
    __shared__ int slots[kBlock], paths[kBlock];
    __shared__ int blocked[kBlock];
    __shared__ int shades[kBlock];    // the thread whose path this one shades, -1 none
    __shared__ uint8_t shaded[kBlock]; // bit 0: the path goes on, bit 1: it left a shadow ray
    __shared__ uint8_t keyCount[kWarps][kShadeKeys];
    __shared__ uint8_t owners[kWarps][64]; // each warp's rays: the lane they belong to, closest hits first
    uint2 stack[walkStack(true)];
    const int n = static_cast<int>(*count);
    const int tid = threadIdx.x, lane = tid & 31, warpBase = tid & ~31;
    const unsigned below = (1u << lane) - 1u;
    uint8_t* own = owners[tid >> 5];
    const int root = rootRef(S);
    const bool scattering = (S.hasVolumes | S.hasSubsurface) != 0;
    uint32_t unused = 0, rays = 0, shRays = 0;
    int slot = -1, path = 0, q = 0;
    bool exhausted = lane >= perWarp; // this lane takes no (more) paths
    bool shadow = false;              // recs[tid] waits to be traced
    bool ended = false;               // ... and is all that its path still waits for
    for (;;) {
        if (slot < 0 && !exhausted) {
            const int i = static_cast<int>(atomicAdd(cursor, 1u));
            if (i < n) {
                slot = queue[i];
                path = pathOfSlot(P, slot);
                q = 0;
            } else {
                exhausted = true;
            }
        }
        slots[tid] = slot;
        paths[tid] = path;
        if (!__syncthreads_or(slot >= 0)) break;
        // the warp's rays
        const bool closest = slot >= 0 && !ended && (q > 0 || !traced);
        const unsigned closestLanes = __ballot_sync(kWarp, closest), shadowLanes = __ballot_sync(kWarp, shadow);
        const int nClosest = __popc(closestLanes), nRays = nClosest + __popc(shadowLanes);
        if (closest) own[__popc(closestLanes & below)] = static_cast<uint8_t>(lane);
        if (shadow) own[nClosest + __popc(shadowLanes & below)] = static_cast<uint8_t>(lane);
        rays += closest ? 1u : 0u;
        shRays += shadow ? 1u : 0u;
        __syncwarp();
        RayWalk w;
        w.cur = kRayDone;
        w.any = false;
        int ray = -1, nextRay = 0; // the block thread this lane's ray belongs to
        for (;;) {
            const unsigned idle = __ballot_sync(kWarp, w.cur == kRayDone);
            if (idle == kWarp || (nextRay < nRays && __popc(idle) >= kRefill)) {
                if (w.cur == kRayDone && ray >= 0) {
                    ScatterRay next;
                    if (w.any) {
                        blocked[ray] = w.prim;
                        ray = -1;
                    } else {
                        if (w.prim == -1) P.hit[slots[ray]] = make_float4(w.tMax, 0.0f, 0.0f, __int_as_float(-1));
                        if ((FEAT & FEAT_MEDIA) && scattering && scatterOn(S, P, W, slots[ray], next)) {
                            w.start(S, root, next.o, next.d, next.mask, 1e30f, -1);
                            ++rays;
                        } else {
                            ray = -1;
                        }
                    }
                }
                const unsigned without = __ballot_sync(kWarp, ray < 0);
                if (ray < 0) {
                    const int i = nextRay + __popc(without & below);
                    if (i < nRays) {
                        ray = warpBase + own[i];
                        w.any = i >= nClosest;
                        if (w.any) {
                            const float4 so = recs[ray].o, sd = recs[ray].d;
                            w.start(S, root, mk(so.x, so.y, so.z), mk(sd.x, sd.y, sd.z), VIS_SHADOW, so.w, 0);
                        } else {
                            const float4 ro = P.rayO[slots[ray]], rd = P.rayD[slots[ray]];
                            w.start(S, root, mk(ro.x, ro.y, ro.z), mk(rd.x, rd.y, rd.z), __float_as_uint(ro.w), 1e30f, -1);
                        }
                    }
                }
                nextRay += __popc(without);
                if (__all_sync(kWarp, ray < 0)) break;
                continue;
            }
            walkTurn<WALK_MIXED, false, true>(
                S, w, stack, unused, unused,
                [&](V3& o, V3& d, uint32_t& mask) {
                    const float4 ro = w.any ? recs[ray].o : P.rayO[slots[ray]], rd = w.any ? recs[ray].d : P.rayD[slots[ray]];
                    o = mk(ro.x, ro.y, ro.z);
                    d = mk(rd.x, rd.y, rd.z);
                    mask = w.any ? static_cast<uint32_t>(VIS_SHADOW) : __float_as_uint(ro.w);
                },
                [&]() { return pathTime(S, P, slots[ray]); },
                [&](float t, float u, float v, int prim, uint32_t) { P.hit[slots[ray]] = make_float4(t, u, v, __int_as_float(prim)); });
            __syncwarp();
        }
        __syncthreads(); // the block shades together; hits and answers are visible
        if (shadow) {
            if (blocked[tid] == 0) {
                const ShadowRec& r = recs[tid];
                const V3 c = neeTerm(mk(r.c.x, r.c.y, r.c.z), mk(1.0f), r.d.w, mk(r.t.x, r.t.y, r.t.z),
                                     (__float_as_uint(r.c.w) & 1u) != 0, r.t.w);
                float4* at = ended && P.direct ? P.Lout + path : P.L + slot;
                float4 L = *at;
                addL(L, c);
                *at = L;
            }
            shadow = false;
            if (ended) slot = -1;
            ended = false;
        }
        // each path to a thread of a warp that shades its key
        int key = -1;
        if (slot >= 0)
            key = shadeKeyOfPrim(S, S.hasSubsurface ? __float_as_uint(P.rayO[slot].w) : 0u, __float_as_int(P.hit[slot].w));
        shades[tid] = -1;
        const unsigned peers = __match_any_sync(kWarp, key);
        if (lane < kShadeKeys) keyCount[tid >> 5][lane] = 0;
        __syncwarp();
        if (key >= 0 && (peers & below) == 0) keyCount[tid >> 5][key] = static_cast<uint8_t>(__popc(peers));
        __syncthreads();
        if (key >= 0) {
            int rank = __popc(peers & below), spare = kWarps, first = 0, firstWarp = 0, mine = 0;
            int most = 0, mostKey = 0;
#pragma unroll
            for (int k = 0; k < kShadeKeys; ++k) {
                int c = 0;
#pragma unroll
                for (int v = 0; v < kWarps; ++v) {
                    if (k == key && v < (tid >> 5)) rank += keyCount[v][k];
                    c += keyCount[v][k];
                }
                const int warps = (c + 31) / 32;
                spare -= warps;
                if (k < key) {
                    first += c;
                    firstWarp += warps;
                }
                if (k == key) mine = warps;
                if (c > most) {
                    most = c;
                    mostKey = k;
                }
            }
            int to = first + rank; // more kinds than warps: the kinds follow each other
            if (spare >= 0) {
                // warps left over go to the most common kind
                if (key == mostKey) mine += spare;
                else if (key > mostKey) firstWarp += spare;
                to = (firstWarp + rank % mine) * 32 + rank / mine;
            }
            shades[to] = tid;
        }
        __syncthreads();
        const int home = shades[tid];
        if (home >= 0) {
            const WaveSeg& A = W.segs[segOfSlot(W, paths[home])];
            bool handed = false;
            const bool cont = shadeSlot<SHADOW_HAND, false, OUT, FEAT>(S, P, A, slots[home], paths[home], unused, unused,
                                                                       unused, &recs[home], &handed);
            shaded[home] = static_cast<uint8_t>((cont ? 1 : 0) | (handed ? 2 : 0));
        }
        __syncthreads();
        if (slot >= 0) {
            const bool cont = shaded[tid] & 1;
            shadow = (shaded[tid] & 2) != 0;
            ended = !cont;
            if (!cont && !shadow) {
                slot = -1;
                ended = false;
            } else if (cont && ++q >= kMaxPathQueries) {
                // as kTail: a path past the per-path query bound is ended and reported
                atomicAdd(&stats[7], 1ull);
                slot = -1;
                shadow = ended = false;
            }
        }
    }
    atomicAdd(&stats[5], static_cast<unsigned long long>(rays));
    atomicAdd(&stats[6], static_cast<unsigned long long>(shRays));
}

// ---- instantiations ---------------------------------------------------------------------------
// The kernels below are compiled in translation units of their own (pe_kernels_*.cu), side by side;
// PE_FULL_KERNELS(K) and its siblings expand K(kernel) over a unit's instantiations.
#define PE_SHADE_ARGS                                                                              \
    (const __grid_constant__ SceneGPU, const __grid_constant__ Paths, const __grid_constant__ Wave, int32_t*)
// one kernel per shading key: K(AOVs or passes, key, blocks per SM)
#define PE_LEAN_KEYS(K, OUT) K(OUT, 0, 1) K(OUT, 1, 5) K(OUT, 2, 6) K(OUT, 3, 5) K(OUT, 4, 5)
#define PE_SHADE_KEY(OUT, KEY, MINB) PE_K(kShadeKey<OUT, KEY, MINB>)
#define PE_FULL_KERNELS(K) K(kShade<FEAT_ALL, false, false>) K(kShade<FEAT_ALL, false, true>)
#define PE_FULL_OUT_KERNELS(K) K(kShade<FEAT_ALL, true, false>) K(kShade<FEAT_ALL, true, true>)
#define PE_MEDIA_KERNELS(K) K(kShade<FEAT_MEDIA, false, false>)
#define PE_GUIDE_KERNELS(K) K(kShade<FEAT_GUIDE, false, false>)
#define PE_TAIL_ARGS                                                                               \
    (const __grid_constant__ SceneGPU, const __grid_constant__ Paths, const __grid_constant__ Wave, const int32_t*, \
     const uint32_t*, uint32_t*, int, unsigned long long*)
#define PE_TAIL_KERNELS(K) K(kTail<false, true>) K(kTail<true, false>) K(kTail<true, true>)
#define PE_LOCKSTEP_KERNELS(K) K(kTailLockstep<false>)
#define PE_TAIL_WARPS_ARGS                                                                         \
    (const __grid_constant__ SceneGPU, const __grid_constant__ Paths, const __grid_constant__ Wave, const int32_t*, \
     const uint32_t*, uint32_t*, int, int, unsigned long long*)
#define PE_TAIL_WARPS_LEAN_KERNELS(K) K(kTailWarps<0, false>) K(kTailWarps<0, true>)
#define PE_TAIL_WARPS_FULL_KERNELS(K) K(kTailWarps<FEAT_ALL, false>) K(kTailWarps<FEAT_ALL, true>)
#define PE_TRACE_ARGS                                                                              \
    (const __grid_constant__ SceneGPU, const __grid_constant__ Paths, const __grid_constant__ Wave, const int32_t*, int, \
     unsigned long long*)
#define PE_TRACE_KERNELS(K)                                                                        \
    K(kTrace<false, false, false>) K(kTrace<false, true, false>) K(kTrace<true, false, false>)     \
    K(kTrace<true, true, false>) K(kTrace<false, false, true>) K(kTrace<false, true, true>)        \
    K(kTrace<true, false, true>) K(kTrace<true, true, true>)
#define PE_BINARY_ARGS                                                                             \
    (const __grid_constant__ SceneGPU, const __grid_constant__ Paths, const int32_t*, unsigned long long*)
#define PE_BINARY_KERNELS(K) K(kIntersectBinary<false>) K(kIntersectBinary<true>)
#define PE_SHADOW_ARGS (const __grid_constant__ SceneGPU, const __grid_constant__ Paths, unsigned long long*)
#define PE_SHADOW_KERNELS(K) K(kShadow<false>) K(kShadow<true>) K(kShadowAny<false>) K(kShadowAny<true>)

} // namespace pe
