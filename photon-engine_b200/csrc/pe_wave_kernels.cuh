// pe_wave_kernels.cuh — the wave's kernels between its traces and shadings: the paths' first rays and the
// slots they take, the bins by shading key, the films.  Included by pe_device.cu alone, which launches
// them, so that the units of the large kernels do not hold copies.
#pragma once

#include "pe_integrator.cuh"

namespace pe {

// ---- path generation and slots ------------------------------------------------------------------
__device__ __forceinline__ void generatePath(const SceneGPU& S, const Paths& P, const Wave& W, int slot, int path) {
    const TablesGPU* T = S.tables;
    const WaveSeg& A = W.segs[segOfSlot(W, path)];
    const int p = (path - A.slotFirst) / A.nSamples, sOff = path - A.slotFirst - p * A.nSamples;
    int x, y;
    tilePixel(A, A.pixelFirst + p, x, y);
    Sobol sb;
    sb.pixelHash = pixelHashOf(A.seed, x, y);
    sb.revIndex = rev32(static_cast<uint32_t>(A.sampleFirst + sOff));
    sb.dim = 0;
    V3 o, d;
    float time;
    cameraRay(T, A.filterCdf, A.cam, A.filterWidth, x, y, A.width, A.height, sb, o, d, (A.flags & SEG_MOTION) != 0, &time);
    if (S.motions && P.time) P.time[slot] = time;
    P.rayO[slot] = make_float4(o.x, o.y, o.z, __uint_as_float(VIS_CAMERA));
    P.rayD[slot] = make_float4(d.x, d.y, d.z, 0.0f);
    P.thr[slot] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    P.L[slot] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    P.lastN[slot] = make_float4(0.0f, 1.0f, 0.0f, __uint_as_float(PF_SPECULAR_BOUNCE | PF_CAMERA_RAY | PF_FIRST_SEGMENT));
    P.lastP[slot] = make_float4(o.x, o.y, o.z, __uint_as_float(sb.dim));
    P.pickP[slot] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(sb.pixelHash));
    P.pickN[slot] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(packCounters(0, 0, 0, 0)));
    if (S.hasVolumes | S.hasSubsurface) P.med[slot] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (P.guiding) {
        P.guideMark[slot] = 0u;
        if (trainOrder(A, path) % P.guideStride == 0) P.guideRec[static_cast<size_t>(slot) * 6 + 4] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    if (S.hasMips && P.cone) P.cone[slot] = make_float2(A.coneWidth, A.coneSpread);
    if (P.pass) {
        float4* b = passBlock(P, path);
        for (int k = 0; k < P.passStride; ++k) b[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        b[PASS_LOBES] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
        b[PASS_HIT] = make_float4(o.x, o.y, o.z, 0.0f);
    }
    if (P.pathOf) P.pathOf[slot] = path;
}

// Hands an ended path's radiance to Lout (and counts it off its segment when those are tracked).
__device__ __forceinline__ void flushPath(const Paths& P, const Wave& W, int slot) {
    const int path = P.pathOf[slot];
    P.Lout[path] = P.L[slot];
    if (P.segLeft) {
        __threadfence(); // the radiance is visible before the segment's count says it is done
        atomicSub(&P.segLeft[segOfSlot(W, path)], 1u);
    }
}

// The wave's first `count` paths into slots [0, count), all queued.
static __global__ void kGenerate(const __grid_constant__ SceneGPU S, const __grid_constant__ Paths P, const __grid_constant__ Wave W, int count) {
    for (int slot = blockIdx.x * blockDim.x + threadIdx.x; slot < count; slot += gridDim.x * blockDim.x) {
        generatePath(S, P, W, slot, slot);
        P.queueA[slot] = slot;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) P.now[BC_QUEUE] = static_cast<uint32_t>(count);
}

// After a bounce of a regenerating wave: every slot freed this bounce hands its path's radiance
// to Lout (its NEE terms are in by now; in direct waves it did so when it ended), and the first
// `fresh` of them take the wave's paths [nextPath, nextPath + fresh), appended to the next
// closest-hit queue after its `queued` entries.
static __global__ void kRecycle(const __grid_constant__ SceneGPU S, const __grid_constant__ Paths P, const __grid_constant__ Wave W, int freed, int fresh, int nextPath, int32_t* queue, int queued,
                         uint32_t* queueCount) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < freed; k += gridDim.x * blockDim.x) {
        const int slot = P.freeQ[k];
        if (!P.direct) flushPath(P, W, slot);
        if (k < fresh) {
            generatePath(S, P, W, slot, nextPath + k);
            queue[queued + k] = slot;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *queueCount = static_cast<uint32_t>(queued + fresh);
}

// The radiance of the paths the tail kernel finished, to Lout.
static __global__ void kFlush(const __grid_constant__ Paths P, const __grid_constant__ Wave W, const int32_t* queue, const uint32_t* count) {
    const int n = static_cast<int>(*count);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) flushPath(P, W, queue[i]);
}

// Continuous waves (the request server): freed slots form a stack (freeQ, its size in
// counters[CNT_FREE]).  kFlushFreed hands over the radiance of the `freed` slots pushed this
// bounce, above `base`; kInject then pops `fresh` slots for the wave's paths [nextPath, +fresh),
// appended to the next closest-hit queue after its `queued` entries.
static __global__ void kFlushFreed(const __grid_constant__ Paths P, const __grid_constant__ Wave W, int base, int freed) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < freed; k += gridDim.x * blockDim.x)
        flushPath(P, W, P.freeQ[base + k]);
}

static __global__ void kInject(const __grid_constant__ SceneGPU S, const __grid_constant__ Paths P, const __grid_constant__ Wave W, int top, int fresh, int nextPath, int32_t* queue, int queued,
                        uint32_t* queueCount) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < fresh; k += gridDim.x * blockDim.x) {
        const int slot = P.freeQ[top - fresh + k];
        generatePath(S, P, W, slot, nextPath + k);
        if (P.born) P.born[slot] = P.iter;
        queue[queued + k] = slot;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *queueCount = static_cast<uint32_t>(queued + fresh);
        P.counters[CNT_FREE] = static_cast<uint32_t>(top - fresh);
    }
}

// Slots of a finished sweep back onto the free stack, above `top`.
static __global__ void kReturnSlots(const __grid_constant__ Paths P, const int32_t* slots, int n, int top) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) P.freeQ[top + k] = slots[k];
    if (blockIdx.x == 0 && threadIdx.x == 0) P.counters[CNT_FREE] = static_cast<uint32_t>(top + n);
}

// Every slot free: the stack holds slots [0, n).
static __global__ void kInitFree(const __grid_constant__ Paths P, int n) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) P.freeQ[k] = k;
    if (blockIdx.x == 0 && threadIdx.x == 0) P.counters[CNT_FREE] = static_cast<uint32_t>(n);
}

// ---- binning -------------------------------------------------------------------------------------
// The queue's slots into the bins of their hits' shading keys.  A pass of its own rather than the
// end of each ray's walk: rays end in any order, and bins in that order made the shading kernels'
// state reads scatter (8.3 against 7.1 ms of shading per 8.3M-path knot wave); here a bin keeps the
// queue's order but for the interleaving of blocks.  Bound by the latency of its loads and of the bins'
// counters: the walk leaves a ray's key in a byte (instances' hits excepted), and a block takes each
// bin's share for 1024 entries at once (traversal and binning of the 256x256 x 64-spp Cornell wave 2.48 ->
// 2.21 ms, of the 1920x1080 x 4-spp knot wave 6.86 -> 6.53 ms).  5 us per million rays over that wave's
// launches, 14 to 17 in launches of 0.4-0.5 M rays.
constexpr int kBinBlock = 256, kBinEach = 4;
static __global__ void __launch_bounds__(kBinBlock) kBin(const __grid_constant__ SceneGPU S, const __grid_constant__ Paths P, const int32_t* queue) {
    constexpr int kWarps = kBinBlock / 32;
    __shared__ uint32_t count[kWarps][kShadeKeys], first[kWarps][kShadeKeys];
    const int n = static_cast<int>(P.now[BC_QUEUE]);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x < kBounceBlock) P.next[threadIdx.x] = 0u; // the next bounce's counters
    for (int base = blockIdx.x * kBinBlock * kBinEach; base < n; base += gridDim.x * kBinBlock * kBinEach) {
        int slot[kBinEach], key[kBinEach];
        uint32_t rank[kBinEach]; // among the warp's entries of the same key
        uint32_t mine = 0;       // lane k: the warp's entries of key k
#pragma unroll
        for (int j = 0; j < kBinEach; ++j) {
            const int i = base + (warp * kBinEach + j) * 32 + lane;
            slot[j] = i < n ? queue[i] : -1;
        }
#pragma unroll
        for (int j = 0; j < kBinEach; ++j) key[j] = slot[j] >= 0 ? P.key[slot[j]] : -1;
#pragma unroll
        for (int j = 0; j < kBinEach; ++j) {
            if (key[j] == kKeyOfPrim) {
                const uint32_t mask = S.hasSubsurface ? __float_as_uint(P.rayO[slot[j]].w) : 0u;
                key[j] = shadeKeyOfPrim(S, mask, __float_as_int(P.hit[slot[j]].w));
            }
            const unsigned peers = __match_any_sync(kWarp, key[j]);
            rank[j] = __popc(peers & ((1u << lane) - 1u)) + __shfl_sync(kWarp, mine, key[j] < 0 ? 0 : key[j]);
#pragma unroll
            for (int k = 0; k < kShadeKeys; ++k) {
                const uint32_t c = __popc(__ballot_sync(kWarp, key[j] == k));
                if (lane == k) mine += c;
            }
        }
        if (lane < kShadeKeys) count[warp][lane] = mine;
        __syncthreads();
        if (threadIdx.x < kShadeKeys) {
            uint32_t total = 0;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) total += count[w][threadIdx.x];
            uint32_t at = total ? atomicAdd(&P.now[BC_KEYS + threadIdx.x], total) : 0u;
#pragma unroll
            for (int w = 0; w < kWarps; ++w) {
                first[w][threadIdx.x] = at;
                at += count[w][threadIdx.x];
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kBinEach; ++j)
            if (key[j] >= 0) P.sortQ[static_cast<size_t>(key[j]) * P.capacity + first[warp][key[j]] + rank[j]] = slot[j];
    }
}

// ---- film: Film::addSample in sample order per pixel (src/core/image/film.cpp:56-69) ----------
// The AOV films of one pixel (addAovs, renderer.cpp:219-224): albedo and alpha by addSample,
// the normal by addSampleSigned (film.cpp:73-85), in sample order.
static __device__ __noinline__ void filmAovs(const Paths& P, const WaveSeg& A, int p, int pix) {
    const size_t n = static_cast<size_t>(A.width) * static_cast<size_t>(A.height);
    for (int f = 0; f < 3; ++f) {
        float* fsum = A.aov + static_cast<size_t>(f) * 5 * n;
        uint32_t* fcnt = reinterpret_cast<uint32_t*>(fsum + 3 * n);
        float* fsq = fsum + 4 * n;
        float r = fsum[3 * pix + 0], g = fsum[3 * pix + 1], b = fsum[3 * pix + 2], q = fsq[pix];
        uint32_t c = fcnt[pix];
        for (int s = 0; s < A.nSamples; ++s) {
            const int path = pathOfSample(A, p, s);
            V3 v;
            if (f == 0) {
                const float4 a = P.aovA[path];
                v = mk(a.x, a.y, a.z);
            } else if (f == 1) {
                const float4 nn = P.aovN[path];
                v = mk(nn.x, nn.y, nn.z);
            } else {
                v = mk(P.aovA[path].w);
            }
            ++c;
            if (!(finitef(v.x) && finitef(v.y) && finitef(v.z))) continue;
            if (f != 1 && !(v.x >= 0.0f && v.y >= 0.0f && v.z >= 0.0f)) continue;
            r += v.x;
            g += v.y;
            b += v.z;
            if (f != 1) {
                const float lum = luminance(v);
                q += lum * lum;
            }
        }
        fsum[3 * pix + 0] = r;
        fsum[3 * pix + 1] = g;
        fsum[3 * pix + 2] = b;
        fsq[pix] = q;
        fcnt[pix] = c;
    }
}

// The render-pass films of one pixel (addPasses, renderer.cpp:206-217), in sample order: light
// passes, depth, ids and light groups by addSample, the position by addSampleSigned.
static __device__ __noinline__ void filmPasses(const Paths& P, const WaveSeg& A, int p, int pix) {
    const size_t n = static_cast<size_t>(A.width) * static_cast<size_t>(A.height);
    const int nFilms = PFILM_GROUPS + (P.passStride - PASS_GROUPS);
    for (int f = 0; f < nFilms; ++f) {
        float* fsum = A.pass + static_cast<size_t>(f) * 5 * n;
        uint32_t* fcnt = reinterpret_cast<uint32_t*>(fsum + 3 * n);
        float* fsq = fsum + 4 * n;
        const int slotOf = f < PFILM_DEPTH ? f
                         : f == PFILM_DEPTH || f == PFILM_POSITION ? PASS_HIT
                         : f == PFILM_OBJECT ? PASS_OBJECT
                         : f == PFILM_MATERIAL ? PASS_MATERIAL
                                               : PASS_GROUPS + (f - PFILM_GROUPS);
        const bool isSigned = f == PFILM_POSITION;
        float r = fsum[3 * pix + 0], g = fsum[3 * pix + 1], b = fsum[3 * pix + 2], q = fsq[pix];
        uint32_t c = fcnt[pix];
        for (int s = 0; s < A.nSamples; ++s) {
            const float4* blk = passBlock(P, pathOfSample(A, p, s));
            const float4 v4 = blk[slotOf];
            V3 v = mk(v4.x, v4.y, v4.z);
            if (f == PFILM_DEPTH || f == PFILM_POSITION) {
                const bool hit = blk[PASS_OBJECT].w != 0.0f;
                v = !hit ? mk(0.0f) : f == PFILM_DEPTH ? mk(v4.w) : v;
            }
            ++c;
            if (!(finitef(v.x) && finitef(v.y) && finitef(v.z))) continue;
            if (!isSigned && !(v.x >= 0.0f && v.y >= 0.0f && v.z >= 0.0f)) continue;
            r += v.x;
            g += v.y;
            b += v.z;
            if (!isSigned) {
                const float lum = luminance(v);
                q += lum * lum;
            }
        }
        fsum[3 * pix + 0] = r;
        fsum[3 * pix + 1] = g;
        fsum[3 * pix + 2] = b;
        fsq[pix] = q;
        fcnt[pix] = c;
    }
    if (A.cryptoObj) {
        // each sample's Cryptomatte ids; the host adds them to its CryptoFilms
        for (int s = 0; s < A.nSamples; ++s) {
            const float4 id = passBlock(P, pathOfSample(A, p, s))[PASS_CRYPTO];
            const size_t o = static_cast<size_t>(A.sampleFirst + s - A.cryptoFirst) * n + static_cast<size_t>(pix);
            A.cryptoObj[o] = id.x;
            A.cryptoMat[o] = id.y;
        }
    }
}

static __global__ void kFilm(const __grid_constant__ Paths P, const __grid_constant__ Wave W, unsigned long long* rejected) {
    unsigned long long rej = 0;
    for (int wp = blockIdx.x * blockDim.x + threadIdx.x; wp < W.nPix; wp += gridDim.x * blockDim.x) {
        const WaveSeg& A = W.segs[segOfPixel(W, wp)];
        const int p = wp - A.pixFirst;
        int px, py;
        tilePixel(A, A.pixelFirst + p, px, py);
        const int pix = py * A.width + px;
        float* sum = A.sum;
        float sr = sum[3 * pix + 0], sg = sum[3 * pix + 1], sbb = sum[3 * pix + 2];
        float sq = A.sq[pix];
        uint32_t c = A.cnt[pix];
        for (int s = 0; s < A.nSamples; ++s) {
            const int path = pathOfSample(A, p, s);
            const float4 L = P.Lout ? P.Lout[path] : P.L[path];
            ++c;
            const bool ok = finitef(L.x) && finitef(L.y) && finitef(L.z) && L.x >= 0.0f && L.y >= 0.0f && L.z >= 0.0f;
            if (!ok) {
                ++rej;
                continue;
            }
            sr += L.x;
            sg += L.y;
            sbb += L.z;
            const float lum = luminance(mk(L.x, L.y, L.z));
            sq += lum * lum;
        }
        sum[3 * pix + 0] = sr;
        sum[3 * pix + 1] = sg;
        sum[3 * pix + 2] = sbb;
        A.sq[pix] = sq;
        A.cnt[pix] = c;
        if (A.aov && P.aovA) filmAovs(P, A, p, pix);
        if (A.pass && P.pass) filmPasses(P, A, p, pix);
    }
    if (rej) atomicAdd(rejected, rej);
}

} // namespace pe
