// pe_wave.h — the wavefront's data layout: per-path state columns in HBM, queue counters, and
// the segment table that lets several render requests share one wave.  Plain structs, so the
// host-side scheduler (compiled without device code) can build waves.
#pragma once

#include "pe_math.h"
#include "pe_sdtree.h"

#include <cstddef>
#include <cstdint>
#include <type_traits>
#include <vector_types.h>

namespace pe {

// Pinhole camera as PerspectiveCamera stores it (perspective_camera.cpp:36-40).
struct CamDev {
    V3 position, lowerLeft, horizontal, vertical;
    V3 u, v, forward;       // lens plane axes and view direction
    float lensRadius;       // > 0: thin lens
    int blades;             // thin lens: polygon aperture sides (0 = disk)
    float bladeRotation;    // radians
    int orthographic;
    // Camera::setShutterEnd: the description at shutter close (hasEnd = 0: none)
    int hasEnd;
    V3 position1, lowerLeft1, horizontal1, vertical1, u1, v1, forward1;
    float lensRadius1;
};

enum VisMask : uint32_t { VIS_CAMERA = 1u, VIS_DIFFUSE = 2u, VIS_GLOSSY = 4u, VIS_TRANSMISSION = 8u, VIS_SHADOW = 16u,
                          VIS_ALL = 0x1Fu };
// Marks a random-walk ray in the ray's mask word.  Triangle masks never carry it, so it does
// not change what the ray can hit; the closest-hit kernel bins such rays under their own key.
constexpr uint32_t RAY_WALK = 1u << 31;
constexpr int kMaxMediumEvents = 1024; // path_tracer.cpp:51
constexpr int kMaxWalkSteps = 256;     // path_tracer.cpp:52
// Closest-hit queries one path can make: at most 255 bounces, each preceded by up to 64 skipped
// camera-invisible hits and 65 pass-throughs and followed by up to 256 walk steps, plus 1025
// medium events, stays below this; a path that reaches it is counted as an error and ended.
constexpr int kMaxPathQueries = 1 << 17;

// path flags (bits of state word)
enum PathFlags : uint32_t {
    PF_SPECULAR_BOUNCE = 1u << 0,
    PF_CAMERA_RAY = 1u << 1,
    PF_PICKER_VALID = 1u << 2,
    PF_FIRST_SEGMENT = 1u << 3,
    PF_WALK = 1u << 4,   // inside a random walk: lastP = σt, lastN = albedo, pickP.x = g
    PF_GUIDE_SNAP = 1u << 5, // the path's guide training record waits for its radiance snapshot
};
// Bits 24..31 of the flags word: the light-link node of the path's last surface vertex.
constexpr uint32_t kPrevNodeShift = 24;
constexpr uint32_t kPrevNodeMask = 0xFFu << kPrevNodeShift;

// Per-slot state columns (capacity P slots).
struct Paths {
    float4* rayO;    // origin xyz, visibility mask (bits)
    float4* rayD;    // direction xyz, lastBsdfPdf
    float4* thr;     // throughput xyz, wavelength
    float4* L;       // radiance xyz, unused
    float4* lastN;   // last shading normal xyz, flags (bits)
    float4* lastP;   // last point xyz, Sobol dimension (bits)
    float4* pickP;   // light-picker point xyz, pixel hash (bits)
    float4* pickN;   // light-picker normal xyz, counters (bits: depth | diffuseBounces<<8 | passThroughs<<16 | skips<<24)
    float4* hit;     // t, u, v, leaf prim (bits)
    float* time;     // shutter time of the path's rays (read where the scene has moving instances)
    float4* med;     // media stack slots 0,1 | slots 2,3 (bits), mediumEvents | walkStep<<16, stack depth
    int32_t* queueA;
    int32_t* queueB;
    int32_t* shadowQ;
    float4* shO;     // shadow origin xyz, tMax
    float4* shD;     // shadow direction xyz, scalar (cos*w/(pdf*n))
    float4* shC;     // f*Li xyz, flags (bit0: indirect)
    float4* shT;     // throughput at NEE xyz
    uint8_t* key;    // shading key of the slot's closest hit, or kKeyOfPrim (kBin)
    int32_t* sortQ;  // kShadeKeys segments of `capacity` slots: rays binned by shading key
    // learned proposal (null / 0 when off)
    float4* guideQ;      // 3 per query row, compacted per bounce: hit point | shading normal | view direction
    int32_t* guideSlot;  // slot of each query row
    float4* guideOut;    // kSlotMixture per slot: this bounce's proposal (putMixture)
    uint32_t* guideMark; // 1 = guideOut holds this bounce's proposal for the slot
    float4* guideRec;    // 6 per slot: training record of the first guidable vertex (see kGuideCollect)
    float4* trainBuf;    // 4 per training sample, compacted per wave
    int32_t guiding;     // 0 off, 1 record training samples, 2 record and sample with the proposal
    int32_t guideStride; // one path in guideStride records a training sample (trainOrder; about 64K per wave)
    // SD-tree guiding (null / 0 when off)
    SdField sd;          // sampling trees (read), building trees (splats)
    int32_t sdMode;      // bit 0: record training vertices, bit 1: sample with the SD-tree
    float4* sdRec;       // kSdRecords × 4 per slot: (point, pdf) | (ω, 0) | (throughput after, 0) | (radiance snapshot, state)
    uint32_t* sdCount;   // recorded vertices per slot
    // path regeneration (null in a wave whose paths are its slots): a wave of more paths than
    // slots refills each slot freed by an ended path with the wave's next path
    int32_t* pathOf;     // wave path index held by each slot
    int32_t* freeQ;      // slots freed by the shading kernel this bounce
    float4* Lout;        // radiance of each ended path, by wave path index (read by the film kernel)
    uint32_t* segLeft;   // per segment: paths not yet ended (null unless the server tracks segments)
    // AOVs of each path (null unless requested): albedo + alpha, primary normal
    float4* aovA;
    float4* aovN;
    // render passes of each path (null unless requested): passStride float4 per path, laid out
    // as PassSlots says; shPass: 3 per shadow record, the lobe shares of a first-vertex NEE term
    float4* pass;
    float4* shPass;
    int32_t passStride;
    // ray cone of each slot's current ray: width, spread (null without; read only in scenes
    // with mipmapped textures)
    float2* cone;
    // sweeps (continuous waves): a path alive for sweepAge bounces leaves the wavefront for a
    // tail-kernel launch on a side stream (sweepAge 0: off)
    int32_t* born;       // bounce at which each slot's path was injected
    int32_t* sweepQ;     // this bounce's swept slots (counted in counters[CNT_SWEEP])
    int32_t sweepAge;
    int32_t iter;        // current bounce of the continuous wave
    uint32_t capacity;
    // bounce counters (BounceCounters): two blocks that the bounces of a wave use in turn.  A bounce
    // traces and shades what `now` counts and appends to what `next` counts; kBin clears `next`.
    uint32_t* blocks;
    uint32_t* now;
    uint32_t* next;
    // 1: a path that ends hands its radiance to Lout at once, and a shadow ray still to be traced
    // for its last vertex adds to Lout (shadowQ holds ~path); its slot is free for another path
    int32_t direct;
    // wave counters (CounterSlots)
    uint32_t* counters;
};

// A path's render-pass block (float4 slots): the eight light passes (LightPass order), the
// lobe shares of the first bounce (firstLobe, path_tracer.cpp:375), the camera ray's origin and
// then the first hit (xyz, w = distance), the object and material id colours (w of the object
// slot: 1 on a hit), the Cryptomatte object and material ids of the hit, then one slot per
// light group.
enum PassSlots { PASS_DIFFUSE_DIRECT = 0, PASS_EMISSION = 6, PASS_BACKGROUND = 7, PASS_LOBES = 8, PASS_HIT = 11,
                 PASS_OBJECT = 12, PASS_MATERIAL = 13, PASS_CRYPTO = 14, PASS_GROUPS = 15 };
// Films of the pass target, 5 floats per pixel each (sum 3n, count n, sum of squares n).
enum PassFilms { PFILM_DEPTH = 8, PFILM_POSITION = 9, PFILM_OBJECT = 10, PFILM_MATERIAL = 11, PFILM_GROUPS = 12 };

// Shading keys: 0 = miss, 1 + material type (Lambert, Disney, Dielectric, Mirror), 5 = random-walk step.
constexpr int kShadeKeys = 6;
// Shading features beyond a plain surface scene's, as instantiations of the shading code carry them.
enum ShadeFeatures {
    FEAT_MEDIA = 1, // media, subsurface walks, dispersion
    FEAT_GUIDE = 2, // the learned proposal, the SD-tree
    FEAT_REST = 4,  // cutouts, rounded edges, ray cones, light and shadow links, shadow catchers, ambient occlusion
    FEAT_ALL = 7
};
constexpr uint8_t kKeyOfPrim = 255; // Paths::key: kBin derives the key from the hit's primitive
// Counters of one bounce: the closest-hit queue's entries, the shadow records, the work cursors of
// the trace and shading kernels, the rays per shading key and their bins' cursors.
enum BounceCounters { BC_QUEUE = 0, BC_SHADOW = 1, BC_WORK_ISECT = 2, BC_WORK_SHADOW = 3, BC_WORK_SHADE = 4, BC_KEYS = 5,
                      BC_WORK_KEYS = BC_KEYS + kShadeKeys, BC_TOTAL = BC_WORK_KEYS + kShadeKeys };
constexpr int kBounceBlock = 32; // counters from one block to the next
static_assert(BC_TOTAL <= kBounceBlock, "a bounce's counters fit its block");
// Counters of a wave, after the two bounce blocks.
enum CounterSlots { CNT_WORK_TAIL = 0, CNT_GUIDE_Q = 1, CNT_TRAIN = 2, CNT_FREE = 3, CNT_SWEEP = 4, CNT_WAVE = 5 };
constexpr int kCounters = 2 * kBounceBlock + CNT_WAVE; // all of them, from Paths::blocks on
// Paths per wave with regeneration, as a multiple of the slots.
constexpr int kStreamFactor = 16;
// Vertices an SD-tree training path records (the reference records up to 32; its paths in these
// workloads rarely pass 8 guidable vertices).
constexpr int kSdRecords = 8;
enum SdModeBits { SD_RECORD = 1, SD_SAMPLE = 2 };
// Training samples of the learned proposal per wave (the record stride is chosen to give about this many).
constexpr int kGuideTrainRows = 1 << 16;

// One request's share of a wave: a rectangle of its film, a range of its sample indices and its
// render settings.  Wave slots [slotFirst, slotFirst + nPix·nSamples) are its paths, pixel by pixel
// (slot = slotFirst + p·nSamples + s; neighbouring paths are samples of one pixel, then of the
// pixels around it: tilePixel), and its pixels are wave pixels [pixFirst, pixFirst + nPix).
struct WaveSeg {
    CamDev cam;
    int width, height;      // film
    int tileX, tileY, tileW, tileH; // rendered rectangle of the film (whole frame: 0, 0, width, height)
    const int32_t* pixList;  // film pixel (y·width + x) of each tile-linear pixel, or null: the rectangle
    int pixelFirst, nPix;   // range of tile-linear pixel indices in this wave
    int sampleFirst, nSamples;
    uint64_t seed;
    float filterWidth;
    int maxDepth, rrDepth, shadowSamples;
    float clampIndirect;
    const float* filterCdf; // inverse-CDF table of the request's pixel filter
    float* sum;             // the request's film on the device
    uint32_t* cnt;
    float* sq;
    float* aov;             // AOV films (albedo, normal, alpha: each sum 3n, count n, sum of squares n), or null
    float* pass;            // render-pass films (PassFilms order, 5n floats each), or null
    float* cryptoObj;       // Cryptomatte ids per (sample − cryptoFirst, film pixel), or null
    float* cryptoMat;
    int cryptoFirst;
    int slotFirst;
    int pixFirst;
    int flags;              // SegFlags
    float aoStrength;       // RenderSettings::aoStrength (contact AO at camera hits)
    float coneWidth, coneSpread; // camera rays' cone (Camera::pixelConeWidth / pixelConeSpread)
};
// SEG_SWEEP: paths of the segment may leave a continuous wave for a sweep; SEG_MOTION:
// RenderSettings::motionBlur (each camera sample draws a shutter time)
enum SegFlags { SEG_SWEEP = 1, SEG_MOTION = 2 };

// The segments of one wave, ordered by slotFirst (and so by pixFirst).
struct Wave {
    const WaveSeg* segs;
    int nSegs;
    int nSlots;
    int nPix;
};

// Path state whose counters start at `p` (kCounters words).
inline void setCounters(Paths& P, uint32_t* p) {
    P.blocks = p;
    P.now = p;
    P.next = p + kBounceBlock;
    P.counters = p + 2 * kBounceBlock;
}
// ... at bounce block b.
inline void setBlock(Paths& P, int b) {
    P.now = P.blocks + b * kBounceBlock;
    P.next = P.blocks + (1 - b) * kBounceBlock;
}

// The columns that every wave reads or writes, each as f(column, entries per slot).  The lanes and the
// fixed scratch of pe_device_render_tile_noalloc both take theirs from this list, so that neither can
// miss one that a kernel takes for granted.
template <typename F>
constexpr void eachWaveColumn(Paths& P, F f) {
    f(P.rayO, 1); f(P.rayD, 1); f(P.thr, 1); f(P.L, 1); f(P.lastN, 1); f(P.lastP, 1); f(P.pickP, 1); f(P.pickN, 1);
    f(P.hit, 1); f(P.med, 1);
    f(P.shO, 1); f(P.shD, 1); f(P.shC, 1); f(P.shT, 1); // shadow records: one per slot (shadow quality 1)
    f(P.queueA, 1); f(P.queueB, 1); f(P.shadowQ, 1); f(P.sortQ, kShadeKeys);
    f(P.key, 1);
}
// Bytes of path state carved by carveWave: the columns of `slots` slots, then every counter.
constexpr size_t kCarveAlign = 256;
constexpr size_t waveBytes(size_t slots) {
    Paths P{};
    size_t bytes = 0;
    eachWaveColumn(P, [&](auto*& column, size_t entries) { bytes += entries * slots * sizeof(*column); });
    return bytes + (kCounters * sizeof(uint32_t) + kCarveAlign - 1) / kCarveAlign * kCarveAlign;
}
// Path state of `slots` (a multiple of kCarveAlign) slots in the waveBytes(slots) bytes at `base`.
inline Paths carveWave(unsigned char* base, size_t slots) {
    Paths P{};
    eachWaveColumn(P, [&](auto*& column, size_t entries) {
        column = reinterpret_cast<std::decay_t<decltype(column)>>(base);
        base += entries * slots * sizeof(*column);
    });
    setCounters(P, reinterpret_cast<uint32_t*>(base));
    P.capacity = static_cast<uint32_t>(slots);
    return P;
}

// Sample (of the segment's nSamples) of a wave path.
PE_HD int sampleOfPath(const WaveSeg& A, int path) {
    const int local = path - A.slotFirst;
    return local - (local / A.nSamples) * A.nSamples;
}
PE_HD int pathOfSample(const WaveSeg& A, int p, int s) { return A.slotFirst + p * A.nSamples + s; }
// Film position of the segment's tile-linear pixel tp.  The rectangle is numbered in bands of four
// rows, down each band's columns, so that the 32 paths of a warp look at a compact patch of the film
// (their camera rays meet the same nodes and their first hits the same surfaces).
PE_HD void tilePixel(const WaveSeg& A, int tp, int& x, int& y) {
    if (A.pixList) {
        const int fp = A.pixList[tp];
        x = fp % A.width;
        y = fp / A.width;
        return;
    }
    const int band = tp / (4 * A.tileW);
    const int rows = A.tileH - 4 * band < 4 ? A.tileH - 4 * band : 4;
    const int in = tp - band * 4 * A.tileW;
    const int col = in / rows;
    x = A.tileX + col;
    y = A.tileY + 4 * band + (in - col * rows);
}
// The learned proposal trains on the paths whose place in this order of the wave's paths is a multiple of
// guideStride: sample by sample, and within a sample the pixels row by row (a wave of part of a rectangle or
// of a pixel list: in the order of its pixels).  In the paths' own order a stride of the samples per
// pixel would train on the first sample of each pixel alone, and smaller ones on one row in four.
PE_HD bool wholeRectangle(const WaveSeg& A) { return !A.pixList && A.nPix == A.tileW * A.tileH; }
PE_HD int trainOrder(const WaveSeg& A, int path) {
    const int p = (path - A.slotFirst) / A.nSamples, s = path - A.slotFirst - p * A.nSamples;
    int r = p;
    if (wholeRectangle(A)) {
        int x, y;
        tilePixel(A, p, x, y);
        r = (y - A.tileY) * A.tileW + x - A.tileX;
    }
    return A.slotFirst + s * A.nPix + r;
}
// The path at place `order`.
PE_HD int pathOfTrainOrder(const WaveSeg& A, int order) {
    const int s = (order - A.slotFirst) / A.nPix, r = order - A.slotFirst - s * A.nPix;
    int p = r;
    if (wholeRectangle(A)) {
        const int y = r / A.tileW, x = r - y * A.tileW, band = y >> 2;
        const int rows = A.tileH - 4 * band < 4 ? A.tileH - 4 * band : 4;
        p = band * 4 * A.tileW + x * rows + (y - 4 * band);
    }
    return pathOfSample(A, p, s);
}
#ifdef __CUDACC__
// Wave path index held by a slot.
__device__ __forceinline__ int pathOfSlot(const Paths& P, int slot) { return P.pathOf ? P.pathOf[slot] : slot; }
// Segment owning a wave path / a wave pixel (binary search; one segment for a lone request).
__device__ __forceinline__ int segOfSlot(const Wave& W, int slot) {
    int lo = 0, hi = W.nSegs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (W.segs[mid].slotFirst <= slot) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}
__device__ __forceinline__ int segOfPixel(const Wave& W, int p) {
    int lo = 0, hi = W.nSegs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (W.segs[mid].pixFirst <= p) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

#endif

} // namespace pe
