// Kernels of the wavefront diffuse path tracer.
//
// The reference GPU path (render/diffuse_renderer_cuda.cu:159-212) runs, per
// pass: generateRaysKernel -> { OptiX Prime closest hit -> cudaMemcpy(counter)
// -> shadeRaysKernel -> cudaMemcpy(count) } per bounce.  Here a wave takes two
// persistent kernels: the first generates, traces and shades the primary rays
// and queues the paths that go on, the second (k_paths) carries those paths
// to their ends; small waves and next-event estimation take one.  Queue sizes
// stay on the device, so a whole render is launched without host synchronisation
// (and, of several waves, is captured as a CUDA graph by the API).
// k_bounce and k_bounce_nee with kFirst = false do one bounce of all paths
// per launch, for prt_render_profile's times per depth.
#include <algorithm>

#include "prt_internal.h"

namespace prt_b200 {

#ifndef PRT_COUNTERS
#define PRT_COUNTERS 0
#endif

// Traversal counters of the bounce kernel, compiled in with -DPRT_COUNTERS=1
// (the reference's RayStats nodeCount/primCount, core/ray_stats.h:23-28):
//   [0] node visits  [1] triangle tests  [2] rays  [3] warp traversal steps
//   [4] running lanes summed over steps  [5] warp triangle-loop iterations
//   (max over the running lanes of a step, summed)
__device__ unsigned long long g_counters[8];

namespace {

__device__ __forceinline__ void morton8x8(int m, int& x, int& y)
{
    // same order as the reference's mortonTableX/Y (image/morton.cpp)
    x = (m & 1) | ((m >> 1) & 2) | ((m >> 2) & 4);
    y = ((m >> 1) & 1) | ((m >> 2) & 2) | ((m >> 3) & 4);
}

// Pixel of item rr (< tilesX * tilesY * 64) of one pass of a wave: 8x8 tiles
// in row order, Morton order inside a tile (image/morton.cpp's tables).
// Returns false for items past the frame's right or bottom edge.
__device__ __forceinline__ bool wave_item_pixel(int rr, int tilesX, int W, int H, int& x, int& y)
{
    int tile = rr >> 6;
    int mx, my;
    morton8x8(rr & 63, mx, my);
    x = (tile % tilesX) * 8 + mx;
    y = (tile / tilesX) * 8 + my;
    return x < W && y < H;
}

// Camera ray i of a wave of `passes` passes: all passes of an item of the frame
// in turn, so that a warp's rays start in few pixels.  A packet then visits far
// fewer nodes than one that spans 8x4 pixels (1080p terrain frame, 16 passes a
// wave: packet kernel 6.72 -> 3.56 ms, frame of 32 passes 44.9 -> 38.6), the long
// packets at the horizon no longer come last, and rays of one warp stay closer
// together in the other kernels too (512x512 at 64 passes on the small scene 5.41 ->
// 5.03, 32 requests in one batch 29.7 -> 28.0, replay 1.62 -> 1.55; a frame of
// nothing but sky, which only makes camera rays, 3.00 -> 3.06).
template <class I>
__device__ __forceinline__ void wave_item(I i, int passes, int& pass, int& item)
{
    const I t = i / passes;
    pass = (int)(i - t * passes);
    item = (int)t;
}

__device__ __forceinline__ PathRec load_path(const PathRec* q, int i)
{
    const float4* p = reinterpret_cast<const float4*>(q + i);
    PathRec r;
    r.w0 = __ldcs(p);
    r.w1 = __ldcs(p + 1);
    return r;
}

__device__ __forceinline__ void store_path(PathRec* q, int i, float3 org, int tag, float3 dir, uint32_t rng)
{
    float4* p = reinterpret_cast<float4*>(q + i);
    __stcs(p, make_float4(org.x, org.y, org.z, __int_as_float(tag)));
    __stcs(p + 1, make_float4(dir.x, dir.y, dir.z, __uint_as_float(rng)));
}

// Adds the camera rays of a warp that end here (dst: their pixel, else nullptr) to
// the accumulation: c from each that left the scene (the same for all rays of a
// pixel), 0 from the others.  A warp holds many passes of few pixels, so with
// several passes it makes one add per pixel.
__device__ __forceinline__ void add_camera_rays(float4* dst, bool left, float c, bool severalPasses, unsigned lane)
{
    const unsigned FULL = 0xffffffffu;
    unsigned count = 1, lit = left ? 1 : 0;
    if (severalPasses)
    {
        const unsigned peers = __match_any_sync(FULL, reinterpret_cast<unsigned long long>(dst));
        lit = __popc(peers & __ballot_sync(FULL, left));
        count = __popc(peers);
        if (lane != (unsigned)(__ffs(peers) - 1)) dst = nullptr;
    }
    if (dst)
    {
        const float sum = __fmul_rn(c, (float)lit);
        red_add_v4(dst, sum, sum, sum, (float)count);
    }
}

// Warp-aggregated append: one atomic per warp, survivors keep lane order.
__device__ __forceinline__ int warp_append(bool pred, int* counter)
{
    const unsigned lane = threadIdx.x & 31u;
    unsigned m = __ballot_sync(0xffffffffu, pred);
    int base = 0;
    if (lane == 0 && m) base = atomicAdd(counter, __popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    return base + __popc(m & ((1u << lane) - 1u));
}

// Deferred triangle tests per kernel (see warp_trav_deferred): the path-replay
// megakernel, the intersector seam and the diffuse2 bounce have their own switches.
#ifndef PRT_DEFER_REPLAY
#define PRT_DEFER_REPLAY PRT_DEFER_TRIS
#endif
#ifndef PRT_DEFER_ISECT
#define PRT_DEFER_ISECT PRT_DEFER_TRIS
#endif
#ifndef PRT_DEFER_NEE
#define PRT_DEFER_NEE PRT_DEFER_TRIS
#endif

// Lanes refill once at least this many of a warp's 32 lanes are idle
// (persistent threads with dynamic ray fetch, Aila & Laine, HPG 2009): fewer
// shade with emptier warps, more traverse with them.  14 against 12: primaries
// per lane of a 33M-path terrain wave 8.10 -> 8.00 ms, a 32-request batch 31.45
// -> 30.95 ms; 16 and 18 lose 0.5-2% on the 1080p terrain.
#ifndef PRT_REFILL_MIN
#define PRT_REFILL_MIN 14
#endif
constexpr int kRefillMin = PRT_REFILL_MIN;

// Paired FP32 FMAs in the node test (node_hits1<true>): the six plane FMAs of
// two children become three fma.rn.f32x2.  First-bounce kernels, per-lane and
// packet: depth 0 of the terrain 4% / 7% faster, of the 10M field 6% / 8%.
#ifndef PRT_PAIRED_FIRST
#define PRT_PAIRED_FIRST 1
#endif
#ifndef PRT_PAIRED_PACKET
#define PRT_PAIRED_PACKET 1
#endif

// Later bounces keep only a path's origin and its traversal terms in registers
// while the warp traverses: the pixel, RNG state and direction are read again
// from the input queue when the lane shades.  That frees the registers the
// paired node test needs there (with the path kept in registers it spilled and
// ran 2-3% slower); with both, bounces 1-5 of the terrain run 3% faster.
#ifndef PRT_RELOAD_PATH
#define PRT_RELOAD_PATH 1
#endif
#ifndef PRT_PAIRED_LATER
#define PRT_PAIRED_LATER 1
#endif

// Paired node test of the next-event-estimation kernels: k_paths_nee and the later
// bounces of k_bounce_nee (diffuse2 on the terrain frame at 16 spp 2281 -> 2319
// Mrays/s); the first bounce of that one keeps single FMAs.
#ifndef PRT_PAIRED_NEE
#define PRT_PAIRED_NEE 1
#endif

// Paired node test in the any-hit ray-query kernel (k_intersect<true>): 4M
// incoherent occlusion queries on the terrain 1.085 -> 1.024 ms.  Closest-hit
// queries and k_batch_first have single FMAs: the former spilled with the paired test
// while they had 64 registers and kept the shear terms in them.  At 72 without those
// neither spills, and paired they would be 1% (4M closest hits 1.199 -> 1.188 ms) and
// 2% faster (three requests of 1000x700 and 4 passes 1.236 -> 1.211 ms).
#ifndef PRT_PAIRED_QUERY
#define PRT_PAIRED_QUERY 1
#endif

// Minimum resident 128-thread blocks per SM requested from the compiler for
// the bounce kernel (8 caps it at 64 registers per thread).
#ifndef PRT_BOUNCE_MIN_BLOCKS
#define PRT_BOUNCE_MIN_BLOCKS 8
#endif
// The kernels that carry more per lane (whole paths, a batch's request, shadow
// rays, gradients, barycentrics, the first bounce) spill at 64 registers and are
// faster with 72 and 7 blocks: 32-request batch 30.8 -> 29.9 ms, diffuse2 1080p 4
// passes 11.08 -> 10.93, 4M closest-hit queries 1.280 -> 1.265, adjoint 512x512 16
// passes 1.95 -> 1.93, the same with albedo forward 1.48 -> 1.44, 1080p 1 pass 1.83 ->
// 1.79 (32 passes 38.6 either way).  The others lose (bounce by bounce 0.7%, any hit
// 1.3%, packets 2%); 6 blocks lose 1-3%, 9 blocks (56 registers) 5%.
constexpr int kWideBlocks = 7;

// Words of shared memory per lane of the per-bounce kernels.
constexpr int bounce_words(bool first) { return kShearWords + (first || !PRT_RELOAD_PATH ? 5 : 0); }

// One bounce of the wavefront over the queue of paths entering `depth`.
// kFirst: the queue is implicit — item i is a pixel (8x8 tile, Morton index) and one
// of its passes (wave_item) — and the primary ray is generated in registers.
//
// Each warp keeps 32 rays in flight.  Traversal advances one 8-wide node per
// step; as soon as kRefillMin lanes have finished, the finished lanes shade
// their hit (or accumulate), append survivors to the next queue with one
// atomic per warp, and fetch fresh rays, so a few long rays do not idle the
// rest of the warp.
template <bool kFirst, bool kAlbedo>
__global__ void __launch_bounds__(128, kFirst ? kWideBlocks : PRT_BOUNCE_MIN_BLOCKS) k_bounce(WaveArgs a, int depth)
{
    extern __shared__ uint2 s_stack[];
    TravStack st;
    st.sh = s_stack + threadIdx.x;
    st.stride = blockDim.x;
    st.overflow = false;
    // the block's stack columns, then its lanes' words (shear terms and, in the
    // first bounce, pixel, RNG state and direction), then the triangle queues
    const int bd = blockDim.x;
    uint32_t* shw = reinterpret_cast<uint32_t*>(s_stack + kShared * blockDim.x) + threadIdx.x;
    TriQueue* tq = reinterpret_cast<TriQueue*>(reinterpret_cast<uint32_t*>(s_stack + kShared * blockDim.x) +
                                               bounce_words(kFirst) * blockDim.x) + (threadIdx.x >> 5);
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned ltMask = (1u << lane) - 1u;
    const int W = a.cam.width, H = a.cam.height;
    const int perPass = a.tilesX * a.tilesY * 64;
    int total;
    int pass0 = 0;
    if (kFirst)
    {
        total = a.passes * perPass;
        pass0 = *a.passBase + a.passOffset;
    }
    else
    {
        total = *(volatile int*)&a.counts[depth];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(a.rays, kFirst ? (unsigned long long)a.passes * (unsigned long long)W * (unsigned long long)H
                                 : (unsigned long long)total);
    const bool final = depth == a.maxDepth;

    bool has = false;         // this lane holds a ray
    bool exhausted = false;   // warp-uniform: every queue entry has been claimed
    uint32_t cNodes = 0, cTris = 0, cRays = 0;                          // per lane (PRT_COUNTERS)
    unsigned long long cSteps = 0, cLaneSteps = 0, cTriIters = 0;       // per warp (PRT_COUNTERS)
    int qi = 0;               // input-queue index of this lane's path (PRT_RELOAD_PATH)
    float thr = 0.f;
    TravRay r;
    TravState ts;
    ts.done = true;
    for (;;)
    {
        // --- refill idle lanes ---------------------------------------------
        unsigned idle = __ballot_sync(FULL, !has);
        if (!exhausted && (__popc(idle) >= kRefillMin || idle == FULL))
        {
            int n = __popc(idle);
            int base = 0;
            if (lane == 0) base = atomicAdd(&a.fetch[depth], n);
            base = __shfl_sync(FULL, base, 0);
            if (base + n >= total) exhausted = true;
            int i = base + __popc(idle & ltMask);
            if (!has && i < total)
            {
                float3 org, dir;
                int pixel = 0;
                uint32_t rng = 0;
                bool ok = true;
                if (kFirst)
                {
                    int pass, item;
                    wave_item(i, a.passes, pass, item);
                    int x, y;
                    if (!wave_item_pixel(item, a.tilesX, W, H, x, y))
                    {
                        ok = false;
                    }
                    else
                    {
                        pixel = x + y * W;
                        rng = rng_seed(pass0 + pass, pixel);
                        camera_ray(a.cam, x, y, rng, org, dir);
                        thr = kAlbedo ? 1.0f : a.thrConst;
                    }
                }
                else if (PRT_RELOAD_PATH)
                {
                    // L2 only: the record is read again (pixel, RNG, direction) when
                    // the lane shades
                    const float4* p = reinterpret_cast<const float4*>(a.qin + i);
                    const float4 w0 = __ldcg(p), w1 = __ldcg(p + 1);
                    org = f3(w0.x, w0.y, w0.z);
                    dir = f3(w1.x, w1.y, w1.z);
                    qi = i;
                    thr = kAlbedo ? __ldcs(a.thrIn + i) : a.thrConst;
                }
                else
                {
                    PathRec pr = load_path(a.qin, i);
                    org = f3(pr.w0.x, pr.w0.y, pr.w0.z);
                    pixel = __float_as_int(pr.w0.w);
                    dir = f3(pr.w1.x, pr.w1.y, pr.w1.z);
                    rng = __float_as_uint(pr.w1.w);
                    thr = kAlbedo ? __ldcs(a.thrIn + i) : a.thrConst;
                }
                if (ok)
                {
                    has = true;
                    if (kFirst || !PRT_RELOAD_PATH)
                    {
                        shw[4 * bd] = (uint32_t)pixel;
                        shw[5 * bd] = rng;
                        shw[6 * bd] = __float_as_uint(dir.x);
                        shw[7 * bd] = __float_as_uint(dir.y);
                        shw[8 * bd] = __float_as_uint(dir.z);
                    }
                    shear_store(shw, bd, shear_of(dir));
                    trav_setup(r, org, dir);
                    trav_init(ts, a.scene, FLT_MAX, st);
                }
            }
        }
        if (__ballot_sync(FULL, has) == 0)
        {
            if (exhausted) break;
            continue;
        }
        // --- traverse until the warp has enough idle lanes ------------------
        if (PRT_DEFER_TRIS && a.scene.deferTris)
        {
            // node visits queue their triangles; the warp tests them 32 at a
            // time, and every pending test is done before any lane shades
            constexpr bool kPair = kFirst ? PRT_PAIRED_FIRST : (PRT_RELOAD_PATH && PRT_PAIRED_LATER);
            warp_trav_deferred<kPair>(*tq, ts, a.scene, r, shw, bd, 0.0f, st, has, !exhausted, kRefillMin, lane,
                                      PRT_COUNTERS ? &cNodes : nullptr, PRT_COUNTERS ? &cTris : nullptr,
                                      PRT_COUNTERS ? &cSteps : nullptr, PRT_COUNTERS ? &cLaneSteps : nullptr,
                                      PRT_COUNTERS ? &cTriIters : nullptr);
        }
        else
        {
            const Shear sh = shear_load(shw, bd);
            for (;;)
            {
                if (PRT_COUNTERS)
                {
                    unsigned run0 = __ballot_sync(FULL, has && !ts.done);
                    uint32_t tris = 0;
                    if (has && !ts.done) trav_step<false>(ts, a.scene, r, sh, 0.0f, st, &cNodes, &tris);
                    cTris += tris;
                    cLaneSteps += __popc(run0);
                    cSteps += 1;
                    cTriIters += __reduce_max_sync(FULL, tris);
                }
                else if (has && !ts.done)
                {
                    trav_step<false>(ts, a.scene, r, sh, 0.0f, st);
                }
                unsigned running = __ballot_sync(FULL, has && !ts.done);
                if (running == 0) break;
                if (!exhausted && 32 - __popc(running) >= kRefillMin) break;
            }
        }
        // --- finish the lanes whose traversal is complete ---------------------
        // (the finished path's pixel, RNG state and rays are iteration-local, so
        // only what traversal needs is carried around the loop)
        const bool fin = has && ts.done;
        bool cont = false;
        float contrib = 0.f;
        int fpix = 0;
        uint32_t frng = 0;
        float3 forg = r.org, fdir = f3(0.f, 0.f, 0.f);
        if (fin)
        {
            if (!kFirst && PRT_RELOAD_PATH)
            {
                const float4* p = reinterpret_cast<const float4*>(a.qin + qi);
                const float4 w1 = __ldcs(p + 1);
                fpix = __float_as_int(__ldcs(reinterpret_cast<const float*>(p) + 3));
                fdir = f3(w1.x, w1.y, w1.z);
                frng = __float_as_uint(w1.w);
            }
            else
            {
                fpix = (int)shw[4 * bd];
                frng = shw[5 * bd];
                fdir = f3(__uint_as_float(shw[6 * bd]), __uint_as_float(shw[7 * bd]), __uint_as_float(shw[8 * bd]));
            }
            if (ts.triHit < 0)
            {
                contrib = __fmul_rn(thr, a.sky);
            }
            else if (!final)
            {
                if (kAlbedo) thr = __fmul_rn(thr, a.scene.albedo ? __ldg(a.scene.albedo + ts.primHit) : 0.8f);
                diffuse_bounce(a.scene.tris, ts.triHit, forg, fdir, ts.tHit, frng);
                cont = true;
            }
        }
        int o = warp_append(cont, &a.counts[depth + 1]);
        if (cont)
        {
            store_path(a.qout, o, forg, fpix, fdir, frng);
            if (kAlbedo) __stcs(a.thrOut + o, thr);
        }
        const bool ends = fin && !cont;
        if (kFirst)
        {
            const float skyContrib = __fmul_rn(kAlbedo ? 1.0f : a.thrConst, a.sky);
            if (__any_sync(FULL, ends))
                add_camera_rays(ends ? a.accum + fpix : nullptr, ends && ts.triHit < 0, skyContrib, a.passes > 1, lane);
        }
        else if (ends)
        {
            red_add_v4(a.accum + fpix, contrib, contrib, contrib, 1.0f);
        }
        if (fin)
        {
            has = false;
            ++cRays;
        }
    }
    if (PRT_COUNTERS)
    {
        unsigned long long n = cNodes, t = cTris, ry = cRays;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
        {
            n += __shfl_down_sync(FULL, n, off);
            t += __shfl_down_sync(FULL, t, off);
            ry += __shfl_down_sync(FULL, ry, off);
        }
        if (lane == 0)
        {
            atomicAdd(&g_counters[0], n);
            atomicAdd(&g_counters[1], t);
            atomicAdd(&g_counters[2], ry);
            atomicAdd(&g_counters[3], cSteps);
            atomicAdd(&g_counters[4], cLaneSteps);
            atomicAdd(&g_counters[5], cTriIters);
        }
    }
}

// All bounces after the first in one launch, for a wave (WaveArgs) or for a
// wave of a batch (BatchArgs).  A lane takes a path from the depth-1 queue and
// carries it to its end, bouncing in place, then takes the next one.  One
// launch per bounce ends in a tail of its own, 60-100 us in which the longest
// rays of that depth run on an emptying chip, and writes and compacts every
// path; here a wave has one tail and a path is written once.  Rays of mixed
// depths share a warp, which costs little: from the second ray on a path's
// neighbours have scattered.  What a path needs only when it is shaded lives in
// shared memory (kPathWords words per lane), so the registers hold what
// traversal needs; a block takes 18 KB.
// Measured against one launch per bounce: 1080p terrain frame of 1 pass 2.12 ->
// 1.88 ms and of 32 passes 46.4 -> 45.2, 256x256 and 16 passes of 82K triangles
// 0.765 -> 0.63 ms, 10.24M-triangle field at 4 passes and 9 bounces 5.17 -> 4.72.
// kPrimary: the lanes generate their paths' camera rays too, so a small wave is
// one launch with one tail and needs no queue (whole_paths below).
// tag (pixel; in a batch request << 24 | pixel), depth, RNG, throughput, direction, shear terms
constexpr int kPathWords = 7 + kShearWords;

__device__ __forceinline__ const SceneDev& path_scene(const WaveArgs& a, int) { return a.scene; }
__device__ __forceinline__ float4* path_accum(const WaveArgs& a, uint32_t tag) { return a.accum + tag; }
__device__ __forceinline__ int path_max_depth(const WaveArgs& a, int) { return a.maxDepth; }
__device__ __forceinline__ const SceneDev& path_scene(const BatchArgs& a, int req) { return a.reqs[req].scene; }
__device__ __forceinline__ float4* path_accum(const BatchArgs& a, uint32_t tag)
{
    return a.reqs[tag >> 24].accum + (tag & 0xffffffu);
}
__device__ __forceinline__ int path_max_depth(const BatchArgs& a, int req) { return a.reqs[req].maxDepth; }
__device__ __forceinline__ bool path_deferred(const WaveArgs& a) { return a.scene.deferTris != 0; }
__device__ __forceinline__ bool path_deferred(const BatchArgs& a) { return a.leaf1 != 0; }

// Idle lanes of a warp at which it leaves traversal, act of its lanes holding a
// ray: kRefillMin of a full warp, the same share of a partly filled one.
__device__ __forceinline__ int stop_idle(unsigned act)
{
    const int n = __popc(act);
    return 32 - n + max(1, n * kRefillMin / 32);
}

template <class Args, bool kBatch, bool kAlbedo, bool kPrimary>
__global__ void __launch_bounds__(128, kWideBlocks) k_paths(Args a)
{
    static_assert(!(kBatch && kPrimary), "a batch's primary rays have their own kernels");
    extern __shared__ uint2 s_stack[];
    TravStack st;
    st.sh = s_stack + threadIdx.x;
    st.stride = blockDim.x;
    st.overflow = false;
    uint32_t* s_path = reinterpret_cast<uint32_t*>(s_stack + kShared * blockDim.x);
    uint32_t* path = s_path + threadIdx.x;   // word k of this lane's path at path[k * bd]
    TriQueue* tq = reinterpret_cast<TriQueue*>(s_path + kPathWords * blockDim.x) + (threadIdx.x >> 5);   // deferred
    const int bd = blockDim.x;
    uint32_t* shw = path + 7 * bd;
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned ltMask = (1u << lane) - 1u;
    int total, perPass = 0, pass0 = 0;
    if constexpr (kPrimary)
    {
        perPass = a.tilesX * a.tilesY * 64;
        total = a.passes * perPass;
        pass0 = *a.passBase + a.passOffset;
        if (blockIdx.x == 0 && threadIdx.x == 0)
            atomicAdd(a.rays, (unsigned long long)a.passes * (unsigned long long)a.cam.width *
                                  (unsigned long long)a.cam.height);
    }
    else
    {
        total = *(volatile int*)&a.counts[1];
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(a.rays, (unsigned long long)total);
    }
    uint32_t more = 0;   // rays of bounces in this kernel, per warp

    bool has = false;         // this lane holds a path
    bool exhausted = false;   // warp-uniform: every queued path has been claimed
    int req = 0;              // kBatch: the request of this lane's path
    TravRay r;
    TravState ts;
    ts.done = true;
    for (;;)
    {
        // --- lanes whose ray is traced: the path ends or bounces -----------------
        bool fresh = false;   // this lane has a new ray (org, dir)
        float3 org, dir;
        if (has && ts.done)
        {
            const int depth = (int)path[bd];
            float thr = __uint_as_float(path[3 * bd]);
            if (ts.triHit < 0 || depth == path_max_depth(a, req))
            {
                const float c = ts.triHit < 0 ? __fmul_rn(thr, a.sky) : 0.0f;
                red_add_v4(path_accum(a, path[0]), c, c, c, 1.0f);
                has = false;
            }
            else
            {
                const SceneDev& sc = path_scene(a, req);
                uint32_t rng = path[2 * bd];
                org = r.org;
                dir = f3(__uint_as_float(path[4 * bd]), __uint_as_float(path[5 * bd]), __uint_as_float(path[6 * bd]));
                thr = __fmul_rn(thr, kAlbedo && sc.albedo ? __ldg(sc.albedo + ts.primHit) : 0.8f);
                diffuse_bounce(sc.tris, ts.triHit, org, dir, ts.tHit, rng);
                path[bd] = (uint32_t)(depth + 1);
                path[2 * bd] = rng;
                path[3 * bd] = __float_as_uint(thr);
                fresh = true;
            }
        }
        more += __popc(__ballot_sync(FULL, fresh));
        // --- lanes without a path take the next ones ------------------------------
        const unsigned idle = __ballot_sync(FULL, !has);
        if (!exhausted && idle)
        {
            const int n = __popc(idle);
            int base = 0;
            if (lane == 0) base = atomicAdd(&a.fetch[kPrimary ? 0 : 1], n);
            base = __shfl_sync(FULL, base, 0);
            exhausted = base + n >= total;
            const int i = base + __popc(idle & ltMask);
            if (!has && i < total)
            {
                if constexpr (kPrimary)
                {
                    int pass, item;
                    wave_item(i, a.passes, pass, item);
                    int x, y;
                    if (wave_item_pixel(item, a.tilesX, a.cam.width, a.cam.height, x, y))
                    {
                        const int pixel = x + y * a.cam.width;
                        uint32_t rng = rng_seed(pass0 + pass, pixel);
                        camera_ray(a.cam, x, y, rng, org, dir);
                        path[0] = (uint32_t)pixel;
                        path[bd] = 0u;
                        path[2 * bd] = rng;
                        path[3 * bd] = __float_as_uint(1.0f);
                        has = fresh = true;
                    }
                }
                else
                {
                    const PathRec pr = load_path(a.qin, i);
                    org = f3(pr.w0.x, pr.w0.y, pr.w0.z);
                    dir = f3(pr.w1.x, pr.w1.y, pr.w1.z);
                    const uint32_t tag = __float_as_uint(pr.w0.w);
                    if (kBatch) req = (int)(tag >> 24);
                    float thr = 0.8f;
                    if constexpr (!kBatch) thr = kAlbedo ? __ldcs(a.thrIn + i) : a.thrConst;
                    path[0] = tag;
                    path[bd] = 1u;
                    path[2 * bd] = __float_as_uint(pr.w1.w);
                    path[3 * bd] = __float_as_uint(thr);
                    has = fresh = true;
                }
            }
        }
        const unsigned act = __ballot_sync(FULL, has);
        if (act == 0)
        {
            if (exhausted) break;
            continue;   // kPrimary: a tile's items outside the frame
        }
        if (fresh)
        {
            path[4 * bd] = __float_as_uint(dir.x);
            path[5 * bd] = __float_as_uint(dir.y);
            path[6 * bd] = __float_as_uint(dir.z);
            shear_store(shw, bd, shear_of(dir));
            trav_setup(r, org, dir);
            trav_init(ts, path_scene(a, req), FLT_MAX, st);
        }
        // --- traverse until enough of the warp's rays are done ---------------------
        const int stopIdle = stop_idle(act);
        if (PRT_DEFER_TRIS && path_deferred(a))
        {
            warp_trav_deferred<PRT_PAIRED_LATER>(*tq, ts, path_scene(a, req), r, shw, bd, 0.0f, st, has, true, stopIdle, lane);
        }
        else
        {
            const Shear sh = shear_load(shw, bd);
            for (;;)
            {
                if (has && !ts.done) trav_step<false>(ts, path_scene(a, req), r, sh, 0.0f, st);
                const unsigned running = __ballot_sync(FULL, has && !ts.done);
                if (32 - __popc(running) >= stopIdle) break;
            }
        }
    }
    if (lane == 0 && more) atomicAdd(a.rays, (unsigned long long)more);
}

// Primary rays as warp packets (trees with one-triangle leaves).  A warp takes
// 32 consecutive wave items, the passes of few pixels (of one pass, half of an 8x8
// tile), and traverses the tree once for all of them: every lane tests its own
// ray against the node all lanes are at (one broadcast load of the node), the
// node's child hits are OR-ed over the warp, and the children are visited in
// the order of one ray octant shared by the warp, from a stack in shared
// memory that the warp shares.  Each lane culls with its own closest hit and
// tests the triangles of the leaves its own ray hits, so its result is its
// closest hit, the same as per-lane traversal gives (exact ties go to the
// lower primitive id either way).  Camera rays of few pixels visit nearly the same
// nodes, so the lanes stay busy together where the per-lane traversal of k_bounce
// runs 20 of 32 lanes per instruction at this depth; with one pass and coarse
// pixels the union of the rays' nodes grows and the packet loses, and so do small
// waves, which end in the longest packet.  prt_tune.primaryPackets asks for packets
// or lanes (the autotuner tries both); without it large waves of many passes take
// packets (primary_packets in wave_plan.h).
#ifndef PRT_PACKET_PRIMARY
#define PRT_PACKET_PRIMARY 1
#endif
constexpr int kPacketStack = 64;   // >= levels of the deepest tree the build accepts (32)

// The child test of a shared-origin packet split over 24 lanes, one axis of
// one child each, combined with shuffles: the same bounds with about half the
// instructions per node (terrain frame 3061 -> 3106 Mrays/s).
#ifndef PRT_PACKET_IA_SPLIT
#define PRT_PACKET_IA_SPLIT 1
#endif

// Interval traversal of a packet whose rays share one direction octant.  The
// warp tests the packet, not each ray, against a node: lane c (of 0..7) takes
// child c (with a shared origin, lanes c, c + 8 and c + 16 take its x, y and
// z axis, PRT_PACKET_IA_SPLIT) and bounds the entry and exit distances of
// every ray of the packet on each axis from the packet's origin and
// inverse-direction ranges (interval
// products of [plane - omax, plane - omin] and [imin, imax]); the child is
// entered if the largest entry bound does not pass the smallest exit bound,
// clipped to [0, the packet's farthest closest hit].  Child planes are widened
// by one quantization step on both sides (the per-ray test's decode error is
// 2^-9 of a step), so a child that any ray's own test would enter is entered:
// the packet visits a superset of the nodes its rays visit, every lane tests
// its ray against every triangle of the entered leaves with the exact test,
// and each lane's result is its own closest hit.  One child test per node
// instead of one per ray and child; packets of a pinhole camera share one
// origin and need half the interval products (the terrain frame 3015 -> 3060
// Mrays/s).  A launch option (LaunchCfg::packet 2) the autotuner chooses: it
// wins where a packet's rays stay close (fine pixels, short rays; the 1080p
// terrain frame: 3021 against 2982 Mrays/s with per-ray packet tests, before
// the shared-origin case) and loses where they spread apart over long, often
// missing rays (the packet culls with its farthest hit; the 10M-triangle
// field: 2286 against 2859).  Testing each lane's own ray against a leaf's box
// before its triangle (planes kept in shared memory) won back part of the
// field (2580) but cost the terrain as much (2979), and also culling children
// with the four side planes of a pinhole packet's frustum (built from the
// camera basis and the packet's pixel block) cost more than it saved (terrain
// 3063 -> 2921, field 2323 -> 2142), so neither is done.

__device__ __forceinline__ float warp_min_f(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ float warp_max_f(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Bounds of (plane - o) * inv over o in [omin, omax], inv in [imin, imax]
// (kPoint: one origin shared by the packet, omin == omax).
template <bool kPoint>
__device__ __forceinline__ float ia_min(float plane, float omin, float omax, float imin, float imax)
{
    if (kPoint)
    {
        const float d = plane - omin;
        return fminf(d * imin, d * imax);
    }
    const float d0 = plane - omax, d1 = plane - omin;
    return fminf(fminf(d0 * imin, d0 * imax), fminf(d1 * imin, d1 * imax));
}

template <bool kPoint>
__device__ __forceinline__ float ia_max(float plane, float omin, float omax, float imin, float imax)
{
    if (kPoint)
    {
        const float d = plane - omin;
        return fmaxf(d * imin, d * imax);
    }
    const float d0 = plane - omax, d1 = plane - omin;
    return fmaxf(fmaxf(d0 * imin, d0 * imax), fmaxf(d1 * imin, d1 * imax));
}

// The traversal loop of packet_closest_hit_ia over the packet's ranges.
template <bool kPoint>
__device__ __forceinline__ void packet_ia_loop(const SceneDev& sc, const TravRay& r, const Shear& sh, bool valid, uint32_t woct,
                                               uint2* stk, unsigned lane, float& tHit, int& primHit, int& triHit,
                                               float oxmin, float oxmax, float oymin, float oymax, float ozmin,
                                               float ozmax, float ixmin, float ixmax, float iymin, float iymax,
                                               float izmin, float izmax)
{
    const unsigned FULL = 0xffffffffu;
    const uint32_t oct = 7u - oct_inv(woct);   // bit k: negative direction on axis k
    const bool nx = (oct & 1u) != 0u, ny = (oct & 2u) != 0u, nz = (oct & 4u) != 0u;
    const int c = (int)(lane & 7u);
    const int cw = c >> 2, cb = c & 3;
    // the axis this lane bounds in the split child test (lanes 24..31 repeat z)
    const int ax = min((int)(lane >> 3), 2);
    const float oa = ax == 0 ? oxmin : (ax == 1 ? oymin : ozmin);
    const float ia0 = ax == 0 ? ixmin : (ax == 1 ? iymin : izmin), ia1 = ax == 0 ? ixmax : (ax == 1 ? iymax : izmax);
    const bool na = ax == 0 ? nx : (ax == 1 ? ny : nz);
    float tfarP = FLT_MAX;
    int sp = 0;
    uint2 ng = make_uint2(0u, 0x80000000u);   // the root: one internal child at base 0
    for (;;)
    {
        const uint32_t nodeIdx = next_child(ng, woct);
        if ((ng.y & 0xff000000u) && sp < kPacketStack)
        {
            if (lane == 0) stk[sp] = ng;
            ++sp;
        }
        const uint4* qp = reinterpret_cast<const uint4*>(sc.nodes + nodeIdx);
        uint4 q[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) q[k] = __ldg(qp + k);
        // child c of the node against the packet; a relative slack of 2^-18 on
        // both bounds is far more than the rounding of either test at any
        // distance the planes' step margin does not cover
        bool enter;
        if constexpr (kPoint && PRT_PACKET_IA_SPLIT)
        {
            // lane (axis a, child c) bounds one axis; lanes c, c + 8, c + 16
            // hold the x, y, z bounds of child c and lane c combines them
            const uint32_t sh = 8u * (uint32_t)ax;
            const float sa = __uint_as_float(((q[0].w >> sh) & 0xffu) << 23);
            const float pa = __uint_as_float(ax == 0 ? q[0].x : (ax == 1 ? q[0].y : q[0].z));
            const uint32_t loW = ax == 0 ? (cw ? q[2].y : q[2].x)
                                          : (ax == 1 ? (cw ? q[2].w : q[2].z) : (cw ? q[3].y : q[3].x));
            const uint32_t hiW = ax == 0 ? (cw ? q[3].w : q[3].z)
                                          : (ax == 1 ? (cw ? q[4].y : q[4].x) : (cw ? q[4].w : q[4].z));
            const float lo = fmaf(byte_f(loW, cb) - 1.0f, sa, pa), hi = fmaf(byte_f(hiW, cb) + 1.0f, sa, pa);
            const float dn = (na ? hi : lo) - oa, df = (na ? lo : hi) - oa;
            const float tn = fminf(dn * ia0, dn * ia1), tf = fmaxf(df * ia0, df * ia1);
            const float tn1 = __shfl_sync(FULL, tn, c + 8), tn2 = __shfl_sync(FULL, tn, c + 16);
            const float tf1 = __shfl_sync(FULL, tf, c + 8), tf2 = __shfl_sync(FULL, tf, c + 16);
            const float t0 = fmaxf(fmax3(tn, tn1, tn2), 0.0f);
            const float t1 = fminf(fmin3(tf, tf1, tf2), tfarP * 1.0000004f);
            enter = t0 * 0.999996f <= t1 * 1.000004f;
        }
        else
        {
            const uint32_t e = q[0].w;
            const float sx = __uint_as_float((e & 0xffu) << 23), sy = __uint_as_float(((e >> 8) & 0xffu) << 23),
                        sz = __uint_as_float(((e >> 16) & 0xffu) << 23);
            const float px = __uint_as_float(q[0].x), py = __uint_as_float(q[0].y), pz = __uint_as_float(q[0].z);
            const float lx = fmaf(byte_f(cw ? q[2].y : q[2].x, cb) - 1.0f, sx, px);
            const float ly = fmaf(byte_f(cw ? q[2].w : q[2].z, cb) - 1.0f, sy, py);
            const float lz = fmaf(byte_f(cw ? q[3].y : q[3].x, cb) - 1.0f, sz, pz);
            const float hx = fmaf(byte_f(cw ? q[3].w : q[3].z, cb) + 1.0f, sx, px);
            const float hy = fmaf(byte_f(cw ? q[4].y : q[4].x, cb) + 1.0f, sy, py);
            const float hz = fmaf(byte_f(cw ? q[4].w : q[4].z, cb) + 1.0f, sz, pz);
            const float t0 = fmaxf(fmax3(ia_min<kPoint>(nx ? hx : lx, oxmin, oxmax, ixmin, ixmax),
                                         ia_min<kPoint>(ny ? hy : ly, oymin, oymax, iymin, iymax),
                                         ia_min<kPoint>(nz ? hz : lz, ozmin, ozmax, izmin, izmax)),
                                   0.0f);
            const float t1 = fminf(fmin3(ia_max<kPoint>(nx ? lx : hx, oxmin, oxmax, ixmin, ixmax),
                                         ia_max<kPoint>(ny ? ly : hy, oymin, oymax, iymin, iymax),
                                         ia_max<kPoint>(nz ? lz : hz, ozmin, ozmax, izmin, izmax)),
                                   tfarP * 1.0000004f);
            enter = t0 * 0.999996f <= t1 * 1.000004f;
        }
        uint32_t c8 = __ballot_sync(FULL, enter) & 0xffu;
        // non-empty slots (bit 5 of each meta byte), leaves and internal children
        const uint32_t ne = ((((q[1].z >> 5) & 0x01010101u) * 0x01020408u) >> 24) |
                            (((((q[1].w >> 5) & 0x01010101u) * 0x01020408u) >> 24) << 4);
        c8 &= ne;
        const uint32_t imask = q[0].w >> 24;
        const uint32_t leafMask = ne & ~imask;
        uint32_t lb = c8 & leafMask;
        if (lb)
        {
            do
            {
                const uint32_t bit = __ffs(lb) - 1u;
                lb &= lb - 1u;
                const int ti = (int)(q[1].y + __popc(leafMask & ((1u << bit) - 1u)));
                if (valid)
                {
                    const float4* tp = reinterpret_cast<const float4*>(sc.tris + ti);
                    const float4 v0 = __ldg(tp), v1 = __ldg(tp + 1), v2 = __ldg(tp + 2);
                    const int prim = __float_as_int(v0.w);
                    float t, u, v;
                    if (tri_test(r.org, sh, f3(v0.x, v0.y, v0.z), f3(v1.x, v1.y, v1.z), f3(v2.x, v2.y, v2.z), 0.0f, tHit,
                                 prim, primHit, t, u, v))
                    {
                        tHit = t;
                        primHit = prim;
                        triHit = ti;
                    }
                }
            } while (lb);
            tfarP = __uint_as_float(__reduce_max_sync(FULL, valid ? __float_as_uint(tHit) : 0u));
        }
        // internal hits: bit slot -> bit slot ^ octinv, as node_hits1 orders them
        const uint32_t in8 = permute_octant(c8 & imask, woct);
        ng = make_uint2(q[1].x, (in8 << 24) | imask);
        if (!(ng.y & 0xff000000u))
        {
            if (sp == 0) break;
            __syncwarp();
            ng = stk[--sp];
            __syncwarp();
        }
    }
}

__device__ __forceinline__ void packet_closest_hit_ia(const SceneDev& sc, const TravRay& r, const Shear& sh,
                                                      bool valid, unsigned vmask, uint32_t woct, uint2* stk, unsigned lane,
                                                      float& tHit, int& primHit, int& triHit)
{
    const unsigned FULL = 0xffffffffu;
    // packet ranges (lanes without a ray take the first ray's values)
    const int lead = __ffs(vmask) - 1;
    const float lox = __shfl_sync(FULL, r.org.x, lead), loy = __shfl_sync(FULL, r.org.y, lead),
                loz = __shfl_sync(FULL, r.org.z, lead);
    const float lix = __shfl_sync(FULL, r.inv.x, lead), liy = __shfl_sync(FULL, r.inv.y, lead),
                liz = __shfl_sync(FULL, r.inv.z, lead);
    const float ox = valid ? r.org.x : lox, oy = valid ? r.org.y : loy, oz = valid ? r.org.z : loz;
    const float ix = valid ? r.inv.x : lix, iy = valid ? r.inv.y : liy, iz = valid ? r.inv.z : liz;
    const float oxmin = warp_min_f(ox), oxmax = warp_max_f(ox);
    const float oymin = warp_min_f(oy), oymax = warp_max_f(oy);
    const float ozmin = warp_min_f(oz), ozmax = warp_max_f(oz);
    const float ixmin = warp_min_f(ix), ixmax = warp_max_f(ix);
    const float iymin = warp_min_f(iy), iymax = warp_max_f(iy);
    const float izmin = warp_min_f(iz), izmax = warp_max_f(iz);
    // pinhole packets share one origin: half the interval products
    if (oxmin == oxmax && oymin == oymax && ozmin == ozmax)
        packet_ia_loop<true>(sc, r, sh, valid, woct, stk, lane, tHit, primHit, triHit, oxmin, oxmax, oymin, oymax, ozmin,
                             ozmax, ixmin, ixmax, iymin, iymax, izmin, izmax);
    else
        packet_ia_loop<false>(sc, r, sh, valid, woct, stk, lane, tHit, primHit, triHit, oxmin, oxmax, oymin, oymax, ozmin,
                              ozmax, ixmin, ixmax, iymin, iymax, izmin, izmax);
}

// Warp-collective closest-hit traversal of the warp's rays as one packet (one-
// triangle leaves; every lane of the warp calls it).  valid: this lane holds a
// ray; vmask: the ballot of valid; stk: the warp's kPacketStack entries of
// shared memory.  Returns this lane's closest hit (triHit -1: none).
template <bool kPair, bool kIA>
__device__ __forceinline__ void packet_closest_hit(const SceneDev& sc, const TravRay& r, const Shear& sh, bool valid,
                                                   unsigned vmask, uint2* stk, unsigned lane, float& tHit, int& primHit, int& triHit)
{
    const unsigned FULL = 0xffffffffu;
    const uint32_t woct = __shfl_sync(FULL, r.oct, __ffs(vmask) - 1);
    tHit = FLT_MAX;
    primHit = 0x7fffffff;
    triHit = -1;
    if (!sc.hasRoot) return;
    if (kIA && __all_sync(FULL, !valid || r.oct == woct))
    {
        packet_closest_hit_ia(sc, r, sh, valid, vmask, woct, stk, lane, tHit, primHit, triHit);
        return;
    }
    int sp = 0;
    uint2 ng = make_uint2(0u, 0x80000000u);   // the root: one internal child at base 0
    for (;;)
    {
        const uint32_t nodeIdx = next_child(ng, woct);
        if ((ng.y & 0xff000000u) && sp < kPacketStack)
        {
            if (lane == 0) stk[sp] = ng;
            ++sp;
        }
        const uint4* qp = reinterpret_cast<const uint4*>(sc.nodes + nodeIdx);
        uint4 q[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) q[k] = __ldg(qp + k);
        uint32_t leafMask = 0;
        const uint32_t hits = valid ? node_hits1<kPair>(r, q, 0.0f, tHit, leafMask, woct) : 0u;
        // this lane's leaf triangles (leaf slot j -> triBase + rank of j among the leaf slots)
        uint32_t lb = hits & 0xffu;
        while (lb)
        {
            const uint32_t bit = __ffs(lb) - 1u;
            lb &= lb - 1u;
            const int ti = (int)(q[1].y + __popc(leafMask & ((1u << bit) - 1u)));
            const float4* tp = reinterpret_cast<const float4*>(sc.tris + ti);
            const float4 v0 = __ldg(tp), v1 = __ldg(tp + 1), v2 = __ldg(tp + 2);
            const int prim = __float_as_int(v0.w);
            float t, u, v;
            if (tri_test(r.org, sh, f3(v0.x, v0.y, v0.z), f3(v1.x, v1.y, v1.z), f3(v2.x, v2.y, v2.z), 0.0f, tHit, prim,
                         primHit, t, u, v))
            {
                tHit = t;
                primHit = prim;
                triHit = ti;
            }
        }
        ng = make_uint2(q[1].x, __reduce_or_sync(FULL, hits & 0xff000000u) | (q[0].w >> 24));
        if (!(ng.y & 0xff000000u))
        {
            if (sp == 0) break;
            __syncwarp();
            ng = stk[--sp];
            __syncwarp();
        }
    }
}

template <bool kAlbedo, bool kIA>
__global__ void __launch_bounds__(128, PRT_BOUNCE_MIN_BLOCKS) k_primary_packet(WaveArgs a)
{
    extern __shared__ uint2 s_packet[];
    uint2* stk = s_packet + (threadIdx.x >> 5) * kPacketStack;
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const int W = a.cam.width, H = a.cam.height;
    const int perPass = a.tilesX * a.tilesY * 64;
    const int total = a.passes * perPass;
    const int pass0 = *a.passBase + a.passOffset;
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(a.rays, (unsigned long long)a.passes * (unsigned long long)W * (unsigned long long)H);
    const bool final = a.maxDepth == 0;
    for (;;)
    {
        int base = 0;
        if (lane == 0) base = atomicAdd(&a.fetch[0], 32);
        base = __shfl_sync(FULL, base, 0);
        if (base >= total) break;
        const int i = base + (int)lane;
        bool valid = false;
        int pixel = 0;
        uint32_t rng = 0;
        float3 org = f3(0.f, 0.f, 0.f), dir = f3(0.f, 0.f, 1.f);
        if (i < total)
        {
            int pass, item;
            wave_item(i, a.passes, pass, item);
            int x, y;
            if (wave_item_pixel(item, a.tilesX, W, H, x, y))
            {
                valid = true;
                pixel = x + y * W;
                rng = rng_seed(pass0 + pass, pixel);
                camera_ray(a.cam, x, y, rng, org, dir);
            }
        }
        const unsigned vmask = __ballot_sync(FULL, valid);
        if (!vmask) continue;
        TravRay r;
        trav_setup(r, org, dir);
        float tHit;
        int primHit, triHit;
        packet_closest_hit<PRT_PAIRED_PACKET, kIA>(a.scene, r, shear_of(dir), valid, vmask, stk, lane, tHit, primHit, triHit);
        // shade / append / accumulate, as k_bounce does at depth 0
        bool cont = false;
        float thr = kAlbedo ? 1.0f : a.thrConst;
        const float skyContrib = __fmul_rn(thr, a.sky);
        const bool left = valid && triHit < 0;
        if (valid && !left && !final)
        {
            if (kAlbedo) thr = __fmul_rn(thr, a.scene.albedo ? __ldg(a.scene.albedo + primHit) : 0.8f);
            diffuse_bounce(a.scene.tris, triHit, org, dir, tHit, rng);
            cont = true;
        }
        const int o = warp_append(cont, &a.counts[1]);
        if (cont)
        {
            store_path(a.qout, o, org, pixel, dir, rng);
            if (kAlbedo) __stcs(a.thrOut + o, thr);
        }
        const bool ends = valid && !cont;
        if (__any_sync(FULL, ends)) add_camera_rays(ends ? a.accum + pixel : nullptr, left, skyContrib, a.passes > 1, lane);
    }
}

// Bounce kernel of the next-event-estimation integrator
// (render/diffuse2_integrator_single.h:41-90, render/diffuse2_renderer_cuda.cu:63-239).
// A lane takes a path's extension ray; at a hit before maxDepth it samples a
// shadow direction and an extension direction from the same frame, traces the
// shadow ray for any occluder in the same lane (+0.5 * throughput * sky if it
// escapes), then appends the extension ray with its gathered radiance.  An
// escaping extension ray adds throughput * sky weighted 1 from the camera and
// 0.5 after a bounce.  Shadow rays are counted as rays.
template <bool kFirst, bool kAlbedo>
__global__ void __launch_bounds__(128, kWideBlocks) k_bounce_nee(WaveArgs a, int depth)
{
    extern __shared__ uint2 s_stack[];
    TravStack st;
    st.sh = s_stack + threadIdx.x;
    st.stride = blockDim.x;
    st.overflow = false;
    const int bd = blockDim.x;
    uint32_t* shw = reinterpret_cast<uint32_t*>(s_stack + kShared * blockDim.x) + threadIdx.x;   // as in k_bounce
    TriQueue* tq = reinterpret_cast<TriQueue*>(reinterpret_cast<uint32_t*>(s_stack + kShared * blockDim.x) +
                                               bounce_words(kFirst) * blockDim.x) + (threadIdx.x >> 5);   // deferTris
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned ltMask = (1u << lane) - 1u;
    const int W = a.cam.width, H = a.cam.height;
    const int perPass = a.tilesX * a.tilesY * 64;
    int total;
    int pass0 = 0;
    if (kFirst)
    {
        total = a.passes * perPass;
        pass0 = *a.passBase + a.passOffset;
    }
    else
    {
        total = *(volatile int*)&a.counts[depth];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(a.rays, kFirst ? (unsigned long long)a.passes * (unsigned long long)W * (unsigned long long)H
                                 : (unsigned long long)total);
    const bool final = depth == a.maxDepth;
    const float missWeight = depth > 0 ? 0.5f : 1.0f;

    bool has = false, exhausted = false, shadow = false;
    int qi = 0;               // input-queue index of this lane's path (PRT_RELOAD_PATH)
    int slot = 0;             // output-queue slot of the extension ray while its shadow ray is traced
    float thr = 0.f, L = 0.f;
    unsigned long long shadowRays = 0;
    TravRay r;
    TravState ts;
    ts.done = true;
    for (;;)
    {
        unsigned idle = __ballot_sync(FULL, !has);
        if (!exhausted && (__popc(idle) >= kRefillMin || idle == FULL))
        {
            int n = __popc(idle);
            int base = 0;
            if (lane == 0) base = atomicAdd(&a.fetch[depth], n);
            base = __shfl_sync(FULL, base, 0);
            if (base + n >= total) exhausted = true;
            int i = base + __popc(idle & ltMask);
            if (!has && i < total)
            {
                float3 org, dir;
                int pixel = 0;
                uint32_t rng = 0;
                bool ok = true;
                if (kFirst)
                {
                    int pass, item;
                    wave_item(i, a.passes, pass, item);
                    int x, y;
                    if (!wave_item_pixel(item, a.tilesX, W, H, x, y))
                    {
                        ok = false;
                    }
                    else
                    {
                        pixel = x + y * W;
                        rng = rng_seed(pass0 + pass, pixel);
                        camera_ray(a.cam, x, y, rng, org, dir);
                        thr = kAlbedo ? 1.0f : a.thrConst;
                        L = 0.0f;
                    }
                }
                else if (PRT_RELOAD_PATH)
                {
                    // pixel, RNG state and direction are read again when the lane shades
                    const float4* p = reinterpret_cast<const float4*>(a.qin + i);
                    const float4 w0 = __ldcg(p), w1 = __ldcg(p + 1);
                    org = f3(w0.x, w0.y, w0.z);
                    dir = f3(w1.x, w1.y, w1.z);
                    qi = i;
                    thr = kAlbedo ? __ldcs(a.thrIn + i) : a.thrConst;
                    L = __ldcs(a.Lin + i);
                }
                else
                {
                    PathRec pr = load_path(a.qin, i);
                    org = f3(pr.w0.x, pr.w0.y, pr.w0.z);
                    pixel = __float_as_int(pr.w0.w);
                    dir = f3(pr.w1.x, pr.w1.y, pr.w1.z);
                    rng = __float_as_uint(pr.w1.w);
                    thr = kAlbedo ? __ldcs(a.thrIn + i) : a.thrConst;
                    L = __ldcs(a.Lin + i);
                }
                if (ok)
                {
                    has = true;
                    shadow = false;
                    if (kFirst || !PRT_RELOAD_PATH)
                    {
                        shw[4 * bd] = (uint32_t)pixel;
                        shw[5 * bd] = rng;
                        shw[6 * bd] = __float_as_uint(dir.x);
                        shw[7 * bd] = __float_as_uint(dir.y);
                        shw[8 * bd] = __float_as_uint(dir.z);
                    }
                    shear_store(shw, bd, shear_of(dir));
                    trav_setup(r, org, dir);
                    trav_init(ts, a.scene, FLT_MAX, st);
                }
            }
        }
        if (__ballot_sync(FULL, has) == 0)
        {
            if (exhausted) break;
            continue;
        }
        if (PRT_DEFER_NEE && a.scene.deferTris)
        {
            // extension rays (closest hit) and shadow rays (any hit) share the queue
            constexpr bool kPair = !kFirst && PRT_RELOAD_PATH && PRT_PAIRED_NEE;
            warp_trav_deferred<kPair>(*tq, ts, a.scene, r, shw, bd, 0.0f, st, has, true, kRefillMin, lane, nullptr, nullptr,
                                      nullptr, nullptr, nullptr, shadow);
        }
        else
        {
            const Shear sh = shear_load(shw, bd);
            for (;;)
            {
                if (has && !ts.done) trav_step<false>(ts, a.scene, r, sh, 0.0f, st, nullptr, nullptr, shadow);
                unsigned running = __ballot_sync(FULL, has && !ts.done);
                if (running == 0) break;
                if (32 - __popc(running) >= kRefillMin) break;
            }
        }
        // Extension-ray lanes that hit sample their shadow and extension rays,
        // append the extension ray at once and keep only its queue slot while
        // the shadow ray is traced; the radiance gathered so far is written to
        // that slot when the shadow ray finishes.  Values of a finished path
        // are iteration-local, so nothing else is carried around the loop.
        const bool finExt = has && ts.done && !shadow;
        const bool finShadow = has && ts.done && shadow;
        bool spawn = false, end = false;
        int fpix = 0;
        uint32_t frng = 0;
        float3 so = f3(0.f, 0.f, 0.f), sd = f3(0.f, 0.f, 1.f), eo = so, ed = sd;
        if (finExt)
        {
            float3 fdir;
            if (!kFirst && PRT_RELOAD_PATH)
            {
                const float4* p = reinterpret_cast<const float4*>(a.qin + qi);
                const float4 w1 = __ldcs(p + 1);
                fpix = __float_as_int(__ldcs(reinterpret_cast<const float*>(p) + 3));
                fdir = f3(w1.x, w1.y, w1.z);
                frng = __float_as_uint(w1.w);
            }
            else
            {
                fpix = (int)shw[4 * bd];
                frng = shw[5 * bd];
                fdir = f3(__uint_as_float(shw[6 * bd]), __uint_as_float(shw[7 * bd]), __uint_as_float(shw[8 * bd]));
            }
            if (ts.triHit < 0)
            {
                L = __fadd_rn(L, __fmul_rn(__fmul_rn(thr, a.sky), missWeight));
                end = true;
            }
            else if (final)
            {
                end = true;
            }
            else
            {
                if (kAlbedo)
                    thr = __fmul_rn(thr, a.scene.albedo ? __ldg(a.scene.albedo + ts.primHit) : 0.8f);
                else
                    thr = __fmul_rn(thr, 0.8f);
                HitFrame hf = hit_frame(a.scene.tris, ts.triHit, r.org, fdir, ts.tHit);
                sample_bounce(hf, frng, so, sd);   // shadow ray
                sample_bounce(hf, frng, eo, ed);   // extension ray
                spawn = true;
            }
        }
        const int o = warp_append(spawn, &a.counts[depth + 1]);
        if (spawn)
        {
            store_path(a.qout, o, eo, fpix, ed, frng);
            if (kAlbedo) __stcs(a.thrOut + o, thr);
            slot = o;
            shear_store(shw, bd, shear_of(sd));
            trav_setup(r, so, sd);
            trav_init(ts, a.scene, FLT_MAX, st);
            shadow = true;
            ++shadowRays;
        }
        else if (end)
        {
            red_add_v4(a.accum + fpix, L, L, L, 1.0f);
            has = false;
        }
        if (finShadow)
        {
            if (ts.triHit < 0) L = __fadd_rn(L, __fmul_rn(__fmul_rn(thr, a.sky), 0.5f));
            __stcs(a.Lout + slot, L);
            has = false;
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) shadowRays += __shfl_down_sync(FULL, shadowRays, off);
    if (lane == 0 && shadowRays) atomicAdd(a.rays, shadowRays);
}

// A whole wave of the next-event-estimation integrator, from the camera rays on,
// as k_paths<kPrimary>: at a hit before maxDepth a
// lane samples its shadow and extension rays from the same frame, traces the
// shadow ray first (any hit; +0.5 * throughput * sky if it escapes) while the
// extension ray waits in shared memory, then the extension ray.  Camera rays are a
// small part of this integrator's rays, so starting them here wins at every size:
// against a first launch that queued the paths (k_bounce_nee), terrain 256x256 1
// pass 0.76 -> 0.64 ms, 1001x563 16 passes 11.92 -> 11.54, 1080p 32 passes 86.5 -> 82.6.
// pixel, depth | shadow << 8, RNG, throughput, radiance, direction, extension origin, shear terms
constexpr int kNeeWords = 11 + kShearWords;

template <bool kAlbedo>
__global__ void __launch_bounds__(128, kWideBlocks) k_paths_nee(WaveArgs a)
{
    extern __shared__ uint2 s_stack[];
    TravStack st;
    st.sh = s_stack + threadIdx.x;
    st.stride = blockDim.x;
    st.overflow = false;
    uint32_t* s_path = reinterpret_cast<uint32_t*>(s_stack + kShared * blockDim.x);
    uint32_t* path = s_path + threadIdx.x;   // word k of this lane's path at path[k * bd]
    TriQueue* tq = reinterpret_cast<TriQueue*>(s_path + kNeeWords * blockDim.x) + (threadIdx.x >> 5);   // deferTris
    const int bd = blockDim.x;
    uint32_t* shw = path + 11 * bd;
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned ltMask = (1u << lane) - 1u;
    const int perPass = a.tilesX * a.tilesY * 64;
    const int total = a.passes * perPass;
    const int pass0 = *a.passBase + a.passOffset;
    if (blockIdx.x == 0 && threadIdx.x == 0)
        atomicAdd(a.rays, (unsigned long long)a.passes * (unsigned long long)a.cam.width *
                              (unsigned long long)a.cam.height);
    uint32_t more = 0;   // shadow rays and extension rays after the camera's, per warp

    bool has = false, exhausted = false;
    bool shadow = false;      // this lane's ray is a shadow ray
    TravRay r;
    TravState ts;
    ts.done = true;
    for (;;)
    {
        // --- lanes whose ray is traced ---------------------------------------------
        bool fresh = false;   // this lane has a new ray (org, dir)
        float3 org, dir;
        if (has && ts.done)
        {
            const int depth = (int)(path[bd] & 0xffu);
            float thr = __uint_as_float(path[3 * bd]), L = __uint_as_float(path[4 * bd]);
            dir = f3(__uint_as_float(path[5 * bd]), __uint_as_float(path[6 * bd]), __uint_as_float(path[7 * bd]));
            if (shadow)
            {
                if (ts.triHit < 0) L = __fadd_rn(L, __fmul_rn(__fmul_rn(thr, a.sky), 0.5f));
                path[4 * bd] = __float_as_uint(L);
                path[bd] = (uint32_t)(depth + 1);
                org = f3(__uint_as_float(path[8 * bd]), __uint_as_float(path[9 * bd]), __uint_as_float(path[10 * bd]));
                shadow = false;
                fresh = true;
            }
            else if (ts.triHit < 0 || depth == a.maxDepth)
            {
                if (ts.triHit < 0)
                    L = __fadd_rn(L, __fmul_rn(__fmul_rn(thr, a.sky), depth == 0 ? 1.0f : 0.5f));
                red_add_v4(a.accum + path[0], L, L, L, 1.0f);
                has = false;
            }
            else
            {
                thr = __fmul_rn(thr, kAlbedo && a.scene.albedo ? __ldg(a.scene.albedo + ts.primHit) : 0.8f);
                uint32_t rng = path[2 * bd];
                const HitFrame hf = hit_frame(a.scene.tris, ts.triHit, r.org, dir, ts.tHit);
                float3 eo, ed;
                sample_bounce(hf, rng, org, dir);   // shadow ray
                sample_bounce(hf, rng, eo, ed);     // extension ray
                path[bd] = (uint32_t)depth | 0x100u;
                path[2 * bd] = rng;
                path[3 * bd] = __float_as_uint(thr);
                path[5 * bd] = __float_as_uint(ed.x);
                path[6 * bd] = __float_as_uint(ed.y);
                path[7 * bd] = __float_as_uint(ed.z);
                path[8 * bd] = __float_as_uint(eo.x);
                path[9 * bd] = __float_as_uint(eo.y);
                path[10 * bd] = __float_as_uint(eo.z);
                shadow = true;
                fresh = true;
            }
        }
        more += __popc(__ballot_sync(FULL, fresh));
        // --- lanes without a path take the next ones ------------------------------
        const unsigned idle = __ballot_sync(FULL, !has);
        if (!exhausted && idle)
        {
            const int n = __popc(idle);
            int base = 0;
            if (lane == 0) base = atomicAdd(&a.fetch[0], n);
            base = __shfl_sync(FULL, base, 0);
            exhausted = base + n >= total;
            const int i = base + __popc(idle & ltMask);
            if (!has && i < total)
            {
                int pass, item;
                wave_item(i, a.passes, pass, item);
                int x, y;
                if (wave_item_pixel(item, a.tilesX, a.cam.width, a.cam.height, x, y))
                {
                    const int pixel = x + y * a.cam.width;
                    uint32_t rng = rng_seed(pass0 + pass, pixel);
                    camera_ray(a.cam, x, y, rng, org, dir);
                    path[0] = (uint32_t)pixel;
                    path[bd] = 0u;
                    path[2 * bd] = rng;
                    path[3 * bd] = __float_as_uint(1.0f);
                    path[4 * bd] = 0u;
                    path[5 * bd] = __float_as_uint(dir.x);
                    path[6 * bd] = __float_as_uint(dir.y);
                    path[7 * bd] = __float_as_uint(dir.z);
                    shadow = false;
                    has = fresh = true;
                }
            }
        }
        const unsigned act = __ballot_sync(FULL, has);
        if (act == 0)
        {
            if (exhausted) break;
            continue;   // a tile's items outside the frame
        }
        if (fresh)
        {
            shear_store(shw, bd, shear_of(dir));
            trav_setup(r, org, dir);
            trav_init(ts, a.scene, FLT_MAX, st);
        }
        // --- traverse until enough of the warp's rays are done ---------------------
        const int stopIdle = stop_idle(act);
        if (PRT_DEFER_NEE && a.scene.deferTris)
        {
            warp_trav_deferred<PRT_PAIRED_NEE>(*tq, ts, a.scene, r, shw, bd, 0.0f, st, has, true, stopIdle, lane, nullptr, nullptr,
                                               nullptr, nullptr, nullptr, shadow);
        }
        else
        {
            const Shear sh = shear_load(shw, bd);
            for (;;)
            {
                if (has && !ts.done) trav_step<false>(ts, a.scene, r, sh, 0.0f, st, nullptr, nullptr, shadow);
                const unsigned running = __ballot_sync(FULL, has && !ts.done);
                if (32 - __popc(running) >= stopIdle) break;
            }
        }
    }
    if (lane == 0 && more) atomicAdd(a.rays, (unsigned long long)more);
}

// The IntersectorStreamCuda seam (core/intersector_stream_cuda.h:32-33):
// closest or any hit for n ray records.  Persistent warps with the same
// dynamic per-lane refill as k_bounce: a lane whose query is complete writes
// its hit record, and once kQueryRefill lanes of the warp are free they claim
// the next rays from the call's work counter, so incoherent queries of very
// different lengths keep the warp's lanes busy.
// Idle lanes at which the query kernel refills: writing a hit costs less than a
// bounce (4M incoherent closest-hit queries 1.277 ms; 1.305 with 14).
constexpr int kQueryRefill = 12;

template <bool kAnyHit>
__global__ void __launch_bounds__(128, kAnyHit ? PRT_BOUNCE_MIN_BLOCKS : kWideBlocks) k_intersect(SceneDev sc, const RayRec* __restrict__ rays,
                                                                         HitRec* __restrict__ hits,
                                                                         float* __restrict__ anyOut, int n, int* fetch)
{
    extern __shared__ uint2 s_stack[];
    TravStack st;
    st.sh = s_stack + threadIdx.x;
    st.stride = blockDim.x;
    st.overflow = false;
    // the block's stack columns, its lanes' shear terms and, deferTris, the warps'
    // triangle queues, then (closest hit) their barycentrics
    const int bd = blockDim.x;
    uint32_t* s_words = reinterpret_cast<uint32_t*>(s_stack + kShared * blockDim.x);
    uint32_t* shw = s_words + threadIdx.x;
    TriQueue* s_queues = reinterpret_cast<TriQueue*>(s_words + kShearWords * blockDim.x);
    TriQueue* tq = s_queues + (threadIdx.x >> 5);
    TriQueueUV* tuv = reinterpret_cast<TriQueueUV*>(s_queues + (blockDim.x >> 5)) + (threadIdx.x >> 5);
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned ltMask = (1u << lane) - 1u;
    bool has = false, exhausted = false;
    int idx = 0;
    float tnear = 0.f;
    TravRay r;
    TravState ts;
    ts.done = true;
    for (;;)
    {
        unsigned idle = __ballot_sync(FULL, !has);
        if (!exhausted && (__popc(idle) >= kQueryRefill || idle == FULL))
        {
            int cnt = __popc(idle);
            int base = 0;
            if (lane == 0) base = atomicAdd(fetch, cnt);
            base = __shfl_sync(FULL, base, 0);
            if (base + cnt >= n) exhausted = true;
            int i = base + __popc(idle & ltMask);
            if (!has && i < n)
            {
                const float4* rp = reinterpret_cast<const float4*>(rays + i);
                float4 a = __ldcs(rp), b = __ldcs(rp + 1);
                const float3 dir = f3(b.x, b.y, b.z);
                shear_store(shw, bd, shear_of(dir));
                trav_setup(r, f3(a.x, a.y, a.z), dir);
                trav_init(ts, sc, b.w, st);
                tnear = a.w;
                idx = i;
                has = true;
            }
        }
        if (__ballot_sync(FULL, has) == 0)
        {
            if (exhausted) break;
            continue;
        }
        if (PRT_DEFER_ISECT && sc.deferTris)
        {
            constexpr bool kPair = kAnyHit && PRT_PAIRED_QUERY;
            warp_trav_deferred<kPair, !kAnyHit, true>(*tq, ts, sc, r, shw, bd, tnear, st, has, !exhausted, kQueryRefill, lane, nullptr,
                                                nullptr, nullptr, nullptr, nullptr, kAnyHit, tuv);
        }
        else
        {
            const Shear sh = shear_load(shw, bd);
            for (;;)
            {
                if (has && !ts.done) trav_step<kAnyHit>(ts, sc, r, sh, tnear, st);
                unsigned running = __ballot_sync(FULL, has && !ts.done);
                if (running == 0) break;
                if (!exhausted && 32 - __popc(running) >= kQueryRefill) break;
            }
        }
        if (has && ts.done)
        {
            const bool hit = ts.triHit >= 0;
            if (kAnyHit)
                __stcs(anyOut + idx, hit ? ts.tHit : -1.0f);
            else
                __stcs(reinterpret_cast<float4*>(hits) + idx,
                       hit ? make_float4(ts.tHit, __int_as_float(ts.primHit), ts.uHit, ts.vHit)
                           : make_float4(-1.0f, __int_as_float(-1), 0.f, 0.f));
            has = false;
        }
    }
}

// Closest or any hit of one ray by a group of 8 lanes, lane j testing child j of
// the node the ray is at and the triangles of that child if it is a leaf (trees
// of any leaf size).  Every lane of the group holds the ray and the traversal
// state; stk: the group's kPacketStack entries of shared memory.  behind: hits at
// negative t count too (a ray may begin behind its origin).  Returns the
// leaf-order index of the hit triangle, or -1, in every lane.
template <bool kAnyHit>
__device__ __forceinline__ int group_trace(const SceneDev& sc, const TravRay& r, const Shear& sh, float tnear, bool behind,
                                           uint2* stk, unsigned lane, float& tHit, int& primHit, float& uHit, float& vHit)
{
    const int j = (int)(lane & 7u);
    const unsigned gshift = lane & 24u, gmask = 0xffu << gshift;
    int triHit = -1;
    if (!sc.hasRoot) return -1;
    // byte offsets of this lane's near and far planes in a node
    const int nX = (r.inv.x < 0.f ? 56 : 32) + j, fX = (r.inv.x < 0.f ? 32 : 56) + j;
    const int nY = (r.inv.y < 0.f ? 64 : 40) + j, fY = (r.inv.y < 0.f ? 40 : 64) + j;
    const int nZ = (r.inv.z < 0.f ? 72 : 48) + j, fZ = (r.inv.z < 0.f ? 48 : 72) + j;
    int sp = 0;
    uint2 ng = make_uint2(0u, 0x80000000u);   // the root: one internal child at base 0
    for (;;)
    {
        const uint32_t nodeIdx = next_child(ng, r.oct);
        if ((ng.y & 0xff000000u) && sp < kPacketStack)
        {
            if (j == 0) stk[sp] = ng;
            ++sp;
        }
        const uint4* qp = reinterpret_cast<const uint4*>(sc.nodes + nodeIdx);
        const unsigned char* bp = reinterpret_cast<const unsigned char*>(qp);
        const uint4 q0 = __ldg(qp), q1 = __ldg(qp + 1);
        const uint32_t bnX = __ldg(bp + nX), bfX = __ldg(bp + fX), bnY = __ldg(bp + nY), bfY = __ldg(bp + fY),
                       bnZ = __ldg(bp + nZ), bfZ = __ldg(bp + fZ);
        // this child's slab test, as node_hits does it
        const uint32_t e = q0.w;
        const float aix = __uint_as_float(((e & 0xffu) + 15u) << 23) * r.inv.x;
        const float aiy = __uint_as_float((((e >> 8) & 0xffu) + 15u) << 23) * r.inv.y;
        const float aiz = __uint_as_float((((e >> 16) & 0xffu) + 15u) << 23) * r.inv.z;
        const float aox = (__uint_as_float(q0.x) - r.org.x) * r.inv.x - aix;
        const float aoy = (__uint_as_float(q0.y) - r.org.y) * r.inv.y - aiy;
        const float aoz = (__uint_as_float(q0.z) - r.org.z) * r.inv.z - aiz;
        const float t0 = fmax3(fmaf(byte_unit(bnX, 0), aix, aox), fmaf(byte_unit(bnY, 0), aiy, aoy),
                               fmaxf(fmaf(byte_unit(bnZ, 0), aiz, aoz), tnear));
        const float t1 = fmin3(fmaf(byte_unit(bfX, 0), aix, aox), fmaf(byte_unit(bfY, 0), aiy, aoy),
                               fminf(fmaf(byte_unit(bfZ, 0), aiz, aoz), tHit * 1.0000004f));
        const uint32_t meta = ((j < 4 ? q1.z : q1.w) >> (8 * (j & 3))) & 0xffu;
        const bool hit = meta != 0 && t0 <= t1 * 1.0000008f;
        const uint32_t imask = e >> 24;
        const uint32_t c8 = (__ballot_sync(gmask, hit) >> gshift) & 0xffu;
        if (c8 & ~imask)
        {
            // the hit leaves' triangles, each lane its own; the group keeps the
            // nearest (ties to the lower primitive id)
            unsigned long long key = signed_hit_key(tHit, primHit);
            const unsigned long long before = key;
            float u = 0.f, v = 0.f;
            int ti = 0;
            if (hit && !((imask >> j) & 1u))
            {
                float tb = tHit;
                int pb = primHit;
                for (uint32_t k = 0; k < (uint32_t)__popc(meta >> 5); ++k)
                {
                    const int idx = (int)(q1.y + (meta & 0x1fu) + k);
                    const float4* tp = reinterpret_cast<const float4*>(sc.tris + idx);
                    const float4 v0 = __ldg(tp), v1 = __ldg(tp + 1), v2 = __ldg(tp + 2);
                    const int prim = __float_as_int(v0.w);
                    float t, uu, vv;
                    if (tri_test(r.org, sh, f3(v0.x, v0.y, v0.z), f3(v1.x, v1.y, v1.z), f3(v2.x, v2.y, v2.z), tnear, tb, prim,
                                 pb, t, uu, vv))
                    {
                        if (!behind && __float_as_int(t) < 0) continue;
                        tb = t;
                        pb = prim;
                        u = uu;
                        v = vv;
                        ti = idx;
                        key = signed_hit_key(t, prim);
                    }
                }
            }
            const unsigned long long mine = key;
#pragma unroll
            for (int off = 1; off < 8; off <<= 1)
            {
                const unsigned long long o = __shfl_xor_sync(gmask, key, off);
                key = o < key ? o : key;
            }
            if (key != before)
            {
                const int win = __ffs(__ballot_sync(gmask, mine == key)) - 1;
                tHit = signed_key_t(key);
                primHit = (int)(uint32_t)key;
                uHit = __shfl_sync(gmask, u, win);
                vHit = __shfl_sync(gmask, v, win);
                triHit = __shfl_sync(gmask, ti, win);
                if (kAnyHit) return triHit;
            }
        }
        // internal hits: bit slot -> bit slot ^ octinv, as node_hits1 orders them
        const uint32_t in8 = permute_octant(c8 & imask, r.oct);
        ng = make_uint2(q1.x, (in8 << 24) | imask);
        if (!(ng.y & 0xff000000u))
        {
            if (sp == 0) return triHit;
            __syncwarp(gmask);
            ng = stk[--sp];
            __syncwarp(gmask);
        }
    }
}

// Few rays: a group of 8 lanes per ray.  One lane per ray leaves the chip idle
// while the longest ray's chain of node visits runs, each some 300 dependent
// instructions and a cache miss; eight lanes cut a visit to about a fifth of
// that.  perWarp (1, 2 or 4) rays share a warp.  As with many rays, hits at
// negative t count where triangles are tested in the lane and not where the
// tests are deferred.
template <bool kAnyHit>
__global__ void __launch_bounds__(128) k_intersect_few(SceneDev sc, const RayRec* __restrict__ rays,
                                                     HitRec* __restrict__ hits, float* __restrict__ anyOut, int n,
                                                     int perWarp)
{
    __shared__ uint2 s_stk[16 * kPacketStack];
    const unsigned lane = threadIdx.x & 31u;
    const int group = (int)(lane >> 3);
    const long long i = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * perWarp + group;
    if (group >= perWarp || i >= n) return;
    const float4* rp = reinterpret_cast<const float4*>(rays + i);
    const float4 a = __ldg(rp), b = __ldg(rp + 1);
    TravRay r;
    const float3 dir = f3(b.x, b.y, b.z);
    trav_setup(r, f3(a.x, a.y, a.z), dir);
    float t = b.w, u = 0.f, v = 0.f;
    int prim = 0x7fffffff;
    const int tri = group_trace<kAnyHit>(sc, r, shear_of(dir), a.w, !sc.deferTris, s_stk + (threadIdx.x >> 3) * kPacketStack, lane, t,
                                          prim, u, v);
    if ((lane & 7u) != 0) return;
    if (kAnyHit) anyOut[i] = tri >= 0 ? t : -1.0f;
    else reinterpret_cast<float4*>(hits)[i] = tri >= 0 ? make_float4(t, __int_as_float(prim), u, v)
                                                       : make_float4(-1.0f, __int_as_float(-1), 0.f, 0.f);
}

// Hit point and geometric normal of one query ray (Renderer::queryRay), by one
// group of 8 lanes.
__global__ void k_query(SceneDev sc, const RayRec* ray, HitRec* hit, float* pNg)
{
    __shared__ uint2 s_stk[kPacketStack];
    const RayRec rr = *ray;
    TravRay r;
    const float3 dir = f3(rr.dx, rr.dy, rr.dz);
    trav_setup(r, f3(rr.ox, rr.oy, rr.oz), dir);
    float t = rr.tfar, u = 0.f, v = 0.f;
    int prim = 0x7fffffff;
    const int ti = group_trace<false>(sc, r, shear_of(dir), rr.tnear, true, s_stk, threadIdx.x, t, prim, u, v);
    if (threadIdx.x != 0) return;
    if (ti < 0)
    {
        *hit = HitRec{-1.0f, -1, 0.f, 0.f};
        return;
    }
    *hit = HitRec{t, prim, u, v};
    float3 p = madd(r.org, t, dir);
    const TriRec tr = sc.tris[ti];
    float3 p0 = f3(tr.v0.x, tr.v0.y, tr.v0.z), p1 = f3(tr.v1.x, tr.v1.y, tr.v1.z), p2 = f3(tr.v2.x, tr.v2.y, tr.v2.z);
    float3 Ng = normalize(cross(sub(p1, p0), sub(p2, p0)));
    if (dot(Ng, dir) > 0.0f) Ng = f3(-Ng.x, -Ng.y, -Ng.z);
    pNg[0] = p.x; pNg[1] = p.y; pNg[2] = p.z;
    pNg[3] = Ng.x; pNg[4] = Ng.y; pNg[5] = Ng.z;
}

// Gamma-2.2 BGRA8 resolve (image/accum_buffer_cuda.cu:22-37; channel order of
// encodeBgr8, image/pixel.h:42-46).
__global__ void k_resolve_ldr(const float4* __restrict__ accum, uint32_t* __restrict__ out, int n)
{
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 a = accum[i];
    float w = a.w > 0.f ? 1.0f / a.w : 0.0f;
    const float g = 1.0f / 2.2f;
    int r = min(max((int)(powf(a.x * w, g) * 255.0f), 0), 255);
    int gg = min(max((int)(powf(a.y * w, g) * 255.0f), 0), 255);
    int b = min(max((int)(powf(a.z * w, g) * 255.0f), 0), 255);
    out[i] = (uint32_t)b | ((uint32_t)gg << 8) | ((uint32_t)r << 16);
}

// Start of a render call: its first pass is the next one (pass[1]), the call
// after it begins spp later; the ray count and the wave counters start at 0.
__global__ void k_begin_render(int* pass, int spp, unsigned long long* rays, int* counters, int words)
{
    if (threadIdx.x == 0)
    {
        pass[0] = pass[1];
        pass[1] += spp;
        *rays = 0;
    }
    for (int i = threadIdx.x; i < words; i += blockDim.x) counters[i] = 0;
}

constexpr int kReplayMaxDepth = 16;
constexpr int kAggSlots = 256;             // block-private gradient slots of the adjoint
// words per lane: pixel, depth, RNG, throughput, direction (as k_paths), shear terms;
// backward: and dL/d(radiance) of the pixel, this lane's sky gradient
constexpr int kReplayWords = 7 + kShearWords;
constexpr int kBackwardWords = kReplayWords + 2;

// Path-replay megakernel: each lane carries whole paths (pass, pixel), from
// the camera ray to escape or maxDepth.  The forward mode accumulates the
// path's radiance; the backward mode re-traces the same path from its seed
// and scatters dL/d(radiance) into the albedo of every triangle the path
// bounced off and into the sky radiance:
//   radiance = sky * prod_k albedo[prim_k]
//   d radiance / d albedo[prim_k] = radiance / albedo[prim_k]
//   d radiance / d sky            = prod_k albedo[prim_k]
// Paths bounce in their lane and are replaced when they end, with the path's
// state in shared memory, as in k_paths.  The bounce arithmetic is the same
// device code as the wavefront renderer's, so both compute bit-identical paths.
// Both modes defer triangle tests and test nodes with paired FMAs; the backward
// mode affords the queues with 256 gradient slots (1024: 6% slower for the shared
// memory).  Traversal latency and issue bound it, as k_paths.  512x512, 16
// passes, 82K triangles: forward 1.94 -> 1.67 ms, backward 2.29 -> 1.95 ms against
// lanes that kept the path in registers, refilled at 12 idle lanes only and (in
// the backward mode) tested triangles in the lane.
template <bool kBackward>
__global__ void __launch_bounds__(128, kWideBlocks) k_replay(SceneDev sc, CameraDev cam, float4* accum, int pass0, int spp,
                                                   int maxDepth, float sky, const float* __restrict__ dL,
                                                   float* dAlbedo, float* dSky, unsigned long long* rays,
                                                   int* fetch)
{
    extern __shared__ uint2 s_stack[];
    // Block-private accumulation of albedo gradients: a few triangles (a
    // ground plane) receive most of the contributions, so per-path global
    // atomics would serialise on them.  Slot = prim mod kAggSlots; a slot
    // holds one triangle, collisions go straight to global memory.
    __shared__ int s_key[kBackward ? kAggSlots : 1];
    __shared__ float s_val[kBackward ? kAggSlots : 1];
    if (kBackward)
    {
        for (int i = threadIdx.x; i < kAggSlots; i += blockDim.x)
        {
            s_key[i] = -1;
            s_val[i] = 0.f;
        }
        __syncthreads();
    }
    TravStack st;
    st.sh = s_stack + threadIdx.x;
    st.stride = blockDim.x;
    st.overflow = false;
    constexpr int kWords = kBackward ? kBackwardWords : kReplayWords;
    uint32_t* s_path = reinterpret_cast<uint32_t*>(s_stack + kShared * blockDim.x);
    uint32_t* path = s_path + threadIdx.x;   // word k of this lane's path at path[k * bd]
    TriQueue* tq = reinterpret_cast<TriQueue*>(s_path + kWords * blockDim.x) + (threadIdx.x >> 5);   // deferTris
    const int bd = blockDim.x;
    uint32_t* shw = path + 7 * bd;
    uint32_t* grad = path + kReplayWords * bd;   // kBackward
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned ltMask = (1u << lane) - 1u;
    const int W = cam.width;
    const long long npix = (long long)W * cam.height;
    const long long total = (long long)spp * npix;
    if (kBackward) grad[bd] = 0u;   // sky gradient 0
    uint32_t traced = 0;      // rays, per warp

    bool has = false, exhausted = false;
    int prims[kBackward ? kReplayMaxDepth : 1];   // the triangles the path bounced off
    TravRay r;
    TravState ts;
    ts.done = true;
    for (;;)
    {
        // --- lanes whose ray is traced: the path ends or bounces -----------------
        bool fresh = false;   // this lane has a new ray (org, dir)
        float3 org, dir;
        traced += __popc(__ballot_sync(FULL, has && ts.done));
        if (has && ts.done)
        {
            const int depth = (int)path[bd];
            float thr = __uint_as_float(path[3 * bd]);
            const bool escaped = ts.triHit < 0;
            if (!escaped && depth < maxDepth)
            {
                uint32_t rng = path[2 * bd];
                org = r.org;
                dir = f3(__uint_as_float(path[4 * bd]), __uint_as_float(path[5 * bd]), __uint_as_float(path[6 * bd]));
                thr = __fmul_rn(thr, sc.albedo ? __ldg(sc.albedo + ts.primHit) : 0.8f);
                if (kBackward) prims[depth] = ts.primHit;
                diffuse_bounce(sc.tris, ts.triHit, org, dir, ts.tHit, rng);
                path[bd] = (uint32_t)(depth + 1);
                path[2 * bd] = rng;
                path[3 * bd] = __float_as_uint(thr);
                fresh = true;
            }
            else
            {
                const float c = escaped ? __fmul_rn(thr, sky) : 0.0f;
                if (!kBackward)
                {
                    red_add_v4(accum + path[0], c, c, c, 1.0f);
                }
                else if (escaped)
                {
                    const float g = __uint_as_float(grad[0]);
                    grad[bd] = __float_as_uint(__uint_as_float(grad[bd]) + g * thr);
                    const float gc = g * c;
                    for (int k = 0; k < depth; ++k)
                    {
                        const int pk = prims[k];
                        const float al = sc.albedo ? __ldg(sc.albedo + pk) : 0.8f;
                        const float v = gc / al;
                        const int slot = pk & (kAggSlots - 1);
                        int key = s_key[slot];
                        if (key == -1) key = atomicCAS(&s_key[slot], -1, pk);   // -1: claimed by us
                        if (key == -1 || key == pk) atomicAdd(&s_val[slot], v);
                        else atomicAdd(dAlbedo + pk, v);
                    }
                }
                has = false;
            }
        }
        // --- lanes without a path take the next ones ------------------------------
        const unsigned idle = __ballot_sync(FULL, !has);
        if (!exhausted && idle)
        {
            const int n = __popc(idle);
            long long base = 0;
            if (lane == 0) base = (long long)atomicAdd(reinterpret_cast<unsigned long long*>(fetch), (unsigned long long)n);
            base = __shfl_sync(FULL, base, 0);
            exhausted = base + n >= total;
            const long long gi = base + __popc(idle & ltMask);
            if (!has && gi < total)
            {
                int pass, pixel;
                wave_item(gi, spp, pass, pixel);
                float g = 1.f;
                if (kBackward)
                {
                    g = dL[3 * (size_t)pixel] + dL[3 * (size_t)pixel + 1] + dL[3 * (size_t)pixel + 2];
                    grad[0] = __float_as_uint(g);
                }
                if (g != 0.f)   // a pixel without a gradient has nothing to replay
                {
                    uint32_t rng = rng_seed(pass0 + pass, pixel);
                    camera_ray(cam, pixel % W, pixel / W, rng, org, dir);
                    path[0] = (uint32_t)pixel;
                    path[bd] = 0u;
                    path[2 * bd] = rng;
                    path[3 * bd] = __float_as_uint(1.0f);
                    has = fresh = true;
                }
            }
        }
        const unsigned act = __ballot_sync(FULL, has);
        if (act == 0)
        {
            if (exhausted) break;
            continue;
        }
        if (fresh)
        {
            path[4 * bd] = __float_as_uint(dir.x);
            path[5 * bd] = __float_as_uint(dir.y);
            path[6 * bd] = __float_as_uint(dir.z);
            shear_store(shw, bd, shear_of(dir));
            trav_setup(r, org, dir);
            trav_init(ts, sc, FLT_MAX, st);
        }
        // --- traverse until enough of the warp's rays are done ---------------------
        const int stopIdle = stop_idle(act);
        if (PRT_DEFER_REPLAY && sc.deferTris)
        {
            warp_trav_deferred<PRT_PAIRED_LATER>(*tq, ts, sc, r, shw, bd, 0.0f, st, has, true, stopIdle, lane);
        }
        else
        {
            const Shear sh = shear_load(shw, bd);
            for (;;)
            {
                if (has && !ts.done) trav_step<false>(ts, sc, r, sh, 0.0f, st);
                const unsigned running = __ballot_sync(FULL, has && !ts.done);
                if (32 - __popc(running) >= stopIdle) break;
            }
        }
    }
    if (kBackward)
    {
        float skyGrad = __uint_as_float(grad[bd]);
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) skyGrad += __shfl_down_sync(FULL, skyGrad, off);
        if (lane == 0 && skyGrad != 0.f) atomicAdd(dSky, skyGrad);
    }
    if (lane == 0 && rays) atomicAdd(rays, (unsigned long long)traced);
    if (kBackward)
    {
        __syncthreads();
        for (int i = threadIdx.x; i < kAggSlots; i += blockDim.x)
            if (s_key[i] >= 0) atomicAdd(dAlbedo + s_key[i], s_val[i]);
    }
}

// First bounce of the batched renderer: the paths of many requests share one
// queue.  Item i of a wave is a global path index resolved to (request, pass,
// tile, Morton index) by a binary search over the requests' path ranges; the
// queued path records carry (request << 24 | pixel).  Lanes refill dynamically
// as in k_bounce; k_paths takes the queue.
__global__ void __launch_bounds__(128, kWideBlocks) k_batch_first(BatchArgs a)
{
    extern __shared__ uint2 s_dyn[];
    uint2* s_stack = s_dyn;
    long long* s_begin = reinterpret_cast<long long*>(s_dyn + kShared * blockDim.x);
    const int bd = blockDim.x;
    // per lane, as in k_bounce: shear terms, pixel, RNG state, direction
    uint32_t* shw = reinterpret_cast<uint32_t*>(s_begin + a.nreq) + threadIdx.x;
    TriQueue* tq = reinterpret_cast<TriQueue*>(reinterpret_cast<uint32_t*>(s_begin + a.nreq) +
                                               bounce_words(true) * blockDim.x) + (threadIdx.x >> 5);   // when a.leaf1
    for (int q = threadIdx.x; q < a.nreq; q += blockDim.x) s_begin[q] = a.reqs[q].pathBegin;
    __syncthreads();
    TravStack st;
    st.sh = s_stack + threadIdx.x;
    st.stride = blockDim.x;
    st.overflow = false;
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned ltMask = (1u << lane) - 1u;
    const long long total = a.waveEnd - a.waveBegin;
    unsigned long long myRays = 0;

    bool has = false;
    bool exhausted = false;
    int req = 0;
    TravRay r;
    TravState ts;
    ts.done = true;
    for (;;)
    {
        unsigned idle = __ballot_sync(FULL, !has);
        if (!exhausted && (__popc(idle) >= kRefillMin || idle == FULL))
        {
            int n = __popc(idle);
            int base = 0;
            if (lane == 0) base = atomicAdd(&a.fetch[0], n);
            base = __shfl_sync(FULL, base, 0);
            if (base + n >= total) exhausted = true;
            int i = base + __popc(idle & ltMask);
            if (!has && i < total)
            {
                float3 org, dir;
                int pixel = 0;
                uint32_t rng = 0;
                bool ok = true;
                long long gi = a.waveBegin + i;
                int lo = 0, hi = a.nreq - 1;
                while (lo < hi)
                {
                    int mid = (lo + hi + 1) >> 1;
                    if (s_begin[mid] <= gi) lo = mid;
                    else hi = mid - 1;
                }
                req = lo;
                const BatchReq& R = a.reqs[req];
                long long local = gi - s_begin[req];
                int pass, item;
                wave_item(local, R.spp, pass, item);
                int x, y;
                if (!wave_item_pixel(item, R.tilesX, R.cam.width,
                                     R.cam.height, x, y))
                {
                    ok = false;
                }
                else
                {
                    pixel = x + y * R.cam.width;
                    rng = rng_seed(pass, pixel);
                    camera_ray(R.cam, x, y, rng, org, dir);
                    ++myRays;
                }
                if (ok)
                {
                    has = true;
                    shw[4 * bd] = (uint32_t)pixel;
                    shw[5 * bd] = rng;
                    shw[6 * bd] = __float_as_uint(dir.x);
                    shw[7 * bd] = __float_as_uint(dir.y);
                    shw[8 * bd] = __float_as_uint(dir.z);
                    shear_store(shw, bd, shear_of(dir));
                    trav_setup(r, org, dir);
                    trav_init(ts, a.reqs[req].scene, FLT_MAX, st);
                }
            }
        }
        if (__ballot_sync(FULL, has) == 0)
        {
            if (exhausted) break;
            continue;
        }
        if (PRT_DEFER_TRIS && a.leaf1)
        {
            warp_trav_deferred(*tq, ts, a.reqs[req].scene, r, shw, bd, 0.0f, st, has, !exhausted, kRefillMin, lane);
        }
        else
        {
            const Shear sh = shear_load(shw, bd);
            for (;;)
            {
                if (has && !ts.done) trav_step<false>(ts, a.reqs[req].scene, r, sh, 0.0f, st);
                unsigned running = __ballot_sync(FULL, has && !ts.done);
                if (running == 0) break;
                if (!exhausted && 32 - __popc(running) >= kRefillMin) break;
            }
        }
        const bool fin = has && ts.done;
        bool cont = false;
        float contrib = 0.f;
        int pixel = 0;
        uint32_t rng = 0;
        float3 forg = r.org, fdir = f3(0.f, 0.f, 0.f);
        if (fin)
        {
            pixel = (int)shw[4 * bd];
            rng = shw[5 * bd];
            fdir = f3(__uint_as_float(shw[6 * bd]), __uint_as_float(shw[7 * bd]), __uint_as_float(shw[8 * bd]));
            const BatchReq& R = a.reqs[req];
            if (ts.triHit < 0)
            {
                contrib = a.sky;   // throughput 1
            }
            else if (R.maxDepth > 0)
            {
                diffuse_bounce(R.scene.tris, ts.triHit, forg, fdir, ts.tHit, rng);
                cont = true;
            }
        }
        int o = warp_append(cont, &a.counts[1]);
        if (cont) store_path(a.qout, o, forg, (req << 24) | pixel, fdir, rng);
        else if (fin) red_add_v4(a.reqs[req].accum + pixel, contrib, contrib, contrib, 1.0f);
        if (fin) has = false;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) myRays += __shfl_down_sync(FULL, myRays, off);
    if (lane == 0 && myRays) atomicAdd(a.rays, myRays);
}

// Depth 0 of the batched renderer as warp packets (k_primary_packet's
// traversal).  The 32 items a warp takes always belong to one request:
// requests own multiples of 64 paths, and the host uses this kernel only when
// waves start at multiples of 32 paths.
template <bool kIA>
__global__ void __launch_bounds__(128, 8) k_batch_primary_packet(BatchArgs a)
{
    extern __shared__ uint2 s_dyn[];
    long long* s_begin = reinterpret_cast<long long*>(s_dyn);
    uint2* stk = reinterpret_cast<uint2*>(s_begin + a.nreq) + (threadIdx.x >> 5) * kPacketStack;
    for (int q = threadIdx.x; q < a.nreq; q += blockDim.x) s_begin[q] = a.reqs[q].pathBegin;
    __syncthreads();
    const unsigned FULL = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31u;
    const long long total = a.waveEnd - a.waveBegin;
    unsigned long long myRays = 0;
    for (;;)
    {
        int base = 0;
        if (lane == 0) base = atomicAdd(&a.fetch[0], 32);
        base = __shfl_sync(FULL, base, 0);
        if (base >= total) break;
        // the warp's request: the one whose path range holds its first item
        const long long g0 = a.waveBegin + base;
        int lo = 0, hi = a.nreq - 1;
        while (lo < hi)
        {
            const int mid = (lo + hi + 1) >> 1;
            if (s_begin[mid] <= g0) lo = mid;
            else hi = mid - 1;
        }
        const int req = lo;
        const BatchReq& R = a.reqs[req];
        bool valid = false;
        int pixel = 0;
        uint32_t rng = 0;
        float3 org = f3(0.f, 0.f, 0.f), dir = f3(0.f, 0.f, 1.f);
        if (base + (long long)lane < total)
        {
            const long long local = g0 + lane - s_begin[req];
            int pass, item;
            wave_item(local, R.spp, pass, item);
            int x, y;
            if (wave_item_pixel(item, R.tilesX, R.cam.width, R.cam.height, x, y))
            {
                valid = true;
                pixel = x + y * R.cam.width;
                rng = rng_seed(pass, pixel);
                camera_ray(R.cam, x, y, rng, org, dir);
                ++myRays;
            }
        }
        const unsigned vmask = __ballot_sync(FULL, valid);
        if (!vmask) continue;
        TravRay r;
        trav_setup(r, org, dir);
        float tHit;
        int primHit, triHit;
        packet_closest_hit<PRT_PAIRED_PACKET, kIA>(R.scene, r, shear_of(dir), valid, vmask, stk, lane, tHit, primHit, triHit);
        bool cont = false;
        const bool left = valid && triHit < 0;
        if (valid && !left && R.maxDepth > 0)
        {
            diffuse_bounce(R.scene.tris, triHit, org, dir, tHit, rng);
            cont = true;
        }
        const int o = warp_append(cont, &a.counts[1]);
        if (cont) store_path(a.qout, o, org, (req << 24) | pixel, dir, rng);
        const bool ends = valid && !cont;
        // throughput 1 at depth 0
        if (__any_sync(FULL, ends)) add_camera_rays(ends ? R.accum + pixel : nullptr, left, a.sky, R.spp > 1, lane);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) myRays += __shfl_down_sync(FULL, myRays, off);
    if (lane == 0 && myRays) atomicAdd(a.rays, myRays);
}

template <class Kernel>
int grid_for(Kernel kernel, int block, size_t shmem, int numSMs, const LaunchCfg& cfg)
{
    int resident = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, block, shmem) != cudaSuccess || resident < 1)
        resident = 1;
    int perSM = cfg.blocksPerSM > 0 ? std::min(cfg.blocksPerSM, resident) : resident;
    return numSMs * perSM;
}

} // namespace

int launch_bounce(const WaveArgs& a, int depth, const LaunchCfg& cfg, int numSMs, cudaStream_t s)
{
    size_t shmem = (sizeof(uint2) * kShared + sizeof(uint32_t) * bounce_words(depth == 0)) * cfg.block;
    if (a.scene.deferTris && (a.Lout ? PRT_DEFER_NEE : PRT_DEFER_TRIS))
        shmem += sizeof(TriQueue) * (cfg.block / 32);   // the bounce kernels' triangle queues
    bool albedo = a.thrIn != nullptr || a.thrOut != nullptr;
    auto go = [&](auto kernel) {
        int grid = grid_for(kernel, cfg.block, shmem, numSMs, cfg);
        kernel<<<grid, cfg.block, shmem, s>>>(a, depth);
    };
    if (a.Lout)
    {
        if (depth == 0)
        {
            if (albedo) go(k_bounce_nee<true, true>);
            else go(k_bounce_nee<true, false>);
        }
        else
        {
            if (albedo) go(k_bounce_nee<false, true>);
            else go(k_bounce_nee<false, false>);
        }
        return 1;
    }
    if (depth == 0 && packet_primaries(a.scene.leafTris, cfg))
    {
        const size_t pshmem = sizeof(uint2) * kPacketStack * (cfg.block / 32);
        auto goPacket = [&](auto kernel) {
            int grid = grid_for(kernel, cfg.block, pshmem, numSMs, cfg);
            kernel<<<grid, cfg.block, pshmem, s>>>(a);
        };
        if (cfg.packet == kPrimaryIntervals)
        {
            if (albedo) goPacket(k_primary_packet<true, true>);
            else goPacket(k_primary_packet<false, true>);
        }
        else
        {
            if (albedo) goPacket(k_primary_packet<true, false>);
            else goPacket(k_primary_packet<false, false>);
        }
        return 1;
    }
    if (depth == 0)
    {
        if (albedo) go(k_bounce<true, true>);
        else go(k_bounce<true, false>);
    }
    else
    {
        if (albedo) go(k_bounce<false, true>);
        else go(k_bounce<false, false>);
    }
    return 1;
}

namespace {

// Paths per SM up to which a wave's primary rays start in k_paths itself.  A
// small wave is mostly tail (the last rays of each launch run on an emptying
// chip) and one tail beats two; a large one loses more by mixing camera rays with
// later bounces, whose neighbours have scattered.  Two launches -> one, 82K / 1.38M
// / 450K triangles: 65K paths 0.29 / 0.46 / 0.28 -> 0.25 / 0.40 / 0.23 ms, 1M paths
// 0.62 / 1.19 / 0.62 -> 0.59 / 1.16 / 0.57, 2.1M 0.93 / 1.93 / 0.95 -> 0.93 / 1.94 / 0.92,
// 4.2M 1.57 / 3.46 / 1.63 -> 1.64 / 3.57 / 1.65.
constexpr int kWholePaths = 10240;

template <class Args, class Kernel>
void run_paths(Kernel kernel, const Args& a, int words, bool deferred, const LaunchCfg& cfg, int numSMs, cudaStream_t s)
{
    size_t shmem = (sizeof(uint2) * kShared + sizeof(uint32_t) * words) * cfg.block;
    if (deferred) shmem += sizeof(TriQueue) * (cfg.block / 32);
    const int grid = grid_for(kernel, cfg.block, shmem, numSMs, cfg);
    kernel<<<grid, cfg.block, shmem, s>>>(a);
}

} // namespace

bool packet_primaries(int leafTris, const LaunchCfg& cfg)
{
    return PRT_PACKET_PRIMARY && (cfg.packet == kPrimaryPackets || cfg.packet == kPrimaryIntervals) && leafTris == 1;
}

bool whole_paths(long long paths, int leafTris, const LaunchCfg& cfg, bool nee, int numSMs)
{
    // primary rays as packets have their own kernel (not with next-event estimation)
    return nee || (!packet_primaries(leafTris, cfg) && paths <= (long long)kWholePaths * numSMs);
}

int launch_whole(const WaveArgs& a, bool albedo, bool nee, const LaunchCfg& cfg, int numSMs, cudaStream_t s)
{
    const bool deferred = (nee ? PRT_DEFER_NEE : PRT_DEFER_TRIS) && a.scene.deferTris;
    auto go = [&](auto kernel, int words) { run_paths(kernel, a, words, deferred, cfg, numSMs, s); };
    if (nee && albedo) go(k_paths_nee<true>, kNeeWords);
    else if (nee) go(k_paths_nee<false>, kNeeWords);
    else if (albedo) go(k_paths<WaveArgs, false, true, true>, kPathWords);
    else go(k_paths<WaveArgs, false, false, true>, kPathWords);
    return 1;
}

int launch_paths(const WaveArgs& a, const LaunchCfg& cfg, int numSMs, cudaStream_t s)
{
    const bool deferred = PRT_DEFER_TRIS && a.scene.deferTris;
    if (a.thrIn) run_paths(k_paths<WaveArgs, false, true, false>, a, kPathWords, deferred, cfg, numSMs, s);
    else run_paths(k_paths<WaveArgs, false, false, false>, a, kPathWords, deferred, cfg, numSMs, s);
    return 1;
}

int launch_batch_paths(const BatchArgs& a, const LaunchCfg& cfg, int numSMs, cudaStream_t s)
{
    run_paths(k_paths<BatchArgs, true, false, false>, a, kPathWords, PRT_DEFER_TRIS && a.leaf1, cfg, numSMs, s);
    return 1;
}

int launch_batch_first(const BatchArgs& a, const LaunchCfg& cfg, int numSMs, cudaStream_t s)
{
    size_t shmem = (sizeof(uint2) * kShared + sizeof(uint32_t) * bounce_words(true)) * cfg.block + sizeof(long long) * a.nreq;
    if (PRT_DEFER_TRIS && a.leaf1) shmem += sizeof(TriQueue) * (cfg.block / 32);
    if (PRT_PACKET_PRIMARY && cfg.packet && a.packet)
    {
        const size_t pshmem = sizeof(long long) * a.nreq + sizeof(uint2) * kPacketStack * (cfg.block / 32);
        auto goPacket = [&](auto kernel) {
            int grid = grid_for(kernel, cfg.block, pshmem, numSMs, cfg);
            kernel<<<grid, cfg.block, pshmem, s>>>(a);
        };
        if (cfg.packet == kPrimaryIntervals) goPacket(k_batch_primary_packet<true>);
        else goPacket(k_batch_primary_packet<false>);
        return 1;
    }
    const int grid = grid_for(k_batch_first, cfg.block, shmem, numSMs, cfg);
    k_batch_first<<<grid, cfg.block, shmem, s>>>(a);
    return 1;
}

// Up to about 192 (closest) or 320 (any hit) rays per SM the longest ray's chain
// of node visits takes longer than the work does, and eight lanes per ray win;
// beyond that their emptier lanes cost more than they save.  Incoherent
// closest-hit calls, one lane -> eight lanes: 1000 rays on 82K triangles 54 -> 39
// us, on 1.38M 66 -> 42; 28000 on 1.38M 84 -> 79, 40000 86 -> 94 (any hit: 82 -> 72,
// and 80000 96 -> 114).
bool intersect_few(int n, bool anyHit, int numSMs) { return n <= (anyHit ? 320 : 192) * numSMs; }

int launch_intersect(const SceneDev& sc, const RayRec* rays, HitRec* hits, int n, bool anyHit, float* anyOut,
                     int* fetch, int numSMs, cudaStream_t s)
{
    if (n <= 0) return 0;
    const int block = 128;
    if (intersect_few(n, anyHit, numSMs))
    {
        // rays of one warp wait for one another, so they share it only once the chip is full
        const int perWarp = n <= 4 * numSMs ? 1 : (n <= 16 * numSMs ? 2 : 4);
        const int blocks = (n + 4 * perWarp - 1) / (4 * perWarp);
        if (anyHit) k_intersect_few<true><<<blocks, block, 0, s>>>(sc, rays, hits, anyOut, n, perWarp);
        else k_intersect_few<false><<<blocks, block, 0, s>>>(sc, rays, hits, anyOut, n, perWarp);
        return 1;
    }
    size_t shmem = (sizeof(uint2) * kShared + sizeof(uint32_t) * kShearWords) * block;
    if (PRT_DEFER_ISECT && sc.deferTris)
        shmem += (sizeof(TriQueue) + (anyHit ? 0 : sizeof(TriQueueUV))) * (block / 32);
    LaunchCfg cfg;
    auto go = [&](auto kernel) {
        // no more warps than rays: 32 rays per warp
        int grid = std::min(grid_for(kernel, block, shmem, numSMs, cfg), (n + block - 1) / block);
        kernel<<<grid, block, shmem, s>>>(sc, rays, hits, anyOut, n, fetch);
    };
    if (anyHit) go(k_intersect<true>);
    else go(k_intersect<false>);
    return 1;
}

int launch_query(const SceneDev& sc, const RayRec* ray, HitRec* hit, float* pNg, cudaStream_t s)
{
    k_query<<<1, 8, 0, s>>>(sc, ray, hit, pNg);
    return 1;
}

int launch_resolve_ldr(const float4* accum, uint32_t* out, int n, cudaStream_t s)
{
    if (n <= 0) return 0;
    k_resolve_ldr<<<(n + 255) / 256, 256, 0, s>>>(accum, out, n);
    return 1;
}

namespace {

// The primary rays of one pass, written per pixel (row-major) as 32-byte ray
// records (org, tnear 0, dir, tfar FLT_MAX): the wave item -> pixel mapping,
// RNG seeding and camera_ray of the bounce kernels' first depth, exposed so
// the generated rays can be compared with a reference one by one.
__global__ void k_primary_rays(CameraDev cam, int tilesX, int tilesY, int pass, RayRec* out)
{
    const int perPass = tilesX * tilesY * 64;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < perPass; i += gridDim.x * blockDim.x)
    {
        int x, y;
        if (!wave_item_pixel(i, tilesX, cam.width, cam.height, x, y)) continue;
        const int pixel = x + y * cam.width;
        uint32_t rng = rng_seed(pass, pixel);
        float3 org, dir;
        camera_ray(cam, x, y, rng, org, dir);
        float4* o = reinterpret_cast<float4*>(out + pixel);
        o[0] = make_float4(org.x, org.y, org.z, 0.0f);
        o[1] = make_float4(dir.x, dir.y, dir.z, FLT_MAX);
    }
}

} // namespace

int launch_primary_rays(const CameraDev& cam, int pass, RayRec* out, cudaStream_t s)
{
    const int tilesX = (cam.width + 7) / 8, tilesY = (cam.height + 7) / 8;
    const int perPass = tilesX * tilesY * 64;
    if (perPass <= 0) return 0;
    k_primary_rays<<<std::min((perPass + 255) / 256, 4096), 256, 0, s>>>(cam, tilesX, tilesY, pass, out);
    return 1;
}

int launch_begin_render(int* pass, int spp, unsigned long long* rays, int* counters, int words, cudaStream_t s)
{
    k_begin_render<<<1, 256, 0, s>>>(pass, spp, rays, counters, words);
    return 1;
}

int launch_replay(const SceneDev& sc, const CameraDev& cam, float4* accum, int pass0, int spp, int maxDepth, float sky,
                  const float* dL, float* dAlbedo, float* dSky, unsigned long long* rays, int* fetch, bool backward,
                  int numSMs, cudaStream_t s)
{
    long long total = (long long)spp * cam.width * cam.height;
    if (total <= 0) return 0;
    const int block = 128;
    const int words = backward ? kBackwardWords : kReplayWords;
    size_t shmem = (sizeof(uint2) * kShared + sizeof(uint32_t) * words) * block;
    if (PRT_DEFER_REPLAY && sc.deferTris) shmem += sizeof(TriQueue) * (block / 32);
    LaunchCfg cfg;
    auto go = [&](auto kernel) {
        int grid = grid_for(kernel, block, shmem, numSMs, cfg);
        kernel<<<grid, block, shmem, s>>>(sc, cam, accum, pass0, spp, maxDepth, sky, dL, dAlbedo, dSky, rays, fetch);
    };
    if (backward) go(k_replay<true>);
    else go(k_replay<false>);
    return 1;
}

int replay_max_depth() { return kReplayMaxDepth; }

int read_counters(unsigned long long* out, bool reset, cudaStream_t s)
{
    if (!PRT_COUNTERS) return -1;
    if (cudaMemcpyFromSymbolAsync(out, g_counters, sizeof(g_counters), 0, cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return 1;
    if (cudaStreamSynchronize(s) != cudaSuccess) return 1;
    if (reset)
    {
        static const unsigned long long zero[8] = {};
        if (cudaMemcpyToSymbolAsync(g_counters, zero, sizeof(zero), 0, cudaMemcpyHostToDevice, s) != cudaSuccess)
            return 1;
        if (cudaStreamSynchronize(s) != cudaSuccess) return 1;
    }
    return 0;
}

} // namespace prt_b200
