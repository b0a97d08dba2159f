// Full SAH binary tree for the high-quality BVH build (build_bvh8 in
// bvh_build.cu groups and collapses it into 8-wide nodes).
//
// From the root (the triangles in Morton order), every task (a node and its
// contiguous range of triangles) with more than kSahLeaves triangles is split
// by binned SAH, its triangles are partitioned into the two halves of the
// range, and the halves become the next level's tasks, subtrees of
// 2..kSahLeaves triangles or leaves; each subtree is then built by one block
// with an exact sweep SAH.  Output: child / range / parent of the n - 1
// internal nodes (root 0; a child reference ~p is the triangle at position p
// of perm) and perm, the triangle order.
#include <algorithm>
#include <cfloat>
#include <vector>

#include "prt_device.cuh"
#include "prt_internal.h"
#include "refit.cuh"

namespace prt_b200 {

// Task and split records of the top-down phase (declared in prt_internal.h).
struct TopTask
{
    int lo, hi, node;
    int firstChunk, chunks;            // its chunks in the level's chunk list
    int bins;                          // of several chunks: its merged bins
    uint32_t cmin[3], cmax[3];         // centroid bounds as order-preserving bits (ford)
};

struct TopSplit
{
    int axis;       // -1: no bin separates the centroids; split the range in the middle
    int bin;        // left: bins 0..bin
    int nl;         // triangles going left
    int task[2];    // the halves' tasks in the next level, -1: a subtree or a leaf
};

namespace {

__device__ __forceinline__ float box_half_area_lh(const float* lo, const float* hi)
{
    const float dx = hi[0] - lo[0], dy = hi[1] - lo[1], dz = hi[2] - lo[2];
    return dx * dy + dy * dz + dz * dx;
}

__device__ __forceinline__ uint32_t ford(float f)
{
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float funord(uint32_t u)
{
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// --- subtrees of at most kSahLeaves triangles: exact sweep SAH, three warps each -
//
// A subtree of 2..kSahLeaves triangles covers a contiguous range [a, b] of the
// triangle order; one block of three warps, a warp per axis, builds it top-down
// to single-triangle leaves, all nodes of a depth at once, permuting the
// triangles only inside [a, b].
// Splits: for each axis the range's triangles sorted by centroid, the split
// after position p costs area(left box) x |left| + area(right box) x |right|;
// the least cost wins (ties to the more balanced split, then the lower axis
// and position).
// The nodes of a depth are segments of the position range.  A warp walks its
// axis' positions in windows of 32, with segmented shuffle scans inside a window
// and a carry between windows, and windows whose segments are all single
// triangles are skipped; the warps meet at six barriers per depth.  The scans'
// shuffles and minima bound it (issue slots 70%, shared-memory pipe 74% in use);
// element indices, segment ids and segment ends are bytes, so a subtree takes 15
// KB of shared memory, and an SM holds 12 (by registers).
// Measured against one 256-thread block per subtree, whose scans stepped over
// shared memory with two barriers a step: prt_build_accel of 1.38M triangles 3.25
// -> 2.55 ms, 10.24M triangles 21.4 -> 15.7 (one warp for all three axes: 2.81 and
// 17.2, and 82K triangles 12% slower).
// The finished subtree's boxes and grouping costs (refit.cuh) follow, a depth at a
// time from the last, with the triangles' boxes still in shared memory, and one
// thread carries on above the root.  As a launch of its own, walking up from every
// triangle with an atomic per node, that took 222 us for 1.38M triangles; here 107
// (prt_build_accel 2.23 -> 2.10 ms, 10.24M 14.2 -> 13.4, 82K 0.69 -> 0.67).
constexpr int kSahLeaves = 256;

struct SahShared
{
    float box[6][kSahLeaves];           // triangle boxes of the range (lo xyz, hi xyz)
    float suffix[3][kSahLeaves];        // per axis list: area of the box from each position to its segment's end
    unsigned long long best[kSahLeaves];    // per segment: least split key, ~0 for a single triangle
    uint8_t list[2][3][kSahLeaves];     // per axis: elements in centroid order (double buffered)
    uint8_t segOf[kSahLeaves];          // per position: its segment
    uint8_t mark[kSahLeaves];           // per element: it goes left
    // per segment: first and last position, node (0: the root, k: the k-th new
    // one), the segment of its right half; per axis: left marks before its start
    uint8_t segStart[kSahLeaves], segEnd[kSahLeaves], segNode[kSahLeaves], segRight[kSahLeaves];
    uint8_t segBase[3][kSahLeaves];
    uint8_t depthFirst[kSahLeaves + 1];     // per depth: its first node, as in segNode
    int first, nseg, maxSeg;            // node index of pool entry 1; segments, and the largest, of this depth
};

__device__ __forceinline__ float area6(const float* v)
{
    const float dx = v[3] - v[0], dy = v[4] - v[1], dz = v[5] - v[2];
    return dx * dy + dy * dz + dz * dx;
}

__device__ __forceinline__ void box_merge(float* v, const float* w)
{
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        v[k] = fminf(v[k], w[k]);
        v[3 + k] = fmaxf(v[3 + k], w[3 + k]);
    }
}

// Sorts the kSahLeaves (key, idx) pairs of a warp, pair lane * 8 + r in
// register r, by key then idx (bitonic; strides below 8 inside a lane).
__device__ __forceinline__ void warp_sort256(uint32_t* key, uint32_t* idx, int lane)
{
#pragma unroll
    for (int size = 2; size <= kSahLeaves; size <<= 1)
    {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1)
        {
            if (stride >= 8)
            {
                const bool lower = (lane & (stride >> 3)) == 0;
#pragma unroll
                for (int r = 0; r < 8; ++r)
                {
                    const uint32_t ko = __shfl_xor_sync(0xffffffffu, key[r], stride >> 3);
                    const uint32_t io = __shfl_xor_sync(0xffffffffu, idx[r], stride >> 3);
                    const bool up = ((lane * 8) & size) == 0;
                    const bool greater = key[r] > ko || (key[r] == ko && idx[r] > io);
                    if (greater == (lower == up))
                    {
                        key[r] = ko;
                        idx[r] = io;
                    }
                }
            }
            else
            {
#pragma unroll
                for (int r = 0; r < 8; ++r)
                {
                    if (r & stride) continue;
                    const bool up = ((lane * 8 + r) & size) == 0;
                    const uint32_t k0 = key[r], k1 = key[r + stride], i0 = idx[r], i1 = idx[r + stride];
                    const bool greater = k0 > k1 || (k0 == k1 && i0 > i1);
                    if (greater == up)
                    {
                        key[r] = k1;
                        key[r + stride] = k0;
                        idx[r] = i1;
                        idx[r + stride] = i0;
                    }
                }
            }
        }
    }
}

// One subtree per block: roots[i] is its root (an internal node whose range
// holds 2..kSahLeaves triangles); its other internal nodes take new indices
// from *nodeCounter.
__global__ void __launch_bounds__(96, 12) k_sah_subtrees(int n, const int* __restrict__ roots,
                                                   const int* __restrict__ numRoots, const float* __restrict__ triBox,
                                                   uint32_t* vals, int2* child, int2* range, int* parent,
                                                   int* nodeCounter, RefitArgs refit)
{
    __shared__ SahShared S;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int ax = threadIdx.x >> 5;   // this warp's axis
    const unsigned lt = (1u << lane) - 1u;
    const int count = *numRoots;
    for (int ri = blockIdx.x; ri < count; ri += gridDim.x)
    {
        const int u = roots[ri];
        const int2 rg = range[u];
        const int a = rg.x, ns = rg.y - rg.x + 1;   // 2 <= ns <= kSahLeaves
        const int nw = (ns + 31) >> 5;
        // --- load the range ---------------------------------------------------
        for (int t = threadIdx.x; t < ns; t += 96)
        {
            const uint32_t tri = vals[a + t];
            const float2* bp = reinterpret_cast<const float2*>(triBox + 6 * (size_t)tri);
            const float2 b0 = __ldg(bp), b1 = __ldg(bp + 1), b2 = __ldg(bp + 2);
            S.box[0][t] = b0.x;
            S.box[1][t] = b0.y;
            S.box[2][t] = b1.x;
            S.box[3][t] = b1.y;
            S.box[4][t] = b2.x;
            S.box[5][t] = b2.y;
            S.segOf[t] = 0;
        }
        if (threadIdx.x == 0)
        {
            S.first = ns > 2 ? atomicAdd(nodeCounter, ns - 2) : 0;
            S.segStart[0] = 0;
            S.segEnd[0] = (uint8_t)(ns - 1);
            S.segNode[0] = 0;
            S.nseg = 1;
            S.maxSeg = ns;
        }
        __syncthreads();
        // --- the axis' elements sorted by (doubled) centroid, ties by element -----
        {
            uint32_t key[8], idx[8];
#pragma unroll
            for (int r = 0; r < 8; ++r)
            {
                const int i = lane * 8 + r;
                idx[r] = (uint32_t)i;
                // + 0: a negative zero ties with a positive one
                key[r] = i < ns ? ford(S.box[ax][i] + S.box[3 + ax][i] + 0.0f) : 0xffffffffu;
            }
            warp_sort256(key, idx, lane);
            uint2 packed;
            packed.x = idx[0] | (idx[1] << 8) | (idx[2] << 16) | (idx[3] << 24);
            packed.y = idx[4] | (idx[5] << 8) | (idx[6] << 16) | (idx[7] << 24);
            *reinterpret_cast<uint2*>(&S.list[0][ax][lane * 8]) = packed;
            __syncwarp();
        }
        int cur = 0, pool = 1;   // pool: warp 0
        int depth = 0;
        // --- one depth of the subtree per pass ------------------------------------
        for (;;)
        {
            const int maxSeg = S.maxSeg, nseg = S.nseg;
            if (maxSeg <= 1) break;
            const int span = min(maxSeg, 32);   // scans inside a window need log2(span) steps
            for (int i = threadIdx.x; i < nseg; i += 96) S.best[i] = ~0ull;
            __syncthreads();
            // suffix areas, last window first
            float carry[6] = {FLT_MAX, FLT_MAX, FLT_MAX, -FLT_MAX, -FLT_MAX, -FLT_MAX};
            for (int w = nw - 1; w >= 0; --w)
            {
                const int t = 32 * w + lane;
                const int s = t < ns ? S.segOf[t] : 0;
                const int st = S.segStart[s], en = S.segEnd[s];
                const bool act = t < ns && en > st;
                if (!__any_sync(FULL, act)) continue;
                const int room = act ? min(en, 32 * w + 31) - t : 0;   // lanes to the segment's end in this window
                float v[6];
                const int e = act ? S.list[cur][ax][t] : 0;
#pragma unroll
                for (int k = 0; k < 6; ++k) v[k] = S.box[k][e];
#pragma unroll
                for (int off = 1; off < 32; off <<= 1)
                {
                    if (off >= span) break;
                    float o[6];
#pragma unroll
                    for (int k = 0; k < 6; ++k) o[k] = __shfl_down_sync(FULL, v[k], off);
                    if (off <= room) box_merge(v, o);
                }
                if (act && en >= 32 * (w + 1)) box_merge(v, carry);
                S.suffix[ax][t] = area6(v);
#pragma unroll
                for (int k = 0; k < 6; ++k) carry[k] = __shfl_sync(FULL, v[k], 0);
            }
            __syncwarp();
            // prefix areas, the costs, and each segment's least
            for (int w = 0; w < nw; ++w)
            {
                const int t = 32 * w + lane;
                const int s = t < ns ? S.segOf[t] : 0;
                const int st = S.segStart[s], en = S.segEnd[s];
                const bool act = t < ns && en > st;
                if (!__any_sync(FULL, act)) continue;
                const int back = act ? t - max(st, 32 * w) : 0;
                const int room = act ? min(en, 32 * w + 31) - t : 0;
                float v[6];
                const int e = act ? S.list[cur][ax][t] : 0;
#pragma unroll
                for (int k = 0; k < 6; ++k) v[k] = S.box[k][e];
#pragma unroll
                for (int off = 1; off < 32; off <<= 1)
                {
                    if (off >= span) break;
                    float o[6];
#pragma unroll
                    for (int k = 0; k < 6; ++k) o[k] = __shfl_up_sync(FULL, v[k], off);
                    if (off <= back) box_merge(v, o);
                }
                if (act && st < 32 * w) box_merge(v, carry);
                unsigned long long key = ~0ull;
                if (act && t < en)
                {
                    // the split after position t
                    const int nl = t - st + 1, nr = en - t;
                    const float c = area6(v) * (float)nl + S.suffix[ax][t + 1] * (float)nr;
                    const unsigned imbalance = (unsigned)abs(nl - nr);
                    key = ((unsigned long long)__float_as_uint(fmaxf(c, 0.f)) << 32) |
                          ((unsigned long long)imbalance << 16) | ((unsigned)ax << 8) | (unsigned)(t - st);
                }
#pragma unroll
                for (int k = 0; k < 6; ++k) carry[k] = __shfl_sync(FULL, v[k], 31);
#pragma unroll
                for (int off = 1; off < 32; off <<= 1)
                {
                    if (off >= span) break;
                    const unsigned long long o = __shfl_down_sync(FULL, key, off);
                    if (off <= room && o < key) key = o;
                }
                // the first lane of a segment's part in this window holds the part's least
                if (act && back == 0 && key != ~0ull) atomicMin(&S.best[s], key);
            }
            __syncthreads();
            // marks: the chosen axis list's prefix goes left
            for (int t = threadIdx.x; t < ns; t += 96)
            {
                const int s = S.segOf[t];
                const unsigned long long b = S.best[s];
                if (b == ~0ull) continue;
                const int sp = S.segStart[s] + (int)(b & 0xff);
                S.mark[S.list[cur][(int)((b >> 8) & 0xff)][t]] = t <= sp ? 1 : 0;
            }
            __syncthreads();
            // stable partition of the axis' list within the splitting segments
            {
                int run = 0;   // left marks in the windows before
                for (int w = 0; w < nw; ++w)
                {
                    const int t = 32 * w + lane;
                    const int s = t < ns ? S.segOf[t] : 0;
                    const unsigned long long b = S.best[s];
                    const int st = S.segStart[s];
                    const bool act = t < ns && b != ~0ull;
                    const int e = t < ns ? S.list[cur][ax][t] : 0;
                    const bool left = act && S.mark[e];
                    const unsigned m = __ballot_sync(FULL, left);
                    const int before = run + __popc(m & lt);
                    run += __popc(m);
                    if (act && t == st) S.segBase[ax][s] = (uint8_t)before;
                    __syncwarp();
                    if (t < ns)
                    {
                        int np = t;
                        if (act)
                        {
                            const int rank = before - S.segBase[ax][s];   // left elements before t in the segment
                            np = left ? st + rank : st + (int)(b & 0xff) + 1 + (t - st - rank);
                        }
                        S.list[cur ^ 1][ax][np] = (uint8_t)e;
                    }
                }
            }
            __syncthreads();
            // nodes: each splitting segment is an internal node with two children
            if (ax == 0)
            {
                int newMax = 1, next = nseg;
                const int first = S.first;
                for (int i0 = 0; i0 < nseg; i0 += 32)
                {
                    const int i = i0 + lane;
                    const unsigned long long b = i < nseg ? S.best[i] : ~0ull;
                    const bool split = b != ~0ull;
                    int st = 0, en = 0, sp = 0;
                    if (split)
                    {
                        st = S.segStart[i];
                        en = S.segEnd[i];
                        sp = st + (int)(b & 0xff);
                    }
                    const int ls = sp - st + 1, rs = en - sp;
                    const unsigned ms = __ballot_sync(FULL, split);
                    const unsigned ml = __ballot_sync(FULL, split && ls > 1), mr = __ballot_sync(FULL, split && rs > 1);
                    if (split)
                    {
                        const int right = next + __popc(ms & lt);
                        const int pl = pool + __popc(ml & lt) + __popc(mr & lt), pr = pl + (ls > 1 ? 1 : 0);
                        const int me = S.segNode[i];
                        const int node = me == 0 ? u : first + me - 1;
                        int2 refs;
                        if (ls > 1)
                        {
                            refs.x = first + pl - 1;
                            parent[refs.x] = node;
                            range[refs.x] = make_int2(a + st, a + sp);
                        }
                        else
                        {
                            refs.x = ~(a + st);
                            parent[(n - 1) + a + st] = node;
                        }
                        if (rs > 1)
                        {
                            refs.y = first + pr - 1;
                            parent[refs.y] = node;
                            range[refs.y] = make_int2(a + sp + 1, a + en);
                        }
                        else
                        {
                            refs.y = ~(a + en);
                            parent[(n - 1) + a + en] = node;
                        }
                        child[node] = refs;
                        S.segEnd[i] = (uint8_t)sp;
                        S.segNode[i] = (uint8_t)pl;   // of no use when the half is a single triangle
                        S.segRight[i] = (uint8_t)right;
                        S.segStart[right] = (uint8_t)(sp + 1);
                        S.segEnd[right] = (uint8_t)en;
                        S.segNode[right] = (uint8_t)pr;
                        newMax = max(newMax, max(ls, rs));
                    }
                    next += __popc(ms);
                    pool += __popc(ml) + __popc(mr);
                }
                newMax = __reduce_max_sync(FULL, newMax);
                if (lane == 0)
                {
                    S.maxSeg = newMax;
                    S.nseg = next;
                    S.depthFirst[depth + 2] = (uint8_t)pool;   // 255 at most
                }
            }
            __syncthreads();
            for (int t = threadIdx.x; t < ns; t += 96)
            {
                const int s = S.segOf[t];
                if (S.best[s] != ~0ull && t > S.segEnd[s]) S.segOf[t] = S.segRight[s];
            }
            cur ^= 1;
            ++depth;
            __syncthreads();
        }
        // --- bounds and grouping costs, last depth first ----------------------------
        const uint8_t* order = S.list[cur][0];
        for (int t = threadIdx.x; t < ns; t += 96)
        {
            float* lb = refit.box + 6 * (size_t)((n - 1) + a + t);
            const int e = order[t];
#pragma unroll
            for (int k = 0; k < 6; ++k) __stcg(lb + k, S.box[k][e]);
        }
        for (int d = depth - 1; d >= 0; --d)
        {
            const int end = d == 0 ? 1 : S.depthFirst[d + 1];
            for (int i = (d == 0 ? 0 : (d == 1 ? 1 : S.depthFirst[d])) + (int)threadIdx.x; i < end; i += 96)
            {
                const int node = i == 0 ? u : S.first + i - 1;
                const int2 ch = child[node], nr = range[node];
                float b[2][6];
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    const int ref = h == 0 ? ch.x : ch.y;
                    if (ref >= 0) load_box(refit, ref, b[h]);
                    else
                    {
                        const int e = order[~ref - a];
#pragma unroll
                        for (int k = 0; k < 6; ++k) b[h][k] = S.box[k][e];
                    }
                }
                if (refit.cost) refit_node<true>(refit, node, ch, nr.y - nr.x + 1, b[0], b[1]);
                else refit_node<false>(refit, node, ch, nr.y - nr.x + 1, b[0], b[1]);
            }
            __syncthreads();
        }
        // the triangles in their new order
        uint32_t tri[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
            const int t = threadIdx.x + 96 * k;
            tri[k] = t < ns ? vals[a + S.list[cur][0][t]] : 0u;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
            const int t = threadIdx.x + 96 * k;
            if (t < ns) vals[a + t] = tri[k];
        }
        // up from the subtree's root: the second arrival at a node finishes it; a
        // child that is a single triangle does not arrive
        if (threadIdx.x == 0)
        {
            for (int node = parent[u]; node >= 0; node = parent[node])
            {
                const int2 ch = child[node], nr = range[node];
                const int single = ch.x < 0 ? ch.x : ch.y;
                float b[2][6];
                if (single < 0)
                {
                    const float* tb = triBox + 6 * (size_t)refit.vals[~single];
                    float* lb = refit.box + 6 * (size_t)((n - 1) + ~single);
#pragma unroll
                    for (int k = 0; k < 6; ++k) __stcg(lb + k, tb[k]);
                }
                else if (arrive(refit.flag + node) == 0)
                {
                    break;
                }
                load_box(refit, ch.x, b[0]);
                load_box(refit, ch.y, b[1]);
                if (refit.cost) refit_node<true>(refit, node, ch, nr.y - nr.x + 1, b[0], b[1]);
                else refit_node<false>(refit, node, ch, nr.y - nr.x + 1, b[0], b[1]);
            }
        }
        __syncthreads();
    }
}

// --- above kSahLeaves triangles: top-down binned SAH ----------------------------
//
// The high-quality build makes a full SAH tree instead of the Morton
// hierarchy.  From the root (the triangles in Morton order), every task (a
// node and its contiguous range of triangles) with more than kSahLeaves
// triangles is split by the least SAH cost over kTopBins centroid bins per axis,
// its triangles are partitioned into the two halves of the range, and the
// halves become the next level's tasks, k_sah_subtrees' subtrees
// (2..kSahLeaves triangles) or leaves.
//
// A level is two launches over the chunks (kTopChunk triangles) of its tasks:
//   k_top_bin        gathers the bins; the block that brings a task's last chunk
//                    evaluates the split and makes the children, with their
//                    tasks and chunks
//   k_top_partition  moves the triangles to their halves, in order, and gathers
//                    the halves' centroid bounds (the next level's bin ranges)
// Task and chunk lists are made on the device, so levels are launched without
// waiting for the host, which reads the task count back once per batch of
// levels.  A level is a few tens of microseconds of work at 1.4M triangles, so
// launches, host round trips and passes over the triangles are what bounds it.
// Measured against nine launches per level (bins, split, count, children, a
// scan, partition, copy back), a read-back per level and a new output block per
// build: prt_build_accel of 82K triangles 2.78 -> 0.96 ms, 1.38M triangles 5.80
// -> 3.25, 10.24M triangles 28.8 -> 21.4.
constexpr int kTopBins = 32;
constexpr int kTopChunk = 2048;        // triangles per block of the two passes
constexpr int kTopBlock = 256;
constexpr int kBinWords = 7;           // count, box lo, box hi (order-preserving float bits)
constexpr int kTaskBins = 3 * kTopBins * kBinWords;
constexpr int kTopSlots = 4;           // level l counts its tasks, chunks and merged bins in slot l & 3
constexpr int kTopCounts = 3;

__device__ __forceinline__ int top_bin(float c, float cmin, float scale)
{
    return min(kTopBins - 1, max(0, (int)((c - cmin) * scale)));
}

__device__ __forceinline__ float top_scale(float cmin, float cmax)
{
    const float e = cmax - cmin;
    return e > 0.f ? (float)kTopBins * 0.99999f / e : 0.f;
}

// The empty value of word i of a task's bins: count 0; lo fields (1-3) start at
// the largest value, hi fields (4-6) at 0.
__device__ __forceinline__ uint32_t bin_empty(int i)
{
    const int w = i % kBinWords;
    return w >= 1 && w <= 3 ? 0xffffffffu : 0u;
}

// What a level reads and what it makes for the next one.
struct TopArgs
{
    int n;
    const float* triBox;
    const uint32_t* src;        // the level's triangles
    uint32_t* dst;              // the next level's
    uint32_t* out;              // the final order: subtrees and leaves
    const TopTask* tasks;
    const int4* chunks;         // {task, first triangle, last triangle, index in the task}
    TopTask* nextTasks;
    int4* nextChunks;
    const int* count;           // [0] tasks, [1] chunks, [2] tasks of several chunks of this level
    int* nextCount;             // of the next level
    int* clearCount;            // of the level after it
    TopSplit* splits;           // per task
    uint32_t* bins;             // merged bins of the tasks of several chunks, last word: the chunks that have arrived
    uint32_t* nextBins;
    uint16_t* cum;              // per chunk of a task of several: [axis][bin] triangles in bins 0..bin
    int* small;                 // subtree roots
    int* numSmall;
    int* nodeCounter;
    int2* child;
    int2* range;
    int* parent;
};

__device__ __forceinline__ float shfl_ud(float v, int off, bool down)
{
    return down ? __shfl_down_sync(0xffffffffu, v, off) : __shfl_up_sync(0xffffffffu, v, off);
}

// Least-cost split over the bins of one axis (a warp, lane = bin; prefix and
// suffix boxes by warp scans): (cost bits << 32) | (axis * 32 + bin), ~0 if no
// bin separates the triangles.
__device__ __forceinline__ unsigned long long axis_split(const uint32_t* bins, int ax, int lane)
{
    const uint32_t* w = bins + (ax * kTopBins + lane) * kBinWords;
    const int cnt = (int)w[0];
    // left: inclusive prefix over bins 0..lane; right: suffix over lane..31
    int lc = cnt, rc = cnt;
    float llo[3], lhi[3], rlo[3], rhi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        llo[k] = rlo[k] = cnt ? funord(w[1 + k]) : FLT_MAX;
        lhi[k] = rhi[k] = cnt ? funord(w[4 + k]) : -FLT_MAX;
    }
#pragma unroll
    for (int off = 1; off < 32; off <<= 1)
    {
        const int ulc = __shfl_up_sync(0xffffffffu, lc, off);
        const int drc = __shfl_down_sync(0xffffffffu, rc, off);
        float ul[3], uh[3], dl[3], dh[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
            ul[k] = shfl_ud(llo[k], off, false);
            uh[k] = shfl_ud(lhi[k], off, false);
            dl[k] = shfl_ud(rlo[k], off, true);
            dh[k] = shfl_ud(rhi[k], off, true);
        }
        if (lane >= off)
        {
            lc += ulc;
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                llo[k] = fminf(llo[k], ul[k]);
                lhi[k] = fmaxf(lhi[k], uh[k]);
            }
        }
        if (lane + off < 32)
        {
            rc += drc;
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                rlo[k] = fminf(rlo[k], dl[k]);
                rhi[k] = fmaxf(rhi[k], dh[k]);
            }
        }
    }
    // split after bin `lane`: the suffix from lane + 1
    const int nrc = __shfl_down_sync(0xffffffffu, rc, 1);
    float nlo[3], nhi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        nlo[k] = __shfl_down_sync(0xffffffffu, rlo[k], 1);
        nhi[k] = __shfl_down_sync(0xffffffffu, rhi[k], 1);
    }
    unsigned long long best = ~0ull;
    if (lane < 31 && lc > 0 && nrc > 0)
    {
        const float c = box_half_area_lh(llo, lhi) * (float)lc + box_half_area_lh(nlo, nhi) * (float)nrc;
        best = ((unsigned long long)__float_as_uint(fmaxf(c, 0.f)) << 32) | (unsigned)(ax * kTopBins + lane);
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
    {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, best, off);
        best = o < best ? o : best;
    }
    return best;
}

// Consecutive triangles of one thread that fall into the same bin of an axis:
// the bin (-1: none), their number and box (order-preserving float bits).
struct BinRun
{
    int bin;
    uint32_t count, lo[3], hi[3];
};

__device__ __forceinline__ void add_run(uint32_t* axisBins, const BinRun& r)
{
    uint32_t* w = axisBins + r.bin * kBinWords;
    atomicAdd(w, r.count);
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        atomicMin(w + 1 + k, r.lo[k]);
        atomicMax(w + 4 + k, r.hi[k]);
    }
}

// Adds the runs of a warp's lanes to the bins of one axis.  Neighbours in the
// triangle order fall into few bins near the root and into many near the
// leaves: up to four bins, each is reduced over the warp and one lane updates
// it; beyond that the lanes update their bins themselves, since atomics on
// different words run side by side and on the same word one by one.
__device__ __forceinline__ void warp_add_runs(uint32_t* axisBins, const BinRun& run, unsigned lane)
{
    const unsigned FULL = 0xffffffffu;
    const unsigned peers = __match_any_sync(FULL, run.bin);
    unsigned leaders = __ballot_sync(FULL, run.bin >= 0 && lane == (unsigned)(__ffs(peers) - 1));
    if (__popc(leaders) <= 4)
    {
        while (leaders)
        {
            const int l = __ffs(leaders) - 1;
            leaders &= leaders - 1;
            const unsigned grp = __shfl_sync(FULL, peers, l);
            const bool in = (grp >> lane) & 1u;
            BinRun all;
            all.bin = run.bin;
            all.count = __reduce_add_sync(FULL, in ? run.count : 0u);
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                all.lo[k] = __reduce_min_sync(FULL, in ? run.lo[k] : 0xffffffffu);
                all.hi[k] = __reduce_max_sync(FULL, in ? run.hi[k] : 0u);
            }
            if ((int)lane == l) add_run(axisBins, all);
        }
    }
    else if (run.bin >= 0) add_run(axisBins, run);
}

// Triangles of a chunk that a thread of the partition loads together: the loads of
// one do not wait for the work on another, and the block meets once per batch.
// 1.38M triangles, a level: 24 -> 20 us.
constexpr int kTopBatch = 4;
static_assert(kTopChunk == 2 * kTopBatch * kTopBlock, "a chunk is two batches");

struct TopBox
{
    float2 a, b, c;   // lo x y, lo z hi x, hi y z
};

// Triangles first, first + kTopBlock, .. up to last: ids (0 past the end) and boxes.
__device__ __forceinline__ void top_load(const TopArgs& a, int first, int last, uint32_t (&tri)[kTopBatch],
                                         TopBox (&box)[kTopBatch])
{
#pragma unroll
    for (int j = 0; j < kTopBatch; ++j) tri[j] = first + j * kTopBlock <= last ? a.src[first + j * kTopBlock] : 0u;
#pragma unroll
    for (int j = 0; j < kTopBatch; ++j)
    {
        const float2* bp = reinterpret_cast<const float2*>(a.triBox + 6 * (size_t)tri[j]);
        box[j] = {__ldg(bp), __ldg(bp + 1), __ldg(bp + 2)};
    }
}

__global__ void __launch_bounds__(kTopBlock, 5) k_top_bin(TopArgs a)
{
    __shared__ uint32_t sb[kTaskBins];
    __shared__ unsigned long long s_best[3];
    __shared__ int s_last, s_task[2], s_chunk[2], s_bins[2];
    const unsigned lane = threadIdx.x & 31u;
    const int warp = threadIdx.x >> 5;
    const int numChunks = a.count[1];
    for (int c = blockIdx.x; c < numChunks; c += gridDim.x)
    {
        const int4 ch = a.chunks[c];
        const TopTask tk = a.tasks[ch.x];
        float cmin[3], sc[3];
#pragma unroll
        for (int k = 0; k < 3; ++k)
        {
            cmin[k] = funord(tk.cmin[k]);
            sc[k] = top_scale(cmin[k], funord(tk.cmax[k]));
        }
        for (int i = threadIdx.x; i < kTaskBins; i += kTopBlock) sb[i] = bin_empty(i);
        __syncthreads();
        // each thread takes neighbours in the triangle order, which mostly fall
        // into the same bins, and adds them run by run: fewer reductions near the
        // root and atomics near the leaves than one per triangle (1.38M triangles, a
        // level: 40 -> 35 us; prt_build_accel with the partition's batches 2.27 -> 2.22
        // ms, 10.24M 14.7 -> 14.2, 82K 0.77 -> 0.69).  48 registers: with 5 blocks per
        // SM the chunks of 1.38M triangles are one wave, with 4 they are two.
        BinRun run[3];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax)
        {
            run[ax].bin = -1;
            run[ax].count = 0;
        }
        const int per = (ch.z - ch.y + kTopBlock) / kTopBlock;
        const int first = ch.y + (int)threadIdx.x * per, end = min(first + per - 1, ch.z);
        uint32_t next = first <= end ? a.src[first] : 0u;   // loaded one triangle ahead
#pragma unroll 1
        for (int i = first; i <= end; ++i)
        {
            const uint32_t tri = next;
            if (i < end) next = a.src[i + 1];
            const float2* bp = reinterpret_cast<const float2*>(a.triBox + 6 * (size_t)tri);
            const float2 b0 = __ldg(bp), b1 = __ldg(bp + 1), b2 = __ldg(bp + 2);
            const float bl[3] = {b0.x, b0.y, b1.x}, bh[3] = {b1.y, b2.x, b2.y};
            uint32_t lo[3], hi[3];
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                lo[k] = ford(bl[k]);
                hi[k] = ford(bh[k]);
            }
#pragma unroll
            for (int ax = 0; ax < 3; ++ax)
            {
                BinRun& rn = run[ax];
                const int bin = top_bin(0.5f * (bl[ax] + bh[ax]), cmin[ax], sc[ax]);
                const bool same = bin == rn.bin;
                if (!same && rn.bin >= 0) add_run(sb + ax * kTopBins * kBinWords, rn);
                rn.bin = bin;
                rn.count = same ? rn.count + 1 : 1;
#pragma unroll
                for (int k = 0; k < 3; ++k)
                {
                    rn.lo[k] = same ? min(rn.lo[k], lo[k]) : lo[k];
                    rn.hi[k] = same ? max(rn.hi[k], hi[k]) : hi[k];
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int ax = 0; ax < 3; ++ax) warp_add_runs(sb + ax * kTopBins * kBinWords, run[ax], lane);
        __syncthreads();
        // a task of several chunks: the partition pass needs each chunk's
        // counts, and the task's bins are merged in global memory
        bool last = true;
        if (tk.chunks > 1)
        {
            if (warp < 3)
            {
                int x = (int)sb[(warp * kTopBins + (int)lane) * kBinWords];
#pragma unroll
                for (int off = 1; off < 32; off <<= 1)
                {
                    const int y = __shfl_up_sync(0xffffffffu, x, off);
                    if ((int)lane >= off) x += y;
                }
                a.cum[(size_t)c * 3 * kTopBins + warp * kTopBins + lane] = (uint16_t)x;
            }
            uint32_t* g = a.bins + (size_t)tk.bins * (kTaskBins + 1);
            for (int i = threadIdx.x; i < kTaskBins; i += kTopBlock)
            {
                const uint32_t v = sb[i];
                if (v == bin_empty(i)) continue;
                const int w = i % kBinWords;
                if (w == 0) atomicAdd(g + i, v);
                else if (w <= 3) atomicMin(g + i, v);
                else atomicMax(g + i, v);
            }
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) s_last = atomicAdd(g + kTaskBins, 1u) == (uint32_t)tk.chunks - 1u;
            __syncthreads();
            last = s_last != 0;
            if (last)
            {
                __threadfence();
                for (int i = threadIdx.x; i < kTaskBins; i += kTopBlock) sb[i] = __ldcg(g + i);
            }
            __syncthreads();
        }
        if (!last) continue;   // block-uniform
        // --- the split ----------------------------------------------------------
        if (warp < 3)
        {
            const unsigned long long b = axis_split(sb, warp, (int)lane);
            if (lane == 0) s_best[warp] = b;
        }
        __syncthreads();
        if (warp == 0)
        {
            unsigned long long best = s_best[0];
            if (s_best[1] < best) best = s_best[1];
            if (s_best[2] < best) best = s_best[2];
            TopSplit sp;
            if (best == ~0ull)
            {
                sp.axis = -1;
                sp.bin = 0;
                sp.nl = (tk.hi - tk.lo + 1) / 2;
            }
            else
            {
                const int code = (int)(best & 0xffffffffu);
                sp.axis = code / kTopBins;
                sp.bin = code % kTopBins;
                const int cnt = (int)sb[(sp.axis * kTopBins + (int)lane) * kBinWords];
                sp.nl = __reduce_add_sync(0xffffffffu, (int)lane <= sp.bin ? cnt : 0);
            }
            // --- the two halves: next-level tasks, subtrees or leaves -----------
            if (lane < 2)
            {
                const int side = (int)lane;
                const int lo = side == 0 ? tk.lo : tk.lo + sp.nl, hi = side == 0 ? tk.lo + sp.nl - 1 : tk.hi;
                const int size = hi - lo + 1;
                int ref = ~lo, task = -1, chunk = 0, bins = -1;
                if (size == 1)
                {
                    a.parent[(a.n - 1) + lo] = tk.node;
                }
                else
                {
                    ref = atomicAdd(a.nodeCounter, 1);
                    a.parent[ref] = tk.node;
                    a.range[ref] = make_int2(lo, hi);
                    if (size <= kSahLeaves)
                    {
                        a.small[atomicAdd(a.numSmall, 1)] = ref;
                    }
                    else
                    {
                        const int nch = (size + kTopChunk - 1) / kTopChunk;
                        task = atomicAdd(a.nextCount, 1);
                        chunk = atomicAdd(a.nextCount + 1, nch);
                        if (nch > 1) bins = atomicAdd(a.nextCount + 2, 1);
                        TopTask t;
                        t.lo = lo;
                        t.hi = hi;
                        t.node = ref;
                        t.firstChunk = chunk;
                        t.chunks = nch;
                        t.bins = bins;
#pragma unroll
                        for (int k = 0; k < 3; ++k)
                        {
                            t.cmin[k] = 0xffffffffu;
                            t.cmax[k] = 0u;
                        }
                        a.nextTasks[task] = t;
                    }
                }
                const int other = __shfl_xor_sync(0x3u, ref, 1);
                const int otherTask = __shfl_xor_sync(0x3u, task, 1);
                s_task[side] = task;
                s_chunk[side] = chunk;
                s_bins[side] = bins;
                if (side == 0)
                {
                    a.child[tk.node] = make_int2(ref, other);
                    sp.task[0] = task;
                    sp.task[1] = otherTask;
                    a.splits[ch.x] = sp;
                }
            }
            if (lane == 0) s_last = sp.nl;
        }
        __syncthreads();
        // the tasks' chunks, and empty bins for those of several
        const int nl = s_last;
        for (int side = 0; side < 2; ++side)
        {
            const int task = s_task[side], chunk = s_chunk[side];
            if (task < 0) continue;
            const int lo = side == 0 ? tk.lo : tk.lo + nl, hi = side == 0 ? tk.lo + nl - 1 : tk.hi;
            const int nch = (hi - lo + kTopChunk) / kTopChunk;
            for (int k = threadIdx.x; k < nch; k += kTopBlock)
                a.nextChunks[chunk + k] =
                    make_int4(task, lo + k * kTopChunk, min(hi, lo + (k + 1) * kTopChunk - 1), k);
            if (nch > 1)
                for (int i = threadIdx.x; i <= kTaskBins; i += kTopBlock)
                    a.nextBins[(size_t)s_bins[side] * (kTaskBins + 1) + i] = i == kTaskBins ? 0u : bin_empty(i);
        }
        __syncthreads();
    }
}

// The triangles of each chunk to their half of the task's range, in their
// order: a half that is a task goes to dst, a subtree or a leaf to its place in
// the final order.  The halves' centroid bounds go to their tasks with integer
// atomics on the order-preserving bits.
__global__ void __launch_bounds__(kTopBlock, 6) k_top_partition(TopArgs a)
{
    constexpr int kWarps = kTopBlock / 32;
    static_assert(kTopBatch * kWarps == 32, "one lane per count");
    __shared__ int s_left[kTopBatch * kWarps];   // left triangles per item of the batch and warp
    __shared__ int s_before;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int numChunks = a.count[1];
    if (blockIdx.x == 0 && threadIdx.x < kTopCounts) a.clearCount[threadIdx.x] = 0;
    for (int c = blockIdx.x; c < numChunks; c += gridDim.x)
    {
        const int4 ch = a.chunks[c];
        const TopTask tk = a.tasks[ch.x];
        const TopSplit sp = a.splits[ch.x];
        float cmin = 0.f, sc = 0.f;
        if (sp.axis >= 0)
        {
            cmin = funord(tk.cmin[sp.axis]);
            sc = top_scale(cmin, funord(tk.cmax[sp.axis]));
        }
        // left triangles of the task before this chunk
        if (threadIdx.x == 0) s_before = 0;
        __syncthreads();
        if (sp.axis < 0)
        {
            if (threadIdx.x == 0) s_before = min(ch.y - tk.lo, sp.nl);
        }
        else if (ch.w > 0)
        {
            int sum = 0;
            for (int k = threadIdx.x; k < ch.w; k += kTopBlock)
                sum += a.cum[(size_t)(tk.firstChunk + k) * 3 * kTopBins + sp.axis * kTopBins + sp.bin];
            sum = __reduce_add_sync(0xffffffffu, sum);
            if (lane == 0 && sum) atomicAdd(&s_before, sum);
        }
        __syncthreads();
        int baseL = s_before;   // left triangles of the task before this batch
        uint32_t bmin[2][3], bmax[2][3];
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                bmin[h][k] = 0xffffffffu;
                bmax[h][k] = 0u;
            }
        uint32_t* const toL = sp.task[0] >= 0 ? a.dst : a.out;
        uint32_t* const toR = sp.task[1] >= 0 ? a.dst : a.out;
        for (int i0 = ch.y; i0 <= ch.z; i0 += kTopBatch * kTopBlock)
        {
            uint32_t tri[kTopBatch];
            TopBox box[kTopBatch];
            unsigned left[kTopBatch];   // this warp's lanes whose triangle goes left
            const int i = i0 + (int)threadIdx.x;
            top_load(a, i, ch.z, tri, box);
#pragma unroll
            for (int j = 0; j < kTopBatch; ++j)
            {
                const int ij = i + j * kTopBlock;
                const bool valid = ij <= ch.z;
                int side = 0;
                const float cen[3] = {0.5f * (box[j].a.x + box[j].b.y), 0.5f * (box[j].a.y + box[j].c.x),
                                      0.5f * (box[j].b.x + box[j].c.y)};
                if (sp.axis < 0) side = ij - tk.lo < sp.nl ? 0 : 1;
                else
                {
                    const float cx = sp.axis == 0 ? cen[0] : (sp.axis == 1 ? cen[1] : cen[2]);
                    side = top_bin(cx, cmin, sc) <= sp.bin ? 0 : 1;
                }
                if (valid)
                {
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                    {
                        const uint32_t o = ford(cen[k]);
                        if (side == 0)
                        {
                            bmin[0][k] = min(bmin[0][k], o);
                            bmax[0][k] = max(bmax[0][k], o);
                        }
                        else
                        {
                            bmin[1][k] = min(bmin[1][k], o);
                            bmax[1][k] = max(bmax[1][k], o);
                        }
                    }
                }
                left[j] = __ballot_sync(0xffffffffu, valid && side == 0);
                if (lane == 0) s_left[j * kWarps + warp] = __popc(left[j]);
            }
            __syncthreads();
            // left triangles before each (item, warp): every warp scans the counts
            const int count = s_left[lane];
            int incl = count;
#pragma unroll
            for (int off = 1; off < 32; off <<= 1)
            {
                const int y = __shfl_up_sync(0xffffffffu, incl, off);
                if (lane >= off) incl += y;
            }
#pragma unroll
            for (int j = 0; j < kTopBatch; ++j)
            {
                const int ij = i + j * kTopBlock;
                const int l = baseL + __shfl_sync(0xffffffffu, incl - count, j * kWarps + warp) +
                              __popc(left[j] & ((1u << lane) - 1u));
                if (ij > ch.z) continue;
                const bool toLeft = (left[j] >> lane) & 1u;
                // those before it that did not go left went right
                const int at = toLeft ? tk.lo + l : tk.lo + sp.nl + (ij - tk.lo - l);
                if (at <= tk.hi) (toLeft ? toL : toR)[at] = tri[j];
            }
            baseL += __shfl_sync(0xffffffffu, incl, 31);
            __syncthreads();
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
        {
            if (sp.task[h] < 0) continue;   // block-uniform
            TopTask* t = a.nextTasks + sp.task[h];
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                const uint32_t lo = __reduce_min_sync(0xffffffffu, bmin[h][k]);
                const uint32_t hi = __reduce_max_sync(0xffffffffu, bmax[h][k]);
                if (lane == 0)
                {
                    if (lo != 0xffffffffu) atomicMin(&t->cmin[k], lo);
                    if (hi != 0u) atomicMax(&t->cmax[k], hi);
                }
            }
        }
    }
}

// The root: node 0 over all n triangles, a task (n > kSahLeaves) or a rebuild
// subtree.  counters: [0] rebuild subtrees, [1] nodes, then the levels' slots.
__global__ void k_top_root(const float* __restrict__ cbounds, int n, TopTask* tasks, int4* chunks, uint32_t* bins,
                           int* small, int* counters, int2* range, int* parent)
{
    const int nch = (n + kTopChunk - 1) / kTopChunk;
    if (threadIdx.x == 0)
    {
        range[0] = make_int2(0, n - 1);
        parent[0] = -1;
        counters[0] = n <= kSahLeaves ? 1 : 0;
        counters[1] = 1;
        for (int i = 0; i < kTopCounts * kTopSlots; ++i) counters[2 + i] = 0;
        if (n <= kSahLeaves)
        {
            small[0] = 0;
        }
        else
        {
            counters[2] = 1;
            counters[3] = nch;
            counters[4] = 1;
            TopTask t;
            t.lo = 0;
            t.hi = n - 1;
            t.node = 0;
            t.firstChunk = 0;
            t.chunks = nch;
            t.bins = 0;
            for (int k = 0; k < 3; ++k)
            {
                t.cmin[k] = ford(cbounds[k]);
                t.cmax[k] = ford(cbounds[3 + k]);
            }
            tasks[0] = t;
        }
    }
    if (n <= kSahLeaves) return;
    for (int k = threadIdx.x; k < nch; k += blockDim.x)
        chunks[k] = make_int4(0, k * kTopChunk, min(n - 1, (k + 1) * kTopChunk - 1), k);
    for (int i = threadIdx.x; i <= kTaskBins; i += blockDim.x) bins[i] = i == kTaskBins ? 0u : bin_empty(i);
}

} // namespace

void sah_tree_carve(Carve& c, int n, SahTreeBuffers& B)
{
    // a level's tasks are disjoint ranges of more than kSahLeaves triangles, each
    // with at most one partly filled chunk; those of several chunks have more
    // than kTopChunk triangles
    B.maxTasks = n / (kSahLeaves + 1) + 2;
    B.maxChunks = n / kTopChunk + B.maxTasks + 2;
    const int maxBins = n / (kTopChunk + 1) + 2;
    for (int i = 0; i < 2; ++i)
    {
        B.task[i] = c.take<TopTask>(B.maxTasks);
        B.chunks[i] = c.take<int4>(B.maxChunks);
        B.bins[i] = c.take<uint32_t>((size_t)maxBins * (kTaskBins + 1));
    }
    B.splits = c.take<TopSplit>(B.maxTasks);
    B.cum = c.take<uint16_t>((size_t)B.maxChunks * 3 * kTopBins);
    B.small = c.take<int>((size_t)n / 2 + 1);
    B.counters = c.take<int>(2 + kTopCounts * kTopSlots);
}

// Top-down binned SAH from the root down to subtrees of kSahLeaves triangles,
// then k_sah_subtrees for those.  perm: the triangles in their starting order;
// out: in the tree's order.
cudaError_t sah_build_tree(int n, const float* triBox, const float* cbounds, const uint32_t* perm, uint32_t* out,
                           int2* child, int2* range, int* parent, const SahTreeBuffers& B, const RefitArgs& refit,
                           int numSMs, cudaStream_t stream)
{
    k_top_root<<<1, 256, 0, stream>>>(cbounds, n, B.task[0], B.chunks[0], B.bins[0], B.small, B.counters, range, parent);
    cudaError_t e = cudaGetLastError();
    if (n <= kSahLeaves)
    {
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(out, perm, sizeof(uint32_t) * (size_t)n, cudaMemcpyDeviceToDevice, stream);
    }
    else
    {
        int binSM = 1, partSM = 1;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&binSM, k_top_bin, kTopBlock, 0);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&partSM, k_top_partition, kTopBlock, 0);
        // enough levels for SAH splits of ordinary scenes, then more at a time
        int batch = 4;
        for (int m = n; m > kSahLeaves; m >>= 1) ++batch;
        int level = 0;
        for (;;)
        {
            for (int l = 0; l < batch && e == cudaSuccess; ++l, ++level)
            {
                TopArgs a;
                a.n = n;
                a.triBox = triBox;
                a.src = level == 0 ? perm : B.order[(level - 1) & 1];
                a.dst = B.order[level & 1];
                a.out = out;
                a.tasks = B.task[level & 1];
                a.chunks = B.chunks[level & 1];
                a.nextTasks = B.task[(level + 1) & 1];
                a.nextChunks = B.chunks[(level + 1) & 1];
                a.count = B.counters + 2 + kTopCounts * (level & (kTopSlots - 1));
                a.nextCount = B.counters + 2 + kTopCounts * ((level + 1) & (kTopSlots - 1));
                a.clearCount = B.counters + 2 + kTopCounts * ((level + 2) & (kTopSlots - 1));
                a.splits = B.splits;
                a.bins = B.bins[level & 1];
                a.nextBins = B.bins[(level + 1) & 1];
                a.cum = B.cum;
                a.small = B.small;
                a.numSmall = B.counters;
                a.nodeCounter = B.counters + 1;
                a.child = child;
                a.range = range;
                a.parent = parent;
                const long long bound =
                    std::min<long long>(B.maxChunks, (long long)n / kTopChunk + 1 + (level < 30 ? 1ll << level : 1ll << 30));
                k_top_bin<<<(int)std::min<long long>(bound, (long long)binSM * numSMs), kTopBlock, 0, stream>>>(a);
                k_top_partition<<<(int)std::min<long long>(bound, (long long)partSM * numSMs), kTopBlock, 0, stream>>>(a);
                e = cudaGetLastError();
            }
            int numTasks = 0;
            if (e == cudaSuccess)
                e = cudaMemcpyAsync(&numTasks, B.counters + 2 + kTopCounts * (level & (kTopSlots - 1)), sizeof(int),
                                    cudaMemcpyDeviceToHost, stream);
            if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
            if (e != cudaSuccess || numTasks == 0) break;
            if (numTasks > B.maxTasks) return cudaErrorInvalidValue;
            batch = 8;
        }
    }
    if (e != cudaSuccess) return e;
    int perSM = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_sah_subtrees, 96, 0);
    k_sah_subtrees<<<std::max(1, perSM) * numSMs, 96, 0, stream>>>(n, B.small, B.counters, triBox, out, child, range,
                                                                parent, B.counters + 1, refit);
    return cudaGetLastError();
}


} // namespace prt_b200
