// Bounds and grouping costs of a binary tree node from its two children, for the
// passes that work bottom-up (bvh_build.cu, sah_build.cu; the dynamic program is
// described in bvh_build.cu).
#pragma once
#include <cfloat>

#include "prt_device.cuh"

namespace prt_b200 {

#ifndef PRT_WIDE_DP
#define PRT_WIDE_DP 1
#endif
#ifndef PRT_SAH_CTRI
#define PRT_SAH_CTRI 0.7f
#endif

__device__ __forceinline__ float box_half_area(const float* b)
{
    float dx = b[3] - b[0], dy = b[4] - b[1], dz = b[5] - b[2];
    return dx * dy + dy * dz + dz * dx;
}

struct RefitArgs
{
    int n;
    const uint32_t* vals;   // sorted triangle ids
    const float* triBox;    // 6 floats per triangle, by triangle id
    const int2* child;
    const int2* range;
    const int* parent;
    float* box;             // 6 floats per node: internal [0, n-1), leaves [n-1, 2n-1)
    int* flag;              // arrivals per internal node, zeroed
    float4* cost;           // kGroup: 2 float4 (C(u, 1..8)) per internal node
    uint2* dec;             // kGroup: 8 decision bytes per internal node
    int leafMax;
};

// C(child, 1..8) of a binary child: loaded for an internal node, its area x
// cTri for a single triangle.
__device__ __forceinline__ void child_costs(const RefitArgs& a, int ref, const float* b, float* c)
{
    if (ref < 0)
    {
        const float leafCost = box_half_area(b) * PRT_SAH_CTRI;
#pragma unroll
        for (int i = 0; i < 8; ++i) c[i] = leafCost;
        return;
    }
    const float4 lo = __ldcg(a.cost + 2 * (size_t)ref), hi = __ldcg(a.cost + 2 * (size_t)ref + 1);
    c[0] = lo.x; c[1] = lo.y; c[2] = lo.z; c[3] = lo.w;
    c[4] = hi.x; c[5] = hi.y; c[6] = hi.z; c[7] = hi.w;
}

// The box of a finished node or of a leaf.
__device__ __forceinline__ void load_box(const RefitArgs& a, int ref, float* b)
{
    const size_t i = ref >= 0 ? ref : (a.n - 1) + ~ref;
#pragma unroll
    for (int c = 0; c < 6; ++c) b[c] = __ldcg(a.box + 6 * i + c);
}

// Node `node` (children ch with boxes ba and bb, cnt triangles) from its two
// finished children: box, and with kGroup its grouping costs and decisions.
template <bool kGroup>
__device__ __forceinline__ void refit_node(const RefitArgs& a, int node, int2 ch, int cnt, const float* ba, const float* bb)
{
    float r[6];
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
        r[c] = fminf(ba[c], bb[c]);
        r[3 + c] = fmaxf(ba[3 + c], bb[3 + c]);
    }
#pragma unroll
    for (int c = 0; c < 6; ++c) __stcg(a.box + 6 * (size_t)node + c, r[c]);
    if (kGroup)
    {
        float ca[8], cb[8];
        child_costs(a, ch.x, ba, ca);
        child_costs(a, ch.y, bb, cb);
        const float area = box_half_area(r);
        float dist[8];
        uint8_t split[8];
        dist[0] = FLT_MAX;
        split[0] = 0;
#pragma unroll
        for (int i = 2; i <= 8; ++i)
        {
            float best = FLT_MAX;
            int bj = 1;
#pragma unroll
            for (int j = 1; j < i; ++j)
            {
                const float v = ca[j - 1] + cb[i - j - 1];
                if (v < best)
                {
                    best = v;
                    bj = j;
                }
            }
            dist[i - 1] = best;
            split[i - 1] = (uint8_t)bj;
        }
        const float leafOpt = cnt <= a.leafMax ? area * PRT_SAH_CTRI * (float)cnt : FLT_MAX;
        const float wideOpt = area + dist[7];
        float cs[8];
        float c = fminf(leafOpt, wideOpt);
        cs[0] = c;
        uint32_t d0 = leafOpt <= wideOpt ? 1u : 0u, d1 = 0;
#pragma unroll
        for (int i = 2; i <= 8; ++i)
        {
            uint32_t d = split[i - 1];
            if (c <= dist[i - 1]) d |= 0x80;
            else c = dist[i - 1];
            cs[i - 1] = c;
            if (i <= 4) d0 |= d << (8 * (i - 1));
            else d1 |= d << (8 * (i - 5));
        }
        __stcg(a.cost + 2 * (size_t)node, make_float4(cs[0], cs[1], cs[2], cs[3]));
        __stcg(a.cost + 2 * (size_t)node + 1, make_float4(cs[4], cs[5], cs[6], cs[7]));
        __stcg(a.dec + node, make_uint2(d0, d1));
    }
}

// Arrival at a node: the atomic increment releases this thread's writes (its
// child's box and costs) and, for the second arrival, acquires the sibling's.
__device__ __forceinline__ unsigned arrive(int* flag)
{
    unsigned old;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(flag) : "memory");
    return old;
}

} // namespace prt_b200
