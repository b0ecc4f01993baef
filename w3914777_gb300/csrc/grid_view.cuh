// grid_view.cuh -- reading the tiered state tile by tile (diagnostics,
// reductions, the resting monitor): a tile has one tier, so the branch on it
// is uniform, addresses need no division per cell, and a thread takes four
// consecutive cells in one or two 16-byte loads.
#pragma once
#include "amps_kernels.h"

namespace amps {

__device__ __forceinline__ int tile_tier(const Grid &g, int x, int y) { return g.tier[(y / g.tile) * g.ntx + x / g.tile]; }

// Four cells at storage offset o (a multiple of 4) of a half or FP32 tile.
__device__ __forceinline__ void load4f(const Grid &g, int tier, int64_t o, float v[4])
{
    if (tier == TIER_FP32) {
        const float4 q = __ldg(reinterpret_cast<const float4 *>((const float *)g.store[TIER_FP32] + o));
        v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    } else {
        const uint2 u = __ldg(reinterpret_cast<const uint2 *>((const __half *)g.store[TIER_HALF] + o));
        const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&u.x));
        const float2 b = __half22float2(*reinterpret_cast<const __half2 *>(&u.y));
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
}

// ... of a tile of any tier, as doubles.
__device__ __forceinline__ void load4d(const Grid &g, int tier, int64_t o, double v[4])
{
    if (tier == TIER_FP64) {
        const double2 *p = reinterpret_cast<const double2 *>((const double *)g.store[TIER_FP64] + o);
        const double2 a = __ldg(p), b = __ldg(p + 1);
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    } else {
        float f[4];
        load4f(g, tier, o, f);
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = (double)f[k];
    }
}

// One cell.
__device__ __forceinline__ float load1f(const Grid &g, int tier, int64_t o)
{
    if (tier == TIER_FP32) return __ldg((const float *)g.store[TIER_FP32] + o);
    return __half2float(__ushort_as_half(__ldg((const unsigned short *)g.store[TIER_HALF] + o)));
}
__device__ __forceinline__ double load1d(const Grid &g, int tier, int64_t o)
{
    return tier == TIER_FP64 ? __ldg((const double *)g.store[TIER_FP64] + o) : (double)load1f(g, tier, o);
}

// v >= level for the float v of a half or FP32 tile and a double level is
// v >= level_f, the smallest float not below the level: no FP64 operation.
struct Level {
    double d;
    float f;
    template <typename D> __device__ explicit Level(D l) : d(l), f(__double2float_ru(l)) {}
};

// The last block of a launch to arrive here (every thread of the block gets
// the answer; what the blocks wrote before is visible to it).  *counter is
// zero before the launch and again after it.
__device__ __forceinline__ bool last_block(unsigned *counter)
{
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicInc(counter, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    __threadfence();
    return last;
}

}  // namespace amps
