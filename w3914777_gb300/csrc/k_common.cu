// k_common.cu -- utility kernels of libamps: tiered state <-> row-major
// arrays, the monitor on a resting state, tile classification with ordered
// per-tier work lists, and deterministic FP64 reductions.
#include "../../include/amps.h"
#include "amps_kernels.h"
#include "grid_view.cuh"

namespace amps {

// ---------------------------------------------------------------- state ----
__device__ __forceinline__ int tier_of(const Grid &g, int x, int y)
{
    return g.tier[(y / g.tile) * g.ntx + x / g.tile];
}

// storage index of domain cell (x, y) of field f
__device__ __forceinline__ int64_t store_index(const Grid &g, int f, int x, int y)
{
    return (int64_t)f * g.fs + (int64_t)y * g.px + x;
}

// c: index of the cell in the row-major domain array
__device__ __forceinline__ double read_cell(const Grid &g, int f, int64_t c)
{
    const int x = (int)(c % g.nx), y = (int)(c / g.nx);
    const int t = tier_of(g, x, y);
    const int64_t k = store_index(g, f, x, y);
    if (t == TIER_FP64) return ((const double *)g.store[2])[k];
    if (t == TIER_FP32) return (double)((const float *)g.store[1])[k];
    return (double)__half2float(((const __half *)g.store[0])[k]);
}

// Row-major [nf][ny][nx] arrays <-> the tiered storage, a CTA per tile and
// kXferFields fields: the tile's tier is one uniform branch, a thread moves
// four cells of a row with 16-byte accesses (V: rows of the array are 16-byte
// aligned) and no address takes a division per cell.  Bound by HBM: 2048^2 Q=8, cold,
// FP64 in 157 us (and an 80 us copy before it) with a division per cell and 8-byte
// accesses, 77 now; FP32 out 157, 40 now.
constexpr int kXferFields = 4;

template <typename S> __device__ __forceinline__ void put4(S *d, const double v[4], int n, bool vec)
{
    if (vec && n == 4) {
        if constexpr (sizeof(S) == 8) {
            reinterpret_cast<double2 *>(d)[0] = make_double2(v[0], v[1]);
            reinterpret_cast<double2 *>(d)[1] = make_double2(v[2], v[3]);
        } else {
            *reinterpret_cast<float4 *>(d) = make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
        }
        return;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (k < n) d[k] = (S)v[k];
}

// The storage of a ragged grid's edge tile reaches past the domain: zeros there.
template <int T, typename S>
__global__ void __launch_bounds__(256) scatter_kernel(Grid g, const S *__restrict__ src, bool vec)
{
    constexpr int TPT = T * T / 4, PER = 256 / TPT;
    const int tile = blockIdx.x, l = threadIdx.x % TPT;
    const int x = tile % g.ntx * T + l % (T / 4) * 4, y = tile / g.ntx * T + l / (T / 4);
    if (x >= g.nx || y >= g.ny) return;
    const int t = g.tier[tile], n = g.nx - x < 4 ? g.nx - x : 4;
#pragma unroll
    for (int j = threadIdx.x / TPT; j < kXferFields; j += PER) {
        const int f = blockIdx.y * kXferFields + j;
        if (f >= g.nf) break;
        const S *p = src + (int64_t)f * g.n + (int64_t)y * g.nx + x;
        const int64_t o = (int64_t)f * g.fs + (int64_t)y * g.px + x;
        S v[4] = {S(0), S(0), S(0), S(0)};
        if (vec && n == 4) {
            if constexpr (sizeof(S) == 8) {
                const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
                v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
            } else {
                const float4 a = *reinterpret_cast<const float4 *>(p);
                v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (k < n) v[k] = p[k];
        }
        if (t == TIER_FP64) {
            double2 *d = reinterpret_cast<double2 *>((double *)g.store[2] + o);
            d[0] = make_double2((double)v[0], (double)v[1]);
            d[1] = make_double2((double)v[2], (double)v[3]);
        } else if (t == TIER_FP32) {
            *reinterpret_cast<float4 *>((float *)g.store[1] + o) =
                make_float4((float)v[0], (float)v[1], (float)v[2], (float)v[3]);
        } else {
            const __half2 a = __floats2half2_rn((float)v[0], (float)v[1]), b = __floats2half2_rn((float)v[2], (float)v[3]);
            uint2 u;
            u.x = *reinterpret_cast<const unsigned *>(&a);
            u.y = *reinterpret_cast<const unsigned *>(&b);
            *reinterpret_cast<uint2 *>((__half *)g.store[0] + o) = u;
        }
    }
}

template <int T, typename S>
__global__ void __launch_bounds__(256) gather_kernel(Grid g, S *dst, int f0, int nfs, bool vec)
{
    constexpr int TPT = T * T / 4, PER = 256 / TPT;
    const int tile = blockIdx.x, l = threadIdx.x % TPT;
    const int x = tile % g.ntx * T + l % (T / 4) * 4, y = tile / g.ntx * T + l / (T / 4);
    if (x >= g.nx || y >= g.ny) return;
    const int t = g.tier[tile], n = g.nx - x < 4 ? g.nx - x : 4;
#pragma unroll
    for (int j = threadIdx.x / TPT; j < kXferFields; j += PER) {
        const int f = blockIdx.y * kXferFields + j;
        if (f >= nfs) break;
        const int64_t o = (int64_t)(f0 + f) * g.fs + (int64_t)y * g.px + x;
        S *p = dst + (int64_t)f * g.n + (int64_t)y * g.nx + x;
        if (sizeof(S) == 4 && t != TIER_FP64) {  // float to float: no FP64 conversion
            float v[4];
            load4f(g, t, o, v);
            if (vec && n == 4) {
                *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (k < n) p[k] = (S)v[k];
            }
            continue;
        }
        double v[4];
        load4d(g, t, o, v);
        put4(p, v, n, vec);
    }
}

template <typename S> static bool rows_aligned(const Grid &g, const void *p)
{
    return g.nx % (16 / (int)sizeof(S)) == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0;
}

template <typename S> static void scatter_t(const Grid &g, const void *src, cudaStream_t s)
{
    const dim3 grid(g.ntx * g.nty, (g.nf + kXferFields - 1) / kXferFields);
    const bool vec = rows_aligned<S>(g, src);
    if (g.tile == 32) scatter_kernel<32, S><<<grid, 256, 0, s>>>(g, (const S *)src, vec);
    else scatter_kernel<16, S><<<grid, 256, 0, s>>>(g, (const S *)src, vec);
}

template <typename S> static void gather_t(const Grid &g, void *dst, int f0, int nfs, cudaStream_t s)
{
    const dim3 grid(g.ntx * g.nty, (nfs + kXferFields - 1) / kXferFields);
    const bool vec = rows_aligned<S>(g, dst);
    if (g.tile == 32) gather_kernel<32, S><<<grid, 256, 0, s>>>(g, (S *)dst, f0, nfs, vec);
    else gather_kernel<16, S><<<grid, 256, 0, s>>>(g, (S *)dst, f0, nfs, vec);
}

cudaError_t scatter_fields(const Grid &g, const void *src, int src_f32, cudaStream_t s)
{
    if (src_f32) scatter_t<float>(g, src, s);
    else scatter_t<double>(g, src, s);
    return cudaGetLastError();
}

cudaError_t gather_fields(const Grid &g, void *dst, int dst_f32, int f0, int nfs, cudaStream_t s)
{
    if (dst_f32) gather_t<float>(g, dst, f0, nfs, s);
    else gather_t<double>(g, dst, f0, nfs, s);
    return cudaGetLastError();
}

__global__ void fill_kernel(double *p, int n, double v)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = v;
}

cudaError_t fill_doubles(double *p, int n, double v, cudaStream_t s)
{
    fill_kernel<<<(n + 1023) / 1024 < 152 ? (n + 1023) / 1024 : 152, 256, 0, s>>>(p, n, v);
    return cudaGetLastError();
}

// ------------------------------------------------------ resting monitor ----
// One CTA per tile, a warp per field: the spatial metric of the current state,
// and/or the temporal snapshot (same lattice and slots as the fused epilogues).
// diff: the temporal metric against snap (max |state - snap|, the fused
// temporal monitor's reduction) in place of the range.  Half and FP32 tiles
// reduce in float (exact; the range is formed in double).  1024^2 Q=8 FP32, cold: 191 us with a
// block reduction per field in double, 22 now; sintering's 17 FP64 fields: 396 and 101.
template <int T>
__global__ void __launch_bounds__(kThreads) monitor_state_kernel(Grid g, int kind, int samples, int mfield,
                                                                 double *metric, double *snap, int write_snap,
                                                                 int *flags, int diff)
{
    __shared__ double red[kThreads / 32];
    constexpr int NV = T * T / 4;  // four-cell groups of a tile
    const int tile = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int x0 = tile % g.ntx * T, y0 = tile / g.ntx * T, tier = g.tier[tile];
    // a ragged grid's edge tile: only its cells inside the domain
    const int vw = min(T, g.nx - x0), vh = min(T, g.ny - y0);
    double result = 0.0;
    bool bad = false;
    for (int f = warp; f < g.nf; f += kThreads / 32) {
        if (mfield >= 0 && f != mfield) continue;
        const int slot = mfield < 0 ? f : 0;
        const int64_t fo = (int64_t)f * g.fs;
        double mn = samples ? INFINITY : 1.0, mx = samples && !diff ? -INFINITY : 0.0;
        float mnf = INFINITY, mxf = -INFINITY;
#pragma unroll 4
        for (int u = lane; u < NV; u += 32) {
            const int j = u / (T / 4), i = u % (T / 4) * 4;
            if (j >= vh || i >= vw) continue;
            const int64_t sc = (int64_t)(y0 + j) * g.px + x0 + i;  // snapshot slot: storage layout
            if (tier != TIER_FP64 && !(samples && (diff || write_snap))) {
                float v[4];
                load4f(g, tier, fo + sc, v);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (i + k < vw) {
                        bad |= !(fabsf(v[k]) < INFINITY);
                        mnf = fminf(mnf, v[k]);
                        mxf = fmaxf(mxf, v[k]);
                    }
                continue;
            }
            double v[4];
            load4d(g, tier, fo + sc, v);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if (i + k >= vw) continue;
                bad |= (__double2hiint(v[k]) & 0x7ff00000) == 0x7ff00000;
                if (!samples) continue;
                if (diff) {
                    mx = fmax(mx, fabs(snap[(int64_t)slot * g.fs + sc + k] - v[k]));
                    continue;
                }
                mn = fmin(mn, v[k]);
                mx = fmax(mx, v[k]);
                if (write_snap) snap[(int64_t)slot * g.fs + sc + k] = v[k];
            }
        }
        if (samples && tier != TIER_FP64 && !diff && !write_snap) {
            mn = (double)mnf;
            mx = (double)mxf;
        }
        if (!samples && lane < 16) {  // the 4x4 lattice
            const int pr = lane / 4, pc = lane % 4;
            const int j = kind == 1 ? (pr * (T - 1) * 2 + 3) / 6 : T / 8 + pr * (T / 4);
            const int i = kind == 1 ? (pc * (T - 1) * 2 + 3) / 6 : T / 8 + pc * (T / 4);
            if (i < vw && j < vh) {
                const double v = load1d(g, tier, fo + (int64_t)(y0 + j) * g.px + x0 + i);
                double *sp = snap + ((int64_t)slot * g.ntx * g.nty + tile) * 16 + lane;
                if (diff) {
                    mx = fmax(mx, fabs(*sp - v));
                } else {
                    mn = fmin(mn, v);
                    mx = fmax(mx, v);
                    if (write_snap) *sp = v;
                }
            }
        }
        mx = warp_max(mx);
        mn = warp_min(mn);
        result = fmax(result, diff ? mx : mx - mn);
    }
    if (lane == 0) red[warp] = result;
    if (__syncthreads_or(bad) && threadIdx.x == 0) atomicOr(flags, 1);
    if (threadIdx.x == 0 && metric) {
        for (int w = 1; w < kThreads / 32; ++w) result = fmax(result, red[w]);
        metric[tile] = result;
    }
}

cudaError_t monitor_state(const Grid &g, int kind, int samples, int mfield, double *metric, double *snap,
                          int write_snap, int *flags, cudaStream_t s, int diff)
{
    const int n = g.ntx * g.nty;
    if (g.tile == 32)
        monitor_state_kernel<32><<<n, kThreads, 0, s>>>(g, kind, samples, mfield, metric, snap, write_snap, flags, diff);
    else
        monitor_state_kernel<16><<<n, kThreads, 0, s>>>(g, kind, samples, mfield, metric, snap, write_snap, flags, diff);
    return cudaGetLastError();
}

// ------------------------------------------------------------ classify ----
// Inclusive scan of 64-bit packed counters over a 1024-thread block.
__device__ __forceinline__ unsigned long long block_scan(unsigned long long v, unsigned long long *ws)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) ws[w] = v;
    __syncthreads();
    if (w == 0) {
        unsigned long long t = lane < (int)(blockDim.x >> 5) ? ws[lane] : 0ull;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long u = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += u;
        }
        ws[lane] = t;
    }
    __syncthreads();
    const unsigned long long r = v + (w > 0 ? ws[w - 1] : 0ull);
    __syncthreads();
    return r;
}

// Inclusive scan of two 64-bit packed counters at once (the barriers of one
// scan); *ta, *tb: the block's totals.
__device__ __forceinline__ void block_scan2(unsigned long long &a, unsigned long long &b, unsigned long long *ws,
                                            unsigned long long *ta, unsigned long long *tb)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long ua = __shfl_up_sync(0xffffffffu, a, o);
        const unsigned long long ub = __shfl_up_sync(0xffffffffu, b, o);
        if (lane >= o) {
            a += ua;
            b += ub;
        }
    }
    if (lane == 31) {
        ws[w] = a;
        ws[32 + w] = b;
    }
    __syncthreads();
    if (w == 0) {
        unsigned long long sa = lane < nw ? ws[lane] : 0ull, sb = lane < nw ? ws[32 + lane] : 0ull;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long ua = __shfl_up_sync(0xffffffffu, sa, o);
            const unsigned long long ub = __shfl_up_sync(0xffffffffu, sb, o);
            if (lane >= o) {
                sa += ua;
                sb += ub;
            }
        }
        ws[lane] = sa;
        ws[32 + lane] = sb;
    }
    __syncthreads();
    if (w > 0) {
        a += ws[w - 1];
        b += ws[32 + w - 1];
    }
    *ta = ws[nw - 1];
    *tb = ws[32 + nw - 1];
    __syncthreads();
}

// Ordered compaction of the tiles of each tier (tier maps are small: one
// 1024-thread CTA loops over them).
__device__ void lists_from_tiers(const uint8_t *tier, int ntiles, int *lists, int *counts, unsigned long long *ws)
{
    __shared__ unsigned long long base;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    for (int t0 = 0; t0 < ntiles; t0 += blockDim.x) {
        const int t = t0 + threadIdx.x;
        const int k = t < ntiles ? tier[t] : -1;
        const unsigned long long mine = k >= 0 ? (1ull << (21 * k)) : 0ull;
        const unsigned long long inc = block_scan(mine, ws);
        const unsigned long long b = base;
        if (k >= 0) {
            const unsigned long long excl = b + inc - mine;
            const int rank = (int)((excl >> (21 * k)) & AMPS_MAX_TILES);
            lists[k * ntiles + rank] = t;
        }
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) base = b + inc;
        __syncthreads();
    }
    if (threadIdx.x < 3) counts[threadIdx.x] = (int)((base >> (21 * threadIdx.x)) & AMPS_MAX_TILES);
}

// The per-tier tile lists and counts, and the launch order of the fused
// grain-growth step: first the tiles that take its slow paths -- FP64 or half
// tiles, and FP32 tiles with a neighbour (after the boundary map) at another
// tier, which stage their neighbourhood with conversions -- then the all-FP32
// neighbourhoods, each group in tile order.  Slow tiles then run in the first
// wave, where their extra time is absorbed, instead of straggling at the end
// of the step.  Scheduling only: every tile is computed by exactly one CTA
// either way.  A thread ranks a tile, or in larger maps a run of consecutive
// tiles, so one scan of two
// packed counters -- the tier ranks, and the slow (low 32 bits) / all-FP32
// (high 32 bits) ranks -- serves maps of any size: a 4096-tile map's
// classification, cold, 27 us with a scan per 1024 tiles and list, 19 now.
__device__ void lists_and_order(const ClassifyArgs &c, const uint8_t *tier, unsigned long long *ws)
{
    const int ntiles = c.ntx * c.nty;
    auto slow_at = [&](int t) {
        const int x = t % c.ntx, y = t / c.ntx;
        bool slow = false;
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx) {
                int yy = y + dy, xx = x + dx;
                if (c.bc == 0) {
                    yy = yy < 0 ? yy + c.nty : (yy >= c.nty ? yy - c.nty : yy);
                    xx = xx < 0 ? xx + c.ntx : (xx >= c.ntx ? xx - c.ntx : xx);
                } else {
                    yy = yy < 0 ? 0 : (yy >= c.nty ? c.nty - 1 : yy);
                    xx = xx < 0 ? 0 : (xx >= c.ntx ? c.ntx - 1 : xx);
                }
                slow |= tier[yy * c.ntx + xx] != TIER_FP32;
            }
        return slow;
    };
    if (ntiles <= (int)blockDim.x) {  // a tile a thread
        const int t = threadIdx.x, k = t < ntiles ? tier[t] : -1;
        const bool slow = k >= 0 && slow_at(t);
        const unsigned long long ma = k >= 0 ? (1ull << (21 * k)) : 0ull;
        const unsigned long long mb = k >= 0 ? (slow ? 1ull : (1ull << 32)) : 0ull;
        unsigned long long a = ma, b = mb, ta, tb;
        block_scan2(a, b, ws, &ta, &tb);
        if (k >= 0) {
            const unsigned long long ea = a - ma, eb = b - mb;
            c.lists[k * ntiles + (int)((ea >> (21 * k)) & AMPS_MAX_TILES)] = t;
            c.order[slow ? (int)(eb & 0xFFFFFFFFull) : (int)(tb & 0xFFFFFFFFull) + (int)(eb >> 32)] = t;
        }
        if (t < 3) c.counts[t] = (int)((ta >> (21 * t)) & AMPS_MAX_TILES);
        return;
    }
    const int per = (ntiles + (int)blockDim.x - 1) / (int)blockDim.x;
    const int t0 = min((int)threadIdx.x * per, ntiles), t1 = min(t0 + per, ntiles);
    unsigned long long ma = 0, mb = 0, slows = 0;  // slows: bit i, tile t0 + i (the first 64 of the run)
    for (int t = t0; t < t1; ++t) {
        const bool slow = slow_at(t);
        if (t - t0 < 64) slows |= (unsigned long long)slow << (t - t0);
        ma += 1ull << (21 * tier[t]);
        mb += slow ? 1ull : (1ull << 32);
    }
    unsigned long long a = ma, b = mb, ta, tb;
    block_scan2(a, b, ws, &ta, &tb);
    unsigned long long ea = a - ma, eb = b - mb;
    const int nslow = (int)(tb & 0xFFFFFFFFull);
    for (int t = t0; t < t1; ++t) {
        const int k = tier[t];
        const bool slow = t - t0 < 64 ? (slows >> (t - t0) & 1ull) != 0ull : slow_at(t);
        c.lists[k * ntiles + (int)((ea >> (21 * k)) & AMPS_MAX_TILES)] = t;
        c.order[slow ? (int)(eb & 0xFFFFFFFFull) : nslow + (int)(eb >> 32)] = t;
        ea += 1ull << (21 * k);
        eb += slow ? 1ull : (1ull << 32);
    }
    if (threadIdx.x < 3) c.counts[threadIdx.x] = (int)((ta >> (21 * threadIdx.x)) & AMPS_MAX_TILES);
}

// Tier maps of up to this many tiles are also kept in the classifying CTA's
// shared memory, so that the lists, the launch order and the log read them
// there instead of from global memory.
constexpr int kClassifyShared = 8192;

__device__ void classify_body(const ClassifyArgs &c)
{
    __shared__ unsigned long long ws[64];
    __shared__ int prom, dem;
    __shared__ uint8_t s_tier[kClassifyShared];
    const int ntiles = c.ntx * c.nty;
    const bool in_smem = ntiles <= kClassifyShared;
    if (threadIdx.x == 0) {
        for (int k = 0; k < 3; ++k) c.stats[k] += (unsigned long long)c.counts[k] * (unsigned long long)c.stat_steps;
        c.stats[3] += 1;
        *c.step_base += c.advance;
        prom = 0;
        dem = 0;
    }
    __syncthreads();
    int np = 0, nd = 0;
    for (int t = threadIdx.x; t < ntiles; t += blockDim.x) {
        const int x = t % c.ntx, y = t / c.ntx;
        double m = c.metric[t];
        if (y < c.nty - 1) m = fmax(m, c.metric[t + c.ntx]);
        if (y > 0) m = fmax(m, c.metric[t - c.ntx]);
        if (x < c.ntx - 1) m = fmax(m, c.metric[t + 1]);
        if (x > 0) m = fmax(m, c.metric[t - 1]);
        // NaN metric (a NaN in the tile) promotes: fmax drops NaN, so test the tile's own
        const bool nan = !(c.metric[t] == c.metric[t]);
        int nt;
        if (nan || m >= c.thr_hi) nt = c.high_tier;
        else if (c.use_mid && m >= c.thr_lo) nt = TIER_FP32;
        else nt = TIER_HALF;
        if (c.sched) nt = c.sched[(int64_t)min(*c.sched_i, c.sched_n - 1) * ntiles + t];
        const int old = c.tier_cur[t];
        c.tier_prev[t] = (uint8_t)old;
        c.tier_cur[t] = (uint8_t)nt;
        if (in_smem) s_tier[t] = (uint8_t)nt;
        np += nt > old;
        nd += nt < old;
    }
    atomicAdd(&prom, np);
    atomicAdd(&dem, nd);
    __syncthreads();
    const uint8_t *tier = in_smem ? s_tier : c.tier_cur;
    lists_and_order(c, tier, ws);
    if (threadIdx.x == 0) {
        c.stats[4] += prom;
        c.stats[5] += dem;
        if (c.sched) *c.sched_i += 1;  // every thread read it before the barriers above
    }
    if (c.log && c.max_log > 0) {
        const int n = *c.log_n;
        __syncthreads();
        if (n < c.max_log) {
            for (int t = threadIdx.x; t < ntiles; t += blockDim.x) c.log[(int64_t)n * ntiles + t] = tier[t];
            if (threadIdx.x == 0) *c.log_n = n + 1;
        }
    }
}

// Launched with programmatic dependent launch after the period's last step:
// its launch overlaps that step's tail, and the next step's launch overlaps
// it; it waits for the step (and its writes) before reading the metric.
__global__ void __launch_bounds__(1024) classify_kernel(ClassifyArgs c)
{
    pdl_trigger();
    pdl_wait();
    classify_body(c);
}

// One CTA per ensemble member; member b's arguments are cs[b].
__global__ void __launch_bounds__(1024) classify_batch_kernel(const ClassifyArgs *cs) { classify_body(cs[blockIdx.x]); }

cudaError_t classify(const ClassifyArgs &c, cudaStream_t s)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(1024);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, classify_kernel, c);
}

cudaError_t classify_batch(const ClassifyArgs *cs, int count, cudaStream_t s)
{
    classify_batch_kernel<<<count, 1024, 0, s>>>(cs);
    return cudaGetLastError();
}

__global__ void __launch_bounds__(1024) build_lists_kernel(const uint8_t *tier, int ntiles, int *lists, int *counts)
{
    __shared__ unsigned long long ws[32];
    lists_from_tiers(tier, ntiles, lists, counts, ws);
}

// graingrowth/function.h:38-39,68-73 (and snowflake/function.h:69-70,106-113):
// at every 10th step the update kernel copies the monitored field into the
// snapshot, but a low tile's second 8-column block returns before the copy,
// so its samples in columns 10 and 14 keep the value of the last step at
// which the tile was high.  Here the monitor step's epilogue has written the
// whole lattice (the state the classification just judged); this puts the
// earlier values back where the reference keeps them.  keep holds the
// snapshot as it stood after the previous classification.
__global__ void snap_ref_kernel(double *snap, double *keep, const uint8_t *tier, int ntiles, int total)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const int si = i % 16, t = (i / 16) % ntiles;
    if (tier[t] == TIER_HALF && (si % 4) >= 2) snap[i] = keep[i];
    keep[i] = snap[i];
}

cudaError_t snap_ref_fixup(double *snap, double *keep, const uint8_t *tier, int ntiles, int nmon, cudaStream_t s)
{
    const int total = nmon * ntiles * 16;
    snap_ref_kernel<<<(total + 255) / 256, 256, 0, s>>>(snap, keep, tier, ntiles, total);
    return cudaGetLastError();
}

cudaError_t build_lists(const uint8_t *tier, int ntiles, int *lists, int *counts, cudaStream_t s)
{
    build_lists_kernel<<<1, 1024, 0, s>>>(tier, ntiles, lists, counts);
    return cudaGetLastError();
}

__global__ void advance_kernel(int64_t *step_base, int advance, int stat_steps, const int *counts,
                               unsigned long long *stats)
{
    for (int k = 0; k < 3; ++k) stats[k] += (unsigned long long)counts[k] * (unsigned long long)stat_steps;
    *step_base += advance;
}

cudaError_t advance_period(int64_t *step_base, int advance, int stat_steps, const int *counts,
                           unsigned long long *stats, cudaStream_t s)
{
    advance_kernel<<<1, 1, 0, s>>>(step_base, advance, stat_steps, counts, stats);
    return cudaGetLastError();
}

// Period bookkeeping of every ensemble member without a classification
// (one thread per member; advance and stat_steps from each member's args).
__global__ void advance_batch_kernel(const ClassifyArgs *cs, int count)
{
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= count) return;
    const ClassifyArgs &c = cs[b];
    for (int k = 0; k < 3; ++k) c.stats[k] += (unsigned long long)c.counts[k] * (unsigned long long)c.stat_steps;
    *c.step_base += c.advance;
}

cudaError_t advance_batch(const ClassifyArgs *cs, int count, cudaStream_t s)
{
    advance_batch_kernel<<<(count + 127) / 128, 128, 0, s>>>(cs, count);
    return cudaGetLastError();
}

// ---------------------------------------------------------- reductions ----
constexpr int kRedBlocks = 1024;

template <int KIND> __device__ __forceinline__ double fold(double a, double b)
{
    return KIND == 1 ? fmin(a, b) : (KIND == 2 ? fmax(a, b) : a + b);
}

// The block's fold of acc in a fixed shape (thread 0 has it): deterministic.
template <int KIND> __device__ __forceinline__ double block_fold(double acc, double none, double *red)
{
    constexpr int NW = kThreads / 32;
    for (int o = 16; o > 0; o >>= 1) acc = fold<KIND>(acc, __shfl_xor_sync(0xffffffffu, acc, o));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        acc = threadIdx.x < NW ? red[threadIdx.x] : none;
        for (int o = NW / 2; o > 0; o >>= 1) acc = fold<KIND>(acc, __shfl_xor_sync(0xffffffffu, acc, o));
    }
    return acc;
}

// One launch: each block folds its tiles in a fixed order, the last one to
// finish folds the blocks' partials (out may be page-locked host memory).
// Bound by the read of the field and the FP64 pipe's share of it (a conversion
// and an addition a cell), so few blocks that loop: every block's tree costs
// its threads five FP64 operations.  1024^2 FP32, cold: 91 us as two launches
// with one thread folding the partials, 12 now.
template <int T, int KIND>
__global__ void __launch_bounds__(kThreads) reduce_kernel(Grid g, int field, double *partials, unsigned *counter,
                                                          double *out)
{
    __shared__ double red[kThreads / 32];
    constexpr int TPT = T * T / 4, PER = kThreads / TPT;  // threads a tile, tiles a block at a time
    const int l = threadIdx.x % TPT;
    const double none = KIND == 1 ? INFINITY : (KIND == 2 ? -INFINITY : 0.0);
    double acc = none;
#pragma unroll 2
    for (int t = blockIdx.x * PER + threadIdx.x / TPT; t < g.ntx * g.nty; t += gridDim.x * PER) {
        const int x = t % g.ntx * T + l % (T / 4) * 4, y = t / g.ntx * T + l / (T / 4);
        if (x >= g.nx || y >= g.ny) continue;
        double v[4];
        load4d(g, g.tier[t], (int64_t)field * g.fs + (int64_t)y * g.px + x, v);
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (x + k < g.nx) acc = KIND == 3 ? fma(v[k], v[k], acc) : fold<KIND>(acc, v[k]);
    }
    acc = block_fold<KIND>(acc, none, red);
    if (threadIdx.x == 0) partials[blockIdx.x] = acc;
    if (!last_block(counter)) return;
    acc = none;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += kThreads) acc = fold<KIND>(acc, __ldcg(partials + k));
    acc = block_fold<KIND>(acc, none, red);
    if (threadIdx.x == 0) *out = acc;
}

template <int T>
static cudaError_t reduce_t(const Grid &g, int field, int kind, double *partials, unsigned *counter, double *out,
                            cudaStream_t s)
{
    constexpr int per = T == 32 ? 1 : 4;
    const int n = (g.ntx * g.nty + per - 1) / per, blocks = n < 304 ? n : 304;
    switch (kind) {
    case 0: reduce_kernel<T, 0><<<blocks, kThreads, 0, s>>>(g, field, partials, counter, out); break;
    case 1: reduce_kernel<T, 1><<<blocks, kThreads, 0, s>>>(g, field, partials, counter, out); break;
    case 2: reduce_kernel<T, 2><<<blocks, kThreads, 0, s>>>(g, field, partials, counter, out); break;
    default: reduce_kernel<T, 3><<<blocks, kThreads, 0, s>>>(g, field, partials, counter, out); break;
    }
    return cudaGetLastError();
}

cudaError_t reduce_field(const Grid &g, int field, int kind, double *partials, unsigned *counter, double *out,
                         cudaStream_t s)
{
    return g.tile == 32 ? reduce_t<32>(g, field, kind, partials, counter, out, s)
                        : reduce_t<16>(g, field, kind, partials, counter, out, s);
}

__global__ void compare_partial_kernel(Grid g, int field, const double *other, double *partials)
{
    __shared__ double red[8];
    double mx = 0.0, ss = 0.0;
    const int64_t chunk = (g.n + gridDim.x - 1) / gridDim.x;
    const int64_t lo = blockIdx.x * chunk, hi = min(g.n, lo + chunk);
    for (int64_t c = lo + threadIdx.x; c < hi; c += blockDim.x) {
        const double d = read_cell(g, field, c) - other[c];
        mx = (fabs(d) > mx || !(d == d)) ? fabs(d) : mx;
        ss += d * d;
    }
    mx = block_max(mx, red);
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += red[w];
        partials[2 * blockIdx.x] = mx;
        partials[2 * blockIdx.x + 1] = t;
    }
}

__global__ void compare_final_kernel(const double *partials, int np, int64_t n, double *out2)
{
    if (threadIdx.x != 0) return;
    double mx = 0.0, ss = 0.0;
    for (int k = 0; k < np; ++k) {
        mx = fmax(mx, partials[2 * k]);
        ss += partials[2 * k + 1];
    }
    out2[0] = mx;
    out2[1] = sqrt(ss / (double)n);
}

cudaError_t compare_field(const Grid &g, int field, const double *other, double *partials, double *out2,
                          cudaStream_t s)
{
    compare_partial_kernel<<<kRedBlocks, kThreads, 0, s>>>(g, field, other, partials);
    compare_final_kernel<<<1, 32, 0, s>>>(partials, kRedBlocks, g.n, out2);
    return cudaGetLastError();
}

}  // namespace amps
