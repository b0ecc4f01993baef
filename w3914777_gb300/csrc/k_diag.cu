// k_diag.cu -- microstructure diagnostics, read straight from the tiered state
// (no gathered copy), all deterministic (integer counts, or fixed-order FP64
// partials):
//  * level-set interface: area, edge-count perimeter and bounding box of
//    {f >= level} (Kobayashi dendrite extent and tip positions);
//  * grains: connected components (4-neighbour, through periodic wraps) of
//    cells labelled by the dominant order parameter argmax_k eta_k where
//    max_k eta_k >= threshold -- grain count, labelled cells, mean area;
//  * grain-boundary length between every pair of labels (grain growth:
//    boundary network; sintering: neck widths, with cells labelled only where
//    the concentration c >= level).
// No reference counterpart: the reference's analysis scripts compare fields
// only (mean absolute error, graingrowth/end2enderror.py:34, which
// amps_compare_all also reports).
#include "amps_internal.cuh"
#include "amps_kernels.h"
#include "grid_view.cuh"

#include <algorithm>

namespace amps {

namespace {

constexpr int kDT = 256;

__device__ __forceinline__ int wrap_or_out(int i, int n, int bc)
{
    if (i >= 0 && i < n) return i;
    if (bc == 0) return i < 0 ? i + n : i - n;
    return -1;  // zero-flux: no neighbour outside the domain
}

// One cell's f >= level, and four cells' as a mask (offsets as in load4f).
__device__ __forceinline__ bool ge1(const Grid &g, int f, int x, int y, const Level &lv)
{
    const int t = tile_tier(g, x, y);
    const int64_t o = (int64_t)f * g.fs + (int64_t)y * g.px + x;
    return t == TIER_FP64 ? load1d(g, t, o) >= lv.d : load1f(g, t, o) >= lv.f;
}
__device__ __forceinline__ unsigned ge4(const Grid &g, int t, int64_t o, const Level &lv)
{
    unsigned m = 0;
    if (t == TIER_FP64) {
        double v[4];
        load4d(g, t, o, v);
#pragma unroll
        for (int k = 0; k < 4; ++k) m |= (unsigned)(v[k] >= lv.d) << k;
    } else {
        float v[4];
        load4f(g, t, o, v);
#pragma unroll
        for (int k = 0; k < 4; ++k) m |= (unsigned)(v[k] >= lv.f) << k;
    }
    return m;
}

// Level set of one field: cells, edges towards the right and lower neighbours,
// bounding box.  A thread holds four cells as a bit mask; the right neighbour of
// the last comes from the next lane, or across the tile's edge.  1024^2,
// cold: 75 us with a gathered copy of the fields and box atomics per cell, 13 now.
template <int T>
__global__ void __launch_bounds__(kDT) interface_kernel(Grid g, int field, int bc, double level,
                                                        unsigned long long *part, unsigned *counter,
                                                        unsigned long long *out)
{
    constexpr int TPT = T * T / 4, PER = kDT / TPT, GPR = T / 4;
    __shared__ unsigned long long scnt[3][kDT / 32];
    __shared__ int sbox[4][kDT / 32];
    const Level lv(level);
    const int l = threadIdx.x % TPT, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned in = 0, ex = 0, ey = 0;
    int x0 = 0x7fffffff, x1 = -1, y0 = 0x7fffffff, y1 = -1;
    for (int t = blockIdx.x * PER + threadIdx.x / TPT; t < g.ntx * g.nty; t += gridDim.x * PER) {
        const int tx = t % g.ntx, ty = t / g.ntx;
        const int x = tx * T + l % GPR * 4, y = ty * T + l / GPR;
        const bool dom = x < g.nx && y < g.ny;
        const unsigned valid = dom ? (g.nx - x >= 4 ? 15u : (1u << (g.nx - x)) - 1u) : 0u;
        const int64_t fo = (int64_t)field * g.fs;
        const unsigned own = dom ? ge4(g, g.tier[t], fo + (int64_t)y * g.px + x, lv) & valid : 0u;
        const unsigned next = __shfl_down_sync(0xffffffffu, own, 1);
        if (!dom) continue;
        unsigned right = own >> 1, rvalid = valid >> 1;  // bit k: the neighbour x + k + 1
        const int n = g.nx - x < 4 ? g.nx - x : 4;       // cells here
        const int xr = wrap_or_out(x + n, g.nx, bc);
        if (xr >= 0) {
            const bool r = x + n < g.nx && l % GPR != GPR - 1 ? (next & 1u) != 0u : ge1(g, field, xr, y, lv);
            right |= (unsigned)r << (n - 1);
            rvalid |= 1u << (n - 1);
        }
        ex += __popc((own ^ right) & rvalid);
        const int yd = wrap_or_out(y + 1, g.ny, bc);
        if (yd >= 0)
            ey += __popc((own ^ ge4(g, g.tier[yd / T * g.ntx + tx], fo + (int64_t)yd * g.px + x, lv)) & valid);
        if (own) {
            in += __popc(own);
            x0 = min(x0, x + __ffs(own) - 1);
            x1 = max(x1, x + 31 - __clz(own));
            y0 = min(y0, y);
            y1 = max(y1, y);
        }
    }
    auto block = [&]() {  // the block's counts and box in slot 0 of each shared array
        __syncthreads();
        if (warp == 0) {
            constexpr int NW = kDT / 32;
            unsigned long long c[3];
            for (int k = 0; k < 3; ++k) {
                c[k] = lane < NW ? scnt[k][lane] : 0ull;
                for (int o = NW / 2; o > 0; o >>= 1) c[k] += __shfl_xor_sync(0xffffffffu, c[k], o);
            }
            const int a = __reduce_min_sync(0xffffffffu, lane < NW ? sbox[0][lane] : 0x7fffffff);
            const int b = __reduce_max_sync(0xffffffffu, lane < NW ? sbox[1][lane] : -1);
            const int d = __reduce_min_sync(0xffffffffu, lane < NW ? sbox[2][lane] : 0x7fffffff);
            const int e = __reduce_max_sync(0xffffffffu, lane < NW ? sbox[3][lane] : -1);
            __syncwarp();
            if (lane == 0) {
                for (int k = 0; k < 3; ++k) scnt[k][0] = c[k];
                sbox[0][0] = a; sbox[1][0] = b; sbox[2][0] = d; sbox[3][0] = e;
            }
        }
        __syncthreads();
    };
    auto put = [&](unsigned long long a, unsigned long long b, unsigned long long c) {  // this warp's
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
            c += __shfl_xor_sync(0xffffffffu, c, o);
        }
        const int p = __reduce_min_sync(0xffffffffu, x0), q = __reduce_max_sync(0xffffffffu, x1);
        const int r = __reduce_min_sync(0xffffffffu, y0), s = __reduce_max_sync(0xffffffffu, y1);
        __syncthreads();
        if (lane == 0) {
            scnt[0][warp] = a; scnt[1][warp] = b; scnt[2][warp] = c;
            sbox[0][warp] = p; sbox[1][warp] = q; sbox[2][warp] = r; sbox[3][warp] = s;
        }
        block();
    };
    put(in, ex, ey);
    if (threadIdx.x < 7)
        part[blockIdx.x * 7 + threadIdx.x] = threadIdx.x < 3 ? scnt[threadIdx.x][0]
                                                             : (unsigned long long)(long long)sbox[threadIdx.x - 3][0];
    if (!last_block(counter)) return;
    unsigned long long a = 0, b = 0, c = 0;
    x0 = y0 = 0x7fffffff;
    x1 = y1 = -1;
    for (int k = threadIdx.x; k < (int)gridDim.x; k += kDT) {
        const unsigned long long *p = part + k * 7;
        a += __ldcg(p);
        b += __ldcg(p + 1);
        c += __ldcg(p + 2);
        x0 = min(x0, (int)__ldcg(p + 3));
        x1 = max(x1, (int)__ldcg(p + 4));
        y0 = min(y0, (int)__ldcg(p + 5));
        y1 = max(y1, (int)__ldcg(p + 6));
    }
    put(a, b, c);
    if (threadIdx.x < 7)
        out[threadIdx.x] = threadIdx.x < 3 ? scnt[threadIdx.x][0]
                                           : (unsigned long long)(long long)sbox[threadIdx.x - 3][0];
}

// Labels of N consecutive cells (N = 4: at an offset that is a multiple of 4):
// argmax_k eta_k (fields e0 .. e0+q-1) where the maximum is >= thr and, with
// cf >= 0, field cf >= clevel; else -1.  Ties go to the lower index.
template <int N>
__device__ __forceinline__ void label_cells(const Grid &g, int tier, int64_t o, int e0, int q, const Level &thr, int cf,
                                            const Level &cl, int *lab)
{
    int best[N];
    bool ok[N];
    if (tier == TIER_FP64) {
        double bv[N];
        for (int k = 0; k < q; ++k) {
            double v[4];
            const int64_t a = (int64_t)(e0 + k) * g.fs + o;
            if (N == 4) load4d(g, tier, a, v);
            else v[0] = load1d(g, tier, a);
#pragma unroll
            for (int j = 0; j < N; ++j)
                if (k == 0 || v[j] > bv[j]) {
                    best[j] = k;
                    bv[j] = v[j];
                }
        }
#pragma unroll
        for (int j = 0; j < N; ++j) ok[j] = bv[j] >= thr.d;
    } else {
        float bv[N];
#pragma unroll 4
        for (int k = 0; k < q; ++k) {
            float v[4];
            const int64_t a = (int64_t)(e0 + k) * g.fs + o;
            if (N == 4) load4f(g, tier, a, v);
            else v[0] = load1f(g, tier, a);
#pragma unroll
            for (int j = 0; j < N; ++j)
                if (k == 0 || v[j] > bv[j]) {
                    best[j] = k;
                    bv[j] = v[j];
                }
        }
#pragma unroll
        for (int j = 0; j < N; ++j) ok[j] = bv[j] >= thr.f;
    }
    if (cf >= 0) {
        const int64_t a = (int64_t)cf * g.fs + o;
        if (N == 4) {
            const unsigned m = ge4(g, tier, a, cl);
#pragma unroll
            for (int j = 0; j < N; ++j) ok[j] &= (m >> j & 1u) != 0u;
        } else {
            ok[0] &= tier == TIER_FP64 ? load1d(g, tier, a) >= cl.d : load1f(g, tier, a) >= cl.f;
        }
    }
#pragma unroll
    for (int j = 0; j < N; ++j) lab[j] = ok[j] ? best[j] : -1;
}

// A non-root always points to a smaller index (links go from the larger root
// to the smaller), so a walk from i ends within i steps; the cap (cells + 1)
// only guards against a corrupted array and raises flag bit 2.
__device__ __forceinline__ int find_root(const int *parent, int i, int64_t cap, int *flags)
{
    for (int64_t it = 0; it < cap; ++it) {
        const int p = ((volatile const int *)parent)[i];
        if (p == i) return i;
        i = p;
    }
    atomicOr(flags, 4);
    return i;
}

// Each retry continues from a strictly smaller index, so this ends within
// `cap` rounds as well.  True if it linked two components (a root got a
// parent): each true lowers the number of roots by one.
__device__ __forceinline__ bool unite(int *parent, int a, int b, int64_t cap, int *flags)
{
    for (int64_t it = 0; it < cap; ++it) {
        a = find_root(parent, a, cap, flags);
        b = find_root(parent, b, cap, flags);
        if (a == b) return false;
        if (a < b) {
            const int t = a;
            a = b;
            b = t;
        }
        const int old = atomicMin(&parent[a], b);  // link the larger root under the smaller
        if (old == a) return true;
        a = old;  // a was re-linked meanwhile: continue from its new parent
    }
    atomicOr(flags, 4);
    return false;
}

// Labels of a tile and its connected components, in shared memory: each row's
// runs of equal labels by a ballot, then one link per contact of two runs of
// neighbouring rows.  To global memory go only the tile's border cells (label
// and component) and its roots -- all that joining the tiles needs -- and the
// counts of components and labelled cells.  1024^2 Q=8, cold: 345 us as a
// gathered copy, labels, links per cell pair and a count; 27 + 13 (joining) now.
template <int T>
__global__ void __launch_bounds__(kDT) grain_tile_kernel(Grid g, int e0, int q, double thr, int cf, double clevel,
                                                         int *lab, int *parent, unsigned long long *acc, int *flags)
{
    constexpr int CPT = T * T / kDT;  // 4 or 1 cells a thread
    __shared__ int sl[T * T], sp[T * T];
    const Level lt(thr), lc(clevel);
    const int tile = blockIdx.x, x0 = tile % g.ntx * T, y0 = tile / g.ntx * T;
    const int vw = min(T, g.nx - x0), vh = min(T, g.ny - y0);
    {
        const int u = threadIdx.x * CPT, i = u % T, j = u / T;
        int l[CPT];
        label_cells<CPT>(g, g.tier[tile], (int64_t)(y0 + j) * g.px + x0 + i, e0, q, lt, cf, lc, l);
#pragma unroll
        for (int k = 0; k < CPT; ++k) sl[u + k] = i + k < vw && j < vh ? l[k] : -1;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    for (int u = threadIdx.x; u < T * T; u += kDT) {  // a warp: one row of 32, or two of 16
        const int i = u % T, l = sl[u];
        const bool start = i == 0 || sl[u - 1] != l;
        const unsigned m = __ballot_sync(0xffffffffu, start) & (0xffffffffu >> (31 - lane));
        sp[u] = u - lane + 31 - __clz(m);  // the run's first cell
    }
    __syncthreads();
    for (int u = threadIdx.x + T; u < T * T; u += kDT) {
        const int i = u % T, l = sl[u];
        if (l < 0 || sl[u - T] != l) continue;
        if (i > 0 && sl[u - 1] == l && sl[u - T - 1] == l) continue;  // the contact's first cell links
        unite(sp, u, u - T, T * T + 1, flags);
    }
    __syncthreads();
    unsigned roots = 0, cells = 0;
    for (int u = threadIdx.x; u < T * T; u += kDT) {
        const int i = u % T, j = u / T, l = sl[u];
        const bool in = i < vw && j < vh;
        const bool border = in && (i == 0 || j == 0 || i == vw - 1 || j == vh - 1);
        const int r = l < 0 ? 0 : find_root(sp, u, T * T + 1, flags);
        const int c = (y0 + j) * g.nx + x0 + i;
        if (border) lab[c] = l;
        if (l >= 0) {
            ++cells;
            roots += r == u;
            if (border || r == u) parent[c] = (y0 + r / T) * g.nx + x0 + r % T;
        }
    }
    roots = __reduce_add_sync(0xffffffffu, roots);
    cells = __reduce_add_sync(0xffffffffu, cells);
    if (lane == 0 && cells) {
        atomicAdd(&acc[0], (unsigned long long)roots);
        atomicAdd(&acc[1], (unsigned long long)cells);
    }
}

// Joins the tiles' components across their right and lower edges (through
// periodic wraps): one link per contact of two equal labels along an edge.
// Every link takes one from the count; the last block reports and clears it.
__global__ void __launch_bounds__(kDT) grain_join_kernel(Grid g, int bc, const int *lab, int *parent,
                                                         unsigned long long *acc, unsigned *counter, int *flags,
                                                         unsigned long long *out)
{
    const int T = g.tile;
    const int64_t n = (int64_t)g.nx * g.ny, units = (int64_t)g.ntx * g.nty * 2 * T;
    unsigned links = 0;
    for (int64_t u = blockIdx.x * (int64_t)kDT + threadIdx.x; u < units; u += (int64_t)gridDim.x * kDT) {
        const int k = (int)(u % T), side = (int)(u / T & 1), tile = (int)(u / (2 * T));
        const int x0 = tile % g.ntx * T, y0 = tile / g.ntx * T;
        const int vw = min(T, g.nx - x0), vh = min(T, g.ny - y0);
        if (k >= (side ? vw : vh)) continue;
        const int x = side ? x0 + k : x0 + vw - 1, y = side ? y0 + vh - 1 : y0 + k;
        const int xn = side ? x : wrap_or_out(x + 1, g.nx, bc), yn = side ? wrap_or_out(y + 1, g.ny, bc) : y;
        if (xn < 0 || yn < 0) continue;
        const int64_t a = (int64_t)y * g.nx + x, b = (int64_t)yn * g.nx + xn, d = side ? 1 : g.nx;
        const int l = lab[a];
        if (l < 0 || lab[b] != l) continue;
        if (k > 0 && lab[a - d] == l && lab[b - d] == l) continue;  // joined by the contact's first cell
        links += unite(parent, (int)a, (int)b, n + 1, flags);
    }
    links = __reduce_add_sync(0xffffffffu, links);
    if ((threadIdx.x & 31) == 0 && links) atomicAdd(&acc[0], 0ull - links);
    if (!last_block(counter) || threadIdx.x != 0) return;
    out[0] = atomicExch(&acc[0], 0ull);
    out[1] = atomicExch(&acc[1], 0ull);
    out[2] = (unsigned long long)*(volatile int *)flags;
}

// Boundary edges between differently labelled neighbours, per unordered
// label pair (a < b): [(a*q + b)*2 + 0] x-edges (length dy each), [.. + 1]
// y-edges.  A block labels its tile and the cells right of and below it, counts
// in shared memory, and adds its nonzero counts; the last block reports the
// totals and clears them.
template <int T>
__global__ void __launch_bounds__(kDT) boundary_kernel(Grid g, int e0, int q, int bc, int cf, double clevel,
                                                       unsigned long long *acc, unsigned *counter,
                                                       unsigned long long *out)
{
    constexpr int CPT = T * T / kDT, P = T + 1;
    extern __shared__ unsigned hist[];
    __shared__ int sl[P * P];
    const Level lt(-1e300), lc(clevel);
    const int tile = blockIdx.x, x0 = tile % g.ntx * T, y0 = tile / g.ntx * T, nh = 2 * q * q;
    const int vw = min(T, g.nx - x0), vh = min(T, g.ny - y0);
    for (int k = threadIdx.x; k < nh; k += kDT) hist[k] = 0;
    {
        const int u = threadIdx.x * CPT, i = u % T, j = u / T;
        int l[CPT];
        label_cells<CPT>(g, g.tier[tile], (int64_t)(y0 + j) * g.px + x0 + i, e0, q, lt, cf, lc, l);
#pragma unroll
        for (int k = 0; k < CPT; ++k)
            if (i + k < vw && j < vh) sl[j * P + i + k] = l[k];
    }
    __syncthreads();  // (a partial tile's edge slots below are not written above)
    for (int u = threadIdx.x; u < vw + vh; u += kDT) {
        const bool side = u >= vh;  // below, else right
        const int k = side ? u - vh : u;
        const int x = side ? x0 + k : wrap_or_out(x0 + vw, g.nx, bc), y = side ? wrap_or_out(y0 + vh, g.ny, bc) : y0 + k;
        int l = -1;
        if (x >= 0 && y >= 0)
            label_cells<1>(g, tile_tier(g, x, y), (int64_t)y * g.px + x, e0, q, lt, cf, lc, &l);
        sl[side ? vh * P + k : k * P + vw] = l;
    }
    __syncthreads();
    for (int u = threadIdx.x; u < T * T; u += kDT) {
        const int i = u % T, j = u / T;
        if (i >= vw || j >= vh) continue;
        const int l = sl[j * P + i], r = sl[j * P + i + 1], d = sl[(j + 1) * P + i];
        if (l < 0) continue;
        if (r >= 0 && r != l) atomicAdd(&hist[(min(l, r) * q + max(l, r)) * 2], 1u);
        if (d >= 0 && d != l) atomicAdd(&hist[(min(l, d) * q + max(l, d)) * 2 + 1], 1u);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nh; k += kDT)
        if (hist[k]) atomicAdd(&acc[k], (unsigned long long)hist[k]);
    if (!last_block(counter)) return;
    for (int k = threadIdx.x; k < nh; k += kDT) out[k] = atomicExch(&acc[k], 0ull);
}

// max |a-b|, sum (a-b)^2, sum |a-b| per block (fixed order within the block)
__global__ void compare3_kernel(const double *a, const double *b, int64_t n, double *partials)
{
    __shared__ double red[3][kDT / 32];
    double mx = 0.0, ss = 0.0, sa = 0.0;
    const int64_t chunk = (n + gridDim.x - 1) / gridDim.x;
    const int64_t lo = blockIdx.x * chunk, hi = min(n, lo + chunk);
    for (int64_t i = lo + threadIdx.x; i < hi; i += kDT) {
        const double d = a[i] - b[i];
        mx = (fabs(d) > mx || !(d == d)) ? fabs(d) : mx;
        ss += d * d;
        sa += fabs(d);
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double m2 = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = (m2 > mx || !(m2 == m2)) ? m2 : mx;
        ss += __shfl_xor_sync(0xffffffffu, ss, o);
        sa += __shfl_xor_sync(0xffffffffu, sa, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = mx;
        red[1][threadIdx.x >> 5] = ss;
        red[2][threadIdx.x >> 5] = sa;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = 0.0, s2 = 0.0, s1 = 0.0;
        for (int w = 0; w < kDT / 32; ++w) {
            m = (red[0][w] > m || !(red[0][w] == red[0][w])) ? red[0][w] : m;
            s2 += red[1][w];
            s1 += red[2][w];
        }
        partials[3 * blockIdx.x] = m;
        partials[3 * blockIdx.x + 1] = s2;
        partials[3 * blockIdx.x + 2] = s1;
    }
}

__global__ void compare3_final_kernel(const double *partials, int np, int64_t n, double *out)
{
    if (threadIdx.x != 0) return;
    double m = 0.0, s2 = 0.0, s1 = 0.0;
    for (int k = 0; k < np; ++k) {
        const double v = partials[3 * k];
        m = (v > m || !(v == v)) ? v : m;
        s2 += partials[3 * k + 1];
        s1 += partials[3 * k + 2];
    }
    out[0] = m;
    out[1] = sqrt(s2 / (double)n);
    out[2] = s1 / (double)n;
}

}  // namespace

cudaError_t diag_interface(const Grid &g, int field, int bc, double level, unsigned long long *part, unsigned *counter,
                           unsigned long long *out, cudaStream_t s)
{
    const int per = g.tile == 32 ? 1 : 4, blocks = std::min((g.ntx * g.nty + per - 1) / per, 1024);
    if (g.tile == 32) interface_kernel<32><<<blocks, kDT, 0, s>>>(g, field, bc, level, part, counter, out);
    else interface_kernel<16><<<blocks, kDT, 0, s>>>(g, field, bc, level, part, counter, out);
    return cudaGetLastError();
}

cudaError_t diag_grains(const Grid &g, int e0, int q, int bc, double thr, int cf, double clevel, int *lab, int *parent,
                        unsigned long long *acc, unsigned *counter, int *flags, unsigned long long *out,
                        cudaStream_t s)
{
    const int tiles = g.ntx * g.nty;
    if (g.tile == 32) grain_tile_kernel<32><<<tiles, kDT, 0, s>>>(g, e0, q, thr, cf, clevel, lab, parent, acc, flags);
    else grain_tile_kernel<16><<<tiles, kDT, 0, s>>>(g, e0, q, thr, cf, clevel, lab, parent, acc, flags);
    const int blocks = (int)std::min<int64_t>(((int64_t)tiles * 2 * g.tile + kDT - 1) / kDT, 152 * 8);
    grain_join_kernel<<<blocks, kDT, 0, s>>>(g, bc, lab, parent, acc, counter, flags, out);
    return cudaGetLastError();
}

cudaError_t diag_boundaries(const Grid &g, int e0, int q, int bc, int cf, double clevel, unsigned long long *acc,
                            unsigned *counter, unsigned long long *out, cudaStream_t s)
{
    const int tiles = g.ntx * g.nty;
    const size_t smem = (size_t)2 * q * q * sizeof(unsigned);
    if (g.tile == 32) boundary_kernel<32><<<tiles, kDT, smem, s>>>(g, e0, q, bc, cf, clevel, acc, counter, out);
    else boundary_kernel<16><<<tiles, kDT, smem, s>>>(g, e0, q, bc, cf, clevel, acc, counter, out);
    return cudaGetLastError();
}

cudaError_t diag_compare3(const double *a, const double *b, int64_t n, double *partials, int np, double *out,
                          cudaStream_t s)
{
    compare3_kernel<<<np, kDT, 0, s>>>(a, b, n, partials);
    compare3_final_kernel<<<1, 32, 0, s>>>(partials, np, n, out);
    return cudaGetLastError();
}

}  // namespace amps
