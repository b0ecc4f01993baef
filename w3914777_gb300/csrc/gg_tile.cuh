// gg_tile.cuh -- the per-tile body of the fused grain-growth step, shared by
// the single-run step kernel (k_graingrowth.cu), its binary16-arithmetic
// instantiations (k_gg_half.cu) and the ensemble's tile-queue kernel.
//
// Reference: graingrowth/function.h:5-30 (kernel1_pure) and
// graingrowth/function.h:33-277 (kernel1_mix), generalised from Q=2 to Q
// fields with cross coefficient gamma:
//   dfd_i = 2*gamma*eta_i*sum_{j!=i} eta_j^2 + eta_i^3 - eta_i
//   eta_i' = eta_i - dt*L*(dfd_i - kappa*lap(eta_i)).
#pragma once
#include "amps_internal.cuh"

namespace amps {

// Half / FP32 tile: staged float neighbourhood, float arithmetic.  Each
// thread advances CPT consecutive cells of one row (CPT = 4 for 32x32 tiles:
// one 128-bit shared load plus two halo scalars per row, shared row sums,
// 128-bit / 64-bit global stores).
template <int TIER, int CPT>
__device__ __forceinline__ void store_cells(const StepArgs &a, int64_t idx, const float *v)
{
    if (CPT == 4 && TIER == TIER_FP32) {
        *reinterpret_cast<float4 *>((float *)a.out[TIER_FP32] + idx) = make_float4(v[0], v[1], v[2], v[3]);
    } else if (CPT == 4 && TIER == TIER_HALF) {
        __half2 h0 = __floats2half2_rn(v[0], v[1]), h1 = __floats2half2_rn(v[2], v[3]);
        uint2 u;
        u.x = *reinterpret_cast<unsigned *>(&h0);
        u.y = *reinterpret_cast<unsigned *>(&h1);
        *reinterpret_cast<uint2 *>((__half *)a.out[TIER_HALF] + idx) = u;
    } else {
#pragma unroll
        for (int k = 0; k < CPT; ++k) store_tier<TIER>(a, idx + k, v[k]);
    }
}

// MON: this step evaluates the monitor (compiled out of the other steps, so
// their loop carries no monitor state).
template <int T, int TIER, bool MON>
__device__ __forceinline__ void gg_tile_lo_impl(const StepArgs &a, const float *sm, int tile, int tx, int ty,
                                                double *red)
{
    using S = Stage<float, T, 1>;
    constexpr int CPT = T * T / kThreads;  // cells per thread, along x
    constexpr int GPR = T / CPT;           // thread groups per row
    const int row = threadIdx.x / GPR;
    const int c0 = (threadIdx.x % GPR) * CPT;
    const int nf = a.nf;
    const Phys &ph = a.ph;
    float *smm = const_cast<float *>(sm);
    float ssum[CPT];
#pragma unroll
    for (int k = 0; k < CPT; ++k) ssum[k] = 0.f;
    for (int f = 0; f < nf; ++f) {
        float c[CPT];
        const float *ctr = &S::at(smm, f, row + 1, S::O + c0);
#pragma unroll
        for (int k = 0; k < CPT; ++k) c[k] = ctr[k];
#pragma unroll
        for (int k = 0; k < CPT; ++k) ssum[k] = fmaf(c[k], c[k], ssum[k]);
    }
    const float dtm = ph.gg_dtm, g2 = ph.gg_g2, kap = ph.gg_kap, inv = ph.gg_inv;
    const int64_t gbase = (int64_t)(ty * T + row) * a.px + tx * T + c0;
    double metric = 0.0;
    MonAccF mon;
    for (int f = 0; f < nf; ++f) {
        const bool mon_f = MON && (a.mfield < 0 || a.mfield == f);
        const int mslot = a.mfield < 0 ? f : 0;
        double snapv[CPT];
        if (mon_f) {
            mon_reset(a, mon);
#pragma unroll
            for (int k = 0; k < CPT; ++k) snapv[k] = snap_prefetch<T>(a, mslot, tile, row, c0 + k, gbase + k);
        }
        float w[3][CPT + 2];
#pragma unroll
        for (int rr = 0; rr < 3; ++rr) {
            const float *p = &S::at(smm, f, row + rr, S::O + c0);
            if (CPT == 4) {
                const float4 q = *reinterpret_cast<const float4 *>(p);
                w[rr][1] = q.x; w[rr][2] = q.y; w[rr][3] = q.z; w[rr][4] = q.w;
            } else {
#pragma unroll
                for (int k = 0; k < CPT; ++k) w[rr][k + 1] = p[k];
            }
            w[rr][0] = p[-1];
            w[rr][CPT + 1] = p[CPT];
        }
        float out[CPT];
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const float e = w[1][k + 1];
            float s;
            if (a.stencil == 0)
                s = (w[0][k] + w[0][k + 1] + w[0][k + 2]) + (w[1][k] + w[1][k + 2]) + (w[2][k] + w[2][k + 1] + w[2][k + 2])
                  - 8.f * e;
            else
                s = (w[1][k] + w[1][k + 2]) + (w[0][k + 1] + w[2][k + 1]) - 4.f * e;
            const float lap = s * inv;
            const float e2 = e * e;
            const float dfd = e * fmaf(g2, ssum[k] - e2, e2 - 1.f);
            out[k] = fmaf(-dtm, fmaf(-kap, lap, dfd), e);
        }
        store_cells<TIER, CPT>(a, (int64_t)f * a.n + gbase, out);
        if (mon_f) {
            // a ragged grid's edge tile: cells past the domain are not samples
            const int vw = min(T, a.nx - tx * T), vh = min(T, a.ny - ty * T);
#pragma unroll
            for (int k = 0; k < CPT; ++k)
                if (row < vh && c0 + k < vw)
                    mon_add<T>(a, mon, mslot, tile, row, c0 + k, gbase + k, round_to_tier<TIER>(out[k]), w[1][k + 1],
                               snapv[k]);
            metric = mon_finish(a, mon, red, metric);
        }
    }
    if (MON && threadIdx.x == 0) a.metric[tile] = metric;
}

template <int T, int TIER>
__device__ __forceinline__ void gg_tile_lo(const StepArgs &a, const float *sm, int tile, int tx, int ty, double *red)
{
    if (a.monitor_now) gg_tile_lo_impl<T, TIER, true>(a, sm, tile, tx, ty, red);
    else gg_tile_lo_impl<T, TIER, false>(a, sm, tile, tx, ty, red);
}

// Half/FP32 tile, 32^2 tiles: the sum of squares over fields is formed once
// per cell into shared memory (ss, 32x32 floats, after the staged fields),
// then each thread advances RPT rows x 4 cells of a field from RPT + 2 staged
// rows with a 3-row register window (RPT = 4: 1.5 row reads per output row,
// 8: 1.25, against 2 for two rows a thread), the CTA's RPT groups on fields
// g, g+RPT, ...  Per cell the arithmetic, and its order, is
// gg_tile_lo_impl's.  MK, the monitor kind of a monitor step (0: none, 2:
// temporal, 3: rate; the spatial range takes gg_tile_lo_impl): the tile
// metric is a maximum over fields and cells, so each thread folds every
// field it computes into one accumulator and the block reduces once.
// PH > 0: one CTA of a split tile -- staging slots 0..PH-1 hold fields
// [f0, f0 + PH), and the caller has formed `ss` over every field.
template <int TIER, int RPT, int MK = 0, int PH = 0>
__device__ __forceinline__ void gg_tile_lo_rows(const StepArgs &a, const float *sm, float *ss, int tile, int tx,
                                                int ty, double *red, int f0 = 0)
{
    static_assert(PH == 0 || MK == 0, "split tiles run the steps without a monitor");
    constexpr int T = 32, CPT = 4, GPR = T / CPT;
    using S = Stage<float, T, 1>;
    float *smm = const_cast<float *>(sm);
    const int nf = PH ? PH : a.nf;
    if constexpr (PH == 0) {
        const int row = threadIdx.x / GPR, c = (threadIdx.x % GPR) * CPT;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int f = 0; f < nf; ++f) {
            const float4 q = *reinterpret_cast<const float4 *>(&S::at(smm, f, row + 1, S::O + c));
            acc.x = fmaf(q.x, q.x, acc.x);
            acc.y = fmaf(q.y, q.y, acc.y);
            acc.z = fmaf(q.z, q.z, acc.z);
            acc.w = fmaf(q.w, q.w, acc.w);
        }
        *reinterpret_cast<float4 *>(ss + row * T + c) = acc;
        __syncthreads();
    }
    static_assert(T % RPT == 0 && (T / RPT) * GPR * RPT == kThreads, "RPT groups of T/RPT x GPR threads");
    const int group = threadIdx.x / (kThreads / RPT), t = threadIdx.x % (kThreads / RPT);
    const int r0 = RPT * (t / GPR), c0 = (t % GPR) * CPT;  // tile-local rows r0 .. r0+RPT-1
    const Phys &ph = a.ph;
    const float dtm = ph.gg_dtm, g2 = ph.gg_g2, kap = ph.gg_kap, inv = ph.gg_inv;
    const int64_t gbase = (int64_t)(ty * T + r0) * a.px + tx * T + c0;
    MonAccF mon;
    if (MK) mon_reset(a, mon);
    for (int f = group; f < nf; f += RPT) {
        const bool mon_f = MK && (a.mfield < 0 || a.mfield == f);
        const int mslot = a.mfield < 0 ? f : 0;
        float w[3][CPT + 2];
        auto load_row = [&](int sr, float *d) {
            const float *p = &S::at(smm, f, sr, S::O + c0);
            const float4 q = *reinterpret_cast<const float4 *>(p);
            d[0] = p[-1];
            d[1] = q.x; d[2] = q.y; d[3] = q.z; d[4] = q.w;
            d[CPT + 1] = p[CPT];
        };
        load_row(r0, w[0]);
        load_row(r0 + 1, w[1]);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            float *up = w[i % 3], *md = w[(i + 1) % 3], *dn = w[(i + 2) % 3];
            load_row(r0 + i + 2, dn);
            const float4 sq = *reinterpret_cast<const float4 *>(ss + (r0 + i) * T + c0);
            const float ssum[CPT] = {sq.x, sq.y, sq.z, sq.w};
            float out[CPT];
#pragma unroll
            for (int k = 0; k < CPT; ++k) {
                const float e = md[k + 1];
                float sv;
                if (a.stencil == 0)
                    sv = (up[k] + up[k + 1] + up[k + 2]) + (md[k] + md[k + 2]) + (dn[k] + dn[k + 1] + dn[k + 2]) -
                         8.f * e;
                else
                    sv = (md[k] + md[k + 2]) + (up[k + 1] + dn[k + 1]) - 4.f * e;
                const float lap = sv * inv;
                const float e2 = e * e;
                const float dfd = e * fmaf(g2, ssum[k] - e2, e2 - 1.f);
                out[k] = fmaf(-dtm, fmaf(-kap, lap, dfd), e);
            }
            const int64_t gi = gbase + (int64_t)i * a.px;
            store_cells<TIER, CPT>(a, (int64_t)(f0 + f) * a.n + gi, out);
            if constexpr (MK != 0) {
                // a ragged grid's edge tile: cells past the domain are not samples
                if (mon_f && r0 + i < min(T, a.ny - ty * T)) {
                    const int vw = min(T, a.nx - tx * T);
#pragma unroll
                    for (int k = 0; k < CPT; ++k)
                        if (c0 + k < vw)
                            mon_add_k<T, MK>(a, mon, mslot, tile, r0 + i, c0 + k, gi + k, round_to_tier<TIER>(out[k]),
                                             md[k + 1]);
                }
            }
        }
    }
    if constexpr (MK != 0) {
        const double metric = mon_finish_k<MK>(a, mon, red);
        if (threadIdx.x == 0) a.metric[tile] = metric;
    }
}

// ---- FP64 tiles --------------------------------------------------------------
// Bound by the FP64 pipe (1.25 TFLOP/s nominal, ~1/60 of FP32): everything
// here is arranged for few FP64 operations a cell and field, and the rest
// (staging, shared-memory traffic, index arithmetic) hides behind them.
//
// A tile is advanced in bands of HB rows: the band's rows and a 1-cell halo of
// every field are staged as doubles in the memory the FP32 tiles stage in
// (half the rows at twice the size: gg_fp64_band), then a lane sweeps RR rows
// x 2 columns of one field.
//
// Library order (REF = false).  With the 3x3 box sum B (eight neighbours plus
// the cell), S = sum_j eta_j^2 and G = 2 gamma S - 1, the update is
//   eta' = eta - dtL*(eta*(G + (1 - 2 gamma) eta^2) - kappa/dxdy*(B - 9 eta)).
// G is formed once per cell for all fields (into shared memory).  B shares its
// partial sums: the middle pair of the two columns' row sums, and the middle
// pair of rows of two output rows: 10.4 FP64 operations a cell and field
// (eight rows a lane) in place of the 18 of eight separate neighbours.  9 eta
// is taken off the pair of rows before the third is added: partial sums stay
// below 6 eta and the last addition is of opposite numbers, so the error
// against extended precision is that of the eight-neighbour form (equal to a
// few percent over 200 steps of a polycrystal).
// Which additions pair up depends on the parity of the tile-local row and
// column, so every launch that computes a cell gets the same bits.
// 5-point stencil: (left + right) + (up + down) - 4 eta.
//
// REF: the reference's expression order, every operation rounded on its own
// (graingrowth/function.h:20-23); 8*eta is exact, so its subtraction is one
// fused operation; the division by dx*dy is div_known; pow(eta, 3) is the
// correctly rounded cube (cube_rn), within an ulp of any library's pow.  About
// 27 FP64 operations a cell and field at Q = 2 in place of ~137 with pow and
// the general division: 30 us a step in place of 103 on the reference's 512^2
// two-field adaptive run, nearly all of whose 16^2 tiles hold a moving boundary.
template <int T> struct Stage64 {
    static constexpr int O = 2, P = T + 2 * O;  // interior at column 2: 16-byte aligned rows
    __host__ __device__ static constexpr int field(int hb) { return (hb + 2) * P; }
};

// Rows of a band of `nf` fields: the most that fit in the FP32 staging of a
// 32^2 tile (16 rows of 36 doubles against 34 of 40 floats, and the sum tile
// in that of the sums of squares); a 16^2 tile whole, up to 12 fields (with 16 an
// SM's four CTAs would take 196 KB: steps without FP64 tiles 2% slower).
__host__ __device__ __forceinline__ int gg_fp64_band(int tile, int nf) { return tile == 32 ? 16 : (nf <= 12 ? 16 : 8); }

// Stage rows [r0 - 1, r0 + hb] of every field (tile-local), each cell read at
// its owner tile's input tier: the tile of the 3x3 neighbourhood at that
// position, or (own: a ragged grid's edge tile, whose boundary-mapped halo
// can lie in another tile) the tile that holds the mapped cell.  FP64 cells by
// asynchronous copies, every field in flight at once.
// ALL64: every cell is at FP64 (no tier is looked up).
template <int T, bool NC, bool ALL64 = false>
__device__ __forceinline__ void gg_stage64(const StepArgs &a, double *sm, const uint8_t *nt, int x0, int y0, int r0,
                                           int hb, bool own, int tid)
{
    using S = Stage64<T>;
    const int nf = a.nf, fs = S::field(hb);
    for (int u = tid; u < (hb + 2) * (T + 2); u += kThreads) {
        const int ly = r0 - 1 + u / (T + 2), lx = u % (T + 2) - 1;
        const int gy = bc_map(y0 + ly, a.ny, a.bc), gx = bc_map(x0 + lx, a.nx, a.bc);
        const int cls = (ly < 0 ? 0 : (ly < T ? 3 : 6)) + (lx < 0 ? 0 : (lx < T ? 1 : 2));
        const int tier = ALL64 ? TIER_FP64 : own ? a.tier_in[(gy / T) * a.ntx + gx / T] : nt[cls];
        const int64_t g = (int64_t)gy * a.px + gx;
        double *d = sm + (ly - r0 + 1) * S::P + S::O + lx;
        if (NC && tier == TIER_FP64) {
            const double *src = (const double *)a.in[TIER_FP64] + g;
            for (int f = 0; f < nf; ++f)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(d + f * fs)),
                             "l"(src + (int64_t)f * a.n)
                             : "memory");
        } else {
#pragma unroll 4
            for (int f = 0; f < nf; ++f) {
                const int64_t k = (int64_t)f * a.n + g;
                if (tier == TIER_FP64) d[f * fs] = __ldcg((const double *)a.in[TIER_FP64] + k);
                else if (tier == TIER_FP32) d[f * fs] = (double)ldro<NC>((const float *)a.in[TIER_FP32] + k);
                else d[f * fs] = (double)__half2float(__ushort_as_half(ldro<NC>((const unsigned short *)a.in[TIER_HALF] + k)));
            }
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    cp_async_wait_all();
}

// The monitor of an FP64 tile, from the values just stored (exact) and the
// tile's input: one pass over the tile after the update, on monitor steps only.
template <int T, int KIND>
__device__ __forceinline__ void gg_monitor64(const StepArgs &a, const uint8_t *nt, int tile, int tx, int ty, double *red, int tid)
{
    const int x0 = tx * T, y0 = ty * T;
    // a ragged grid's edge tile: cells past the domain are not samples
    const int vw = min(T, a.nx - x0), vh = min(T, a.ny - y0);
    constexpr bool range = KIND == 1;  // one reduction per field; the other kinds are maxima over fields
    double metric = 0.0;
    MonAcc mon;
    mon_reset(a, mon);
    for (int f = 0; f < a.nf; ++f) {
        if (a.mfield >= 0 && a.mfield != f) continue;
        const int mslot = a.mfield < 0 ? f : 0;
        if (range) mon_reset(a, mon);
        for (int u = tid; u < T * T; u += kThreads) {
            const int row = u / T, col = u % T;
            if (row >= vh || col >= vw) continue;
            const int64_t g = (int64_t)(y0 + row) * a.px + x0 + col, k = (int64_t)f * a.n + g;
            const double v = ((const double *)a.out[TIER_FP64])[k];
            if constexpr (KIND == 3) {
                if ((__double2hiint(v) & 0x7ff00000) == 0x7ff00000) mon.bad = 1;
                if (sample_index<T>(2, a.samples, row, col) >= 0)
                    mon.dmaxf = fmaxf(mon.dmaxf, fabsf((float)v - load_tier<float>(a, nt[4], k)));
            } else {
                mon_add<T>(a, mon, mslot, tile, row, col, g, v, 0.0, snap_prefetch<T>(a, mslot, tile, row, col, g));
            }
        }
        if (range) metric = mon_finish(a, mon, red, metric);
    }
    if (!range) metric = mon_finish(a, mon, red, metric);
    if (tid == 0) a.metric[tile] = metric;
}

// The update of every field in one band (rows [r0, r0 + hb) of the tile) from
// its staging; a lane takes RR rows x 2 columns.  rot: added to a warp's index
// where it picks its fields.
template <int T, bool REF, int RR>
__device__ __forceinline__ void gg_band64(const StepArgs &a, const double *sm, double *ss, int x0, int y0, int r0,
                                          int hb, int rot, int tid)
{
    using S = Stage64<T>;
    constexpr int GPR = T / 2, RG = 32 / GPR;  // column pairs a row, row groups a warp
    const int nf = a.nf, fs = S::field(hb);
    const Phys &ph = a.ph;
    if (!REF) {
        // G = 2 gamma S - 1 at every cell of the band
        for (int u = tid; u < hb * GPR; u += kThreads) {
            const int row = u / GPR, c = 2 * (u % GPR);
            const double *p = sm + (row + 1) * S::P + S::O + c;
            double s0 = 0.0, s1 = 0.0;
            for (int f = 0; f < nf; ++f) {
                const double2 v = *reinterpret_cast<const double2 *>(p + f * fs);
                s0 = fma(v.x, v.x, s0);
                s1 = fma(v.y, v.y, s1);
            }
            *reinterpret_cast<double2 *>(ss + row * T + c) =
                make_double2(fma(ph.kd[GG_G2], s0, -1.0), fma(ph.kd[GG_G2], s1, -1.0));
        }
        __syncthreads();
    }
    const int lane = tid & 31, warp = (tid >> 5) + rot;
    const int c = 2 * (lane % GPR);
    const int parts = hb / (RG * RR);  // warps that share a field
    for (int u = warp & 7; u < nf * parts; u += kThreads / 32) {
        const int f = u / parts, rb = (u % parts) * RG * RR + (lane / GPR) * RR;  // band-local first row
        const double *p = sm + f * fs + rb * S::P + S::O + c;                     // staged row rb: one above
        double *out = (double *)a.out[TIER_FP64] + (int64_t)f * a.n + (int64_t)(y0 + r0 + rb) * a.px + x0 + c;
        auto load = [&](int r, double *w) {
            const double2 m = *reinterpret_cast<const double2 *>(p + r * S::P);
            w[0] = p[r * S::P - 1];
            w[1] = m.x;
            w[2] = m.y;
            w[3] = p[r * S::P + 2];
        };
        if constexpr (REF) {
            double w[3][4];
            load(0, w[0]);
            load(1, w[1]);
#pragma unroll
            for (int i = 0; i < RR; ++i) {
                const double *rd = w[i % 3], *rc = w[(i + 1) % 3];
                double *ru = w[(i + 2) % 3];
                load(i + 2, ru);
                double v2[2];
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const double e = rc[k + 1];
                    double s;
                    if (a.stencil == 0) {
                        s = __dadd_rn(__dadd_rn(__dadd_rn(rd[k], rd[k + 1]), rd[k + 2]), rc[k]);
                        s = __dadd_rn(__dadd_rn(__dadd_rn(__dadd_rn(s, rc[k + 2]), ru[k]), ru[k + 1]), ru[k + 2]);
                        s = __fma_rn(-8.0, e, s);
                    } else {
                        s = __fma_rn(-4.0, e, __dadd_rn(__dadd_rn(__dadd_rn(rc[k], rc[k + 2]), rd[k + 1]), ru[k + 1]));
                    }
                    const double lap = div_known(s, ph.dxdy, ph.inv_dxdy, ph.dxdy_div);
                    const double *q = sm + (rb + i + 1) * S::P + S::O + c + k;  // field 0 at this cell
                    const int b0 = f == 0;                                    // the first other field
                    double sum = 0.0;
                    if (b0 < nf) sum = __dmul_rn(q[b0 * fs], q[b0 * fs]);
                    for (int b = b0 + 1; b < nf; ++b)
                        if (b != f) sum = __dadd_rn(sum, __dmul_rn(q[b * fs], q[b * fs]));
                    const double dfd = __dsub_rn(__dadd_rn(__dmul_rn(__dmul_rn(ph.kd[GG_G2], e), sum), cube_rn(e)), e);
                    v2[k] = __dsub_rn(e, __dmul_rn(ph.kd[GG_DTM], __dsub_rn(dfd, __dmul_rn(ph.grcoef, lap))));
                }
                *reinterpret_cast<double2 *>(out + (int64_t)i * a.px) = make_double2(v2[0], v2[1]);
            }
        } else {
            const double m2 = ph.kd[GG_M2], ki = ph.kd[GG_KI], dtm = ph.kd[GG_DTM];
            // lap: the stencil's sum; g: G at the cell
            auto update = [&](double e, double lap, double g) {
                return fma(-dtm, fma(-ki, lap, e * fma(m2, e * e, g)), e);
            };
            if (a.stencil == 0) {
                // h0, h1: row sums of rows i-1, i; e1: the centre values of row i
                double w[4], h0[2], h1[2], e1[2];
                auto sums = [&](double *h) {
                    const double pr = w[1] + w[2];
                    h[0] = w[0] + pr;
                    h[1] = pr + w[3];
                };
                load(0, w);
                sums(h0);
                load(1, w);
                sums(h1);
                e1[0] = w[1];
                e1[1] = w[2];
#pragma unroll
                for (int i = 0; i < RR; i += 2) {
                    double h2[2], h3[2], e2[2], e3[2];
                    load(i + 2, w);
                    sums(h2);
                    e2[0] = w[1];
                    e2[1] = w[2];
                    load(i + 3, w);
                    sums(h3);
                    e3[0] = w[1];
                    e3[1] = w[2];
                    const double2 ga = *reinterpret_cast<const double2 *>(ss + (rb + i) * T + c);
                    const double2 gb = *reinterpret_cast<const double2 *>(ss + (rb + i + 1) * T + c);
                    double oa[2], ob[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const double q = h1[k] + h2[k];
                        oa[k] = update(e1[k], h0[k] + fma(-9.0, e1[k], q), k ? ga.y : ga.x);
                        ob[k] = update(e2[k], fma(-9.0, e2[k], q) + h3[k], k ? gb.y : gb.x);
                        h0[k] = h2[k];
                        h1[k] = h3[k];
                        e1[k] = e3[k];
                    }
                    *reinterpret_cast<double2 *>(out + (int64_t)i * a.px) = make_double2(oa[0], oa[1]);
                    *reinterpret_cast<double2 *>(out + (int64_t)(i + 1) * a.px) = make_double2(ob[0], ob[1]);
                }
            } else {
#pragma unroll 2
                for (int i = 0; i < RR; ++i) {
                    double w[4];
                    load(i + 1, w);
                    const double2 up = *reinterpret_cast<const double2 *>(p + i * S::P);
                    const double2 dn = *reinterpret_cast<const double2 *>(p + (i + 2) * S::P);
                    const double2 g = *reinterpret_cast<const double2 *>(ss + (rb + i) * T + c);
                    *reinterpret_cast<double2 *>(out + (int64_t)i * a.px) =
                        make_double2(update(w[1], fma(-4.0, w[1], (w[0] + w[2]) + (up.x + dn.x)), g.x),
                                     update(w[2], fma(-4.0, w[2], (w[1] + w[3]) + (up.y + dn.y)), g.y));
                }
            }
        }
    }
}

// Rows [row0, row1) of an FP64 tile in bands of hb rows (the whole tile but
// for a CTA of a split tile), by the whole CTA, in the CTA's staging memory
// (no copy into it may be in flight).
template <int T, bool REF, bool NC = true>
__device__ __forceinline__ void gg_tile_fp64(const StepArgs &a, float *smf, const uint8_t *nt, int tile, int tx, int ty,
                                          double *red, int row0, int row1, int hb, int tid)
{
    double *sm = reinterpret_cast<double *>(smf);
    double *ss = sm + a.nf * Stage64<T>::field(hb);
    const int x0 = tx * T, y0 = ty * T;
    const bool own = (tx + 1) * T > a.nx || (ty + 1) * T > a.ny;  // a ragged grid's edge tile
    for (int r0 = row0; r0 < row1; r0 += hb) {
        gg_stage64<T, NC>(a, sm, nt, x0, y0, r0, hb, own, tid);
        __syncthreads();
        // the warps' fields rotate with the tile, so that CTAs with fewer
        // fields than warps load every SM sub-partition's FP64 pipe
        const int rot = 2 * (tile & 3);
        if (T == 32 && hb == 16 && a.nf % 8 == 0) gg_band64<T, REF, T == 32 ? 8 : 2>(a, sm, ss, x0, y0, r0, hb, rot, tid);
        else if (T == 32 && hb == 16) gg_band64<T, REF, T == 32 ? 4 : 2>(a, sm, ss, x0, y0, r0, hb, rot, tid);
        // (one row a lane keeps all eight warps of a two-field 16^2 tile busy:
        // 32.4 -> 30.1 us a step of the reference's 512^2 adaptive run)
        else if (REF && a.nf <= 2) gg_band64<T, REF, REF ? 1 : 2>(a, sm, ss, x0, y0, r0, hb, rot, tid);
        else gg_band64<T, REF, 2>(a, sm, ss, x0, y0, r0, hb, rot, tid);
        __syncthreads();  // the next band overwrites the staging; the monitor reads the stored tile
    }
    if (a.monitor_now) {
        if (a.monitor_kind == 3) gg_monitor64<T, 3>(a, nt, tile, tx, ty, red, tid);
        else if (a.monitor_kind == 2) gg_monitor64<T, 2>(a, nt, tile, tx, ty, red, tid);
        else gg_monitor64<T, 1>(a, nt, tile, tx, ty, red, tid);
    }
}

// The speculative staging copies have landed (false: a bounded wait on the
// tensor copy gave up -- flagged; the CTA waits once more for it and returns).
__device__ __forceinline__ bool gg_copies_landed(const StepArgs &a, bool bulk, uint64_t *bar)
{
    if (!bulk) {
        cp_async_wait_all();
        return true;
    }
    const bool ok = mbar_wait_bounded(bar, 0);
    if (__syncthreads_or(!ok)) {
        if (threadIdx.x == 0) {
            atomicOr(a.flags, 2);
            if (!ok) mbar_wait_bounded(bar, 0);
        }
        return false;
    }
    return true;
}

// The same out of line, after the discarded copies (see gg_tile_step).
template <int T, bool REF, bool NC = true>
__device__ __noinline__ void gg_tile_fp64_call(const StepArgs &a, float *smf, const uint8_t *nt, int tile, int tx, int ty,
                                               double *red, bool spec, bool bulk, uint64_t *bar)
{
    if (spec && !gg_copies_landed(a, bulk, bar)) return;
    if (spec && !bulk) __syncthreads();  // every thread's own copies
    gg_tile_fp64<T, REF, NC>(a, smf, nt, tile, tx, ty, red, 0, T, gg_fp64_band(T, a.nf), (int)threadIdx.x);
}

__device__ __forceinline__ __half2 gg_hconst(const Phys &ph, int i)
{
    const __half h = __ushort_as_half(ph.gg_h[i]);
    return __halves2half2(h, h);
}

// Half tile in binary16 arithmetic on pairs of adjacent columns, packed as
// the reference packs its half2 tiles (graingrowth/tools.h:165).  Each cell
// enters as the half rounding of its staged float, itself the float rounding
// of the owner tile's input -- the reference's __float2half(double) halo
// patching and its __floats2half2_rn demotion (graingrowth/function.h:87-161,
// graingrowth/tools.h:256-271).
//   HA == AMPS_HALF_REF: graingrowth/function.h:163-166 as written, every
//     +, -, *, / rounded on its own (the _rn intrinsics are never contracted
//     into fused multiply-adds) and in the reference's order; Q fields
//     generalise `hetab*hetab` to the left-to-right sum over j != i, and
//     `htwo*hone` to 2*gamma.  The 5-point stencil follows the FP64
//     reference-order tiles' order.
//   HA == AMPS_HALF_HFMA2: the same update as packed fused multiply-adds,
//     eta*(2*gamma*S + eta^2 - 1) and eta - dt*L*(dfd - kappa/dxdy * s).
// MK != 0: a monitor step; the epilogue folds each stored value (exact in
// double) into the per-field accumulator as the other tiers do.
template <int T, int MK, int HA>
__device__ __forceinline__ void gg_tile_half2(const StepArgs &a, const float *sm, int tile, int tx, int ty, double *red)
{
    using S = Stage<float, T, 1>;
    constexpr int PPR = T / 2, NP = T * PPR;  // pairs per row, per tile
    float *smm = const_cast<float *>(sm);
    const int nf = a.nf;
    const Phys &ph = a.ph;
    const __half2 h1 = __float2half2_rn(1.f), h2 = __float2half2_rn(2.f), h4 = __float2half2_rn(4.f),
                  h8 = __float2half2_rn(8.f);
    auto pair = [&](int f, int sr, int c) {  // staged row sr, tile columns c and c+1
        return __floats2half2_rn(S::at(smm, f, sr, S::O + c), S::at(smm, f, sr, S::O + c + 1));
    };
    double metric = 0.0;
    for (int f = 0; f < nf; ++f) {
        const bool mon_f = MK != 0 && (a.mfield < 0 || a.mfield == f);
        const int mslot = a.mfield < 0 ? f : 0;
        MonAcc mon;
        if (mon_f) mon_reset(a, mon);
        for (int p = threadIdx.x; p < NP; p += kThreads) {
            const int row = p / PPR, c = 2 * (p % PPR);
            const __half2 dl = pair(f, row, c - 1), dc = pair(f, row, c), dr = pair(f, row, c + 1);
            const __half2 ml = pair(f, row + 1, c - 1), ctr = pair(f, row + 1, c), mr = pair(f, row + 1, c + 1);
            const __half2 ul = pair(f, row + 2, c - 1), uc = pair(f, row + 2, c), ur = pair(f, row + 2, c + 1);
            __half2 out;
            if constexpr (HA == 1) {
                __half2 s;
                if (a.stencil == 0) {
                    s = __hadd2_rn(dl, dc);
                    s = __hadd2_rn(s, dr);
                    s = __hadd2_rn(s, ml);
                    s = __hadd2_rn(s, mr);
                    s = __hadd2_rn(s, ul);
                    s = __hadd2_rn(s, uc);
                    s = __hadd2_rn(s, ur);
                    s = __hsub2_rn(s, __hmul2_rn(h8, ctr));
                } else {
                    s = __hsub2_rn(__hadd2_rn(__hadd2_rn(__hadd2_rn(ml, mr), dc), uc), __hmul2_rn(h4, ctr));
                }
                const __half2 lap = __h2div(s, gg_hconst(ph, GH_DXDY));
                __half2 sum = __float2half2_rn(0.f);
                bool first = true;
                for (int b = 0; b < nf; ++b) {
                    if (b == f) continue;
                    const __half2 v = pair(b, row + 1, c);
                    const __half2 s2 = __hmul2_rn(v, v);
                    sum = first ? s2 : __hadd2_rn(sum, s2);
                    first = false;
                }
                __half2 dfd = __hmul2_rn(__hmul2_rn(__hmul2_rn(h2, gg_hconst(ph, GH_GAM)), ctr), sum);
                dfd = __hsub2_rn(__hadd2_rn(dfd, __hmul2_rn(__hmul2_rn(ctr, ctr), ctr)), ctr);
                dfd = __hmul2_rn(h1, dfd);
                out = __hsub2_rn(ctr, __hmul2_rn(__hmul2_rn(gg_hconst(ph, GH_DT), gg_hconst(ph, GH_MOB)),
                                                 __hsub2_rn(dfd, __hmul2_rn(gg_hconst(ph, GH_KAP), lap))));
            } else {
                __half2 s = a.stencil == 0 ? __hadd2(__hadd2(__hadd2(dl, dc), dr), __hadd2(ml, mr)) +
                                                 __hadd2(__hadd2(ul, uc), ur)
                                           : __hadd2(__hadd2(ml, mr), __hadd2(dc, uc));
                s = __hfma2(a.stencil == 0 ? __hneg2(h8) : __hneg2(h4), ctr, s);
                __half2 sum = __float2half2_rn(0.f);
                for (int b = 0; b < nf; ++b) {
                    if (b == f) continue;
                    const __half2 v = pair(b, row + 1, c);
                    sum = __hfma2(v, v, sum);
                }
                const __half2 dfd = __hmul2(ctr, __hfma2(gg_hconst(ph, GH_G2), sum, __hfma2(ctr, ctr, __hneg2(h1))));
                out = __hfma2(__hneg2(gg_hconst(ph, GH_DTM)), __hfma2(__hneg2(gg_hconst(ph, GH_KINV)), s, dfd), ctr);
            }
            const int64_t g = (int64_t)(ty * T + row) * a.px + tx * T + c;
            *reinterpret_cast<__half2 *>((__half *)a.out[TIER_HALF] + (int64_t)f * a.n + g) = out;
            if (mon_f) {
                const double s0 = snap_prefetch<T>(a, mslot, tile, row, c, g);
                const double s1 = snap_prefetch<T>(a, mslot, tile, row, c + 1, g + 1);
                mon_add<T>(a, mon, mslot, tile, row, c, g, (double)__low2float(out), (double)__low2float(ctr), s0);
                mon_add<T>(a, mon, mslot, tile, row, c + 1, g + 1, (double)__high2float(out),
                           (double)__high2float(ctr), s1);
            }
        }
        if (mon_f) metric = mon_finish(a, mon, red, metric);
    }
    if (MK != 0 && threadIdx.x == 0) a.metric[tile] = metric;
}

// ---- ragged grids ----------------------------------------------------------------
// A grid whose sides are not multiples of the tile keeps whole tiles in
// storage (row pitch px = ntx*T, nty*T rows): the last tile column and row
// reach past the domain into that padding.  Such a partial tile is staged and
// computed as a whole tile -- its cells past the domain compute from padding
// and store into padding, which no cell inside the domain ever reads, and
// the monitor skips them -- with one correction: the staged slots of column
// w and row h (w x h: the tile's cells inside the domain), the right and
// lower halo of its last valid cells, held padding and are re-read across
// the boundary map (periodic: column 0 / row 0 of the domain) at the input
// tier of the tile that owns them.  Every access stays inside the storage:
// rows and halo columns are boundary-mapped (nx, ny >= T), interior row
// segments end at most at the padded pitch.
__device__ __forceinline__ bool gg_partial_tile(const StepArgs &a, int T, int tx, int ty)
{
    return (tx + 1) * T > a.nx || (ty + 1) * T > a.ny;
}

// The patch of a partial tile's staging (Stage<CT, T, 1> layout, fields
// [f0, f0 + nfs) in slots 0..nfs-1; nfs < 0: all); the caller synchronises
// before and after.
template <typename CT, int T>
__device__ __noinline__ void patch_ragged(const StepArgs &a, CT *sm, int tx, int ty, int f0 = 0, int nfs = -1)
{
    using S = Stage<CT, T, 1>;
    const int x0 = tx * T, y0 = ty * T;
    const int w = min(T, a.nx - x0), h = min(T, a.ny - y0);
    // column w for rows -1..h (when w < T); row h for columns -1..w-1, or
    // -1..T when the tile is whole in x (the corner (w, h) once)
    const int nc = w < T ? h + 2 : 0;
    const int nr = h < T ? (w < T ? w + 1 : w + 2) : 0;
    for (int u = threadIdx.x; u < nc + nr; u += kThreads) {
        const int lx = u < nc ? w : u - nc - 1, ly = u < nc ? u - 1 : h;
        const int gx = bc_map(x0 + lx, a.nx, a.bc), gy = bc_map(y0 + ly, a.ny, a.bc);
        const int tier = a.tier_in[(gy / T) * a.ntx + gx / T];
        const int64_t o = (int64_t)gy * a.px + gx;
        CT *d = &S::at(sm, 0, ly + 1, S::O + lx);
        const int nl = nfs < 0 ? a.nf : nfs;
        for (int f = 0; f < nl; ++f) d[f * S::FIELD] = load_tier<CT>(a, tier, (int64_t)(f0 + f) * a.n + o);
    }
}

// Fused all-tier step: at most 64 registers, so that four CTAs share an SM
// and the half/FP32 tiles (the common case) keep their occupancy.
// every tile of the 3x3 neighbourhood (after the boundary map) holds FP32 input
__device__ __forceinline__ bool all_fp32(const uint8_t *nt)
{
    bool ok = true;
#pragma unroll
    for (int k = 0; k < 9; ++k) ok &= nt[k] == TIER_FP32;
    return ok;
}

// One tile of the fused step (every tier), by the whole CTA: neighbourhood
// tiers, staging, update (and the monitor on monitor steps).  Shared by the
// single-run step kernel and the ensemble's tile-queue kernel, so that a
// member of an ensemble gets exactly the results of a single run.  MK: 0 for
// a step without the monitor, 1/2/3 a monitor step of that monitor kind
// (spatial / temporal / rate), -1 a monitor step of the kind in `a`.
// NC = false: no read-only-path loads (the persistent multi-step kernel
// reads values that other CTAs of the same launch wrote).  RG: the grid may
// be ragged (its edge tiles partial); compiled out of the whole-tile grids'
// kernels, whose registers it would otherwise spill.
// F64 = false: no tile of the run is ever at FP64 (and REF says nothing).
// How the FP64 path is kept off the other tiles' way: out of line (the
// ensemble, ragged steps without a monitor, 16^2 tiles), or, in the reference's
// order, where a call costs 8-15% of an all-FP64 step, behind opaque copies of
// what its addresses and indices come from, which the compiler otherwise
// forms ahead of the branch.  512^2, 16^2 tiles, us a step without / with
// all tiles at FP64: plainly inlined 7.80 / 29.3, called 7.19 / 32.9, opaque
// 7.45 / 29.2; the library's order, half tiles of 8 fields: 11.35 inlined, 11.15
// called.  (32^2 tiles in the library's order: 13.9 us a 1024^2 step inlined
// plainly, 14.1 with opaque copies, up to 4% more called.)
// TT: the thread that issues the tensor copy.  The ensemble's launches take one
// that loads no neighbour's tier: thread 0 waits for its tier first (1000 steady
// steps of 64 members: 298 ms with thread 0, 292 with thread 32; a single run's
// small grids are faster with thread 0).
// tm, bar (T = 32): a tensor map of this step's FP32 input and an mbarrier;
// tiles whose halo needs no wrap or mirror then fetch the whole FP32
// neighbourhood -- every field, 34 rows x 40 columns, the staging layout --
// by one bulk tensor copy issued by one thread (sm 128-byte aligned).
template <int T, bool REF, int MK, int HA = 0, bool NC = true, bool RG = false, bool F64 = true,
          int TT = 0>
__device__ __forceinline__ void gg_tile_step(const StepArgs &a, float *sm, uint8_t *ntier, double *red, int tile,
                                             const CUtensorMap *tm = nullptr, uint64_t *bar = nullptr)
{
    constexpr bool MON = MK != 0;
    constexpr bool kFp64Call = (T == 16 && !REF) || (RG && MK <= 0);
    const int tx = tile % a.ntx, ty = tile / a.ntx;
    load_neighbour_tiers(a, tx, ty, ntier);
    // the copy of the FP32 neighbourhood (the common case) starts before the
    // tiers are known, so that its latency overlaps theirs; where the tile
    // turns out FP64 or its neighbourhood mixed, the copies are drained and
    // their data (in-bounds reads of the full-size FP32 store) discarded
    // (not when every tile is known to be FP64)
    const bool spec = T == 32 && a.in[TIER_FP32] != nullptr && !(F64 && a.all64);
    const bool bulk = spec && tm != nullptr && tx >= 1 && ty >= 1 && tx <= a.ntx - 2 && ty <= a.nty - 2;
    if (bulk) {
        if (threadIdx.x == TT) {
            mbar_init(bar, 1);
            fence_mbar_init();
            mbar_arrive_expect_tx(bar, (uint32_t)(Stage<float, T, 1>::FIELD * a.nf * sizeof(float)));
            tma_load_3d(sm, tm, tx * T - Stage<float, T, 1>::O, ty * T - 1, 0, bar);
        }
    } else if (spec) {
        stage_tile_async32<T, 1, false>(a, sm, tx, ty, a.nf);
    }
    auto spec_done = [&]() -> bool { return gg_copies_landed(a, bulk, bar); };
    const int tier = a.tier_out[tile];
    __syncthreads();
    if (F64 && tier == TIER_FP64) {
        // the FP64 bands are staged in the same memory: the discarded copies land first
        if constexpr (kFp64Call) {
            gg_tile_fp64_call<T, REF, NC>(a, sm, ntier, tile, tx, ty, red, spec, bulk, bar);
        } else {
            int tid = (int)threadIdx.x, x = tx, y = ty;
            if constexpr (REF) asm volatile("" : "+r"(tid), "+r"(tile), "+r"(x), "+r"(y), "+l"(sm)::"memory");
            if (spec && !spec_done()) return;
            if (spec && !bulk) __syncthreads();  // every thread's own copies
            gg_tile_fp64<T, REF, NC>(a, sm, ntier, tile, x, y, red, 0, T, gg_fp64_band(T, a.nf), tid);
        }
        return;
    }
    const bool all32 = all_fp32(ntier);
    if (spec) {
        if (!spec_done()) return;
        // mixed neighbourhood: the FP32-owned slots are in place; each thread
        // overwrites its own other slots with their converted values
        if (!all32) stage_tile<float, T, 1, true, NC>(a, sm, ntier, tx, ty, 0, a.nf);
    } else if (all32) {
        stage_tile_async32<T, 1>(a, sm, tx, ty, a.nf);
    } else {
        stage_tile<float, T, 1, false, NC>(a, sm, ntier, tx, ty, 0, a.nf);
    }
    __syncthreads();
    if (RG && gg_partial_tile(a, T, tx, ty)) {  // a ragged grid's edge tile: its wrapped halo
        patch_ragged<float, T>(a, sm, tx, ty);
        __syncthreads();
    }
    if constexpr (HA != 0) {
        if (tier == TIER_HALF) {
            gg_tile_half2<T, MK, HA>(a, sm, tile, tx, ty, red);
            return;
        }
    }
    if constexpr (T == 32) {
        // the spatial range needs one reduction per field: gg_tile_lo_impl
        float *ss = sm + a.nf * Stage<float, T, 1>::FIELD;  // gg_smem_bytes reserves it
        if (!MON) {
            // 8 rows a thread when the fields come in eights (one warp a field)
            if (a.nf % 8 == 0) {
                if (tier == TIER_FP32) gg_tile_lo_rows<TIER_FP32, 8>(a, sm, ss, tile, tx, ty, red);
                else gg_tile_lo_rows<TIER_HALF, 8>(a, sm, ss, tile, tx, ty, red);
            } else {
                if (tier == TIER_FP32) gg_tile_lo_rows<TIER_FP32, 4>(a, sm, ss, tile, tx, ty, red);
                else gg_tile_lo_rows<TIER_HALF, 4>(a, sm, ss, tile, tx, ty, red);
            }
            return;
        }
        if (MK == 3 && a.nf % 8 == 0) {
            if (tier == TIER_FP32) gg_tile_lo_rows<TIER_FP32, 8, 3>(a, sm, ss, tile, tx, ty, red);
            else gg_tile_lo_rows<TIER_HALF, 8, 3>(a, sm, ss, tile, tx, ty, red);
            return;
        }
        if (MK == 3 || (MK == -1 && a.monitor_kind == 3)) {
            if (tier == TIER_FP32) gg_tile_lo_rows<TIER_FP32, 4, 3>(a, sm, ss, tile, tx, ty, red);
            else gg_tile_lo_rows<TIER_HALF, 4, 3>(a, sm, ss, tile, tx, ty, red);
            return;
        }
        if (MK == 2 || (MK == -1 && a.monitor_kind == 2)) {
            if (tier == TIER_FP32) gg_tile_lo_rows<TIER_FP32, 4, 2>(a, sm, ss, tile, tx, ty, red);
            else gg_tile_lo_rows<TIER_HALF, 4, 2>(a, sm, ss, tile, tx, ty, red);
            return;
        }
    }
    if (tier == TIER_FP32) gg_tile_lo_impl<T, TIER_FP32, MON>(a, sm, tile, tx, ty, red);
    else gg_tile_lo_impl<T, TIER_HALF, MON>(a, sm, tile, tx, ty, red);
}

// Fused all-tier step: at most 64 registers, so that four CTAs share an SM.
// The monitor steps (one in `cadence`) are separate instantiations, one per
// monitor kind MK, so the other steps' kernel carries no monitor code and
// each monitor step's kernel only its own kind's.  Half/FP32 tiles stage
// their neighbourhood in shared memory (reading it directly through L1
// measured 18.1 against 15.8 us per adaptive 1024^2 Q=8 step).
// tm: the tensor map of the step's FP32 input, valid when a.tma_stage.
template <int T, bool REF, int MK, int HA = 0, bool RG = false, bool F64 = true>
__global__ void __launch_bounds__(kThreads, 4) gg_step_kernel(const __grid_constant__ StepArgs a, const __grid_constant__ CUtensorMap tm)
{
    extern __shared__ __align__(128) unsigned char smraw[];
    __shared__ double red[kThreads / 32];
    __shared__ uint8_t ntier[9];
    __shared__ __align__(8) uint64_t bar;
    // 128-byte aligned staging (gg_smem_bytes adds the slack), as tensor copies need
    float *sm = reinterpret_cast<float *>((reinterpret_cast<uintptr_t>(smraw) + 127) & ~uintptr_t(127));
    // programmatic dependent launch (gg_launch): the next step's CTAs may be
    // scheduled into the slots this grid's last wave leaves free; every CTA
    // waits for the previous grid to complete, its writes visible, before
    // its first global read (both are no-ops for a plain launch)
    pdl_trigger();
    pdl_wait();
    const int tile = a.order ? a.order[blockIdx.x] : (int)blockIdx.x;
    gg_tile_step<T, REF, MK, HA, true, RG, F64>(a, sm, ntier, red, tile, a.tma_stage ? &tm : nullptr, &bar);
}


}  // namespace amps
