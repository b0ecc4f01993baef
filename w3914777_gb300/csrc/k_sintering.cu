// k_sintering.cu -- fused solid-state sintering step: Cahn-Hilliard density c
// plus one Allen-Cahn order parameter per particle.
//
// The reference runs four kernels per step with full-size intermediates
// (sintering/function.h:51-79 con1_pure: mu; :80-108 con2_pure: c update;
// :110-159 phi1/phi2_pure: eta updates; sequenced in sintering/main.cu:136-147).
// Here one CTA per tile stages c with a 2-cell halo and every eta with a
// 1-cell halo, computes the chemical potential mu on the tile plus a 1-cell
// ring (phase A), then c' from lap(mu) and every eta' from c' and the old
// etas (phase B) -- the reference's operator splitting, in one pass.
// Generalised to N particles: sum_{i<j} 2 eta_i eta_j for the grain-boundary
// mobility term (the reference's 2*eta1*eta2, sintering/function.h:97) and
// sums over all eta in the bulk terms.
#include "amps_internal.cuh"
#include "amps_kernels.h"
#include <type_traits>

namespace amps {

// ---- per-cell arithmetic (non-reference order), shared by the whole-tile
// and the row-band paths.  C points at a cell's c with row stride cs; E at the
// cell's eta_0, field stride es, row stride rs.

// FP64 tiles are bound by the FP64 pipe, so their forms are arranged for few
// operations on it: constants folded on the host, per-cell factors formed once
// for all particles, clamps by integer tests, absent particles (+0 over the
// stencil) skipped -- 3 + 1 + 8 operations a present particle for mu, c and eta
// where the direct forms take 3 + 2 + 12.

// v clamped to [0, 1] (sintering/function.h:100-101): for 0 <= v < 1 an
// integer test of the high word.
__device__ __forceinline__ double clamp01(double v)
{
    if ((unsigned)__double2hiint(v) < 0x3ff00000u) return v;
    return v >= 1.0 ? 1.0 : (v < 0.0 ? 0.0 : v);
}
__device__ __forceinline__ float clamp01(float v) { return v >= 1.f ? 1.f : (v < 0.f ? 0.f : v); }

// Chemical potential mu at one cell (sintering/function.h:67-71) of an FP64
// tile; s2: the cell's sum of eta^2.
__device__ __forceinline__ double sint_mu64(const double *C, int cs, const double *E, int es, int np, const Phys &ph,
                                            double &s2)
{
    const double cc = C[0];
    const double lap = fma(-4.0, cc, C[-1] + C[1] + C[-cs] + C[cs]);
    double s3 = 0.0;
    s2 = 0.0;
    for (int k = 0; k < np; ++k) {
        const double e = E[k * es];
        if (pos_zero(e)) continue;  // adds +0 to sums that never hold -0
        s2 = fma(e, e, s2);
        s3 = fma(e * e, e, s3);
    }
    const double t = fma(2.0, cc, fma(4.0, s3, -6.0 * s2));
    const double c1 = 1.0 - cc;
    const double dfdc = fma(ph.kd[SN_B], t, ph.kd[SN_A2] * (cc * c1 * (c1 - cc)));
    return fma(-ph.kd[SN_HCMI], lap, dfdc);
}

// c' at one cell (sintering/function.h:90-100) of an FP64 tile, from the mu
// region M (row stride ms, M at the cell), s2 and the old etas.
__device__ __forceinline__ double sint_c64(double cc, const double *M, int ms, const double *E, int es, int np,
                                           const Phys &ph, double s2)
{
    const double lapm = fma(-4.0, M[0], M[-1] + M[1] + M[-ms] + M[ms]);
    const double c2 = cc * cc;
    const double phi = c2 * cc * fma(6.0, c2, fma(-15.0, cc, 10.0));
    double se = 0.0;
    for (int k = 0; k < np; ++k) {
        const double e = E[k * es];
        if (!pos_zero(e)) se += e;
    }
    const double sum = fma(se, se, -s2);  // sum_{i != j} eta_i eta_j
    const double mob = fma(ph.kd[SN_DGRB], sum,
                           fma(ph.kd[SN_DSUR], cc * (1.0 - cc), fma(ph.kd[SN_DVD], phi, ph.kd[SN_DVAP])));
    return clamp01(fma(ph.kd[SN_DTI] * mob, lapm, cc));
}

// The sum of eta^2 at one cell, as sint_mu64 forms it.
__device__ __forceinline__ double sint_s2(const double *E, int es, int np)
{
    double s2 = 0.0;
    for (int k = 0; k < np; ++k) {
        const double e = E[k * es];
        if (!pos_zero(e)) s2 = fma(e, e, s2);
    }
    return s2;
}

// The per-cell factors of the eta updates: 12B(2 - c') and 12B(s2 + 1 - c').
struct SintCell {
    double b2, bt;
    __device__ __forceinline__ SintCell(double cn, double s2, const Phys &ph)
        : b2(ph.kd[SN_B12] * (2.0 - cn)), bt(ph.kd[SN_B12] * (s2 + (1.0 - cn)))
    {
    }
};

// eta' of one particle at one cell (sintering/function.h:126-131) of an FP64
// tile; Ep at the cell's eta, row stride rs.
__device__ __forceinline__ double sint_eta64(const double *Ep, int rs, const SintCell &q, const Phys &ph)
{
    const double e = Ep[0];
    // a particle absent from the whole stencil stays absent (+0)
    if (pos_zero(e) && pos_zero(Ep[-1]) && pos_zero(Ep[1]) && pos_zero(Ep[-rs]) && pos_zero(Ep[rs])) return 0.0;
    const double lap = fma(-4.0, e, Ep[-1] + Ep[1] + Ep[-rs] + Ep[rs]);
    const double x = fma(e, fma(-e, q.b2, q.bt), -(ph.kd[SN_HCKI] * lap));
    return clamp01(fma(-ph.kd[SN_DTL], x, e));
}

// ---- half and FP32 tiles: float fields, mu in MT (double: mu_lap_fp64).

template <typename MT>
__device__ __forceinline__ MT sint_mu(const float *C, int cs, const float *E, int es, int np, const Phys &ph)
{
    const float cc = C[0];
    MT lap, s2 = 0, s3 = 0;
    bool exact = false;
    if constexpr (sizeof(MT) == 8) {
        // double mu from float inputs.  Where c and every eta are 0 or 1
        // (the bulk), the sums below are small integers, exact in float:
        // form them there and keep the FP64 pipe for the other cells.
        // The results are the double path's to the bit.  Where both are zero
        // -- in a particle and in a pore alike -- mu is +0, and no FP64
        // operation is left.
        bool bin = (cc == 0.f || cc == 1.f);
        float s2f = 0.f, s3f = 0.f;
        for (int k = 0; k < np; ++k) {
            const float e = E[k * es];
            bin &= (e == 0.f || e == 1.f);
            const float e2 = e * e;
            s2f += e2;
            s3f = fmaf(e2, e, s3f);
        }
        const float csum = C[-1] + C[1] + C[-cs] + C[cs];
        bin &= (C[-1] == 0.f || C[-1] == 1.f) && (C[1] == 0.f || C[1] == 1.f) && (C[-cs] == 0.f || C[-cs] == 1.f) &&
               (C[cs] == 0.f || C[cs] == 1.f);
        if (bin) {
            if (csum == 4.f * cc && 2.f * cc + 4.f * s3f == 6.f * s2f) return MT(0);
            exact = true;
            s2 = s2f;
            s3 = s3f;
            lap = ((MT)csum - MT(4) * (MT)cc) * kc<MT>(ph, SN_INV);
        }
    }
    if (!exact) {
        lap = ((MT)C[-1] + (MT)C[1] + (MT)C[-cs] + (MT)C[cs] - MT(4) * (MT)cc) * kc<MT>(ph, SN_INV);
        for (int k = 0; k < np; ++k) {
            const MT e = E[k * es];
            const MT e2 = e * e;
            s2 += e2;
            s3 = fma(e2, e, s3);
        }
    }
    const MT c1 = MT(1) - (MT)cc;
    const MT A2 = kc<MT>(ph, SN_A2);
    const MT dfdc = kc<MT>(ph, SN_B) * (MT(2) * (MT)cc + MT(4) * s3 - MT(6) * s2) + A2 * (MT)cc * c1 * (c1 - (MT)cc);
    return dfdc - kc<MT>(ph, SN_HCM) * lap;
}

// c' from the mu region M (row stride ms, M at the cell) and the old etas;
// s2f: sum of eta^2 at the cell.
template <typename MT>
__device__ __forceinline__ float sint_c_new(float cc, const MT *M, int ms, const float *E, int es, int np, const Phys &ph,
                                            float &s2f)
{
    const float phi = cc * cc * cc * fma(6.f * cc, cc, 10.f - 15.f * cc);
    float se = 0.f;
    s2f = 0.f;
    for (int k = 0; k < np; ++k) {
        const float e = E[k * es];
        se += e;
        s2f = fma(e, e, s2f);
    }
    if constexpr (sizeof(MT) == 8) {
        // mu +0 over the stencil (the bulk): its Laplacian is 0 and c stays,
        // without an FP64 operation
        if (pos_zero(M[0]) && pos_zero(M[-1]) && pos_zero(M[1]) && pos_zero(M[-ms]) && pos_zero(M[ms])) return clamp01(cc);
    }
    const MT lapm = (M[-1] + M[1] + M[-ms] + M[ms] - MT(4) * M[0]) * kc<MT>(ph, SN_INV);
    const float sum = se * se - s2f;  // sum_{i != j} eta_i eta_j
    const float mob = kc<float>(ph, SN_DVOL) * phi + kc<float>(ph, SN_DVAP) * (1.f - phi) +
                      kc<float>(ph, SN_DSUR) * cc * (1.f - cc) + kc<float>(ph, SN_DGRB) * sum;
    return clamp01((float)((MT)cc + (MT)(kc<float>(ph, SN_DT) * mob) * lapm));
}

// eta' of one particle; Ep at the cell's eta, row stride rs.
__device__ __forceinline__ float sint_eta_new(const float *Ep, int rs, float cn, float s2f, const Phys &ph)
{
    const float e = Ep[0];
    const float lap = (Ep[-1] + Ep[1] + Ep[-rs] + Ep[rs] - 4.f * e) * kc<float>(ph, SN_INV);
    const float dfd = kc<float>(ph, SN_B12) * e * (s2f + (1.f - cn) - e * (2.f - cn));
    return clamp01(fma(-kc<float>(ph, SN_DTL), fma(-kc<float>(ph, SN_HCK), lap, dfd), e));
}

// Threads of a tile CTA: the staging of a 32^2 tile with 16 particles leaves
// room for two CTAs an SM (one at FP64), so 512 threads a CTA, for warps that
// hide the serial sums over the particles (1024^2 with 16: 131 us a step with
// 256, 120 with 512 and the FP64 bands' changes).  Plain FP64 runs in the
// reference's order, which take whole tiles at every step, of 256^2 to 1024^2
// cells and 2 or 4 particles: 0.70 to 1.005 of the time with 256.
// One tile of one step at tier TIER (smraw: the kernel's dynamic shared
// memory, sint_smem<T, TIER, MU64> bytes; red / ntier: its static scratch).
// NT: the CTA's threads (sint_threads).
template <int T> constexpr int sint_threads() { return T == 32 ? 512 : 256; }

template <int T, int TIER, bool REF, bool MU64, int NT = sint_threads<T>()>
__device__ __forceinline__ void sint_tile(const StepArgs &a, unsigned char *smraw, double *red, uint8_t *ntier,
                                          int tile)
{
    using CT = typename std::conditional<TIER == TIER_FP64, double, float>::type;
    using MT = typename std::conditional<MU64, double, CT>::type;  // type of mu and lap(mu)
    using SC = Stage<CT, T, 2>;
    using SE = Stage<CT, T, 1>;
    constexpr int E = T + 2;
    MT *mu = reinterpret_cast<MT *>(smraw);                       // [E*E]
    CT *smc = reinterpret_cast<CT *>(smraw + sizeof(MT) * E * E);  // c, 2-cell halo
    CT *sme = smc + SC::FIELD;                                     // etas, 1-cell halo
    const int tx = tile % a.ntx, ty = tile / a.ntx;
    const int x0 = tx * T, y0 = ty * T;
    const int np = a.nf - 1;
    load_neighbour_tiers(a, tx, ty, ntier);
    __syncthreads();
    stage_tile<CT, T, 2, false, true, NT>(a, smc, ntier, tx, ty, 0, 1);
    stage_tile<CT, T, 1, false, true, NT>(a, sme, ntier, tx, ty, 1, np);
    __syncthreads();
    const Phys &ph = a.ph;

    // phase A: mu on the tile + ring (sintering/function.h:67-71)
    for (int u = threadIdx.x; u < E * E; u += NT) {
        int i = u % E - 1, j = u / E - 1;
        if (a.bc != 0) {
            i = bc_map(x0 + i, a.nx, 1) - x0;
            j = bc_map(y0 + j, a.ny, 1) - y0;
        }
        const CT *C = &SC::at(smc, 0, j + 2, i + SC::O);
        const CT cc = C[0];
        MT m;
        if (REF) {
            const double lap = __ddiv_rn(__dsub_rn(__dadd_rn(__dadd_rn(__dadd_rn(C[-1], C[1]), C[-SC::P]), C[SC::P]),
                                                   __dmul_rn(4.0, cc)), ph.dxdy);
            double e0 = SE::at(sme, 0, j + 1, i + SE::O);
            double s2 = __dmul_rn(e0, e0), s3 = cube_rn(e0);
            for (int k = 1; k < np; ++k) {
                const double e = SE::at(sme, k, j + 1, i + SE::O);
                s2 = __dadd_rn(s2, __dmul_rn(e, e));
                s3 = __dadd_rn(s3, cube_rn(e));
            }
            const double A2 = 2.0 * ph.A;
            const double dfdc = __dadd_rn(
                __dsub_rn(__dmul_rn(ph.B, __dsub_rn(__dadd_rn(__dmul_rn(2.0, cc), __dmul_rn(4.0, s3)), __dmul_rn(6.0, s2))),
                          __dmul_rn(__dmul_rn(A2, __dmul_rn(cc, cc)), __dsub_rn(1.0, cc))),
                __dmul_rn(__dmul_rn(A2, cc), __dmul_rn(__dsub_rn(1.0, cc), __dsub_rn(1.0, cc))));
            m = __dsub_rn(dfdc, __dmul_rn(0.5 * ph.coefm, lap));
        } else if constexpr (TIER == TIER_FP64) {
            double s2;
            m = sint_mu64(C, SC::P, &SE::at(sme, 0, j + 1, i + SE::O), SE::FIELD, np, ph, s2);
        } else {
            m = sint_mu<MT>(C, SC::P, &SE::at(sme, 0, j + 1, i + SE::O), SE::FIELD, np, ph);
        }
        mu[u] = m;
    }
    __syncthreads();

    // phase B: c' (sintering/function.h:90-100), then eta_i' (:126-131)
    double metric = 0.0;
    // half/FP32 tiles fold their float values into a float accumulator (the
    // same metric, without FP64 operations per cell)
    using MA = typename std::conditional<TIER == TIER_FP64, MonAcc, MonAccF>::type;
    MA mon;
    const bool mon_on = a.monitor_now != 0;
    if (mon_on) mon_reset(a, mon);
    for (int u = threadIdx.x; u < T * T; u += NT) {
        const int i = u % T, j = u / T;
        const int o = (j + 1) * E + (i + 1);
        const int64_t g = (int64_t)(y0 + j) * a.nx + x0 + i;
        const CT cc = SC::at(smc, 0, j + 2, i + SC::O);
        CT cn;
        double s2ref = 0.0;
        CT s2f = 0;
        if (REF) {
            const double lapm = __ddiv_rn(__dsub_rn(__dadd_rn(__dadd_rn(__dadd_rn(mu[o - 1], mu[o + 1]), mu[o - E]), mu[o + E]),
                                                    __dmul_rn(4.0, mu[o])), ph.dxdy);
            const double phi = __dmul_rn(cube_rn((double)cc),
                                         __dadd_rn(__dsub_rn(10.0, __dmul_rn(15.0, cc)), __dmul_rn(6.0, __dmul_rn(cc, cc))));
            double sum = 0.0;
            for (int p = 0; p < np; ++p)
                for (int q = p + 1; q < np; ++q)
                    sum = __dadd_rn(sum, __dmul_rn(__dmul_rn(SE::at(sme, p, j + 1, i + SE::O), SE::at(sme, q, j + 1, i + SE::O)), 2.0));
            const double mob = __dadd_rn(__dadd_rn(__dadd_rn(__dmul_rn(ph.dvol, phi), __dmul_rn(ph.dvap, __dsub_rn(1.0, phi))),
                                                   __dmul_rn(__dmul_rn(ph.dsur, cc), __dsub_rn(1.0, cc))),
                                         __dmul_rn(ph.dgrb, sum));
            double v = __dadd_rn(cc, __dmul_rn(__dmul_rn(ph.dt, mob), lapm));
            if (v >= 1) v = 1;
            else if (v < 0) v = 0;
            cn = v;
            double e0 = SE::at(sme, 0, j + 1, i + SE::O);
            s2ref = __dmul_rn(e0, e0);
            for (int k = 1; k < np; ++k) {
                const double e = SE::at(sme, k, j + 1, i + SE::O);
                s2ref = __dadd_rn(s2ref, __dmul_rn(e, e));
            }
        } else if constexpr (TIER == TIER_FP64) {
            const double *Ec = &SE::at(sme, 0, j + 1, i + SE::O);
            s2f = sint_s2(Ec, SE::FIELD, np);
            cn = sint_c64(cc, mu + o, E, Ec, SE::FIELD, np, ph, s2f);
        } else {
            cn = sint_c_new<MT>(cc, mu + o, E, &SE::at(sme, 0, j + 1, i + SE::O), SE::FIELD, np, ph, s2f);
        }
        store_tier<TIER>(a, g, cn);
        if (mon_on && a.mfield <= 0)
            mon_add<T>(a, mon, 0, tile, j, i, g, (CT)round_to_tier<TIER>(cn), cc,
                       snap_prefetch<T>(a, 0, tile, j, i, g));
        for (int k = 0; k < np; ++k) {
            const CT *Ep = &SE::at(sme, k, j + 1, i + SE::O);
            const CT e = Ep[0];
            CT en;
            if (REF) {
                const double lap = __ddiv_rn(__dsub_rn(__dadd_rn(__dadd_rn(__dadd_rn(Ep[-1], Ep[1]), Ep[-SE::P]), Ep[SE::P]),
                                                       __dmul_rn(4.0, e)), ph.dxdy);
                const double cnd = cn;
                const double dfd = __dmul_rn(ph.B, __dadd_rn(__dadd_rn(
                    __dmul_rn(__dmul_rn(-12.0, __dmul_rn(e, e)), __dsub_rn(2.0, cnd)),
                    __dmul_rn(__dmul_rn(12.0, e), __dsub_rn(1.0, cnd))), __dmul_rn(__dmul_rn(12.0, e), s2ref)));
                double v = __dsub_rn(e, __dmul_rn(ph.dt * ph.coefl, __dsub_rn(dfd, __dmul_rn(0.5 * ph.coefk, lap))));
                if (v >= 1) v = 1;
                else if (v < 0) v = 0;
                en = v;
            } else if constexpr (TIER == TIER_FP64) {
                en = sint_eta64(Ep, SE::P, SintCell(cn, s2f, ph), ph);
            } else {
                en = sint_eta_new(Ep, SE::P, cn, s2f, ph);
            }
            store_tier<TIER>(a, (int64_t)(k + 1) * a.n + g, en);
        }
    }
    if (mon_on) {
        metric = mon_finish<NT>(a, mon, red, metric);
        if (threadIdx.x == 0) a.metric[tile] = metric;
    }
}

// A half or FP32 tile of 32^2 with mu in double (the default), 512 threads, four
// cells of a row a thread where the work is per particle: one 16-byte load
// brings four cells, so an eta update reads five words of shared memory where
// a cell at a time reads twenty, and a particle that is +0 over a thread's
// stencil (most particles, nearly everywhere) is left at +0 after one integer
// test.  The per-cell arithmetic is sint_mu's, sint_c_new's and sint_eta_new's.
//   A  mu on the tile + ring: rows of four-cell groups, then the two side columns;
//   B1 c' and the sum of eta^2, two cells a thread; the per-cell factors of
//      the eta updates replace mu in shared memory;
//   B2 eta', half of the threads the even particles, half the odd.
// 1024^2, 16 particles (85% bulk), the half/FP32 launch alone: 98 us with FP64
// in every cell's mu, 72 with none in the bulk, 60 in this form.
__device__ __forceinline__ void sint_tile_lo32(const StepArgs &a, unsigned char *smraw, double *red, uint8_t *ntier,
                                               int tile, bool half)
{
    constexpr int T = 32, NT = 512, E = T + 2;
    using SC = Stage<float, T, 2>;
    using SE = Stage<float, T, 1>;
    double *mu = reinterpret_cast<double *>(smraw);                            // [E*E]
    float *smc = reinterpret_cast<float *>(smraw + sizeof(double) * E * E);  // c, 2-cell halo
    float *sme = smc + SC::FIELD;                                              // etas, 1-cell halo
    float *sq = reinterpret_cast<float *>(smraw), *st = sq + T * T;           // after B1: 2 - c', s2 + (1 - c')
    const int tx = tile % a.ntx, ty = tile / a.ntx;
    const int x0 = tx * T, y0 = ty * T;
    const int np = a.nf - 1, tid = threadIdx.x;
    load_neighbour_tiers(a, tx, ty, ntier);
    __syncthreads();
    {  // each half of the CTA stages half of the particles, the first also c
        const int n0 = (np - 1) / 2;
        if (tid < 256) {
            stage_tile<float, T, 2, false, true, 256>(a, smc, ntier, tx, ty, 0, 1, tid);
            stage_tile<float, T, 1, false, true, 256>(a, sme, ntier, tx, ty, 1, n0, tid);
        } else {
            stage_tile<float, T, 1, false, true, 256>(a, sme + n0 * SE::FIELD, ntier, tx, ty, 1 + n0, np - n0, tid - 256);
        }
    }
    __syncthreads();
    const Phys &ph = a.ph;

    // A
    for (int u = tid; u < E * 8 + 2 * E; u += NT) {
        const bool group = u < E * 8;
        const int r = group ? u / 8 : (u - E * 8) / 2;
        int j = r - 1, i = group ? u % 8 * 4 : ((u - E * 8) % 2 ? T : -1);
        const int o = r * E + i + 1;
        if (a.bc != 0) {
            j = bc_map(y0 + j, a.ny, 1) - y0;
            if (!group) i = bc_map(x0 + i, a.nx, 1) - x0;
        }
        const float *C = &SC::at(smc, 0, j + 2, i + SC::O), *Ec = &SE::at(sme, 0, j + 1, i + SE::O);
        if (!group) {
            mu[o] = sint_mu<double>(C, SC::P, Ec, SE::FIELD, np, ph);
            continue;
        }
        // the bulk, four cells at once: c, its neighbours and every eta 0 or 1
        // (x*x == x) and both sums zero -> mu = +0; other cells one by one
        const float4 cm = *reinterpret_cast<const float4 *>(C), cu = *reinterpret_cast<const float4 *>(C - SC::P),
                     cd = *reinterpret_cast<const float4 *>(C + SC::P);
        const float w[6] = {C[-1], cm.x, cm.y, cm.z, cm.w, C[4]};
        const float up[4] = {cu.x, cu.y, cu.z, cu.w}, dn[4] = {cd.x, cd.y, cd.z, cd.w};
        bool bin[4];
        float s2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < 4; ++k)
            bin[k] = w[k] * w[k] == w[k] && w[k + 1] * w[k + 1] == w[k + 1] && w[k + 2] * w[k + 2] == w[k + 2] &&
                     up[k] * up[k] == up[k] && dn[k] * dn[k] == dn[k];
#pragma unroll 4
        for (int f = 0; f < np; ++f) {
            const float4 q = *reinterpret_cast<const float4 *>(Ec + f * SE::FIELD);
            const float e[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float e2 = e[k] * e[k];
                bin[k] = bin[k] && e2 == e[k];
                s2[k] += e2;
            }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            // (where every eta is 0 or 1 the sums of squares and cubes are equal;
            // x*x == x holds for +infinity too, which the sums then show)
            const bool zero = bin[k] && w[k + 1] < INFINITY && w[k] + w[k + 2] + dn[k] + up[k] == 4.f * w[k + 1] && w[k + 1] == s2[k];
            mu[o + k] = zero ? 0.0 : sint_mu<double>(C + k, SC::P, Ec + k, SE::FIELD, np, ph);
        }
    }
    __syncthreads();

    // B1
    double metric = 0.0;
    MonAccF mon;
    const bool mon_on = a.monitor_now != 0;
    if (mon_on) mon_reset(a, mon);
    {
        const int j = tid / 16, i = tid % 16 * 2;
        const int64_t g = (int64_t)(y0 + j) * a.nx + x0 + i;
        float cn[2], s2[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float cc = SC::at(smc, 0, j + 2, i + k + SC::O);
            cn[k] = sint_c_new<double>(cc, mu + (j + 1) * E + i + k + 1, E, &SE::at(sme, 0, j + 1, i + k + SE::O),
                                       SE::FIELD, np, ph, s2[k]);
            if (mon_on && a.mfield <= 0)
                mon_add<T>(a, mon, 0, tile, j, i + k, g + k, half ? __half2float(__float2half_rn(cn[k])) : cn[k], cc,
                           snap_prefetch<T>(a, 0, tile, j, i + k, g + k));
        }
        if (half) *reinterpret_cast<__half2 *>((__half *)a.out[TIER_HALF] + g) = __floats2half2_rn(cn[0], cn[1]);
        else *reinterpret_cast<float2 *>((float *)a.out[TIER_FP32] + g) = make_float2(cn[0], cn[1]);
        __syncthreads();  // mu is read no more
        *reinterpret_cast<float2 *>(sq + j * T + i) = make_float2(2.f - cn[0], 2.f - cn[1]);
        *reinterpret_cast<float2 *>(st + j * T + i) = make_float2(s2[0] + (1.f - cn[0]), s2[1] + (1.f - cn[1]));
    }
    __syncthreads();

    // B2
    {
        const int j = tid % 256 / 8, i = tid % 8 * 4;
        const int64_t g = (int64_t)(y0 + j) * a.nx + x0 + i;
        const float4 q4 = *reinterpret_cast<const float4 *>(sq + j * T + i);
        const float4 t4 = *reinterpret_cast<const float4 *>(st + j * T + i);
        const float q[4] = {q4.x, q4.y, q4.z, q4.w}, t[4] = {t4.x, t4.y, t4.z, t4.w};
        // (a NaN or infinity in the factors reaches every particle)
        const bool finite = fabsf(t[0]) < INFINITY && fabsf(t[1]) < INFINITY && fabsf(t[2]) < INFINITY && fabsf(t[3]) < INFINITY;
        const float inv = kc<float>(ph, SN_INV), b12 = kc<float>(ph, SN_B12), dtl = kc<float>(ph, SN_DTL),
                    hck = kc<float>(ph, SN_HCK);
#pragma unroll 2
        for (int f = tid / 256; f < np; f += 2) {
            const float *Ep = &SE::at(sme, f, j + 1, i + SE::O);
            const float4 m = *reinterpret_cast<const float4 *>(Ep), u = *reinterpret_cast<const float4 *>(Ep - SE::P),
                         d = *reinterpret_cast<const float4 *>(Ep + SE::P);
            const float w[6] = {Ep[-1], m.x, m.y, m.z, m.w, Ep[4]};
            const float up[4] = {u.x, u.y, u.z, u.w}, dn[4] = {d.x, d.y, d.z, d.w};
            unsigned any = __float_as_uint(w[0]) | __float_as_uint(w[5]);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                any |= __float_as_uint(w[k + 1]) | __float_as_uint(up[k]) | __float_as_uint(dn[k]);
            float o[4] = {0.f, 0.f, 0.f, 0.f};
            if (any != 0u || !finite) {
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float e = w[k + 1];
                    const float lap = (w[k] + w[k + 2] + up[k] + dn[k] - 4.f * e) * inv;
                    const float dfd = b12 * e * (t[k] - e * q[k]);
                    o[k] = clamp01(fmaf(-dtl, fmaf(-hck, lap, dfd), e));
                }
            }
            const int64_t go = (int64_t)(f + 1) * a.n + g;
            if (half) {
                const __half2 h0 = __floats2half2_rn(o[0], o[1]), h1 = __floats2half2_rn(o[2], o[3]);
                uint2 v;
                v.x = *reinterpret_cast<const unsigned *>(&h0);
                v.y = *reinterpret_cast<const unsigned *>(&h1);
                *reinterpret_cast<uint2 *>((__half *)a.out[TIER_HALF] + go) = v;
            } else {
                *reinterpret_cast<float4 *>((float *)a.out[TIER_FP32] + go) = make_float4(o[0], o[1], o[2], o[3]);
            }
        }
    }
    if (mon_on) {
        metric = mon_finish<NT>(a, mon, red, metric);
        if (tid == 0) a.metric[tile] = metric;
    }
}

// ---- FP64 tiles in row bands ----------------------------------------------
// An FP64 tile of a non-monitor step (non-reference order) is split into
// T / kBandRows row bands, one CTA each: 4x the parallelism on the
// latency-bound FP64 arithmetic, and ~50 KB of shared memory instead of the
// whole tile's ~176 KB, so half/FP32 CTAs share the SM.  A band stages its
// rows of c (2-cell halo) and of every eta (1-cell halo) in double, forms mu on
// its rows + a 1-cell ring, then c' and every eta' -- the whole-tile path's
// per-cell arithmetic (sint_mu64, sint_c64, sint_eta64), so the same bits.

template <int T> struct SintBand {
    static constexpr int BR = kBandRows, NB = T / BR;
    static constexpr int W1 = T + 4, H1 = BR + 2, FE = W1 * H1;  // etas (tile column 0 at column 2, as c)
    static constexpr int W2 = T + 4, H2 = BR + 4;                // c
    static constexpr int WM = T + 2, HM = BR + 2;                // mu, and sum of eta^2
    static size_t smem(int np) { return sizeof(double) * ((size_t)np * FE + W2 * H2 + 2 * WM * HM); }
};

// Threads: the band and its ring (10 x 34 or 10 x 18 cells) in one pass.
template <int T> constexpr int sint_band_threads() { return T == 32 ? 352 : 192; }

template <int T>
__global__ void __launch_bounds__(sint_band_threads<T>(), 4)
    sint_step_f64_band_kernel(const __grid_constant__ StepArgs a)
{
    using B = SintBand<T>;
    constexpr int NT = sint_band_threads<T>();
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ uint8_t ntier[9];
    // launched programmatically after the previous step's last grid: wait
    // for it, then release the step's half/FP32 launch (FP64 launch first)
    pdl_wait();
    pdl_trigger();
    const int np = a.nf - 1, items = a.count[TIER_FP64] * B::NB;
    double *sme = reinterpret_cast<double *>(smraw);  // [np][H1][W1]
    double *smc = sme + np * B::FE;                   // [H2][W2]
    double *mu = smc + B::W2 * B::H2, *sum2 = mu + B::WM * B::HM;  // [HM][WM]
    const Phys &ph = a.ph;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int tile = a.list[it / B::NB], band = it % B::NB;
        const int tx = tile % a.ntx, ty = tile / a.ntx;
        const int x0 = tx * T, y0 = ty * T, ly0 = band * B::BR;
        load_neighbour_tiers(a, tx, ty, ntier);
        __syncthreads();  // (also: the previous item's reads of the staging)
        stage_band<T, 2, NT>(a, smc, ntier, tx, ty, ly0 - 2, B::H2, 0, 1);
        stage_band<T, 1, NT>(a, sme, ntier, tx, ty, ly0 - 1, B::H1, 1, np);
        stage_band_wait();
        __syncthreads();
        // mu on the band + ring; with zero flux an out-of-domain ring cell takes
        // the mu of the cell it mirrors, which lies in the same band
        for (int u = threadIdx.x; u < B::WM * B::HM; u += NT) {
            int ly = ly0 - 1 + u / B::WM, lx = u % B::WM - 1;
            if (a.bc != 0) {
                lx = bc_map(x0 + lx, a.nx, 1) - x0;
                ly = bc_map(y0 + ly, a.ny, 1) - y0;
            }
            const double *C = smc + (ly - (ly0 - 2)) * B::W2 + lx + 2;
            const double *E = sme + (ly - (ly0 - 1)) * B::W1 + lx + 2;
            mu[u] = sint_mu64(C, B::W2, E, B::FE, np, ph, sum2[u]);
        }
        __syncthreads();
        for (int u = threadIdx.x; u < B::BR * T; u += NT) {
            const int jb = u / T, i = u % T;
            const int64_t g = (int64_t)(y0 + ly0 + jb) * a.nx + x0 + i;
            const double cc = smc[(jb + 2) * B::W2 + i + 2];
            const double *E = sme + (jb + 1) * B::W1 + i + 2;
            const int m = (jb + 1) * B::WM + i + 1;
            const double cn = sint_c64(cc, mu + m, B::WM, E, B::FE, np, ph, sum2[m]);
            store_tier<TIER_FP64>(a, g, cn);
            const SintCell q(cn, sum2[m], ph);
            for (int k = 0; k < np; ++k)
                store_tier<TIER_FP64>(a, (int64_t)(k + 1) * a.n + g, sint_eta64(E + k * B::FE, B::W1, q, ph));
        }
    }
}

// The tiles of one tier (list / count built by the classification).
// Launched programmatically after the previous step's last grid: its CTAs
// wait for that grid, then release the step's half/FP32 launch, which runs
// alongside (FP64 launch first).
template <int T, int TIER, bool REF, bool MU64>
__global__ void __launch_bounds__(sint_threads<T>()) sint_step_kernel(StepArgs a)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double red[sint_threads<T>() / 32];
    __shared__ uint8_t ntier[9];
    pdl_wait();
    pdl_trigger();
    if ((int)blockIdx.x >= a.count[TIER]) return;
    sint_tile<T, TIER, REF, MU64>(a, smraw, red, ntier, a.list[blockIdx.x]);
}

// The half and FP32 tiles of a step in one launch (one CTA per tile; FP64
// tiles, whose double staging needs more shared memory, are left to the FP64
// launch).  Separate half and FP32 launches would each cover only part of
// the grid and run one after the other.  After the step's FP64 launch it is
// launched to run alongside it (disjoint tiles and output stores; both read
// the previous step's state only); its last CTA waits for the FP64 grid
// before it exits, so this grid completes after both.
template <int T, bool MU64>
__global__ void __launch_bounds__(sint_threads<T>()) sint_step_lo_kernel(const __grid_constant__ StepArgs a)
{
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double red[sint_threads<T>() / 32];
    __shared__ uint8_t ntier[9];
    const int tile = blockIdx.x;
    const int tier = a.tier_out[tile];
    if constexpr (T == 32 && MU64) {
        if (tier != TIER_FP64) sint_tile_lo32(a, smraw, red, ntier, tile, tier == TIER_HALF);
    } else {
        if (tier == TIER_FP32) sint_tile<T, TIER_FP32, false, MU64>(a, smraw, red, ntier, tile);
        else if (tier == TIER_HALF) sint_tile<T, TIER_HALF, false, MU64>(a, smraw, red, ntier, tile);
    }
    if (blockIdx.x == gridDim.x - 1) pdl_wait();
}

template <int T, int TIER, bool MU64> static size_t sint_smem(int nf)
{
    using CT = typename std::conditional<TIER == TIER_FP64, double, float>::type;
    using MT = typename std::conditional<MU64, double, CT>::type;
    return sizeof(MT) * (T + 2) * (T + 2) + sizeof(CT) * ((size_t)Stage<CT, T, 2>::FIELD
                                                          + (size_t)(nf - 1) * Stage<CT, T, 1>::FIELD);
}

template <int T, int TIER, bool REF, bool MU64>
static cudaError_t sint_launch_t(const StepArgs &a, int grid, cudaStream_t s, bool pdl)
{
    return launch_kernel_nt(sint_step_kernel<T, TIER, REF, MU64>, grid, sint_threads<T>(), sint_smem<T, TIER, MU64>(a.nf),
                            s, pdl, a);
}

size_t sint_smem_bytes(int tile, int tier, int nf, bool mu64)
{
    if (tile == 32) {
        if (tier == TIER_FP64) return sint_smem<32, TIER_FP64, true>(nf);
        return mu64 ? sint_smem<32, TIER_FP32, true>(nf) : sint_smem<32, TIER_FP32, false>(nf);
    }
    if (tier == TIER_FP64) return sint_smem<16, TIER_FP64, true>(nf);
    return mu64 ? sint_smem<16, TIER_FP32, true>(nf) : sint_smem<16, TIER_FP32, false>(nf);
}

// Where other tiers are in use most tiles are not FP64: CTAs enough to fill
// the SMs once, which loop over the bands, instead of a CTA for every band
// of the grid (4096 CTAs of which 572 had a band, 1024^2 with 16 particles: the
// FP64 launch alone 64 us, 59 with 608).
template <int T> static cudaError_t sint_launch_band(const StepArgs &a, int grid, int np, cudaStream_t s, bool pdl)
{
    const bool mixed = a.in[TIER_HALF] != nullptr || a.in[TIER_FP32] != nullptr;
    const int n = grid * SintBand<T>::NB, ctas = mixed && n > 4 * 152 ? 4 * 152 : n;
    return launch_kernel_nt(sint_step_f64_band_kernel<T>, ctas, sint_band_threads<T>(), SintBand<T>::smem(np), s, pdl, a);
}

cudaError_t sint_launch(int tile, int tier, bool ref, bool mu64, const StepArgs &a, int grid, cudaStream_t s,
                        bool pdl)
{
    if (tier == TIER_FP64 && !ref && !a.monitor_now) {  // row bands (the monitor needs whole tiles)
        const int np = a.nf - 1;
        return tile == 32 ? sint_launch_band<32>(a, grid, np, s, pdl) : sint_launch_band<16>(a, grid, np, s, pdl);
    }
#define AMPS_SINT(TT)                                                                              \
    switch (tier) {                                                                                \
    case TIER_HALF:                                                                                \
        return mu64 ? sint_launch_t<TT, TIER_HALF, false, true>(a, grid, s, pdl)                        \
                    : sint_launch_t<TT, TIER_HALF, false, false>(a, grid, s, pdl);                      \
    case TIER_FP32:                                                                                \
        return mu64 ? sint_launch_t<TT, TIER_FP32, false, true>(a, grid, s, pdl)                        \
                    : sint_launch_t<TT, TIER_FP32, false, false>(a, grid, s, pdl);                      \
    default:                                                                                       \
        return ref ? sint_launch_t<TT, TIER_FP64, true, true>(a, grid, s, pdl)                          \
                   : sint_launch_t<TT, TIER_FP64, false, true>(a, grid, s, pdl);                        \
    }
    if (tile == 32) { AMPS_SINT(32) }
    AMPS_SINT(16)
#undef AMPS_SINT
}

cudaError_t sint_launch_lo(int tile, bool mu64, const StepArgs &a, int grid, cudaStream_t s, bool after64)
{
#define AMPS_SLO(TT, MM) \
    return launch_kernel_nt(sint_step_lo_kernel<TT, MM>, grid, sint_threads<TT>(), sint_smem<TT, TIER_FP32, MM>(a.nf), s, \
                            after64, a)
    if (tile == 32) {
        if (mu64) AMPS_SLO(32, true);
        AMPS_SLO(32, false);
    }
    if (mu64) AMPS_SLO(16, true);
    AMPS_SLO(16, false);
#undef AMPS_SLO
}

cudaError_t sint_prepare_lo(int tile, bool mu64)
{
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if (tile == 32)
        return mu64 ? cudaFuncSetAttribute(sint_step_lo_kernel<32, true>, attr, kMaxDynSmem)
                    : cudaFuncSetAttribute(sint_step_lo_kernel<32, false>, attr, kMaxDynSmem);
    return mu64 ? cudaFuncSetAttribute(sint_step_lo_kernel<16, true>, attr, kMaxDynSmem)
                : cudaFuncSetAttribute(sint_step_lo_kernel<16, false>, attr, kMaxDynSmem);
}

cudaError_t sint_prepare(int tile, int tier, bool ref, bool mu64)
{
    const int lim = kMaxDynSmem;
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if (tier == TIER_FP64 && !ref) {
        const cudaError_t e = tile == 32 ? cudaFuncSetAttribute(sint_step_f64_band_kernel<32>, attr, lim)
                                         : cudaFuncSetAttribute(sint_step_f64_band_kernel<16>, attr, lim);
        if (e != cudaSuccess) return e;
    }
#define AMPS_SP(TT)                                                                                      \
    switch (tier) {                                                                                      \
    case TIER_HALF:                                                                                      \
        return mu64 ? cudaFuncSetAttribute(sint_step_kernel<TT, TIER_HALF, false, true>, attr, lim)      \
                    : cudaFuncSetAttribute(sint_step_kernel<TT, TIER_HALF, false, false>, attr, lim);    \
    case TIER_FP32:                                                                                      \
        return mu64 ? cudaFuncSetAttribute(sint_step_kernel<TT, TIER_FP32, false, true>, attr, lim)      \
                    : cudaFuncSetAttribute(sint_step_kernel<TT, TIER_FP32, false, false>, attr, lim);    \
    default:                                                                                             \
        return ref ? cudaFuncSetAttribute(sint_step_kernel<TT, TIER_FP64, true, true>, attr, lim)        \
                   : cudaFuncSetAttribute(sint_step_kernel<TT, TIER_FP64, false, true>, attr, lim);      \
    }
    if (tile == 32) { AMPS_SP(32) }
    AMPS_SP(16)
#undef AMPS_SP
}

}  // namespace amps
