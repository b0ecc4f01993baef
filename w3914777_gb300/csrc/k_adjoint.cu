// k_adjoint.cu -- explicit time step, its hand-written adjoint, and a
// checkpointed rollout for the Kobayashi dendrite and grain growth, on
// row-major device arrays (float or double).  No reference counterpart (the
// reference is forward-only); the step restated is snowflake/function.h:5-60
// and graingrowth/function.h:5-30.
//
// Kobayashi step, per cell (periodic or zero-flux neighbour map M):
//   px = (phi[M(x+1)] - phi[M(x-1)]) / 2dx,  py likewise,  a = aniso*(atan2(py,px) - theta0)
//   eps = epsb*(1 + delta*cos a),  epd = -epsb*aniso*delta*sin a
//   lap = (sum of phi at the 8 radius-2 cross neighbours - 8 phi) / dxdy
//   term1 = ((eps*epd*px)[M(y+1)] - (eps*epd*px)[M(y-1)]) / 2dy
//   term2 = -((eps*epd*py)[M(x+1)] - (eps*epd*py)[M(x-1)]) / 2dx
//   m = alpha/pi*atan(gama*(teq - T)),  g = phi*(1-phi)*(phi - 1/2 + m + noise*chi)
//   phi' = phi + dt/tau*(term1 + term2 + eps^2*lap + g),  T' = T + dt*lapT + K*(phi' - phi)
// The adjoint maps output cotangents (gphi', gT') to input cotangents and adds
// dL/d(delta, K, epsb) into a device double[3].  Each step is ONE fused
// kernel: a CTA stages its tile plus halo (radius 2 forward, 3 adjoint) in
// shared memory, computes the intermediates there, and applies the stencil
// transposes from shared memory.  Zero-flux (mirror) boundaries are
// differentiated exactly: about a face the mirror makes a symmetric sum over
// offsets +-k a symmetric matrix, and the transpose of a central difference the
// negative difference of the odd extension (f(-1) = -f(0)), so a transpose is a
// stencil on cotangents extended by even or odd reflection.
//
// Grain growth: eta_k' = eta_k - dt*L*(dfd_k - kappa*lap eta_k),
//   dfd_k = eta_k*(eta_k^2 - 1 + 2*gamma*(S - eta_k^2)),  S = sum_j eta_j^2;
// gradients w.r.t. (L, kappa, gamma).
//
// Parameter values and the noise step origin can come from device memory
// (ParamSrc), so a captured CUDA graph of a whole rollout stays valid when
// they change between calls.
#include "../../include/amps.h"
#include "amps_internal.cuh"

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include <new>
#include <type_traits>
#include <vector>

namespace {

using amps::pdl_trigger;
using amps::pdl_wait;

constexpr int kAdjThreads = 256;
constexpr int kMaxAdjSmem = 226 * 1024;  // dynamic shared memory opt-in limit

// Constants of the Kobayashi kernels in the compute type, rounded on the host.
template <typename R> struct KobAdj {
    int nx, ny, bc;
    int mode;          // FP64: the anisotropy mode where it is an even integer 2..16, else 0
    bool noisy;
    uint64_t seed;
    double aniso_d;
    R hx, hy, aniso, theta0, c0, s0;  // 0.5/dx, 0.5/dy, mode, theta0, cos and sin of aniso*theta0
    R dtt, inv, m, gama, teq, noise, dt, dtinv;  // dt/tau, 1/(dx*dy), alpha/pi, ..., dt/(dx*dy)
};

// The constants that depend on the differentiable parameters, formed by one
// thread while the staging loads are in flight: each thread's own kept the
// FP64 pipe busier than the rest of an FP32 step.
template <typename R> struct KobPar {
    R epsb, delta, kappa, ebd, meb, mea, mad;  // ..., -epsb*aniso*delta, -epsb*delta, -epsb*aniso, -aniso*delta
    uint64_t nkey;                             // the noise's per-step part
};

struct GgAdj {
    int nx, ny, bc, q, stencil;
    bool vin, vg, vout;  // 16-byte accesses to the state, the output cotangents, the result
    double inv, dt;  // 1/(dx*dy)
};

// The three differentiable parameters and the noise step index: by value,
// or (dev / dstep non-null) read from device memory at kernel start.
struct ParamSrc {
    double v[3];
    const double *dev;
    int64_t step;          // step index, or offset added to *dstep
    const int64_t *dstep;
};

__device__ __forceinline__ void load_params(const ParamSrc &s, double &a, double &b, double &c, int64_t &step)
{
    if (s.dev) {
        a = s.dev[0];
        b = s.dev[1];
        c = s.dev[2];
    } else {
        a = s.v[0];
        b = s.v[1];
        c = s.v[2];
    }
    step = s.dstep ? *s.dstep + s.step : s.step;
}

__device__ __forceinline__ int nbmap(int i, int n, int bc)
{
    if (bc == 0) return i < 0 ? i + n : (i >= n ? i - n : i);
    return i < 0 ? -i - 1 : (i >= n ? 2 * n - i - 1 : i);
}

// The driving term's noise: uniform in [0, 1) by (step, cell), as amps_run's.
__device__ __forceinline__ uint64_t mix64(uint64_t z)
{
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
// float: the 53-bit integer rounded once and scaled exactly, the double value rounded to float
template <typename R> __device__ __forceinline__ R u01(uint64_t nkey, uint64_t cell)
{
    const uint64_t v = mix64(nkey + cell) >> 11;
    if constexpr (sizeof(R) == 4) return __ull2float_rn(v) * 0x1.0p-53f;
    else return (double)v * 0x1.0p-53;
}

template <typename R> __device__ __forceinline__ void kob_params(const KobAdj<R> &p, const ParamSrc &ps, KobPar<R> &k)
{
    double delta, kappa, epsb;
    int64_t step;
    load_params(ps, delta, kappa, epsb, step);
    k.epsb = R(epsb);
    k.delta = R(delta);
    k.kappa = R(kappa);
    k.ebd = R(-epsb * p.aniso_d * delta);
    k.meb = R(-epsb * delta);
    k.mea = R(-epsb * p.aniso_d);
    k.mad = R(-p.aniso_d * delta);
    k.nkey = mix64(p.seed ^ mix64((uint64_t)step));
}

// cos and sin of the anisotropy angle a = aniso*(atan2(py, px) - theta0).
// FP64 with an even integer mode: the power of the unit gradient vector (de
// Moivre's formula; a zero gradient counts as angle 0, as atan2 has it for an
// even mode), about 40 FP64 operations against ~110 of atan2, sin and cos.
template <typename R> __device__ __forceinline__ void kob_angle(const KobAdj<R> &p, R px, R py, R &ca, R &sa)
{
    if constexpr (sizeof(R) == 8) {
        if (p.mode) {
            double c = 1.0, s = 0.0;
            if (px != 0.0 || py != 0.0) {
                // scaled by a power of two (exact), so that the squares stay in range
                const int ex = max(__double2hiint(px) >> 20 & 0x7ff, __double2hiint(py) >> 20 & 0x7ff);
                const double k = __hiloint2double(max(1, min(2046, 2046 - ex)) << 20, 0);
                const double x = px * k, y = py * k;
                const double ir = rsqrt(fma(x, x, y * y));
                c = x * ir;
                s = y * ir;
            }
            double pr = 1.0, pi = 0.0;
            bool one = true;  // the product so far is 1
            for (int n = p.mode;;) {
                if (n & 1) {
                    const double t = one ? c : fma(pr, c, -pi * s);
                    pi = one ? s : fma(pr, s, pi * c);
                    pr = t;
                    one = false;
                }
                n >>= 1;
                if (!n) break;
                const double t = fma(c, c, -s * s);
                s = 2.0 * c * s;
                c = t;
            }
            ca = fma(pr, p.c0, pi * p.s0);
            sa = fma(pi, p.c0, -pr * p.s0);
            return;
        }
        sincos(p.aniso * (atan2(py, px) - p.theta0), &sa, &ca);
    } else {
        sincosf(p.aniso * (atan2f(py, px) - p.theta0), &sa, &ca);
    }
}

// s += v exactly: returns the rounding error of the sum (Knuth's two-sum).
__device__ __forceinline__ float two_sum(float &s, float v)
{
    const float t = s + v, b = t - s, e = (s - (t - b)) + (v - b);
    s = t;
    return e;
}

// The block's sums of three values a thread, each scaled and added into out[k].
// FP64 addition is what costs (a warp's takes 16 cycles of an SM's pipe): the
// threads' values meet in shared memory, three warps fold one value each (NT/32 a
// lane, floats as s + e + f with every rounding error kept: more than FP64's 53
// bits without its pipe), and only their trees are FP64.  A sum that leaves the
// floats' range makes e NaN: folded again in FP64.  buf: 3 * NT values of shared
// memory, free once every thread of the block's NT is here.
template <int NT, typename R>
__device__ __forceinline__ void block_sums(R *buf, R a, R b, R c, double sa, double sb, double sc, double *out)
{
    __syncthreads();
    buf[threadIdx.x] = a;
    buf[NT + threadIdx.x] = b;
    buf[2 * NT + threadIdx.x] = c;
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (w >= 3) return;
    const R *p = buf + w * NT + lane;
    double d;
    if constexpr (sizeof(R) == 4) {
        float s = p[0], e = 0.f, f = 0.f;
#pragma unroll
        for (int k = 1; k < NT / 32; ++k) f += two_sum(e, two_sum(s, p[32 * k]));
        d = (double)s + ((double)e + (double)f);
        if (!(fabsf(e) < INFINITY)) {
            d = p[0];
#pragma unroll 1
            for (int k = 1; k < NT / 32; ++k) d += (double)p[32 * k];
        }
    } else {
        d = p[0];
#pragma unroll
        for (int k = 1; k < NT / 32; ++k) d += p[32 * k];
    }
    for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
    if (lane == 0) atomicAdd(&out[w], d * (w == 0 ? sa : (w == 1 ? sb : sc)));
}

// An asynchronous copy of one element, or of 16 bytes (both sides aligned),
// from global to shared memory; in flight until gg_stage_wait.
template <typename R> __device__ __forceinline__ void cp_elem(R *d, const R *g)
{
    const unsigned sa = (unsigned)__cvta_generic_to_shared(d);
    if constexpr (sizeof(R) == 4)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(g) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sa), "l"(g) : "memory");
}
template <typename R> __device__ __forceinline__ void cp_16(R *d, const R *g)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(d)), "l"(g)
                 : "memory");
}

__device__ __forceinline__ void gg_stage_wait()
{
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// A tile of TX x TY cells with a halo of H cells, row-major in shared memory.
template <int TX, int TY, int H> struct Reg {
    static constexpr int W = TX + 2 * H, HT = TY + 2 * H, N = W * HT;
};

// ------------------------------------------------------------ Kobayashi ----
// Threads of a CTA.  32x8 tiles (grids of few tiles, where a step is latency):
// the widest region in one pass, the forward's 34x10 or the adjoint's 36x12.
template <int TY> constexpr int kob_fwd_threads() { return TY == 8 ? 352 : 256; }
template <int TY> constexpr int kob_adj_threads() { return TY == 8 ? 448 : 256; }

// Forward step.  Shared: phi, T over the halo-2 region; eps*epd*px,
// eps*epd*py and eps over the halo-1 region (at an out-of-domain zero-flux
// position: the values of the mirrored cell, as the map M looks them up).
// FP32 bound by latency at moderate sizes, FP64 by the pipe.  us a step,
// forward / adjoint, before (constants, noise and parameter sums in FP64 per
// thread, atan2 and sin and cos in FP64) and now: FP32 256^2 12.3/26.7, under
// 7.4/8.2; 1024^2 65.6/143, 14.0/32.0; FP64 1024^2 398/749, 256/549.
template <typename R, int TX, int TY>
__global__ void __launch_bounds__(kob_fwd_threads<TY>()) kob_fwd_kernel(const __grid_constant__ KobAdj<R> p, ParamSrc ps,
                                                                        const R *__restrict__ in, R *__restrict__ out)
{
    using R2 = Reg<TX, TY, 2>;
    using R1 = Reg<TX, TY, 1>;
    constexpr int NT = kob_fwd_threads<TY>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ KobPar<R> k;
    R *sphi = reinterpret_cast<R *>(smem_raw), *sT = sphi + R2::N;
    R *sP1 = sT + R2::N, *sP2 = sP1 + R1::N, *seps = sP2 + R1::N;
    const int nx = p.nx, ny = p.ny, bc = p.bc;
    const int64_t n = (int64_t)nx * ny;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
    const R *phi = in, *T = in + n;
    // launched programmatically after the stream's previous grid: wait for it
    // (and its writes) before the first global read
    pdl_trigger();
    pdl_wait();
    for (int u = threadIdx.x; u < R2::N; u += NT) {
        const int gx = x0 - 2 + u % R2::W, gy = y0 - 2 + u / R2::W;
        if (gx < nx + 2 && gy < ny + 2) {
            const int64_t j = (int64_t)nbmap(gy, ny, bc) * nx + nbmap(gx, nx, bc);
            cp_elem(sphi + u, phi + j);
            cp_elem(sT + u, T + j);
        } else {
            sphi[u] = sT[u] = R(0);
        }
    }
    if (threadIdx.x == NT - 1) kob_params(p, ps, k);
    gg_stage_wait();
    __syncthreads();
    for (int u = threadIdx.x; u < R1::N; u += NT) {
        int gx = x0 - 1 + u % R1::W, gy = y0 - 1 + u / R1::W;
        R P1 = R(0), P2 = R(0), e = R(0);
        if (gx <= nx && gy <= ny) {
            if (bc == 1) {
                gx = nbmap(gx, nx, 1);
                gy = nbmap(gy, ny, 1);
            }
            const int o = (gy - y0 + 2) * R2::W + (gx - x0 + 2);
            const R px = (sphi[o + 1] - sphi[o - 1]) * p.hx;
            const R py = (sphi[o + R2::W] - sphi[o - R2::W]) * p.hy;
            R ca, sa;
            kob_angle(p, px, py, ca, sa);
            e = k.epsb * (R(1) + k.delta * ca);
            const R ed = k.ebd * sa;
            P1 = e * ed * px;
            P2 = e * ed * py;
        }
        sP1[u] = P1;
        sP2[u] = P2;
        seps[u] = e;
    }
    __syncthreads();
    for (int u = threadIdx.x; u < TX * TY; u += NT) {
        const int i = u % TX, jj = u / TX, gx = x0 + i, gy = y0 + jj;
        if (gx >= nx || gy >= ny) continue;
        const int o = (jj + 2) * R2::W + i + 2, o1 = (jj + 1) * R1::W + i + 1;
        constexpr int W = R2::W;
        const R ph = sphi[o], t0 = sT[o];
        const R sp = (sphi[o - 1] + sphi[o + 1]) + (sphi[o - 2] + sphi[o + 2]) + (sphi[o - W] + sphi[o + W]) +
                     (sphi[o - 2 * W] + sphi[o + 2 * W]);
        const R lap = (sp - R(8) * ph) * p.inv;
        const R st = (sT[o - 1] + sT[o + 1]) + (sT[o - 2] + sT[o + 2]) + (sT[o - W] + sT[o + W]) +
                     (sT[o - 2 * W] + sT[o + 2 * W]);
        const R lapT = (st - R(8) * t0) * p.inv;
        const R term1 = (sP1[o1 + R1::W] - sP1[o1 - R1::W]) * p.hy;
        const R term2 = -(sP2[o1 + 1] - sP2[o1 - 1]) * p.hx;
        const R m = p.m * atan(p.gama * (p.teq - t0));
        R drive = ph - R(0.5) + m;
        const int64_t g = (int64_t)gy * nx + gx;
        if (p.noisy) drive += p.noise * (u01<R>(k.nkey, (uint64_t)g) - R(0.5));
        const R e = seps[o1];
        const R d = p.dtt * (term1 + term2 + e * e * lap + ph * (R(1) - ph) * drive);
        out[g] = ph + d;
        out[n + g] = t0 + p.dt * lapT + k.kappa * d;
    }
}

// Adjoint step.  Shared (halo 3 for phi, 2 for the rest, 1 for the
// anisotropy cotangents), with a zero-flux domain's cotangents extended past
// its faces -- even where a symmetric sum's transpose reads them, odd where a
// difference's does:
//   phi (R3); mu = gphi' + K gT' (R2, odd) and gT' (R2, even);
//   sin a, cos a, px, py (R2, at out-of-domain positions the mirrored cell's;
//   eps and epd are rebuilt from them exactly as the forward computes them);
//   Q = dt/tau*mu*eps^2/dxdy (R2, even); lpx (R1, odd in x), lpy (R1, odd in
//   y): the cotangents of px, py including the path through theta = atan2(py, px).
template <typename R, int TX, int TY>
__global__ void __launch_bounds__(kob_adj_threads<TY>())
    kob_adj_kernel(const __grid_constant__ KobAdj<R> p, ParamSrc ps, const R *__restrict__ in,
                   const R *__restrict__ gout, R *__restrict__ gin, double *__restrict__ gparams)
{
    using R3 = Reg<TX, TY, 3>;
    using R2 = Reg<TX, TY, 2>;
    using R1 = Reg<TX, TY, 1>;
    constexpr int NT = kob_adj_threads<TY>();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ KobPar<R> k;
    R *sphi = reinterpret_cast<R *>(smem_raw);
    R *smu = sphi + R3::N, *sgT = smu + R2::N, *ssa = sgT + R2::N, *sca = ssa + R2::N;
    R *spx = sca + R2::N, *spy = spx + R2::N, *sQ = spy + R2::N, *slpx = sQ + R2::N, *slpy = slpx + R1::N;
    const int nx = p.nx, ny = p.ny, bc = p.bc;
    const int64_t n = (int64_t)nx * ny;
    const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
    const R *phi = in, *T = in + n, *gpo = gout, *gTo = gout + n;
    pdl_trigger();
    pdl_wait();
    for (int u = threadIdx.x; u < R3::N; u += NT) {
        const int gx = x0 - 3 + u % R3::W, gy = y0 - 3 + u / R3::W;
        if (gx < nx + 3 && gy < ny + 3) cp_elem(sphi + u, phi + (int64_t)nbmap(gy, ny, bc) * nx + nbmap(gx, nx, bc));
        else sphi[u] = R(0);
    }
    for (int u = threadIdx.x; u < R2::N; u += NT) {
        const int gx = x0 - 2 + u % R2::W, gy = y0 - 2 + u / R2::W;
        if (gx < nx + 2 && gy < ny + 2) {
            const int64_t j = (int64_t)nbmap(gy, ny, bc) * nx + nbmap(gx, nx, bc);
            cp_elem(sgT + u, gTo + j);
            cp_elem(smu + u, gpo + j);
        } else {
            sgT[u] = smu[u] = R(0);
        }
    }
    if (threadIdx.x == NT - 1) kob_params(p, ps, k);
    gg_stage_wait();
    __syncthreads();
    const R K = k.kappa;
    auto EPS = [&](R ca) { return k.epsb * (R(1) + k.delta * ca); };
    auto EPD = [&](R sa) { return k.ebd * sa; };
    // mu, sin a, cos a, px, py and Q over R2
    for (int u = threadIdx.x; u < R2::N; u += NT) {
        const int gx = x0 - 2 + u % R2::W, gy = y0 - 2 + u / R2::W;
        R sa = R(0), ca = R(0), px = R(0), py = R(0), q = R(0), mu = R(0);
        if (gx <= nx + 1 && gy <= ny + 1) {
            const bool dom = gx >= 0 && gx < nx && gy >= 0 && gy < ny;
            const int sx = bc == 1 ? nbmap(gx, nx, 1) : gx, sy = bc == 1 ? nbmap(gy, ny, 1) : gy;
            const int o = (sy - y0 + 3) * R3::W + (sx - x0 + 3);
            px = (sphi[o + 1] - sphi[o - 1]) * p.hx;
            py = (sphi[o + R3::W] - sphi[o - R3::W]) * p.hy;
            kob_angle(p, px, py, ca, sa);
            const R e = EPS(ca);
            mu = smu[u] + K * sgT[u];
            q = p.dtt * mu * e * e * p.inv;
            if (bc == 1 && !dom) mu = -mu;
        }
        smu[u] = mu;
        ssa[u] = sa;
        sca[u] = ca;
        spx[u] = px;
        spy[u] = py;
        sQ[u] = q;
    }
    __syncthreads();
    // anisotropy cotangents over R1; parameter gradients of the tile's own cells
    R gd = R(0), ge = R(0), gk = R(0);
    for (int u = threadIdx.x; u < R1::N; u += NT) {
        const int rx = u % R1::W, ry = u / R1::W, gx = x0 - 1 + rx, gy = y0 - 1 + ry;
        R lpx = R(0), lpy = R(0);
        if (gx <= nx && gy <= ny) {
            // an out-of-domain zero-flux position: minus the mirrored cell's lpx, lpy
            const bool dom = gx >= 0 && gx < nx && gy >= 0 && gy < ny, out = bc == 1 && !dom;
            const int mx = out ? nbmap(gx, nx, 1) - x0 + 1 : rx, my = out ? nbmap(gy, ny, 1) - y0 + 1 : ry;
            const int o3 = (my + 2) * R3::W + mx + 2, o2 = (my + 1) * R2::W + mx + 1;
            constexpr int W = R3::W;
            const R sp = (sphi[o3 - 1] + sphi[o3 + 1]) + (sphi[o3 - 2] + sphi[o3 + 2]) + (sphi[o3 - W] + sphi[o3 + W]) +
                         (sphi[o3 - 2 * W] + sphi[o3 + 2 * W]);
            const R lap = (sp - R(8) * sphi[o3]) * p.inv;
            const R A = p.dtt * p.hy * (smu[o2 - R2::W] - smu[o2 + R2::W]);
            const R B = p.dtt * p.hx * (smu[o2 + 1] - smu[o2 - 1]);
            const R C = p.dtt * smu[o2] * lap;
            const R sa = ssa[o2], ca = sca[o2], px = spx[o2], py = spy[o2];
            const R e = EPS(ca), ed = EPD(sa);
            const R le = A * ed * px + B * ed * py + R(2) * C * e;
            const R led = A * e * px + B * e * py;
            lpx = A * e * ed;
            lpy = B * e * ed;
            const R la = le * k.meb * sa + led * k.ebd * ca;
            const R lth = p.aniso * la;
            const R r2 = px * px + py * py;
            if (r2 > R(0)) {  // atan2 has no derivative where the gradient vanishes
                lpx += lth * (-py / r2);
                lpy += lth * (px / r2);
            }
            if (out) {
                lpx = -lpx;
                lpy = -lpy;
            }
            if (rx >= 1 && rx <= TX && ry >= 1 && ry <= TY && gx < nx && gy < ny) {
                gd += le * k.epsb * ca + led * k.mea * sa;
                ge += le * (R(1) + k.delta * ca) + led * k.mad * sa;
            }
        }
        slpx[u] = lpx;
        slpy[u] = lpy;
    }
    __syncthreads();
    for (int u = threadIdx.x; u < TX * TY; u += NT) {
        const int i = u % TX, jj = u / TX, gx = x0 + i, gy = y0 + jj;
        if (gx >= nx || gy >= ny) continue;
        const int o3 = (jj + 3) * R3::W + i + 3, o2 = (jj + 2) * R2::W + i + 2, o1 = (jj + 1) * R1::W + i + 1;
        constexpr int W = R3::W, W2 = R2::W;
        // transposes: radius-2 cross of Q (eps^2 lap phi) and of gT' (lap T)
        R lq = -R(8) * sQ[o2], lt = -R(8) * sgT[o2];
        const int off[4] = {2, 1, -1, -2};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            lq += sQ[o2 + off[j]] + sQ[o2 + off[j] * W2];
            lt += sgT[o2 + off[j]] + sgT[o2 + off[j] * W2];
        }
        const R dpx = (slpx[o1 - 1] - slpx[o1 + 1]) * p.hx;
        const R dpy = (slpy[o1 - R1::W] - slpy[o1 + R1::W]) * p.hy;
        // the forward increment d = phi' - phi at this cell (for dL/dK)
        auto P1 = [&](int o) { return EPS(sca[o]) * EPD(ssa[o]) * spx[o]; };
        auto P2 = [&](int o) { return EPS(sca[o]) * EPD(ssa[o]) * spy[o]; };
        const R term1 = (P1(o2 + W2) - P1(o2 - W2)) * p.hy;
        const R term2 = -(P2(o2 + 1) - P2(o2 - 1)) * p.hx;
        const R ph = sphi[o3];
        const R sp = (sphi[o3 - 1] + sphi[o3 + 1]) + (sphi[o3 - 2] + sphi[o3 + 2]) + (sphi[o3 - W] + sphi[o3 + W]) +
                     (sphi[o3 - 2 * W] + sphi[o3 + 2 * W]);
        const R lap = (sp - R(8) * ph) * p.inv;
        const int64_t g = (int64_t)gy * nx + gx;
        const R t0 = T[g];
        const R m = p.m * atan(p.gama * (p.teq - t0));
        R drive = ph - R(0.5) + m;
        if (p.noisy) drive += p.noise * (u01<R>(k.nkey, (uint64_t)g) - R(0.5));
        const R e = EPS(sca[o2]);
        const R d = p.dtt * (term1 + term2 + e * e * lap + ph * (R(1) - ph) * drive);
        const R mu = smu[o2];
        const R dg = (R(1) - R(2) * ph) * drive + ph * (R(1) - ph);
        const R gT = sgT[o2];
        gin[g] = gpo[g] + p.dtt * mu * dg + lq + dpx + dpy;
        const R z = p.gama * (p.teq - t0);
        const R dm = p.m * (-p.gama) / (R(1) + z * z);
        gin[n + g] = gT + p.dtinv * lt + p.dtt * mu * ph * (R(1) - ph) * dm;
        gk += gT * d;
    }
    static_assert(R3::N + 7 * R2::N + 2 * R1::N >= 3 * NT, "room of the parameter sums");
    block_sums<NT>(sphi, gd, gk, ge, 1.0, 1.0, 1.0, gparams);
}

// --------------------------------------------------------- grain growth ----
// One 32 x TY tile per CTA (any sides, both boundaries): every field (the
// adjoint: and every output cotangent) with a 1-cell halo staged by
// asynchronous copies, the per-cell sums S = sum e^2 (and P = sum g e) formed
// once into shared tiles, then a warp advances one field, a lane sweeping
// TY/4 rows x 4 cells with running row sums (with fewer than 8 fields two or
// four warps share a field's rows).
//
// The zero-flux map mirrors about the domain's faces (-1 -> 0, n -> n-1).  On
// each axis the three-point sum is then a symmetric matrix (the mirrored
// neighbour adds to the diagonal), so both stencils' Laplacians are symmetric
// for either boundary: the adjoint applies the forward Laplacian to the
// cotangents, staged through the same map.
//
// FP32 bound: issue slots and the latency of one partial wave at moderate
// sizes, so TY = 16 (four adjoint CTAs an SM at 8 fields, against two of 32
// rows); FP64 bound: the FP64 pipe, hence the shared row sums and the factored
// formulas (about 11 operations a cell and field forward, 28 adjoint, where
// the direct forms take 18 and 45).  us a step, forward / adjoint, before and now:
// FP32 1024^2 Q=8 periodic 22.6/51.2, 13.7/39.3; 605x443 Q=8 zero-flux 14.6/44.3,
// 8.4/14.3; FP64 1024^2 Q=8 271/739, 189/503.
// The kernels' constants, formed by one thread while the copies are in flight
// (each thread's own would keep the FP64 pipe busier than the step itself).
template <typename R> struct GgConst {
    R dtm, g2, g4, m2, ki;      // dt*L, 2 gamma, 4 gamma, 1 - 2 gamma, kappa/(dx*dy)
    double sl, sk, sg;          // scales of the parameter sums
    __device__ void set(const GgAdj &p, double mobil, double grcoef, double gamma)
    {
        dtm = R(p.dt * mobil);
        g2 = R(2.0 * gamma);
        g4 = R(4.0 * gamma);
        m2 = R(1.0 - 2.0 * gamma);
        ki = R(grcoef * p.inv);
        sl = -p.dt;
        sk = p.dt * mobil * p.inv;
        sg = -2.0 * p.dt * mobil;
    }
};

template <typename R, int TY> struct G32 {
    static constexpr int T = 32, O = 16 / (int)sizeof(R), P = T + 2 * O, ROWS = TY + 2, FIELD = ROWS * P;
    static size_t smem(int nfields, int sums) { return sizeof(R) * ((size_t)nfields * FIELD + (size_t)sums * TY * T); }
};

// Stage q fields of f (row-major [q][ny][nx]) over the tile at (x0, y0) and its
// halo through the boundary map; cells past the one that a last valid cell
// reads are zero.  A thread owns a slot -- a 16-byte chunk, a halo cell -- of
// every field.  vec: nx * sizeof(R) and the base are multiples of 16 bytes.
template <typename R, int TY>
__device__ __forceinline__ void gg_stage32(R *s, const R *f, int q, int x0, int y0, const GgAdj &p, bool vec)
{
    using L = G32<R, TY>;
    constexpr int V = 16 / (int)sizeof(R), CH = L::T / V, UI = L::ROWS * CH;
    const int64_t n = (int64_t)p.nx * p.ny;
    const int units = vec ? UI + L::ROWS * 2 : L::ROWS * (L::T + 2);
    for (int u = threadIdx.x; u < units; u += kAdjThreads) {
        int ry, c;  // staged row, tile column
        bool chunk = false;
        if (vec && u < UI) {
            ry = u / CH;
            c = u % CH * V;
            chunk = x0 + c < p.nx;
        } else if (vec) {
            ry = (u - UI) / 2;
            c = (u - UI) % 2 ? L::T : -1;
        } else {
            ry = u / (L::T + 2);
            c = u % (L::T + 2) - 1;
        }
        const bool wide = vec && u < UI;  // the slot is V elements
        const int gx = x0 + c, gy = y0 - 1 + ry;
        const bool ok = gx <= p.nx && gy <= p.ny;
        R *d = s + ry * L::P + L::O + c;
        const R *g = f;
        if (ok) g += (int64_t)nbmap(gy, p.ny, p.bc) * p.nx + nbmap(gx, p.nx, p.bc);
        for (int k = 0; k < q; ++k, d += L::FIELD, g += n) {
            if (ok && chunk) {
                cp_16(d, g);
                continue;
            }
            if (ok) cp_elem(d, g);
            else *d = R(0);
            if (wide)
                for (int j = 1; j < V; ++j) d[j] = R(0);
        }
    }
}

// Four cells (16-byte aligned) of a staged row: v; with their outer neighbours
// w[0..5].
template <typename R> __device__ __forceinline__ void ld4(const R *p, R *v)
{
    if constexpr (sizeof(R) == 4) {
        const float4 a = *reinterpret_cast<const float4 *>(p);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    } else {
        const double2 a = *reinterpret_cast<const double2 *>(p), b = *reinterpret_cast<const double2 *>(p + 2);
        v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
    }
}

// The rows of one field that a lane sweeps: its stencil's sum at four cells,
// row by row.  Stencil 0: three-cell row sums, the middle pair of each four
// shared; 9 e is taken off before the last row is added (see gg_tile.cuh).
template <typename R, int ST> struct LapRows {
    R a[4], b[4], e[4];  // ST 0: the row sums of the two rows above the next; ST 1: the rows themselves
    R l, r;              // ST 1: the outer neighbours of row e
    __device__ __forceinline__ static void sums(const R *p, R *v, R *h)
    {
        ld4(p, v);
        const R x = v[0] + v[1], y = v[2] + v[3];
        h[0] = p[-1] + x;
        h[1] = x + v[2];
        h[2] = v[1] + y;
        h[3] = y + p[4];
    }
    // p: the staged row above the lane's first, row pitch P
    __device__ __forceinline__ void start(const R *p, int P)
    {
        if (ST == 0) {
            R t[4];
            sums(p, t, a);
            sums(p + P, e, b);
        } else {
            ld4(p, a);
            ld4(p + P, e);
            l = p[P - 1];
            r = p[P + 4];
        }
    }
    // dn: the staged row below the current one.  c: the current row's cells, m: their stencil sums; moves on.
    __device__ __forceinline__ void step(const R *dn, R *c, R *m)
    {
        R v[4];
        if (ST == 0) {
            R h[4];
            sums(dn, v, h);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                c[k] = e[k];
                m[k] = a[k] + (b[k] + h[k] - R(9) * e[k]);
                a[k] = b[k];
                b[k] = h[k];
                e[k] = v[k];
            }
        } else {
            ld4(dn, v);
            const R l2 = dn[-1], r2 = dn[4];
            const R w[6] = {l, e[0], e[1], e[2], e[3], r};
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                c[k] = e[k];
                m[k] = (w[k] + w[k + 2]) + (a[k] + v[k]) - R(4) * e[k];
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                a[k] = e[k];
                e[k] = v[k];
            }
            l = l2;
            r = r2;
        }
    }
};

// Four results to global memory: the first nv of them (vec: 16-byte stores).
template <typename R> __device__ __forceinline__ void st4(R *d, const R *v, int nv, bool vec)
{
    if (vec && nv >= 4) {
        if constexpr (sizeof(R) == 4) {
            *reinterpret_cast<float4 *>(d) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
            *reinterpret_cast<double2 *>(d) = make_double2(v[0], v[1]);
            *reinterpret_cast<double2 *>(d + 2) = make_double2(v[2], v[3]);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < nv) d[k] = v[k];
    }
}

// PARTS warps share a field's rows.
template <typename R, int TY, int PARTS, int ST>
__global__ void __launch_bounds__(kAdjThreads) gg_fwd32_kernel(GgAdj p, ParamSrc ps, const R *__restrict__ eta,
                                                               R *__restrict__ out)
{
    using L = G32<R, TY>;
    constexpr int RPT = TY / 4 / PARTS;  // rows a lane
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ GgConst<R> sc;
    R *se = reinterpret_cast<R *>(smem_raw), *sG = se + p.q * L::FIELD;
    const int ntx = (p.nx + 31) / 32, x0 = blockIdx.x % ntx * 32, y0 = blockIdx.x / ntx * TY;
    pdl_trigger();
    pdl_wait();
    gg_stage32<R, TY>(se, eta, p.q, x0, y0, p, p.vin);
    if (threadIdx.x == kAdjThreads - 1) {
        double mobil, grcoef, gamma;
        int64_t step;
        load_params(ps, mobil, grcoef, gamma, step);
        sc.set(p, mobil, grcoef, gamma);
    }
    gg_stage_wait();
    __syncthreads();
    const R dtm = sc.dtm, g2 = sc.g2, m2 = sc.m2, ki = sc.ki;
    // FP64: G = 2 gamma S - 1 and dfd = e*(G + (1 - 2 gamma) e^2), two operations a
    // field fewer; FP32 keeps S and the form whose terms cancel exactly in a grain's
    // interior (there the separately rounded 2 gamma and 1 - 2 gamma would not)
    constexpr bool D = sizeof(R) == 8;
    {
        constexpr int C = TY / 8;  // cells a thread: every thread, for the serial sum over the fields
        const int row = threadIdx.x / (L::T / C), c = threadIdx.x % (L::T / C) * C;
        R acc[C] = {};
        for (int k = 0; k < p.q; ++k) {
            const R *v = se + k * L::FIELD + (row + 1) * L::P + L::O + c;
#pragma unroll
            for (int j = 0; j < C; ++j) acc[j] += v[j] * v[j];
        }
#pragma unroll
        for (int j = 0; j < C; ++j) sG[row * L::T + c + j] = D ? g2 * acc[j] - R(1) : acc[j];
    }
    __syncthreads();
    const int64_t n = (int64_t)p.nx * p.ny;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c0 = (lane & 7) * 4;
    const int nv = p.nx - x0 - c0;  // valid cells from the lane's first on
    for (int u = warp; u < p.q * PARTS; u += kAdjThreads / 32) {
        const int f = u / PARTS, r0 = ((lane >> 3) + u % PARTS * 4) * RPT;
        const R *fs = se + f * L::FIELD + r0 * L::P + L::O + c0;
        LapRows<R, ST> w;
        w.start(fs, L::P);
        R *dst = out + f * n + (int64_t)(y0 + r0) * p.nx + x0 + c0;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            R e[4], m[4], G[4], o[4];
            w.step(fs + (i + 2) * L::P, e, m);
            ld4(sG + (r0 + i) * L::T + c0, G);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const R e2 = e[k] * e[k], b = D ? G[k] + m2 * e2 : (e2 - R(1)) + g2 * (G[k] - e2);
                o[k] = e[k] - dtm * (e[k] * b - ki * m[k]);
            }
            if (y0 + r0 + i < p.ny) st4(dst + (int64_t)i * p.nx, o, nv, p.vout);
        }
    }
}

// Input cotangents of all q fields and dL/d(L, kappa, gamma) into gparams:
//   b = e^2 - 1 + 2 gamma (S - e^2),  dfd_k = e*b,
//   gin_k = g_k - dtL*(g_k*(b + 2 e^2) + 4 gamma e (P - g_k e) - kappa lap g_k).
template <typename R, int TY, int PARTS, int ST>
__global__ void __launch_bounds__(kAdjThreads, sizeof(R) == 4 ? 4 : 2)
    gg_adj32_kernel(GgAdj p, ParamSrc ps, const R *__restrict__ eta, const R *__restrict__ gout, R *__restrict__ gin,
                    double *__restrict__ gparams)
{
    using L = G32<R, TY>;
    constexpr int RPT = TY / 4 / PARTS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ GgConst<R> sc;
    R *se = reinterpret_cast<R *>(smem_raw), *sg = se + p.q * L::FIELD;
    R *sS = sg + p.q * L::FIELD, *sP = sS + TY * L::T;
    const int ntx = (p.nx + 31) / 32, x0 = blockIdx.x % ntx * 32, y0 = blockIdx.x / ntx * TY;
    pdl_trigger();
    pdl_wait();
    gg_stage32<R, TY>(se, eta, p.q, x0, y0, p, p.vin);
    gg_stage32<R, TY>(sg, gout, p.q, x0, y0, p, p.vg);
    if (threadIdx.x == kAdjThreads - 1) {
        double mobil, grcoef, gamma;
        int64_t step;
        load_params(ps, mobil, grcoef, gamma, step);
        sc.set(p, mobil, grcoef, gamma);
    }
    gg_stage_wait();
    __syncthreads();
    {
        constexpr int C = TY / 8;
        const int row = threadIdx.x / (L::T / C), c = threadIdx.x % (L::T / C) * C;
        R S[C] = {}, P[C] = {};
        for (int k = 0; k < p.q; ++k) {
            const int o = k * L::FIELD + (row + 1) * L::P + L::O + c;
#pragma unroll
            for (int j = 0; j < C; ++j) {
                const R e = se[o + j];
                S[j] += e * e;
                P[j] += sg[o + j] * e;
            }
        }
#pragma unroll
        for (int j = 0; j < C; ++j) {
            sS[row * L::T + c + j] = S[j];
            sP[row * L::T + c + j] = P[j];
        }
    }
    __syncthreads();
    const int64_t n = (int64_t)p.nx * p.ny;
    const R dtm = sc.dtm, g2 = sc.g2, g4 = sc.g4, ki = sc.ki;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c0 = (lane & 7) * 4;
    const int nv = p.nx - x0 - c0;
    R gl = R(0), gkap = R(0), ggam = R(0);  // sums of g*(dfd - kappa lap e), g*(stencil sum of e), g*e*(S - e^2)
    for (int u = warp; u < p.q * PARTS; u += kAdjThreads / 32) {
        const int f = u / PARTS, r0 = ((lane >> 3) + u % PARTS * 4) * RPT;
        const int o0 = f * L::FIELD + r0 * L::P + L::O + c0;
        LapRows<R, ST> we, wg;
        we.start(se + o0, L::P);
        wg.start(sg + o0, L::P);
        R *dst = gin + f * n + (int64_t)(y0 + r0) * p.nx + x0 + c0;
#pragma unroll 1  // (unrolled, the next rows' loads are hoisted and spill)
        for (int i = 0; i < RPT; ++i) {
            R e[4], g[4], me[4], mg[4], S[4], P[4], o[4];
            we.step(se + o0 + (i + 2) * L::P, e, me);
            wg.step(sg + o0 + (i + 2) * L::P, g, mg);
            ld4(sS + (r0 + i) * L::T + c0, S);
            ld4(sP + (r0 + i) * L::T + c0, P);
            const bool row = y0 + r0 + i < p.ny;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const R e2 = e[k] * e[k], s1 = S[k] - e2, b = (e2 - R(1)) + g2 * s1, x = g[k] * e[k];
                o[k] = g[k] - dtm * (g[k] * (b + R(2) * e2) + (g4 * e[k]) * (P[k] - x) - ki * mg[k]);
                if (row && k < nv) {
                    gl += g[k] * (e[k] * b - ki * me[k]);
                    gkap += g[k] * me[k];
                    ggam += x * s1;
                }
            }
            if (row) st4(dst + (int64_t)i * p.nx, o, nv, p.vout);
        }
    }
    // (the staging and the sum tiles behind it, no longer read, hold 3 * kAdjThreads values for any q)
    static_assert(2 * L::FIELD + 2 * TY * L::T >= 3 * kAdjThreads, "room of the parameter sums");
    block_sums<kAdjThreads>(se, gl, gkap, ggam, sc.sl, sc.sk, sc.sg, gparams);
}

// ------------------------------------------------------------- launches ----
constexpr int kTX = 32;

template <typename R, int TY> constexpr size_t kob_fwd_smem()
{
    return (2 * Reg<kTX, TY, 2>::N + 3 * Reg<kTX, TY, 1>::N) * sizeof(R);
}
template <typename R, int TY> constexpr size_t kob_adj_smem()
{
    return (Reg<kTX, TY, 3>::N + 7 * Reg<kTX, TY, 2>::N + 2 * Reg<kTX, TY, 1>::N) * sizeof(R);
}

// 32x16 tiles, or 32x8 where that leaves fewer than two CTAs per SM.
bool small_tiles(int nx, int ny) { return (int64_t)((nx + 31) / 32) * ((ny + 15) / 16) < 2 * 152; }

template <typename R> cudaError_t kob_prepare()
{
    const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(kob_adj_kernel<R, kTX, 16>, attr, (int)kob_adj_smem<R, 16>());
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kob_adj_kernel<R, kTX, 8>, attr, (int)kob_adj_smem<R, 8>());
    return e;
}

// Calls fn(TY, PARTS, ST as integral constants) for a grain-growth launch
// (kernel: `sets` staged states, `sums` sum tiles): 16 rows, or 8 where those
// of all fields do not fit or would leave SMs without a tile; a field to 1, 2
// or 4 warps by the fields.
template <typename R, typename F> auto gg_dispatch(int nx, int ny, int q, int stencil, int sets, int sums, F fn)
{
    using std::integral_constant;
    auto st = [&](auto ty, auto parts) {
        return stencil == 0 ? fn(ty, parts, integral_constant<int, 0>()) : fn(ty, parts, integral_constant<int, 1>());
    };
    const integral_constant<int, 1> one;
    const integral_constant<int, 2> two;
    if (G32<R, 16>::smem(sets * q, sums) > (size_t)kMaxAdjSmem ||
        (int64_t)((nx + 31) / 32) * ((ny + 15) / 16) < 152) {
        const integral_constant<int, 8> ty;
        return q > 4 ? st(ty, one) : st(ty, two);
    }
    const integral_constant<int, 16> ty;
    if (q >= 8) return st(ty, one);
    if (q >= 4) return st(ty, two);
    return st(ty, integral_constant<int, 4>());
}

template <typename R> cudaError_t gg_prepare_adj()
{
    const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaSuccess;
    for (int stencil = 0; stencil < 2; ++stencil)
        for (int q : {1, 4, 8})
            for (int side : {8, 4096})  // few tiles, many
                gg_dispatch<R>(side, side, q, stencil, 1, 1, [&](auto ty, auto parts, auto st) {
                    const auto fwd = gg_fwd32_kernel<R, ty(), parts(), st()>;
                    const auto adj = gg_adj32_kernel<R, ty(), parts(), st()>;
                    if (e == cudaSuccess) e = cudaFuncSetAttribute(fwd, attr, kMaxAdjSmem);
                    if (e == cudaSuccess) e = cudaFuncSetAttribute(adj, attr, kMaxAdjSmem);
                });
    return e;
}

template <typename R> KobAdj<R> kob_args(const amps_params *p)
{
    KobAdj<R> k;
    k.nx = p->nx; k.ny = p->ny; k.bc = p->bc;
    const bool even = p->aniso >= 2 && p->aniso <= 16 && p->aniso == 2 * floor(p->aniso / 2);
    k.mode = even ? (int)p->aniso : 0;
    k.noisy = p->noise != 0.0;
    k.seed = p->seed;
    k.aniso_d = p->aniso;
    k.hx = R(0.5 / p->dx); k.hy = R(0.5 / p->dy); k.aniso = R(p->aniso); k.theta0 = R(p->theta0);
    k.c0 = R(cos(p->aniso * p->theta0)); k.s0 = R(sin(p->aniso * p->theta0));
    k.dtt = R(p->dt / p->tau); k.inv = R(1.0 / (p->dx * p->dy)); k.m = R(p->alpha / p->pi); k.gama = R(p->gama);
    k.teq = R(p->teq); k.noise = R(p->noise); k.dt = R(p->dt); k.dtinv = R(p->dt * k.inv);
    return k;
}

// whether 16-byte accesses to rows of `ptr` are aligned
template <typename R> bool vec_ok(const amps_params *p, const void *ptr)
{
    return p->nx % (16 / (int)sizeof(R)) == 0 && (uintptr_t)ptr % 16 == 0;
}

template <typename R> GgAdj gg_args(const amps_params *p, const void *in, const void *gout, const void *out)
{
    GgAdj g;
    g.vin = vec_ok<R>(p, in); g.vg = vec_ok<R>(p, gout); g.vout = vec_ok<R>(p, out);
    g.nx = p->nx; g.ny = p->ny; g.bc = p->bc; g.q = p->nfields; g.stencil = p->stencil;
    g.inv = 1.0 / (p->dx * p->dy); g.dt = p->dt;
    return g;
}

ParamSrc param_src(const amps_params *p, int64_t step)
{
    ParamSrc s;
    if (p->model == AMPS_KOBAYASHI) {
        s.v[0] = p->delta; s.v[1] = p->kappa; s.v[2] = p->epsb;
    } else {
        s.v[0] = p->mobil; s.v[1] = p->grcoef; s.v[2] = p->gamma;
    }
    s.dev = nullptr; s.step = step; s.dstep = nullptr;
    return s;
}

int check(const amps_params *p, int dtype)
{
    if (!p || (dtype != AMPS_F64 && dtype != AMPS_F32) || p->nx < 5 || p->ny < 5) return AMPS_ERR_INVALID;
    if (p->model == AMPS_SINTERING) return AMPS_ERR_UNSUPPORTED;
    if (p->model != AMPS_KOBAYASHI && p->model != AMPS_GRAINGROWTH) return AMPS_ERR_INVALID;
    if (p->model == AMPS_GRAINGROWTH && (p->nfields < 1 || p->nfields > 32)) return AMPS_ERR_INVALID;
    if (p->bc != AMPS_BC_PERIODIC && p->bc != AMPS_BC_NOFLUX) return AMPS_ERR_INVALID;
    if (p->model == AMPS_KOBAYASHI && (p->tau == 0.0 || p->pi == 0.0 || p->dx == 0.0 || p->dy == 0.0))
        return AMPS_ERR_INVALID;
    return AMPS_OK;
}

int64_t state_elems(const amps_params *p)
{
    return (int64_t)p->nx * p->ny * (p->model == AMPS_KOBAYASHI ? 2 : p->nfields);
}

// A launch that may start while the stream's previous grid drains: every
// kernel here waits for it (griddepcontrol.wait) before its first global read.
template <typename K, typename... Args>
void launch2(K kernel, dim3 grid, int threads, size_t smem, cudaStream_t s, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);  // (the callers read cudaGetLastError)
}

template <typename R>
void launch_forward(const amps_params *p, const ParamSrc &ps, const void *in, void *out, cudaStream_t s)
{
    const int nx = p->nx, ny = p->ny;
    if (p->model == AMPS_KOBAYASHI) {
        if (small_tiles(nx, ny)) {
            const dim3 grid((nx + kTX - 1) / kTX, (ny + 7) / 8);
            launch2(kob_fwd_kernel<R, kTX, 8>, grid, kob_fwd_threads<8>(), kob_fwd_smem<R, 8>(), s, kob_args<R>(p), ps,
                    (const R *)in, (R *)out);
        } else {
            const dim3 grid((nx + kTX - 1) / kTX, (ny + 15) / 16);
            launch2(kob_fwd_kernel<R, kTX, 16>, grid, kob_fwd_threads<16>(), kob_fwd_smem<R, 16>(), s, kob_args<R>(p),
                    ps, (const R *)in, (R *)out);
        }
    } else {
        const GgAdj g = gg_args<R>(p, in, nullptr, out);
        gg_dispatch<R>(nx, ny, p->nfields, p->stencil, 1, 1, [&](auto ty, auto parts, auto st) {
            launch2(gg_fwd32_kernel<R, ty(), parts(), st()>, dim3((nx + 31) / 32 * ((ny + ty() - 1) / ty())), kAdjThreads,
                    G32<R, ty()>::smem(p->nfields, 1), s, g, ps, (const R *)in, (R *)out);
        });
    }
}

template <typename R>
void launch_adjoint(const amps_params *p, const ParamSrc &ps, const void *in, const void *gout, void *gin,
                    double *gparams, cudaStream_t s)
{
    const int nx = p->nx, ny = p->ny;
    if (p->model == AMPS_KOBAYASHI) {
        if (small_tiles(nx, ny)) {
            const dim3 grid((nx + kTX - 1) / kTX, (ny + 7) / 8);
            launch2(kob_adj_kernel<R, kTX, 8>, grid, kob_adj_threads<8>(), kob_adj_smem<R, 8>(), s, kob_args<R>(p), ps,
                    (const R *)in, (const R *)gout, (R *)gin, gparams);
        } else {
            const dim3 grid((nx + kTX - 1) / kTX, (ny + 15) / 16);
            launch2(kob_adj_kernel<R, kTX, 16>, grid, kob_adj_threads<16>(), kob_adj_smem<R, 16>(), s, kob_args<R>(p), ps,
                    (const R *)in, (const R *)gout, (R *)gin, gparams);
        }
    } else {
        const GgAdj g = gg_args<R>(p, in, gout, gin);
        gg_dispatch<R>(nx, ny, p->nfields, p->stencil, 2, 2, [&](auto ty, auto parts, auto st) {
            launch2(gg_adj32_kernel<R, ty(), parts(), st()>, dim3((nx + 31) / 32 * ((ny + ty() - 1) / ty())), kAdjThreads,
                    G32<R, ty()>::smem(2 * p->nfields, 2), s, g, ps, (const R *)in, (const R *)gout, (R *)gin, gparams);
        });
    }
}

cudaError_t prepare(int dtype)
{
    static cudaError_t done[2] = {cudaErrorNotReady, cudaErrorNotReady};
    const int k = dtype == AMPS_F64 ? 0 : 1;
    if (done[k] != cudaSuccess) {
        done[k] = k == 0 ? kob_prepare<double>() : kob_prepare<float>();
        if (done[k] == cudaSuccess) done[k] = k == 0 ? gg_prepare_adj<double>() : gg_prepare_adj<float>();
    }
    return done[k];
}

void forward_any(int dtype, const amps_params *p, const ParamSrc &ps, const void *in, void *out, cudaStream_t s)
{
    if (dtype == AMPS_F64) launch_forward<double>(p, ps, in, out, s);
    else launch_forward<float>(p, ps, in, out, s);
}

void adjoint_any(int dtype, const amps_params *p, const ParamSrc &ps, const void *in, const void *gout, void *gin,
                 double *gparams, cudaStream_t s)
{
    if (dtype == AMPS_F64) launch_adjoint<double>(p, ps, in, gout, gin, gparams, s);
    else launch_adjoint<float>(p, ps, in, gout, gin, gparams, s);
}

}  // namespace

extern "C" int amps_step_forward(const amps_params *p, int dtype, const void *state_in, void *state_out, int64_t step,
                                 void *stream)
{
    if (int r = check(p, dtype)) return r;
    if (!state_in || !state_out || state_in == state_out) return AMPS_ERR_INVALID;
    if (prepare(dtype) != cudaSuccess) return AMPS_ERR_CUDA;
    forward_any(dtype, p, param_src(p, step), state_in, state_out, (cudaStream_t)stream);
    return cudaGetLastError() == cudaSuccess ? AMPS_OK : AMPS_ERR_CUDA;
}

extern "C" int amps_step_adjoint(const amps_params *p, int dtype, const void *state_in, const void *grad_out,
                                 void *grad_in, double *grad_params, int64_t step, void *stream)
{
    if (int r = check(p, dtype)) return r;
    if (!state_in || !grad_out || !grad_in || !grad_params || grad_in == grad_out || grad_in == state_in)
        return AMPS_ERR_INVALID;
    if (prepare(dtype) != cudaSuccess) return AMPS_ERR_CUDA;
    adjoint_any(dtype, p, param_src(p, step), state_in, grad_out, grad_in, grad_params, (cudaStream_t)stream);
    return cudaGetLastError() == cudaSuccess ? AMPS_OK : AMPS_ERR_CUDA;
}

// ------------------------------------------------------ rollout handle ----
namespace {

__global__ void set_params_kernel(double *pv, double a, double b, double c, int64_t *dstep, int64_t step0)
{
    pv[0] = a;
    pv[1] = b;
    pv[2] = c;
    *dstep = step0;
}

int auto_segment(int nsteps)
{
    int s = 1;
    while ((int64_t)s * s < nsteps) ++s;
    return s;
}

}  // namespace

struct amps_adjoint {
    amps_params p;
    int dtype = AMPS_F64, nsteps = 0, seg = 1, nseg = 1;
    size_t state_bytes = 0;
    cudaStream_t stream = nullptr, capture = nullptr;
    char *mem = nullptr;  // one allocation: checkpoints, replay states, ping-pong, params
    std::vector<char *> ckpt, segbuf;
    char *tmp[2] = {nullptr, nullptr}, *g[2] = {nullptr, nullptr};
    double *dpv = nullptr, *dgp = nullptr;
    int64_t *dstep = nullptr;
    const char *final_state = nullptr, *final_grad = nullptr;
    bool graphs = true, have_forward = false;
    cudaGraphExec_t exec[2] = {nullptr, nullptr};  // forward sweep, backward sweep
    char err[160] = "";

    ParamSrc src(int64_t off) const
    {
        ParamSrc s;
        s.v[0] = s.v[1] = s.v[2] = 0.0;
        s.dev = dpv;
        s.step = off;
        s.dstep = dstep;
        return s;
    }

    // The whole forward sweep; step k reads the previous output, checkpoint
    // slots take every seg-th state so nothing is copied.
    void enqueue_forward(cudaStream_t s)
    {
        const char *src_p = ckpt[0];
        for (int k = 0; k < nsteps; ++k) {
            char *dst = ((k + 1) % seg == 0 && k + 1 < nsteps) ? ckpt[(k + 1) / seg]
                                                                : (src_p == tmp[0] ? tmp[1] : tmp[0]);
            forward_any(dtype, &p, src(k), src_p, dst, s);
            src_p = dst;
        }
        final_state = src_p;
    }

    // Segments in reverse: replay the segment from its checkpoint (keeping
    // every step's input), then run its adjoint steps backwards.
    void enqueue_backward(cudaStream_t s)
    {
        int cur = 0;
        std::vector<const char *> st(seg);
        for (int sg = nseg - 1; sg >= 0; --sg) {
            const int first = sg * seg, count = nsteps - first < seg ? nsteps - first : seg;
            st[0] = ckpt[sg];
            for (int k = 1; k < count; ++k) {
                forward_any(dtype, &p, src(first + k - 1), st[k - 1], segbuf[k - 1], s);
                st[k] = segbuf[k - 1];
            }
            for (int k = count - 1; k >= 0; --k) {
                adjoint_any(dtype, &p, src(first + k), st[k], g[cur], g[cur ^ 1], dgp, s);
                cur ^= 1;
            }
        }
        final_grad = g[cur];
    }

    int fail(int code, const char *what)
    {
        snprintf(err, sizeof err, "%s", what);
        return code;
    }

    int run_sweep(int which)
    {
        if (!graphs) {
            if (which == 0) enqueue_forward(stream);
            else enqueue_backward(stream);
            return cudaGetLastError() == cudaSuccess ? AMPS_OK : fail(AMPS_ERR_CUDA, cudaGetErrorString(cudaGetLastError()));
        }
        if (!exec[which]) {
            cudaGraph_t graph = nullptr;
            if (cudaStreamBeginCapture(capture, cudaStreamCaptureModeThreadLocal) != cudaSuccess)
                return fail(AMPS_ERR_CUDA, "cudaStreamBeginCapture failed");
            if (which == 0) enqueue_forward(capture);
            else enqueue_backward(capture);
            const cudaError_t e1 = cudaStreamEndCapture(capture, &graph);
            if (e1 != cudaSuccess || !graph) return fail(AMPS_ERR_CUDA, cudaGetErrorString(e1));
            const cudaError_t e2 = cudaGraphInstantiate(&exec[which], graph, 0);
            cudaGraphDestroy(graph);
            if (e2 != cudaSuccess) {
                exec[which] = nullptr;
                return fail(AMPS_ERR_CUDA, cudaGetErrorString(e2));
            }
        }
        return cudaGraphLaunch(exec[which], stream) == cudaSuccess ? AMPS_OK : fail(AMPS_ERR_CUDA, "cudaGraphLaunch failed");
    }

    ~amps_adjoint()
    {
        for (auto &e : exec)
            if (e) cudaGraphExecDestroy(e);
        if (capture) cudaStreamDestroy(capture);
        if (mem) cudaFree(mem);
    }
};

namespace {

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

size_t layout_bytes(const amps_params *p, int dtype, int nsteps, int seg, size_t *state_bytes, int *nseg)
{
    const size_t sb = align256((size_t)state_elems(p) * (dtype == AMPS_F64 ? 8 : 4));
    const int ns = (nsteps + seg - 1) / seg;
    if (state_bytes) *state_bytes = sb;
    if (nseg) *nseg = ns;
    // checkpoints + (seg - 1) replay states + 2 forward + 2 cotangent buffers + params/step/grads
    return sb * ((size_t)ns + (size_t)(seg - 1) + 4) + 256;
}

}  // namespace

extern "C" size_t amps_adjoint_memory_bytes(const amps_params *p, int dtype, int nsteps, int segment)
{
    if (check(p, dtype) != AMPS_OK || nsteps < 1 || segment < 0) return 0;
    const int seg = segment == 0 ? auto_segment(nsteps) : (segment > nsteps ? nsteps : segment);
    return layout_bytes(p, dtype, nsteps, seg, nullptr, nullptr);
}

extern "C" int amps_adjoint_create(const amps_params *p, int dtype, int nsteps, int segment, amps_adjoint **out)
{
    if (!out) return AMPS_ERR_INVALID;
    *out = nullptr;
    if (int r = check(p, dtype)) return r;
    if (nsteps < 1 || segment < 0) return AMPS_ERR_INVALID;
    if (prepare(dtype) != cudaSuccess) return AMPS_ERR_CUDA;
    amps_adjoint *a = new (std::nothrow) amps_adjoint;
    if (!a) return AMPS_ERR_ALLOC;
    a->p = *p;
    a->dtype = dtype;
    a->nsteps = nsteps;
    a->seg = segment == 0 ? auto_segment(nsteps) : (segment > nsteps ? nsteps : segment);
    const size_t total = layout_bytes(p, dtype, nsteps, a->seg, &a->state_bytes, &a->nseg);
    if (cudaMalloc(&a->mem, total) != cudaSuccess) {
        cudaGetLastError();
        delete a;
        return AMPS_ERR_ALLOC;
    }
    char *q = a->mem;
    for (int i = 0; i < a->nseg; ++i, q += a->state_bytes) a->ckpt.push_back(q);
    for (int i = 0; i < a->seg - 1; ++i, q += a->state_bytes) a->segbuf.push_back(q);
    a->tmp[0] = q; q += a->state_bytes;
    a->tmp[1] = q; q += a->state_bytes;
    a->g[0] = q; q += a->state_bytes;
    a->g[1] = q; q += a->state_bytes;
    a->dpv = (double *)q;
    a->dgp = a->dpv + 4;
    a->dstep = (int64_t *)(a->dpv + 8);
    if (cudaStreamCreateWithFlags(&a->capture, cudaStreamNonBlocking) != cudaSuccess) {
        delete a;
        return AMPS_ERR_CUDA;
    }
    *out = a;
    return AMPS_OK;
}

extern "C" int amps_adjoint_destroy(amps_adjoint *a)
{
    if (!a) return AMPS_ERR_INVALID;
    if (a->stream) cudaStreamSynchronize(a->stream);
    else cudaDeviceSynchronize();
    delete a;
    return AMPS_OK;
}

extern "C" int amps_adjoint_set_stream(amps_adjoint *a, void *stream)
{
    if (!a) return AMPS_ERR_INVALID;
    a->stream = (cudaStream_t)stream;
    return AMPS_OK;
}

extern "C" int amps_adjoint_set_graphs(amps_adjoint *a, int enable)
{
    if (!a) return AMPS_ERR_INVALID;
    a->graphs = enable != 0;
    return AMPS_OK;
}

extern "C" int amps_adjoint_segment(const amps_adjoint *a) { return a ? a->seg : -1; }

extern "C" const char *amps_adjoint_last_error(const amps_adjoint *a) { return a ? a->err : "null handle"; }

extern "C" int amps_adjoint_forward(amps_adjoint *a, const double *param_values, const void *state0,
                                    void *state_final, int64_t step0)
{
    if (!a || !param_values || !state0) return AMPS_ERR_INVALID;
    set_params_kernel<<<1, 1, 0, a->stream>>>(a->dpv, param_values[0], param_values[1], param_values[2], a->dstep,
                                             step0);
    if (cudaMemcpyAsync(a->ckpt[0], state0, (size_t)state_elems(&a->p) * (a->dtype == AMPS_F64 ? 8 : 4),
                        cudaMemcpyDeviceToDevice, a->stream) != cudaSuccess)
        return a->fail(AMPS_ERR_CUDA, "state0 copy failed");
    if (int r = a->run_sweep(0)) return r;
    if (state_final &&
        cudaMemcpyAsync(state_final, a->final_state, (size_t)state_elems(&a->p) * (a->dtype == AMPS_F64 ? 8 : 4),
                        cudaMemcpyDeviceToDevice, a->stream) != cudaSuccess)
        return a->fail(AMPS_ERR_CUDA, "final state copy failed");
    a->have_forward = true;
    return AMPS_OK;
}

extern "C" int amps_adjoint_backward(amps_adjoint *a, const void *grad_final, void *grad_state0, double *grad_params)
{
    if (!a || !grad_final) return AMPS_ERR_INVALID;
    if (!a->have_forward) return a->fail(AMPS_ERR_INVALID, "amps_adjoint_backward before amps_adjoint_forward");
    const size_t bytes = (size_t)state_elems(&a->p) * (a->dtype == AMPS_F64 ? 8 : 4);
    if (cudaMemsetAsync(a->dgp, 0, 3 * sizeof(double), a->stream) != cudaSuccess ||
        cudaMemcpyAsync(a->g[0], grad_final, bytes, cudaMemcpyDeviceToDevice, a->stream) != cudaSuccess)
        return a->fail(AMPS_ERR_CUDA, "cotangent copy failed");
    if (int r = a->run_sweep(1)) return r;
    if (grad_state0 &&
        cudaMemcpyAsync(grad_state0, a->final_grad, bytes, cudaMemcpyDeviceToDevice, a->stream) != cudaSuccess)
        return a->fail(AMPS_ERR_CUDA, "gradient copy failed");
    if (grad_params &&
        cudaMemcpyAsync(grad_params, a->dgp, 3 * sizeof(double), cudaMemcpyDeviceToDevice, a->stream) != cudaSuccess)
        return a->fail(AMPS_ERR_CUDA, "parameter gradient copy failed");
    return AMPS_OK;
}
