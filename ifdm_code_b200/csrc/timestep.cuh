// timestep.cuh -- Timestep_criteria (src/CosmoBEC_MPI.cpp:19-78) on the device.
//
// One warp turns the max reductions of the previous passes into the three
// step criteria, advances the scale factor and integrates
//   dt_KE = int da/(H a^3), dt_PE = int da/(H a^2), dt_QI = int da/(H a^4)
// (integrands src/struct3D.h:127-146) with the QUADPACK method the reference
// gets from GSL's qags: one 21-point Gauss-Kronrod rule, accepted when its
// error estimate meets epsrel = 1e-10, else bisection of the worst interval.
// It writes the merged kick coefficients for the next kick; the block's
// threads then fill the separable drift tables exp(-i s kappa_i^2).
#pragma once

#include "step_kernels.cuh"

namespace ifdm {

// ------------------------------------------------------------ quadrature --
__device__ __forceinline__ double qk_integrand(int n, double x, double H0, double Om) {
    const double H = H0 * sqrt(Om / pow(x, 3) + (1.0 - Om));
    return 1. / (H * pow(x, (double)n));
}

// 21-point Kronrod abscissae/weights and the embedded 10-point Gauss weights
// (QUADPACK qk21; x[1],x[3],..,x[9] are the Gauss nodes, x[10] = 0).
__device__ __constant__ double c_gk_x[11] = {
    0.995657163025808080735527280689003, 0.973906528517171720077964012084452,
    0.930157491355708226001207180059508, 0.865063366688984510732096688423493,
    0.780817726586416897063717578345042, 0.679409568299024406234327365114874,
    0.562757134668604683339000099272694, 0.433395394129247190799265943165784,
    0.294392862701460198131126603103866, 0.148874338981631210884826001129720,
    0.0};
__device__ __constant__ double c_gk_wk[11] = {
    0.011694638867371874278064396062192, 0.032558162307964727478818972459390,
    0.054755896574351996031381300244580, 0.075039674810919952767043140916190,
    0.093125454583697605535065465083366, 0.109387158802297641899210590325805,
    0.123491976262065851077958109831074, 0.134709217311473325928054001771707,
    0.142775938577060080797094273138717, 0.147739104901338491374841515972068,
    0.149445554002916905664936468389821};
__device__ __constant__ double c_gk_wg[5] = {
    0.066671344308688137593568809893332, 0.149451349150580593145776339657697,
    0.219086362515982043995534934228163, 0.269266719309996355091226921569469,
    0.295524224714752870173892994651338};

static __device__ void qk21(int n, double H0, double Om, double a, double b, double *res, double *abserr, double *resasc) {
    const double c = 0.5 * (a + b), h = 0.5 * (b - a);
    const double fc = qk_integrand(n, c, H0, Om);
    double kron = fc * c_gk_wk[10], gauss = 0.0, sabs = fabs(kron);
    double fl[10], fr[10];
    for (int j = 0; j < 10; ++j) {
        const double dxj = h * c_gk_x[j];
        fl[j] = qk_integrand(n, c - dxj, H0, Om);
        fr[j] = qk_integrand(n, c + dxj, H0, Om);
    }
    for (int j = 1; j < 10; j += 2) {
        const double s = fl[j] + fr[j];
        gauss += c_gk_wg[j / 2] * s;
        kron += c_gk_wk[j] * s;
        sabs += c_gk_wk[j] * (fabs(fl[j]) + fabs(fr[j]));
    }
    for (int j = 0; j < 10; j += 2) {
        const double s = fl[j] + fr[j];
        kron += c_gk_wk[j] * s;
        sabs += c_gk_wk[j] * (fabs(fl[j]) + fabs(fr[j]));
    }
    const double mean = 0.5 * kron;
    double sasc = c_gk_wk[10] * fabs(fc - mean);
    for (int j = 0; j < 10; ++j) sasc += c_gk_wk[j] * (fabs(fl[j] - mean) + fabs(fr[j] - mean));
    double err = fabs((kron - gauss) * h);
    kron *= h;
    sabs *= fabs(h);
    sasc *= fabs(h);
    if (sasc != 0.0 && err != 0.0) {
        const double scale = pow(200.0 * err / sasc, 1.5);
        err = (scale < 1.0) ? sasc * scale : sasc;
    }
    const double eps = 2.220446049250313e-16, dmin = 2.2250738585072014e-308;
    if (sabs > dmin / (50.0 * eps)) err = fmax(err, 50.0 * eps * sabs);
    *res = kron;
    *abserr = err;
    *resasc = sasc;
}

// The same rule evaluated by a whole warp: lanes 0-9 take the left nodes,
// 10-19 the right ones, 20 the centre (the integrand's two pow calls are the
// cost), then every lane sums the 21 values in qk21's order, so the results
// are bit-identical to qk21 and equal on all lanes.  Called by all 32 lanes.
static __device__ void qk21_warp(int n, double H0, double Om, double a, double b, double *res, double *abserr,
                                 double *resasc) {
    const int lane = threadIdx.x & 31;
    const double c = 0.5 * (a + b), h = 0.5 * (b - a);
    double x = c;
    if (lane < 20) {
        const double dxj = h * c_gk_x[lane % 10];
        x = lane < 10 ? c - dxj : c + dxj;
    }
    const double f = lane <= 20 ? qk_integrand(n, x, H0, Om) : 0.0;
    const double fc = __shfl_sync(0xffffffffu, f, 20);
    double kron = fc * c_gk_wk[10], gauss = 0.0, sabs = fabs(kron);
    double fl[10], fr[10];
#pragma unroll
    for (int j = 0; j < 10; ++j) {
        fl[j] = __shfl_sync(0xffffffffu, f, j);
        fr[j] = __shfl_sync(0xffffffffu, f, 10 + j);
    }
    for (int j = 1; j < 10; j += 2) {
        const double s = fl[j] + fr[j];
        gauss += c_gk_wg[j / 2] * s;
        kron += c_gk_wk[j] * s;
        sabs += c_gk_wk[j] * (fabs(fl[j]) + fabs(fr[j]));
    }
    for (int j = 0; j < 10; j += 2) {
        const double s = fl[j] + fr[j];
        kron += c_gk_wk[j] * s;
        sabs += c_gk_wk[j] * (fabs(fl[j]) + fabs(fr[j]));
    }
    const double mean = 0.5 * kron;
    double sasc = c_gk_wk[10] * fabs(fc - mean);
    for (int j = 0; j < 10; ++j) sasc += c_gk_wk[j] * (fabs(fl[j] - mean) + fabs(fr[j] - mean));
    double err = fabs((kron - gauss) * h);
    kron *= h;
    sabs *= fabs(h);
    sasc *= fabs(h);
    if (sasc != 0.0 && err != 0.0) {
        const double scale = pow(200.0 * err / sasc, 1.5);
        err = (scale < 1.0) ? sasc * scale : sasc;
    }
    const double eps = 2.220446049250313e-16, dmin = 2.2250738585072014e-308;
    if (sabs > dmin / (50.0 * eps)) err = fmax(err, 50.0 * eps * sabs);
    *res = kron;
    *abserr = err;
    *resasc = sasc;
}

#define IFDM_QLIMIT 64
// Returns 0 on success, 1 when the interval limit was reached.  WARP: the
// rule is evaluated by the calling warp (all 32 lanes call, every lane gets
// the result); else by the calling thread alone.
template <bool WARP = false>
static __device__ int qags_dev(int n, double H0, double Om, double a, double b, int limit, double *result) {
    auto rule = [&](double lo_, double hi_, double *r, double *e, double *sc) {
        if constexpr (WARP) qk21_warp(n, H0, Om, lo_, hi_, r, e, sc);
        else qk21(n, H0, Om, lo_, hi_, r, e, sc);
    };
    double r0, e0, s0;
    rule(a, b, &r0, &e0, &s0);
    if ((e0 <= 1e-10 * fabs(r0) && e0 != s0) || e0 == 0.0) {
        *result = r0;
        return 0;
    }
    double lo[IFDM_QLIMIT], hi[IFDM_QLIMIT], rr[IFDM_QLIMIT], ee[IFDM_QLIMIT];
    if (limit > IFDM_QLIMIT) limit = IFDM_QLIMIT;
    int cnt = 1;
    lo[0] = a; hi[0] = b; rr[0] = r0; ee[0] = e0;
    double tot = r0;
    while (cnt < limit) {
        int w = 0;
        for (int i = 1; i < cnt; ++i) if (ee[i] > ee[w]) w = i;
        const double m = 0.5 * (lo[w] + hi[w]);
        double r1, e1, r2, e2, t;
        rule(lo[w], m, &r1, &e1, &t);
        rule(m, hi[w], &r2, &e2, &t);
        lo[cnt] = m; hi[cnt] = hi[w]; rr[cnt] = r2; ee[cnt] = e2;
        hi[w] = m; rr[w] = r1; ee[w] = e1;
        ++cnt;
        double te = 0.0;
        tot = 0.0;
        for (int i = 0; i < cnt; ++i) { tot += rr[i]; te += ee[i]; }
        if (te <= 1e-10 * fabs(tot)) { *result = tot; return 0; }
    }
    *result = tot;
    return 1;
}

__device__ __forceinline__ double bits_to_double(unsigned long long b) { return __longlong_as_double((long long)b); }

// After the initial density pass: partial sums (3 per block, fixed order) ->
// first offset c = mean psi_s and the conserved mean mu = <|psi_s|^2>.
static __global__ void k_reduce_init(TState *__restrict__ ts, const double *__restrict__ part, int nblocks, double n3) {
    __shared__ double red[3][256];
    double a = 0, b = 0, c = 0;
    for (int i = threadIdx.x; i < nblocks; i += blockDim.x) {
        a += part[3 * i];
        b += part[3 * i + 1];
        c += part[3 * i + 2];
    }
    red[0][threadIdx.x] = a;
    red[1][threadIdx.x] = b;
    red[2][threadIdx.x] = c;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) {
            red[0][threadIdx.x] += red[0][threadIdx.x + s];
            red[1][threadIdx.x] += red[1][threadIdx.x + s];
            red[2][threadIdx.x] += red[2][threadIdx.x + s];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        ts->cnext_re = red[0][0] / n3;
        ts->cnext_im = red[1][0] / n3;
        ts->mu = red[2][0] / n3;
    }
}

// Append the current step to a log.
__device__ __forceinline__ void log_step(const TState *ts, StepLog *lg) {
    StepLog e;
    e.coefP = ts->coefP;
    e.coefQ = ts->coefQ;
    e.alpha = ts->alpha;
    e.drift_s = ts->drift_s;
    e.cre = ts->cre;
    e.cim = ts->cim;
    e.pendP = ts->pendP;
    e.pendQ = ts->pendQ;
    e.gphase = ts->gphase;
    e.a = ts->a;
    e.dt_KE = ts->dt_KE;
    e.dt_PE = ts->dt_PE;
    e.dt_QI = ts->dt_QI;
    e.steps = ts->steps;
    *lg = e;
}

// The 21-point rule laid out by lane (0-9 left nodes, 10-19 right, 20 centre,
// the rest zero): signed abscissa, Kronrod weight, Gauss weight.
struct GkNodes {
    double x[32], wk[32], wg[32];
};
__device__ __forceinline__ void gk_fill(GkNodes *g) {  // threads 0..31; the caller syncs
    const int i = threadIdx.x;
    if (i >= 32) return;
    const int j = i < 20 ? i % 10 : 10;
    g->x[i] = i < 10 ? -c_gk_x[j] : (i < 20 ? c_gk_x[j] : 0.0);
    g->wk[i] = i < 21 ? c_gk_wk[j] : 0.0;
    g->wg[i] = i < 20 && j % 2 ? c_gk_wg[j / 2] : 0.0;
}
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The timestep, by one full warp, in two parts: the kinetic criterion depends
// on a alone, so the integrals over a kinetic-limited step can be computed
// before the reductions of the previous step are complete (the one-launch
// kernels do it while they wait for them) and are used when that criterion
// limits the step.  One warp takes the three integrals together: each lane evaluates its
// node's H once, the powers a^2, a^3, a^4 by multiplication and the three
// quotients side by side, and the sums run over the warp in parallel (the
// same rule, sums in another order; an interval whose error estimate misses
// 1e-10 goes to the bisecting qags_dev).  Latency is all that counts here, one
// warp's dependent FP64 chain: with pow() per node, the integrals on three
// warps and sequential 21-term sums the kernel took 12-14 us of every step.
struct StepIntegrals {
    double dt;       // the criterion's step before the scale
    double da, r[3]; // int da/(H a^n) over [a, a + da], n = 3, 2, 4
    int bad;
};
static __device__ __noinline__ int qags_warp(int n, double H0, double Om, double a, double b, int limit, double *r) {
    return qags_dev<true>(n, H0, Om, a, b, limit, r);
}
__device__ __forceinline__ double kinetic_dt(double ai, const Phys &ph) { return ph.A_KE * (ai * ai); }
static __device__ __noinline__ void step_integrals(double ai, double max_dt, const Phys &ph, const GkNodes *gk,
                                                   StepIntegrals *out) {
    const int lane = threadIdx.x & 31;
    const double H = ph.H0 * sqrt(ph.Om / (ai * ai * ai) + (1.0 - ph.Om));
    const double da = H * ai * (max_dt * ph.dt_scale);
    const double lo = ai, hi = ai + da, c = 0.5 * (lo + hi), h = 0.5 * (hi - lo);
    const double x = c + h * gk->x[lane], wk = gk->wk[lane], wg = gk->wg[lane];
    const double x2 = x * x, x3 = x2 * x, Hx = ph.H0 * sqrt(ph.Om / x3 + (1.0 - ph.Om));
    const double f[3] = {1.0 / (Hx * x3), 1.0 / (Hx * x2), 1.0 / (Hx * (x2 * x2))};
    double kron[3], gauss[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        kron[q] = warp_sum(wk * f[q]);
        gauss[q] = warp_sum(wg * f[q]);
    }
    // QUADPACK's estimate sasc min(1, (200 |K - G| / sasc)^1.5) is at most
    // 200 |K - G|: where that meets the tolerance the rule is accepted without it
    int bad = 0;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        double r = kron[q] * h;
        if (!(200.0 * fabs((kron[q] - gauss[q]) * h) <= 1e-10 * fabs(r)))
            bad |= qags_warp(q == 0 ? 3 : (q == 1 ? 2 : 4), ph.H0, ph.Om, lo, hi, ph.limit, &r);
        if (lane == 0) out->r[q] = r;
    }
    if (lane == 0) {
        out->dt = max_dt;
        out->da = da;
        out->bad = bad;
    }
    __syncwarp();
}

// *ts and *si in shared memory, *si the integrals of the kinetic step of
// ts->a; the reductions and the mean of the kicked field (cn_re, cn_im) come
// from the previous step.  Written by lane 0; the caller syncs.
static __device__ __noinline__ void timestep_warp(TState *ts, const Phys &ph, const GkNodes *gk, StepIntegrals *si,
                                                  unsigned long long phi_bits, unsigned long long rho_bits, double cn_re,
                                                  double cn_im) {
    const double maxphi = ph.Phi0 * bits_to_double(phi_bits);
    const double maxrho = ph.S2 * bits_to_double(rho_bits);
    const double ai = ts->a;
    const double dt_KE = si->dt;
    const double dt_PE = ph.B_PE / maxphi * ai;
    double dt_QI = ph.C_QI / maxrho * (ai * ai * ai);
    if (ph.g == 0) dt_QI = 0.0;
    double max_dt = dt_KE;
    int crit = 3;
    if (max_dt > dt_PE) { max_dt = dt_PE; crit = 2; }
    if ((max_dt > dt_QI) && (ph.g != 0)) { max_dt = dt_QI; crit = 4; }
    if (crit != 3) step_integrals(ai, max_dt, ph, gk, si);
    __syncwarp();  // every lane has read *ts and *si before lane 0 rewrites *ts
    if ((threadIdx.x & 31) != 0) return;
    if (si->bad) ts->err |= 1;
    ts->maxphi = maxphi;
    ts->maxrho = maxrho;
    ts->cand_KE = dt_KE;
    ts->cand_PE = dt_PE;
    ts->cand_QI = dt_QI;
    ts->da = si->da;
    ts->crit = crit;
    const double iKE = si->r[0], iPE = si->r[1], iQI = si->r[2];
    ts->dt_KE = iKE;
    ts->dt_PE = iPE;
    ts->dt_QI = iQI;
    ts->a = ai + si->da;
    const double hp = 0.5 * iPE * ph.kP, hq = 0.5 * iQI * ph.kQ;
    const double pp = ts->pendP, pq = ts->pendQ;
    ts->snapP = pp;
    ts->snapQ = pq;
    ts->coefP = pp + hp;
    ts->coefQ = pq + hq;
    ts->pendP = hp;
    ts->pendQ = hq;
    ts->drift_s = ph.kin * iKE;
    // global-phase dither (FP32 mode): psi is stored as exp(-i gphase) psi
    // and this step's kick adds alpha, a pseudo-random phase in [0, 2 pi)
    // from the step count, so consecutive steps round different numbers;
    // the offset c (a mean of psi) rotates with it
    double alpha = 0.0, sa = 0.0, ca = 1.0;
    if (ph.dither) {
        const unsigned long long k = (unsigned long long)ts->steps * 0x9e3779b97f4a7c15ull + 0x632be59bd9b4e019ull;
        const unsigned long long m = (k ^ (k >> 31)) * 0xbf58476d1ce4e5b9ull;
        alpha = 6.283185307179586476925286766559 * (double)((m ^ (m >> 29)) >> 11) * 0x1.0p-53;
        sincos(alpha, &sa, &ca);
    }
    const double g0 = ts->gphase, gp = g0 + alpha, twopi = 6.283185307179586476925286766559;
    ts->alpha = alpha;
    ts->gphase_prev = g0;
    ts->gphase = gp >= twopi ? gp - twopi : gp;  // both in [0, 2 pi): the subtraction is exact
    ts->cre = cn_re * ca + cn_im * sa;
    ts->cim = cn_im * ca - cn_re * sa;
    ts->steps += 1;
}

// The timestep of *ts (global memory) by one block; all threads fill the
// tables exp(-i s kappa_i^2), i < N.
__device__ __forceinline__ void timestep_body(TState *ts, const Phys &ph, double2 *drift64, float2 *drift32) {
    __shared__ TState st;
    __shared__ GkNodes gk;
    __shared__ StepIntegrals si;
    // the state's words a thread each, both ways (by one thread: kernel 15.6 us, so 13.2)
    static_assert(sizeof(TState) % 8 == 0 && sizeof(TState) / 8 <= 64, "words of the state");
    unsigned long long *const sw = reinterpret_cast<unsigned long long *>(&st), *const gw = reinterpret_cast<unsigned long long *>(ts);
    gk_fill(&gk);
    for (unsigned i = threadIdx.x; i < sizeof(TState) / 8; i += blockDim.x) sw[i] = gw[i];
    __syncthreads();
    if (threadIdx.x < 32) {
        step_integrals(st.a, kinetic_dt(st.a, ph), ph, &gk, &si);
        timestep_warp(&st, ph, &gk, &si, st.maxphi_bits, st.maxrho_bits, st.cnext_re, st.cnext_im);
        if (threadIdx.x == 0) st.maxphi_bits = st.maxrho_bits = 0ull;
    }
    __syncthreads();
    for (unsigned i = threadIdx.x; i < sizeof(TState) / 8; i += blockDim.x) gw[i] = sw[i];
    const double s = st.drift_s;
    const double twopi = 6.283185307179586476925286766559;
    for (int i = threadIdx.x; i < ph.N; i += blockDim.x) {
        const double k = (double)kappa(i, ph.N);
        double p = s * (k * k);
        p -= twopi * rint(p * (1.0 / twopi));
        double sn, cs;
        sincos(p, &sn, &cs);
        drift64[i] = make_double2(cs, -sn);
        drift32[i] = make_float2((float)cs, (float)-sn);
    }
}

constexpr int kTimestepThreads = 512;
static __global__ void __launch_bounds__(kTimestepThreads) k_timestep(TState *__restrict__ ts, Phys ph, double2 *__restrict__ drift64,
                           float2 *__restrict__ drift32) {
    timestep_body(ts, ph, drift64, drift32);
}

}  // namespace ifdm
