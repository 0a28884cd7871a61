// box_kernels.cuh -- whole runs of one small box (N <= 128) in one launch.
//
// The ten passes of step_kernels.cuh cost ten launches a step, and up to 64^3
// a pass is shorter than its launch (measured: 72-78 us a step from 16^3 to
// 64^3 whatever the size, host-launch bound).  Here a group of CTAs owns a box and runs all its
// steps in one kernel.  A CTA transforms a whole N x N plane in shared memory,
// so a step has five phases instead of nine passes (144 instead of 240 bytes a
// cell in FP64), separated by a barrier over the group:
//
//   A  x planes: [timestep] kick, FFT along y
//   B  y planes: FFT along x and z, drift, inverse FFT along z and x
//   C  x planes: inverse FFT along y -> psi; density; real FFT along z; FFT along y
//   D  y planes of the half spectrum: FFT along x, -1/kappa^2, inverse FFT
//   E  x planes: inverse FFT along y, half-to-real FFT along z -> phi; max |phi|
//
// A plane is [row][N + 1] in shared memory: with the odd pitch both the lines
// along a row and those across rows are conflict-free with the line index
// fastest over the threads, and the threads of a warp then share one twiddle
// (a broadcast).  Global loads and stores run along z in the phases' own
// register layout (element t + T b + r N/R of column l), so a plane needs no
// staging copies; A's and C's first and last stages read and write global
// memory directly.  The inverse transforms use the forward plan reversed: the last
// stage of one leaves each thread with the first-stage inputs of the other.
//
// The barrier over the group is barrier.cluster when the group is one
// thread-block cluster (hardware keeps a cluster resident together), or a
// counter in global memory when the kernel is a cooperative launch (the
// runtime keeps the grid resident).  The counter wait is bounded.
// Every CTA of the group computes the timestep for itself from the same
// reductions (the same code and inputs, so the same values), which saves a barrier.
#pragma once

#include "angles.cuh"
#include "step_kernels.cuh"
#include "timestep.cuh"
#include "tma.cuh"

namespace ifdm {

// ------------------------------------------------------------------ plans --
// Even first and last radices (C and E pair the rows y and y + N/2 that one
// thread holds), few exchanges, and a power of two first: a smooth line (the
// density is its mean plus a few percent) then leaves the first stage's odd
// outputs by exact differences, which keeps the lowest wave numbers, those
// that carry the potential, 20 times more accurate than radix 12 first
// (48^3 FP32: phi 2.7e-6 against 1e-7 off).  V = 1: another order for the batch tuner.
template <int N, int V> struct BoxPlan;
template <int V> struct BoxPlan<16, V> { static constexpr int E = 4, NST = 2; static constexpr int R[4] = {4, 4, 1, 1}; };
template <> struct BoxPlan<32, 0> { static constexpr int E = 8, NST = 2; static constexpr int R[4] = {4, 8, 1, 1}; };
template <> struct BoxPlan<32, 1> { static constexpr int E = 8, NST = 2; static constexpr int R[4] = {8, 4, 1, 1}; };
template <> struct BoxPlan<48, 0> { static constexpr int E = 12, NST = 2; static constexpr int R[4] = {4, 12, 1, 1}; };
template <> struct BoxPlan<48, 1> { static constexpr int E = 12, NST = 3; static constexpr int R[4] = {4, 4, 3, 1}; };
template <> struct BoxPlan<64, 0> { static constexpr int E = 8, NST = 2; static constexpr int R[4] = {8, 8, 1, 1}; };
template <> struct BoxPlan<64, 1> { static constexpr int E = 8, NST = 3; static constexpr int R[4] = {4, 4, 4, 1}; };
template <> struct BoxPlan<96, 0> { static constexpr int E = 24, NST = 2; static constexpr int R[4] = {8, 12, 1, 1}; };
template <> struct BoxPlan<96, 1> { static constexpr int E = 12, NST = 3; static constexpr int R[4] = {4, 4, 6, 1}; };
template <int V> struct BoxPlan<128, V> { static constexpr int E = 16, NST = 2; static constexpr int R[4] = {16, 8, 1, 1}; };

template <class P> struct RevPlan {
    static constexpr int E = P::E, NST = P::NST;
    static constexpr int rad(int s) { return s < P::NST ? P::R[P::NST - 1 - s] : 1; }
    static constexpr int R[4] = {rad(0), rad(1), rad(2), rad(3)};
};

template <int DIR> struct Bfly<6, DIR> {
    // 6 = 2 * 3 without twiddles (prime factor indexing): n = 2 n1 + 3 n2 mod 6
    template <typename C> __device__ __forceinline__ static void run(C *v) {
        C a[3] = {v[0], v[2], v[4]}, b[3] = {v[3], v[5], v[1]};
        Bfly<3, DIR>::run(a);
        Bfly<3, DIR>::run(b);
        v[0] = a[0] + b[0];
        v[3] = a[0] - b[0];
        v[4] = a[1] + b[1];
        v[1] = a[1] - b[1];
        v[2] = a[2] + b[2];
        v[5] = a[2] - b[2];
    }
};

template <int DIR> struct Bfly<12, DIR> {
    // 12 = 3 * 4 without twiddles (prime factor indexing): n = 4 n1 + 3 n2 mod 12
    template <typename C> __device__ __forceinline__ static void run(C *v) {
        C a[4][3];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int p = 0; p < 3; ++p) a[q][p] = v[(4 * p + 3 * q) % 12];
            Bfly<3, DIR>::run(a[q]);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            C b[4] = {a[0][k], a[1][k], a[2][k], a[3][k]};
            Bfly<4, DIR>::run(b);
            // output index = k mod 3 and q mod 4
#pragma unroll
            for (int q = 0; q < 4; ++q) v[(4 * k + 9 * q) % 12] = b[q];
        }
    }
};

// a * exp(DIR i q), q the angle of the real constants (c, s) = (cos, sin)
template <int DIR, typename C, typename KS> __device__ __forceinline__ C mul_const(C a, KS c, KS s) {
    using R = decltype(a.x);
    if constexpr (sizeof(R) == 8) {
        return DIR > 0 ? mkc(a.x * c.hi - a.y * s.hi, a.x * s.hi + a.y * c.hi)
                       : mkc(a.x * c.hi + a.y * s.hi, a.y * c.hi - a.x * s.hi);
    } else {  // with the constants' rounding remainders, as twmul
        const R sh = DIR > 0 ? s.hi : -s.hi, sl = DIR > 0 ? s.lo : -s.lo;
        const R cr = fmaf(a.x, c.lo, -a.y * sl), ci = fmaf(a.x, sl, a.y * c.lo);
        return mkc(fmaf(a.x, c.hi, fmaf(-a.y, sh, cr)), fmaf(a.x, sh, fmaf(a.y, c.hi, ci)));
    }
}

template <int DIR> struct Bfly<16, DIR> {
    // 16 = 4 * 4: four radix-4 columns, the twiddles w16^(j k), four radix-4 rows
    template <typename C> __device__ __forceinline__ static void run(C *v) {
        using R = decltype(v[0].x);
        constexpr KSplit<R> c1(0.92387953251128675612818318939679), s1(0.38268343236508977172845998403040);
        constexpr KSplit<R> h(0.70710678118654752440084436210485), mh(-0.70710678118654752440084436210485);
        constexpr KSplit<R> mc1(-0.92387953251128675612818318939679), ms1(-0.38268343236508977172845998403040);
        C a[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int q = 0; q < 4; ++q) a[j][q] = v[j + 4 * q];
            Bfly<4, DIR>::run(a[j]);
        }
        a[1][1] = mul_const<DIR>(a[1][1], c1, s1);
        a[1][2] = mul_const<DIR>(a[1][2], h, h);
        a[1][3] = mul_const<DIR>(a[1][3], s1, c1);
        a[2][1] = mul_const<DIR>(a[2][1], h, h);
        a[2][2] = mul_i<DIR>(a[2][2]);
        a[2][3] = mul_const<DIR>(a[2][3], mh, h);
        a[3][1] = mul_const<DIR>(a[3][1], s1, c1);
        a[3][2] = mul_const<DIR>(a[3][2], mh, h);
        a[3][3] = mul_const<DIR>(a[3][3], mc1, ms1);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            C b[4] = {a[0][k], a[1][k], a[2][k], a[3][k]};
            Bfly<4, DIR>::run(b);
#pragma unroll
            for (int q = 0; q < 4; ++q) v[k + 4 * q] = b[q];
        }
    }
};

// ------------------------------------------------------------- arguments ---
// Words the CTAs of a group share in global memory.
struct BoxScratch {
    unsigned long long ctr[2];    // barrier arrivals of groups of N and of N/2 CTAs (a multiple of the
                                  // group's size between launches)
    unsigned long long mx[2][2];  // max |phi|, max |psi|^2 of the previous step, by step parity
    double cnext[2];              // mean of the kicked field (the next offset c)
    double part[128][4];          // initial pass: sums of psi, |psi|^2 and max |psi|^2 per plane
};

struct BoxRun {
    void *psi, *phi, *rhok;
    const void *tw;
    TState *ts;
    BoxScratch *scr;
    Phys ph;
    long win_rows;
    int win_tail;
    int timestep;          // 1: compute each step's timestep; 0: *ts holds it (one step)
    StepLog *log;          // timestep 1: append each step (may be null); 2: replay them
    void *seg_psi, *seg_phi;  // replay: the state before each step is copied here
    double a0;             // initial pass: scale factor
};

// Backward sweep over the recorded steps start .. end-1.
struct BoxSweep {
    void *g, *rhok;
    const void *tw;
    BoxScratch *scr;
    int *err;
    const StepLog *log;
    int start, end;
    const void *seg_psi, *seg_phi;    // states start .. end-2
    const void *last_psi, *last_phi;  // state end-1, or the output map's state (end == start)
    double a, b, alpha;               // the output map's kick
};

// Barrier over the CTAs of a group.
struct GroupBarrier {
    unsigned long long *ctr = nullptr;  // null: the group is a cluster
    unsigned long long target = 0;
    unsigned n = 0;
    int *err = nullptr;
    int *ok = nullptr;  // shared memory

    // all threads; the counter is a multiple of n when a launch starts, and the
    // group cannot pass its first barrier before this CTA has arrived there
    __device__ __forceinline__ void init(unsigned long long *c, unsigned group, bool cluster, int *e, int *sh) {
        n = group;
        err = e;
        ok = sh;
        if (cluster) return;
        ctr = c;
        unsigned long long v = 0;
        if (threadIdx.x == 0) {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(c) : "memory");
            target = v / group * group;
        }
    }
    __device__ __forceinline__ void arrive() {
        if (!ctr) {
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            return;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            target += n;
            asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(ctr), "l"(1ull) : "memory");
        }
    }
    // false for the whole CTA when the bounded wait gave up (bit 2 of *err)
    __device__ __forceinline__ bool wait() {
        if (!ctr) {
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
            __syncthreads();
            return true;
        }
        if (threadIdx.x == 0) {
            int good = 0;
            for (uint32_t i = 0; i < kMaxSpins; ++i) {
                unsigned long long v;
                asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(ctr) : "memory");
                if (v >= target) {
                    good = 1;
                    break;
                }
                if (i > 4096) __nanosleep(128);
            }
            if (!good) atomicOr(err, 2);
            *ok = good;
        }
        __syncthreads();
        return *ok != 0;
    }
    __device__ __forceinline__ bool sync() {
        arrive();
        return wait();
    }
};

// v exp(-i p) - c0, the kicked field less the offset, rounded to K once.
template <typename K> struct BoxKick;
template <> struct BoxKick<double> {
    __device__ __forceinline__ static double2 run(double2 v, double p, double2 c0) {
        double s, c;
        sincos_pi(p, s, c);
        return cmul(v, mkc(c, -s)) - c0;
    }
};
// FP32: the pair, its product with psi and the difference in FP64, so the
// rounding is relative to psi - c too and nothing changes |psi| one way (an
// FP32 pair put back on the unit circle lost 6e-9 of the norm a step).
template <> struct BoxKick<float> {
    __device__ __forceinline__ static float2 run(double2 v, double p, float2 c0) {
        double s, c;
        const int j = sincos_quarter(p, s, c);
        const double x = v.x, y = v.y;
        // exp(-i p) = (-i)^j (c - i s): turn psi by the quarter turns instead of the pair
        const double a = (j & 1) ? y : x, b = (j & 1) ? -x : y;
        const double sg = (j & 2) ? -1.0 : 1.0, cc = c * sg, ss = s * sg;
        return mkc((float)fma(a, cc, fma(b, ss, -(double)c0.x)), (float)fma(b, cc, fma(-a, ss, -(double)c0.y)));
    }
};

template <typename R, typename K, int N> constexpr bool box_fits() {
    // a plane of the arithmetic type and its tables in 227 KB, at most 1024 threads
    return N <= 128 && !(N == 128 && sizeof(K) == 8);
}

// --------------------------------------------------------------- phases ----
// Register arrays that only active threads fill start at zero: filled under a
// condition alone they count as live from the loop's start, through all the
// other phases, and the run kernels spilled 1-7 KB a thread.

template <typename R_, typename K_, int N, int V> struct BoxOps {
    using R = R_;
    using K = K_;
    using G = cx<R>;
    using C = cx<K>;
    using F = BoxPlan<N, V>;
    using B = RevPlan<F>;
    static constexpr int SIZE = N, E = F::E, T = N / E;
    static constexpr int NF = N * T, NT = NF < 128 ? 128 : NF;  // threads (16^3 needs 64)
    // Line l of a transform over `lines` lines and part t of it, the line
    // fastest over the threads.  (Named barriers over groups of 32 lines
    // instead of block barriers measured slower: 128^3 FP32 150 -> 166 thousand
    // cycles a step, the groups run in step anyway.)
    struct Lane {
        int l, t;
        bool act;
        __device__ __forceinline__ explicit Lane(int lines) {
            l = threadIdx.x % lines;
            t = threadIdx.x / lines;
            act = t < T;
        }
    };
    // resident CTAs the registers must allow: 1024 threads an SM in FP32 (64
    // registers), 512 in FP64 arithmetic (128); one box of 64^3 or more has
    // at most one CTA an SM anyway.  (Batch of 24 64^3 FP32 boxes, a launch a phase: one CTA an SM 266 us a step.)
    static constexpr int FIT = (sizeof(K) == 4 ? 1024 : 512) / NT > 1 ? (sizeof(K) == 4 ? 1024 : 512) / NT : 1;
    static constexpr int MINB = N >= 64 ? 1 : FIT, MINBP = FIT;
    static constexpr int H = N / 2, HC = H + 1, NHP = half_pitch<R>(N), P = N + 1;
    static constexpr int F0 = F::R[0], FL = F::R[F::NST - 1];
    // FP32: the stages on either side of the drift in FP64.  There a mode is one
    // number (or FL), so a rounding is a change of the mode itself, while the
    // roundings of the other stages average out over many; the lowest modes,
    // which carry most of a box, set the error (20 steps, 5e-24 eV).
    static constexpr bool CENTRE64 = sizeof(K) == 4 && N <= 96;
    static constexpr int CH = E % 8 == 0 && sizeof(K) == 4 ? 8 : 4;
    static constexpr bool COL = false, ROW = true;
    static_assert(F0 % 2 == 0 && E % F0 == 0 && E % FL == 0, "paired rows, whole butterflies");
    static_assert(HC * T <= NT && NT <= 1024, "threads");

    // shared memory: plane, twiddles, drift table, quadrature nodes, state
    struct Tail {
        TState st;
        StepIntegrals si;
        double red[2][32];
        int ok;
    };
    static constexpr size_t TILE = (size_t(N) * P * sizeof(C) + 15) / 16 * 16;
    static constexpr size_t OFF_TW = TILE, OFF_DR = OFF_TW + size_t(N) * 16, OFF_GK = OFF_DR + size_t(N) * 16;
    static constexpr size_t OFF_TAIL = OFF_GK + sizeof(GkNodes);
    static constexpr size_t SMEM = OFF_TAIL + sizeof(Tail);
    static_assert(SMEM <= 227 * 1024, "shared memory per block");

    template <bool RW> __device__ __forceinline__ static int ad(int l, int n) { return RW ? l * P + n : n * P + l; }

    template <int RAD, bool RW> __device__ __forceinline__ static void get(const C *sm, C *v, int l, int t) {
#pragma unroll
        for (int b = 0; b < E / RAD; ++b)
#pragma unroll
            for (int r = 0; r < RAD; ++r) v[b * RAD + r] = sm[ad<RW>(l, t + T * b + r * (N / RAD))];
    }
    template <int RAD, int NS, bool RW> __device__ __forceinline__ static void put(C *sm, const C *v, int l, int t) {
#pragma unroll
        for (int b = 0; b < E / RAD; ++b) {
            const int j = t + T * b;
            const int base = (j / NS) * NS * RAD + j % NS;
#pragma unroll
            for (int r = 0; r < RAD; ++r) sm[ad<RW>(l, base + r * NS)] = v[b * RAD + r];
        }
    }
    // stages S .. of a transform; OPEN: the last one is left at its loaded inputs
    template <class PL, int DIR, bool RW, int S, int NS, bool OPEN = false>
    __device__ __forceinline__ static void chain(C *sm, C *v, SmemTw<C> tw, const Lane &q) {
        if constexpr (S < PL::NST) {
            constexpr int RP = PL::R[S - 1], RAD = PL::R[S];
            __syncthreads();
            if (q.act) put<RP, NS / RP, RW>(sm, v, q.l, q.t);
            __syncthreads();
            if (q.act) {
                get<RAD, RW>(sm, v, q.l, q.t);
                if constexpr (!OPEN || S + 1 < PL::NST) stage_compute<C, N, E, DIR, RAD, NS>(v, tw, q.t);
            }
            chain<PL, DIR, RW, S + 1, NS * RAD, OPEN>(sm, v, tw, q);
        }
    }
    // v: stage-0 inputs of line l -> outputs v[b RL + r] = element t + T b + r N/RL
    template <class PL, int DIR, bool RW>
    __device__ __forceinline__ static void fft(C *sm, C *v, SmemTw<C> tw, const Lane &q) {
        constexpr int R0 = PL::R[0];
        if (q.act) stage_compute<C, N, E, DIR, R0, 1>(v, tw, q.t);
        chain<PL, DIR, RW, 1, R0>(sm, v, tw, q);
    }
    // store outputs (last radix RL) along RA, sync; the caller loads
    template <int RL, bool RA> __device__ __forceinline__ static void turn(C *sm, const C *v, const Lane &q) {
        __syncthreads();
        if (q.act) put<RL, N / RL, RA>(sm, v, q.l, q.t);
        __syncthreads();
    }

    // block maximum -> one atomic per CTA (called by all threads)
    __device__ __forceinline__ static void block_max(double m, double *red, unsigned long long *dst) {
        m = warp_max(m);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
        __syncthreads();
        if (threadIdx.x < 32) {
            m = threadIdx.x < NT / 32 ? red[threadIdx.x] : 0.0;
            m = warp_max(m);
            if (threadIdx.x == 0) atomic_max_nonneg(dst, m);
        }
    }

    // packed density rows (y in .x, y + N/2 in .y of w[b F0/2 + r]) -> half
    // spectrum of plane p, transformed along z and y
    __device__ __forceinline__ static void rho_to_half(C *sm, const C *w, SmemTw<C> tw, G *rhok, int p, uint32_t salt) {
        {
            const Lane q(N);
            __syncthreads();
            if (q.act) {
#pragma unroll
                for (int b = 0; b < E / F0; ++b)
#pragma unroll
                    for (int r = 0; r < F0 / 2; ++r) sm[t_row(q.t, b, r) * P + q.l] = w[b * (F0 / 2) + r];
            }
            __syncthreads();
        }
        C v[E] = {};
        {
            const Lane q(H);
            if (q.act) get<F0, ROW>(sm, v, q.l, q.t);
            fft<F, -1, ROW>(sm, v, tw, q);
            turn<FL, ROW>(sm, v, q);
        }
        const Lane q(HC);
        if (q.act) {
            const int m = q.l ? N - q.l : 0;
#pragma unroll
            for (int b = 0; b < E / F0; ++b)
#pragma unroll
                for (int r = 0; r < F0 / 2; ++r) {
                    const int y = t_row(q.t, b, r);
                    const C zk = sm[y * P + q.l], zc = cconj(sm[y * P + m]);
                    const C s = cscale(zk + zc, K(0.5)), d = cscale(zk - zc, K(0.5));
                    v[b * F0 + r] = s;
                    v[b * F0 + r + F0 / 2] = mkc(d.y, -d.x);
                }
        }
        fft<F, -1, COL>(sm, v, tw, q);
        if (q.act) {
#pragma unroll
            for (int b = 0; b < E / FL; ++b)
#pragma unroll
                for (int r = 0; r < FL; ++r) {
                    const size_t gi = (size_t(p) * N + (q.t + T * b + r * (N / FL))) * NHP + q.l;
                    rhok[gi] = Cvt<R, K>::out(v[b * FL + r], salt, gi);
                }
        }
    }
    __device__ __forceinline__ static int t_row(int t, int b, int r) { return t + T * b + r * (N / F0); }

    // D: plane ky = p of the half spectrum
    __device__ __forceinline__ static void poisson_x(C *sm, SmemTw<C> tw, G *rhok, int p, uint32_t salt) {
        const Lane q(HC);
        C v[E] = {};
        if (q.act) {
#pragma unroll
            for (int b = 0; b < E / F0; ++b)
#pragma unroll
                for (int r = 0; r < F0; ++r)
                    v[b * F0 + r] = cin<K>(__ldcg(rhok + (size_t(t_row(q.t, b, r)) * N + p) * NHP + q.l));
        }
        fft<F, -1, COL>(sm, v, tw, q);
        if (q.act) {
            const int ky = kappa(p, N), kz = kappa(q.l, N), k2yz = ky * ky + kz * kz;
#pragma unroll
            for (int b = 0; b < E / FL; ++b)
#pragma unroll
                for (int r = 0; r < FL; ++r) {
                    const int kx = kappa(q.t + T * b + r * (N / FL), N), k2 = kx * kx + k2yz;
                    v[b * FL + r] = cscale(v[b * FL + r], k2 == 0 ? K(0) : K(-1) / K(k2));
                }
        }
        fft<B, +1, COL>(sm, v, tw, q);
        if (q.act) {
#pragma unroll
            for (int b = 0; b < E / F0; ++b)
#pragma unroll
                for (int r = 0; r < F0; ++r) {
                    const size_t gi = (size_t(t_row(q.t, b, r)) * N + p) * NHP + q.l;
                    rhok[gi] = Cvt<R, K>::out(v[b * F0 + r], salt, gi);
                }
        }
    }

    // E: half spectrum of x plane p -> real plane in shared memory: element
    // (y, z) is .x (y < N/2) or .y (row y - N/2) of sm[(y % H) P + z], the value
    // as it is stored (rounded to R); global when out != null.  Returns this
    // thread's max over the scan window.
    __device__ __forceinline__ static double half_to_real(C *sm, SmemTw<C> tw, const G *rhok, R *out, int p, uint32_t salt,
                                                          long win_rows, int win_tail) {
        const int tid = threadIdx.x;
        C v[E] = {};
        {
            const Lane q(HC);
            if (q.act) {
#pragma unroll
                for (int b = 0; b < E / FL; ++b)
#pragma unroll
                    for (int r = 0; r < FL; ++r)
                        v[b * FL + r] =
                            cin<K>(__ldcg(rhok + (size_t(p) * N + (q.t + T * b + r * (N / FL))) * NHP + q.l));
            }
            fft<B, +1, COL>(sm, v, tw, q);
            turn<F0, COL>(sm, v, q);
        }
        {
            const Lane q(H);
            if (q.act) {
#pragma unroll
                for (int b = 0; b < E / FL; ++b)
#pragma unroll
                    for (int r = 0; r < FL; ++r) {
                        const int n = q.t + T * b + r * (N / FL), m = n <= H ? n : N - n;
                        C x = sm[q.l * P + m], y = sm[(q.l + H) * P + m];
                        if (m == 0 || m == H) x.y = y.y = K(0);  // c2r ignores these imaginary parts
                        v[b * FL + r] = n <= H ? mkc(x.x - y.y, x.y + y.x) : mkc(x.x + y.y, y.x - x.y);
                    }
            }
            fft<B, +1, ROW>(sm, v, tw, q);
            turn<F0, ROW>(sm, v, q);
        }
        constexpr KSplit<K> inv(1.0 / ((double)N * N * N));
        double mx = 0.0;
        for (int f = tid; f < H * N; f += NT) {
            const int y = f / N, z = f % N;
            const long ra = long(p) * N + y, rb = ra + H;
            const C q = sm[y * P + z];
            const R a = Cvt<R, K>::outr(mulk(q.x, inv.hi, inv.lo), salt, size_t(ra) * N + z);
            const R b = Cvt<R, K>::outr(mulk(q.y, inv.hi, inv.lo), salt, size_t(rb) * N + z);
            sm[y * P + z] = mkc((K)a, (K)b);
            if (out) {
                out[size_t(ra) * N + z] = a;
                out[size_t(rb) * N + z] = b;
            }
            if (ra < win_rows || (ra == win_rows && z < win_tail)) mx = fmax(mx, fabs((double)a));
            if (rb < win_rows || (rb == win_rows && z < win_tail)) mx = fmax(mx, fabs((double)b));
        }
        return mx;
    }
    // this thread's i-th stage-0 element of column l in x plane p
    __device__ __forceinline__ static int row_of(int t, int i) { return t + T * (i / F0) + (i % F0) * (N / F0); }
    __device__ __forceinline__ static size_t elem(int p, int t, int i, int l) {
        return (size_t(p) * N + row_of(t, i)) * N + l;
    }
    // the real plane's value there (half_to_real's layout)
    __device__ __forceinline__ static R real_at(const C *sm, int t, int i, int l) {
        const int r = i % F0, i2 = r < F0 / 2 ? i : i - F0 / 2;
        const C q = sm[row_of(t, i2) * P + l];
        return (R)(r < F0 / 2 ? q.x : q.y);
    }

    // A: columns y of x plane p; KICK: psi with the merged kick (phi null: the
    // real plane in shared memory), else the field as it is
    template <bool KICK>
    __device__ __forceinline__ static void kick_y(C *sm, SmemTw<C> tw, G *psi, const R *phi, const TState *st, int p,
                                                  G *seg_psi, R *seg_phi) {
        const Lane q(N);
        const int l = q.l, t = q.t;
        const bool act = q.act;
        const uint32_t salt = pass_salt(st, 1);
        C v[E] = {};
        if (act) {
            const double cp = st->coefP, cq = st->coefQ, alpha = st->alpha;
            const C c0 = mkc((K)st->cre, (K)st->cim);
            // CH elements' loads at a time: all E at once do not fit the registers
#pragma unroll
            for (int i0 = 0; i0 < E; i0 += CH) {
                G g[CH];
                R ph[CH];
#pragma unroll
                for (int i = 0; i < CH; ++i) g[i] = __ldcg(psi + elem(p, t, i0 + i, l));
                if constexpr (KICK) {
#pragma unroll
                    for (int i = 0; i < CH; ++i)
                        ph[i] = phi ? __ldcg(phi + elem(p, t, i0 + i, l)) : real_at(sm, t, i0 + i, l);
                }
#pragma unroll
                for (int i = 0; i < CH; ++i) {
                    if constexpr (!KICK) {
                        v[i0 + i] = cin<K>(g[i]);
                    } else {
                        const double2 x = cin<double>(g[i]);
                        const double q = cp * (double)ph[i] + cq * cnorm2(x) + alpha;
                        v[i0 + i] = BoxKick<K>::run(x, q, c0);
                        if (seg_psi) {
                            seg_psi[elem(p, t, i0 + i, l)] = g[i];
                            seg_phi[elem(p, t, i0 + i, l)] = ph[i];
                        }
                    }
                }
            }
        }
        fft<F, -1, COL>(sm, v, tw, q);
        if (act) {
#pragma unroll
            for (int b = 0; b < E / FL; ++b)
#pragma unroll
                for (int r = 0; r < FL; ++r) {
                    const size_t gi = (size_t(p) * N + (t + T * b + r * (N / FL))) * N + l;
                    psi[gi] = Cvt<R, K>::out(v[b * FL + r], salt, gi);
                }
        }
    }

    // B: y plane p.  dr: exp(-i s kappa^2) per axis index.  cn: receives the
    // mean of the field from the k = 0 coefficient (plane 0; may be null)
    __device__ __forceinline__ static void drift_xz(C *sm, SmemTw<C> tw, G *psi, const double2 *dr, int p,
                                                    uint32_t salt, double2 c, double *cn) {
        const Lane q(N);
        const int l = q.l, t = q.t;
        const bool act = q.act;
        C v[E] = {};
        if (act) {
#pragma unroll
            for (int b = 0; b < E / F0; ++b)
#pragma unroll
                for (int r = 0; r < F0; ++r) v[b * F0 + r] = cin<K>(__ldcg(psi + (size_t(t_row(t, b, r)) * N + p) * N + l));
        }
        fft<F, -1, COL>(sm, v, tw, q);
        turn<FL, COL>(sm, v, q);
        if (act) get<F0, ROW>(sm, v, l, t);
        if (act) stage_compute<C, N, E, -1, F0, 1>(v, tw, t);
        chain<F, -1, ROW, 1, F0, CENTRE64>(sm, v, tw, q);
        if (act) {
            // the factor and its product with the field in FP64 whatever the storage type, rounded once
            const double inv = 1.0 / ((double)N * N * N);
            double2 f0 = cmul(dr[l], dr[p]);
            f0 = mkc(f0.x * inv, f0.y * inv);
            const bool k0 = cn && p == 0 && threadIdx.x == 0;
            if constexpr (CENTRE64) {
#pragma unroll
                for (int b = 0; b < E / FL; ++b) {
                    double2 d[FL];
#pragma unroll
                    for (int r = 0; r < FL; ++r) {
                        d[r] = cin<double>(v[b * FL + r]);
                        if (r > 0) {  // last stage: twiddle (t + T b) r / N
                            const float4 w = reinterpret_cast<const float4 *>(tw.p)[(t + T * b) * r];
                            d[r] = cmul(d[r], make_double2((double)w.x + (double)w.z, (double)w.y + (double)w.w));
                        }
                    }
                    Bfly<FL, -1>::run(d);
                    if (b == 0 && k0) {
                        cn[0] = c.x + d[0].x * inv;
                        cn[1] = c.y + d[0].y * inv;
                    }
#pragma unroll
                    for (int r = 0; r < FL; ++r) d[r] = cmul(d[r], cmul(f0, dr[t + T * b + r * (N / FL)]));
                    Bfly<FL, +1>::run(d);
#pragma unroll
                    for (int r = 0; r < FL; ++r) v[b * FL + r] = mkc((K)d[r].x, (K)d[r].y);
                }
            } else {
                if (k0) {
                    cn[0] = c.x + (double)v[0].x * inv;
                    cn[1] = c.y + (double)v[0].y * inv;
                }
#pragma unroll
                for (int b = 0; b < E / FL; ++b)
#pragma unroll
                    for (int r = 0; r < FL; ++r) {
                        const double2 w = cmul(cin<double>(v[b * FL + r]), cmul(f0, dr[t + T * b + r * (N / FL)]));
                        v[b * FL + r] = mkc((K)w.x, (K)w.y);
                    }
                stage_compute<C, N, E, +1, FL, 1>(v, tw, t);
            }
        }
        chain<B, +1, ROW, 1, FL>(sm, v, tw, q);
        turn<F0, ROW>(sm, v, q);
        if (act) get<FL, COL>(sm, v, l, t);
        fft<B, +1, COL>(sm, v, tw, q);
        if (act) {
#pragma unroll
            for (int b = 0; b < E / F0; ++b)
#pragma unroll
                for (int r = 0; r < F0; ++r) {
                    const size_t gi = (size_t(t_row(t, b, r)) * N + p) * N + l;
                    psi[gi] = Cvt<R, K>::out(v[b * F0 + r], salt, gi);
                }
        }
    }

    // first half of C: inverse FFT along y of plane p into v (element t_row of column l)
    __device__ __forceinline__ static void inverse_y(C *sm, SmemTw<C> tw, const G *psi, int p, C *v) {
        const Lane q(N);
        const int l = q.l, t = q.t;
        const bool act = q.act;
        if (act) {
#pragma unroll
            for (int b = 0; b < E / FL; ++b)
#pragma unroll
                for (int r = 0; r < FL; ++r)
                    v[b * FL + r] = cin<K>(__ldcg(psi + (size_t(p) * N + (t + T * b + r * (N / FL))) * N + l));
        }
        fft<B, +1, COL>(sm, v, tw, q);
    }
    // C
    __device__ __forceinline__ static double density(C *sm, SmemTw<C> tw, G *psi, G *rhok, const TState *st, int p) {
        const Lane q(N);
        const int l = q.l, t = q.t;
        C v[E] = {};
        inverse_y(sm, tw, psi, p, v);
        double mx = 0.0;
        const uint32_t salt = pass_salt(st, 5);
        C w[E / 2] = {};
        if (q.act) {
            const double mu = st->mu;
            const C c0 = mkc((K)st->cre, (K)st->cim);
            K rho[E];
#pragma unroll
            for (int b = 0; b < E / F0; ++b)
#pragma unroll
                for (int r = 0; r < F0; ++r) {
                    const size_t gi = (size_t(p) * N + t_row(t, b, r)) * N + l;
                    const G g = Cvt<R, K>::out(v[b * F0 + r] + c0, salt, gi);
                    psi[gi] = g;
                    const double n2 = cnorm2(cin<double>(g));  // the stored value defines the density
                    mx = fmax(mx, n2);
                    rho[b * F0 + r] = (K)(n2 - mu);
                }
#pragma unroll
            for (int b = 0; b < E / F0; ++b)
#pragma unroll
                for (int r = 0; r < F0 / 2; ++r) w[b * (F0 / 2) + r] = mkc(rho[b * F0 + r], rho[b * F0 + r + F0 / 2]);
        }
        rho_to_half(sm, w, tw, rhok, p, pass_salt(st, 10));
        return mx;
    }

    // kick adjoint pieces at this thread's elements: theta's sine and cosine
    __device__ __forceinline__ static void kick_angle(G s, R f, double a, double b, double alpha, double &sn, double &cs) {
        const double px = (double)s.x, py = (double)s.y;
        const double th = a * (double)f + b * (px * px + py * py) + alpha;
        // both to FP64's last bits; FP32, 128^3, 20 steps, replay and sweep: 3.69 ms with sincos_pi, 3.51 with the series
        if constexpr (sizeof(K) == 8) sincos_pi(th, sn, cs);
        else sincos_series<true>(th, sn, cs);
    }
    // w = Im(conj(g) psi exp(-i theta)), rounded as it is stored
    __device__ __forceinline__ static R adj_w(G g, G s, double sn, double cs) {
        const double px = (double)s.x, py = (double)s.y;
        const double qx = px * cs + py * sn, qy = py * cs - px * sn;
        return (R)((double)g.x * qy - (double)g.y * qx);
    }
    // source of the adjoint's Poisson solve: INV: g' = inverse FFT along y first
    template <bool INV>
    __device__ __forceinline__ static void adj_source(C *sm, SmemTw<C> tw, G *g, G *rhok, const G *psi, const R *phi, double a,
                                                      double b, double alpha, int p, uint32_t salt) {
        const Lane q(N);
        const int l = q.l, t = q.t;
        C v[E] = {}, w[E / 2] = {};
        if constexpr (INV) inverse_y(sm, tw, g, p, v);
        if (q.act) {
            K rho[E];
#pragma unroll
            for (int q = 0; q < E / F0; ++q)
#pragma unroll
                for (int r = 0; r < F0; ++r) {
                    const size_t gi = (size_t(p) * N + t_row(t, q, r)) * N + l;
                    G x;
                    if constexpr (INV) {
                        x = Cvt<R, K>::out(v[q * F0 + r], salt, gi);
                        g[gi] = x;
                    } else {
                        x = __ldcg(g + gi);
                    }
                    const G s = psi[gi];
                    double sn, cs;
                    kick_angle(s, phi[gi], a, b, alpha, sn, cs);
                    rho[q * F0 + r] = (K)adj_w(x, s, sn, cs);
                }
#pragma unroll
            for (int q = 0; q < E / F0; ++q)
#pragma unroll
                for (int r = 0; r < F0 / 2; ++r) w[q * (F0 / 2) + r] = mkc(rho[q * F0 + r], rho[q * F0 + r + F0 / 2]);
        }
        rho_to_half(sm, w, tw, rhok, p, salt ^ 0x3c6ef372u);
    }
    // g <- exp(+i theta) g + 2 (a phi_s[w] + b w) psi, phi_s[w] in shared memory
    __device__ __forceinline__ static void adj_combine(const C *sm, G *g, const G *psi, const R *phi, double a, double b,
                                                       double alpha, int p, uint32_t salt) {
        const Lane q(N);
        const int l = q.l, t = q.t;
        if (!q.act) return;
#pragma unroll
        for (int q = 0; q < E / F0; ++q)
#pragma unroll
            for (int r = 0; r < F0; ++r) {
                const size_t gi = (size_t(p) * N + t_row(t, q, r)) * N + l;
                const G s = psi[gi], x = g[gi];
                double sn, cs;
                kick_angle(s, phi[gi], a, b, alpha, sn, cs);
                const double u = a * (double)real_at(sm, t, q * F0 + r, l) + b * (double)adj_w(x, s, sn, cs);
                const double gx = (double)x.x, gy = (double)x.y;
                g[gi] = Cvt<R, double>::out(make_double2(gx * cs - gy * sn + 2.0 * u * (double)s.x,
                                                         gy * cs + gx * sn + 2.0 * u * (double)s.y),
                                            salt, gi);
            }
    }

    // initial pass: the sums of plane p
    __device__ __forceinline__ static void initial_sums(const BoxRun &a, int p) {
        const Lane q(N);
        const int l = q.l, t = q.t, tid = threadIdx.x;
        const G *psi = (const G *)a.psi;
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, mx = 0.0;
        if (q.act) {
#pragma unroll
            for (int i = 0; i < E; ++i) {
                const G g = psi[elem(p, t, i, l)];
                const double n2 = cnorm2(cin<double>(g));
                s0 += (double)g.x;
                s1 += (double)g.y;
                s2 += n2;
                mx = fmax(mx, n2);
            }
        }
        __shared__ unsigned long long s_mx;
        if (tid == 0) s_mx = 0ull;
        block_sum3(s0, s1, s2, a.scr->part[p]);
        mx = warp_max(mx);
        if ((tid & 31) == 0) atomic_max_nonneg(&s_mx, mx);
        __syncthreads();
        if (tid == 0) a.scr->part[p][3] = bits_to_double(s_mx);
        __syncthreads();
    }
    // and the half spectrum of the density less a constant (the k = 0 mode is
    // dropped) near its mean: what is rounded to K (FP32), or to the stored half
    // spectrum (mixed), is then small where the density is near its mean.  The
    // constant is the first cell's density, held to within a factor of two of the
    // mean so that no cell's rounding depends on a halo or a void there.  phi
    // against FP64, 64^3, contrast 0.02: nothing subtracted 1.6e-6 (FP32) and
    // 2.1e-6 (mixed), so 2.4e-7 and 1.9e-7, the mean itself 2.2e-7 and 1.8e-7.
    __device__ __forceinline__ static void initial_density(C *sm, SmemTw<C> tw, const BoxRun &a, const TState *st, int p) {
        const Lane q(N);
        const G *psi = (const G *)a.psi;
        const double mu = st->mu, ref = fmin(fmax(cnorm2(cin<double>(psi[0])), 0.5 * mu), 2.0 * mu);
        C w[E / 2] = {};
        if (q.act) {
            K rho[E];
#pragma unroll
            for (int i = 0; i < E; ++i) rho[i] = (K)(cnorm2(cin<double>(psi[elem(p, q.t, i, q.l)])) - ref);
#pragma unroll
            for (int b = 0; b < E / F0; ++b)
#pragma unroll
                for (int r = 0; r < F0 / 2; ++r) w[b * (F0 / 2) + r] = mkc(rho[b * F0 + r], rho[b * F0 + r + F0 / 2]);
        }
        rho_to_half(sm, w, tw, (G *)a.rhok, p, pass_salt(st, 10));
    }
};

// exp(-i s kappa^2) per axis index (conj: +i), all threads of the block
static __device__ __noinline__ void box_drift_table(double2 *dr, double s, int N, bool conj) {
    const double twopi = 6.283185307179586476925286766559;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        const double k = (double)kappa(i, N);
        double p = s * (k * k);
        p -= twopi * rint(p * (1.0 / twopi));
        double sn, cs;
        sincos_pi(p, sn, cs);
        dr[i] = make_double2(cs, conj ? sn : -sn);
    }
}

// shared-memory pieces of a block
template <class O> struct BoxShared {
    typename O::C *sm;
    SmemTw<typename O::C> tw;
    double2 *dr;
    GkNodes *gk;
    typename O::Tail *tail;
    __device__ __forceinline__ BoxShared(unsigned char *raw, const void *table) {
        using C = typename O::C;
        sm = reinterpret_cast<C *>(raw);
        C *t = reinterpret_cast<C *>(raw + O::OFF_TW);
        tw.p = t;
        dr = reinterpret_cast<double2 *>(raw + O::OFF_DR);
        gk = reinterpret_cast<GkNodes *>(raw + O::OFF_GK);
        tail = reinterpret_cast<typename O::Tail *>(raw + O::OFF_TAIL);
        stage_twiddles(t, reinterpret_cast<const C *>(table), O::SIZE);
    }
};

// Load recorded step `e` as the current one (replay of a segment).
__device__ __forceinline__ void box_replay(TState *st, const StepLog &e) {
    st->steps = e.steps;
    st->coefP = e.coefP;
    st->coefQ = e.coefQ;
    st->alpha = e.alpha;
    st->drift_s = e.drift_s;
    st->cre = e.cre;
    st->cim = e.cim;
    st->pendP = e.pendP;
    st->pendQ = e.pendQ;
    st->gphase = e.gphase;
    st->a = e.a;
}

// nsteps leap-frog steps of each box; gridDim.x = boxes * group
template <typename R, typename K, int N, int V>
__global__ void __launch_bounds__(BoxOps<R, K, N, V>::NT, BoxOps<R, K, N, V>::MINB)
    k_box_run(const __grid_constant__ BoxRun one, const BoxRun *many, int nsteps, int group, int cluster) {
    using O = BoxOps<R, K, N, V>;
    using G = typename O::G;
    extern __shared__ __align__(16) unsigned char smraw[];
    const BoxRun &a = many ? many[blockIdx.x / group] : one;
    const int rank = blockIdx.x % group, tid = threadIdx.x;
    BoxShared<O> s(smraw, a.tw);
    TState *st = &s.tail->st;
    gk_fill(s.gk);
    if (tid == 0) *st = *a.ts;
    GroupBarrier bar;
    bar.init(&a.scr->ctr[group != N], group, cluster != 0, &a.ts->err, &s.tail->ok);
    __syncthreads();
    G *psi = (G *)a.psi, *rhok = (G *)a.rhok;
    R *phi = (R *)a.phi;
    BoxScratch *scr = a.scr;
    const bool keep = group == N;  // phi stays in shared memory from E to the next A
    const size_t n3 = size_t(N) * N * N;
    if (a.timestep == 1 && tid < 32) step_integrals(st->a, kinetic_dt(st->a, a.ph), a.ph, s.gk, &s.tail->si);
    for (int n = 0; n < nsteps; ++n) {
        const bool last = n + 1 == nsteps;
        unsigned long long *mphi = last ? &a.ts->maxphi_bits : &scr->mx[(n + 1) & 1][0];
        unsigned long long *mrho = last ? &a.ts->maxrho_bits : &scr->mx[(n + 1) & 1][1];
        if (a.timestep == 1) {
            if (tid < 32) {
                unsigned long long b0 = st->maxphi_bits, b1 = st->maxrho_bits;
                double c0 = st->cnext_re, c1 = st->cnext_im;
                if (n) {
                    b0 = __ldcg(&scr->mx[n & 1][0]);
                    b1 = __ldcg(&scr->mx[n & 1][1]);
                    c0 = __ldcg(&scr->cnext[0]);
                    c1 = __ldcg(&scr->cnext[1]);
                }
                timestep_warp(st, a.ph, s.gk, &s.tail->si, b0, b1, c0, c1);
                if (a.log && rank == 0 && tid == 0) log_step(st, a.log + n);
            }
            __syncthreads();
        } else if (a.timestep == 2) {
            if (tid == 0) box_replay(st, a.log[n]);
            __syncthreads();
        }
        for (int p = rank; p < N; p += group) {
            G *sp = a.seg_psi ? (G *)a.seg_psi + n * n3 : nullptr;
            R *sf = a.seg_phi ? (R *)a.seg_phi + n * n3 : nullptr;
            O::template kick_y<true>(s.sm, s.tw, psi, keep && n ? nullptr : phi, st, p, sp, sf);
        }
        bar.arrive();
        box_drift_table(s.dr, st->drift_s, N, false);
        if (!bar.wait()) return;
        const double2 c = make_double2(st->cre, st->cim);
        for (int p = rank; p < N; p += group)
            O::drift_xz(s.sm, s.tw, psi, s.dr, p, pass_salt(st, 3), c, &st->cnext_re);
        if (rank == 0 && tid == 0) {
            // the sums of this step, or the whole state after the last one
            // (every CTA has read the previous ones before the barrier above)
            if (last) {
                st->maxphi_bits = st->maxrho_bits = 0ull;
                *a.ts = *st;
            } else {
                *mphi = 0ull;
                *mrho = 0ull;
                scr->cnext[0] = st->cnext_re;
                scr->cnext[1] = st->cnext_im;
            }
        }
        if (!bar.sync()) return;
        double mx = 0.0;
        for (int p = rank; p < N; p += group) mx = fmax(mx, O::density(s.sm, s.tw, psi, rhok, st, p));
        O::block_max(mx, s.tail->red[0], mrho);
        if (!bar.sync()) return;
        for (int p = rank; p < N; p += group) O::poisson_x(s.sm, s.tw, rhok, p, pass_salt(st, 7));
        if (!bar.sync()) return;
        mx = 0.0;
        for (int p = rank; p < N; p += group)
            mx = fmax(mx, O::half_to_real(s.sm, s.tw, rhok, keep && !last ? nullptr : phi, p, pass_salt(st, 9), a.win_rows,
                                          a.win_tail));
        O::block_max(mx, s.tail->red[1], mphi);
        if (!last) {
            bar.arrive();
            // the next kinetic step's integrals while the others arrive, on a
            // warp that does not poll
            if (a.timestep == 1 && tid >= 32 && tid < 64)
                step_integrals(st->a, kinetic_dt(st->a, a.ph), a.ph, s.gk, &s.tail->si);
            if (!bar.wait()) return;
        }
    }
}

// the initial density and potential of psi, the state at a0
template <typename R, typename K, int N, int V>
__global__ void __launch_bounds__(BoxOps<R, K, N, V>::NT, BoxOps<R, K, N, V>::MINB)
    k_box_load(const __grid_constant__ BoxRun a, int group, int cluster) {
    using O = BoxOps<R, K, N, V>;
    using G = typename O::G;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int rank = blockIdx.x % group, tid = threadIdx.x;
    BoxShared<O> s(smraw, a.tw);
    TState *st = &s.tail->st;
    if (tid == 0) {
        *st = TState{};
        st->a = a.a0;
    }
    GroupBarrier bar;
    bar.init(&a.scr->ctr[group != N], group, cluster != 0, &a.ts->err, &s.tail->ok);
    __syncthreads();
    G *rhok = (G *)a.rhok;
    for (int p = rank; p < N; p += group) O::initial_sums(a, p);
    if (!bar.sync()) return;
    if (tid < 32) {
        // every CTA: lane l adds planes l, l + 32, ... in order, then the lanes in a fixed tree
        double v[3] = {0.0, 0.0, 0.0}, m = 0.0;
        for (int p = tid; p < N; p += 32) {
            for (int q = 0; q < 3; ++q) v[q] += __ldcg(&a.scr->part[p][q]);
            m = fmax(m, __ldcg(&a.scr->part[p][3]));
        }
        m = warp_max(m);
        for (int q = 0; q < 3; ++q)
            for (int o = 16; o > 0; o >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], o);
        if (tid == 0) {
            const double n3 = (double)N * N * N;
            st->cnext_re = v[0] / n3;
            st->cnext_im = v[1] / n3;
            st->mu = v[2] / n3;
            st->maxrho_bits = (unsigned long long)__double_as_longlong(m);
            if (rank == 0) *a.ts = *st;
        }
    }
    __syncthreads();
    for (int p = rank; p < N; p += group) O::initial_density(s.sm, s.tw, a, st, p);
    if (!bar.sync()) return;
    for (int p = rank; p < N; p += group) O::poisson_x(s.sm, s.tw, rhok, p, pass_salt(st, 7));
    if (!bar.sync()) return;
    double mx = 0.0;
    for (int p = rank; p < N; p += group)
        mx = fmax(mx, O::half_to_real(s.sm, s.tw, rhok, (R *)a.phi, p, pass_salt(st, 9), a.win_rows, a.win_tail));
    O::block_max(mx, s.tail->red[1], &a.ts->maxphi_bits);
}

// The adjoint of steps end-1 .. start on g, or (end == start) of the output map alone.
template <typename R, typename K, int N, int V>
__global__ void __launch_bounds__(BoxOps<R, K, N, V>::NT, BoxOps<R, K, N, V>::MINB)
    k_box_sweep(const __grid_constant__ BoxSweep a, int group, int cluster) {
    using O = BoxOps<R, K, N, V>;
    using G = typename O::G;
    extern __shared__ __align__(16) unsigned char smraw[];
    const int rank = blockIdx.x % group, tid = threadIdx.x;
    BoxShared<O> s(smraw, a.tw);
    TState *st = &s.tail->st;
    GroupBarrier bar;
    bar.init(&a.scr->ctr[group != N], group, cluster != 0, a.err, &s.tail->ok);
    __syncthreads();
    G *g = (G *)a.g, *rhok = (G *)a.rhok;
    const size_t n3 = size_t(N) * N * N;
    const bool map = a.end == a.start;
    for (int n = map ? a.start : a.end - 1; n >= a.start; --n) {
        const uint32_t key = mix32((uint32_t)n * 0x85ebca6bu ^ (map ? 0x51ed270bu : 0xc2b2ae35u));
        double ka = a.a, kb = a.b, kal = a.alpha, drift_s = 0.0;
        const G *psi = (const G *)a.last_psi;
        const R *phi = (const R *)a.last_phi;
        if (!map) {
            const StepLog *e = a.log + n;
            ka = e->coefP;
            kb = e->coefQ;
            kal = e->alpha;
            drift_s = e->drift_s;
            if (n + 1 < a.end) {
                psi = (const G *)a.seg_psi + size_t(n - a.start) * n3;
                phi = (const R *)a.seg_phi + size_t(n - a.start) * n3;
            }
            if (tid == 0) {
                st->steps = (1ll << 32) + n;
                st->cre = st->cim = 0.0;
            }
            __syncthreads();
            for (int p = rank; p < N; p += group)
                O::template kick_y<false>(s.sm, s.tw, g, nullptr, st, p, nullptr, nullptr);
            bar.arrive();
            box_drift_table(s.dr, drift_s, N, true);
            if (!bar.wait()) return;
            for (int p = rank; p < N; p += group)
                O::drift_xz(s.sm, s.tw, g, s.dr, p, key ^ 0x1b873593u, make_double2(0.0, 0.0), nullptr);
            if (!bar.sync()) return;
        }
        for (int p = rank; p < N; p += group) {
            if (map) O::template adj_source<false>(s.sm, s.tw, g, rhok, psi, phi, ka, kb, kal, p, key);
            else O::template adj_source<true>(s.sm, s.tw, g, rhok, psi, phi, ka, kb, kal, p, key);
        }
        if (!bar.sync()) return;
        for (int p = rank; p < N; p += group) O::poisson_x(s.sm, s.tw, rhok, p, key ^ 0x2545f491u);
        if (!bar.sync()) return;
        for (int p = rank; p < N; p += group) {
            O::half_to_real(s.sm, s.tw, rhok, nullptr, p, key ^ 0x6a09e667u, 0, 0);
            __syncthreads();
            O::adj_combine(s.sm, g, psi, phi, ka, kb, kal, p, key ^ 0x7f4a7c15u);
            __syncthreads();
        }
        // the next step's first phase reads this CTA's own planes of g, and
        // rhok is next written after its barriers
    }
}

// One phase (0 timestep, 1..5 A..E) of every box (blockIdx.y), plane blockIdx.x:
// the batch's other schedule, one launch per phase and size.
template <typename R, typename K, int N, int V, int PH>
__global__ void __launch_bounds__(BoxOps<R, K, N, V>::NT, BoxOps<R, K, N, V>::MINBP) k_box_phase(const BoxRun *many) {
    using O = BoxOps<R, K, N, V>;
    using G = typename O::G;
    extern __shared__ __align__(16) unsigned char smraw[];
    const BoxRun &a = many[blockIdx.y];
    const int p = blockIdx.x, tid = threadIdx.x;
    BoxShared<O> s(smraw, a.tw);
    TState *st = &s.tail->st;
    if (PH == 0) gk_fill(s.gk);
    if (tid == 0) *st = *a.ts;
    __syncthreads();
    G *psi = (G *)a.psi, *rhok = (G *)a.rhok;
    if constexpr (PH == 0) {
        if (tid < 32) {
            step_integrals(st->a, kinetic_dt(st->a, a.ph), a.ph, s.gk, &s.tail->si);
            timestep_warp(st, a.ph, s.gk, &s.tail->si, st->maxphi_bits, st->maxrho_bits, st->cnext_re, st->cnext_im);
            if (tid == 0) {
                st->maxphi_bits = st->maxrho_bits = 0ull;
                *a.ts = *st;
            }
        }
    } else if constexpr (PH == 1) {
        O::template kick_y<true>(s.sm, s.tw, psi, (const R *)a.phi, st, p, nullptr, nullptr);
    } else if constexpr (PH == 2) {
        box_drift_table(s.dr, st->drift_s, N, false);
        __syncthreads();
        O::drift_xz(s.sm, s.tw, psi, s.dr, p, pass_salt(st, 3), make_double2(st->cre, st->cim), &a.ts->cnext_re);
    } else if constexpr (PH == 3) {
        O::block_max(O::density(s.sm, s.tw, psi, rhok, st, p), s.tail->red[0], &a.ts->maxrho_bits);
    } else if constexpr (PH == 4) {
        O::poisson_x(s.sm, s.tw, rhok, p, pass_salt(st, 7));
    } else {
        O::block_max(O::half_to_real(s.sm, s.tw, rhok, (R *)a.phi, p, pass_salt(st, 9), a.win_rows, a.win_tail),
                     s.tail->red[1], &a.ts->maxphi_bits);
    }
}

}  // namespace ifdm
