// diagnostics.cu -- power spectrum and energy means of a box on the device.
//
// P(k) of delta = rho / <rho> - 1, rho = |psi|^2, estimated on the full FFT
// grid: P(k_b) = <|delta_k|^2>_b L^3 / N^6 averaged over the modes of
// bin b, with integer wave numbers kappa (|kappa| in [edge_b, edge_{b+1}),
// k = 2 pi kappa / L).  The reference has no such output; it is the measure
// the precision comparisons of the step use, so it runs where psi lives.
//
//   1. z pass: rho from psi as it is stored (a kick does not change it), its
//      sum, the real-to-half FFT along z in FP64;
//   2. FFTs along y and x of the half spectrum;
//   3. the bins: a warp takes whole (x, y) lines in a fixed order; the modes of a
//      bin within 32 consecutive kz are added by a warp tree, the bin's sums in
//      line order (kz between 0 and N/2 stands for -kz too);
//   4. one block per bin adds the partial sums in order.
// 66 bytes a cell (FP64 psi); a full complex transform of rho after writing psi
// out took 184.  Every sum has a fixed order, so the result does not change between runs.
//
// Energy means: the gradient's mean by Parseval, one axis at a time: sum over k of kappa_z^2
// |psi_k|^2 is N^2 times the sum over the lines along z of their own
// transforms, so three one-axis transforms that write nothing replace the
// three-dimensional one (72 bytes a cell instead of 176).
#include "diagnostics.hpp"
#include "step_kernels.cuh"

#include <algorithm>
#include <cmath>
#include <vector>

namespace ifdm {

#define DG_TRY(expr)                                                                     \
    do {                                                                                 \
        cudaError_t e_ = (expr);                                                         \
        if (e_ != cudaSuccess) return std::string(#expr) + ": " + cudaGetErrorString(e_); \
    } while (0)

namespace {

const char *const kGaveUp = "a device-side wait gave up";

constexpr int kBinBlocks = 592, kBinThreads = 256;  // 4 blocks per SM
constexpr int kBinWarps = kBinThreads / 32;

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double block_sum(double v, double *red) {
    v = wsum(v);
    const int w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[w] = v;
    __syncthreads();
    double t = 0.0;
    for (int i = 0; i < nw; ++i) t += red[i];  // every thread, same order
    return t;
}

// FP64 row tiles whatever psi's storage type R
template <int N> using DTile = TileZ<double, double, N>;

// rho = |psi_s|^2, part[block] its sum, real-to-half FFT along z -> rk [row][NHP]
template <typename R, int N>
__global__ void __launch_bounds__(DTile<N>::NT)
    k_rho_half_z(const cx<R> *__restrict__ psi, double2 *__restrict__ rk, double *__restrict__ part,
                 const double2 *__restrict__ tw, const double2 *__restrict__ twh) {
    using TL = DTile<N>;
    constexpr int NH = N / 2 + 1, NHP = half_pitch<double>(N), M = N / 2, PER = TL::L * N / TL::NT;
    static_assert(PER * TL::NT == TL::L * N, "whole rows per thread block");
    extern __shared__ __align__(16) unsigned char smraw[];
    double2 *sm = reinterpret_cast<double2 *>(smraw);
    double *smr = reinterpret_cast<double *>(smraw);
    const size_t row0 = size_t(blockIdx.x) * TL::L, base = row0 * N;
    cx<R> g[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) g[i] = psi[base + threadIdx.x + i * TL::NT];
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int f = threadIdx.x + i * TL::NT, l = f / N, n = f % N;
        const double n2 = cnorm2(cin<double>(g[i]));
        s += n2;
        smr[2 * ((n >> 1) * TL::LP + l) + (n & 1)] = n2;
    }
    __shared__ double out[3];
    block_sum3(s, 0.0, 0.0, out);  // syncs
    if (threadIdx.x == 0) part[blockIdx.x] = out[0];
    fft_tile<double2, M, TL::EH, -1, TL::L, TL::LP, typename TL::HP>(sm, twh);
    constexpr int TPR = TL::NT / TL::L;  // threads per row
    const int l = threadIdx.x / TPR;
    for (int k = threadIdx.x % TPR; k < NH; k += TPR) {
        const double2 zk = sm[(k % M) * TL::LP + l];
        const double2 zc = cconj(sm[((M - k) % M) * TL::LP + l]);
        const double2 e = cscale(zk + zc, 0.5);
        const double2 wo = post_tw<-1, N>(tw, k % N, cscale(zk - zc, 0.5));
        rk[(row0 + l) * NHP + k] = mkc(e.x + wo.y, e.y - wo.x);
    }
}

// psi with the pending half kick (as ifdm_get_psi, in storage units) -> out;
// part[5 block ..]: sums of |psi|^2, |psi|^4, phi |psi|^2, kappa_z^2 |FFT_z|^2
template <typename R, int N>
__global__ void __launch_bounds__(DTile<N>::NT)
    k_energy_z(const cx<R> *__restrict__ psi, const R *__restrict__ phi, const TState *__restrict__ ts,
               double2 *__restrict__ out, double *__restrict__ part, const double2 *__restrict__ tw) {
    using TL = DTile<N>;
    extern __shared__ __align__(16) unsigned char smraw[];
    double2 *sm = reinterpret_cast<double2 *>(smraw);
    const size_t base = size_t(blockIdx.x) * TL::L * N;
    const double cp = ts->pendP, cq = ts->pendQ, g = ts->gphase;
    double a = 0.0, b = 0.0, c = 0.0, k2 = 0.0;
    for (int f = threadIdx.x; f < TL::L * N; f += TL::NT) {
        const double2 v = cin<double>(psi[base + f]);
        const double p = (double)phi[base + f], r = cnorm2(v);
        double sn, cs;
        sincos(cp * p + cq * r - g, &sn, &cs);
        const double2 w = mkc(v.x * cs + v.y * sn, v.y * cs - v.x * sn);
        out[base + f] = w;
        sm[(f % N) * TL::LP + f / N] = w;
        a += r;
        b += r * r;
        c += p * r;
    }
    __syncthreads();
    fft_tile<double2, N, TL::E, -1, TL::L, TL::LP>(sm, tw);
    for (int f = threadIdx.x; f < TL::L * N; f += TL::NT) {
        const double k = (double)kappa(f % N, N);
        k2 = fma(k * k, cnorm2(sm[(f % N) * TL::LP + f / N]), k2);
    }
    __shared__ double o[6];
    block_sum3(a, b, c, o);
    __syncthreads();  // the second sum reuses block_sum3's words
    block_sum3(k2, 0.0, 0.0, o + 3);
    if (threadIdx.x == 0)
        for (int i = 0; i < 4; ++i) part[5 * size_t(blockIdx.x) + i] = o[i];
}

// out[c] = sum over blocks b (in order) of part[stride b + c], c < nv; the error
// bits beside them, *err_out (one copy brings back the results and the bits)
__global__ void k_sum_cols(const double *__restrict__ part, int nb, int stride, int nv, double *__restrict__ out,
                           const TState *__restrict__ ts, double *__restrict__ err_out) {
    __shared__ double red[32];
    if (threadIdx.x == 0) *err_out = (double)ts->err;
    for (int c = 0; c < nv; ++c) {
        double a = 0.0;
        for (int b = threadIdx.x; b < nb; b += blockDim.x) a += part[size_t(stride) * b + c];
        a = block_sum(a, red);
        if (threadIdx.x == 0) out[c] = a;
    }
}

struct BinEdges {
    double e[kMaxBins + 1];
};

__device__ __forceinline__ int bin_of(double kk, const double *e, int nb) {
    if (!(kk >= e[0]) || !(kk < e[nb])) return -1;
    int lo = 0, hi = nb;  // e[lo] <= kk < e[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (kk >= e[mid]) lo = mid;
        else hi = mid;
    }
    return lo;
}

// part[(block * nb + b) * 3 + {0,1,2}] = sum |rho_k|^2, sum |kappa|, modes
__global__ void __launch_bounds__(kBinThreads)
    k_bin_half(const double2 *__restrict__ rk, int N, int pitch, int nb, BinEdges ed, double *__restrict__ part) {
    __shared__ double e[kMaxBins + 1];
    __shared__ double acc[kBinWarps][3 * kMaxBins];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = threadIdx.x; i <= nb; i += blockDim.x) e[i] = ed.e[i];
    for (int i = lane; i < 3 * nb; i += 32) acc[w][i] = 0.0;
    __syncthreads();
    const int M = N / 2;
    const long lines = long(N) * N;
    for (long line = long(blockIdx.x) * kBinWarps + w; line < lines; line += long(gridDim.x) * kBinWarps) {
        const int ix = int(line / N), iy = int(line % N);
        const double kx = ix < M ? ix : ix - N, ky = iy < M ? iy : iy - N;
        const double2 *row = rk + line * pitch;
        for (int k0 = 0; k0 <= M; k0 += 32) {
            const int iz = k0 + lane;
            int b = -1, m = 0;
            double p = 0.0, kk = 0.0;
            if (iz <= M) {
                const double kz = iz < M ? iz : iz - N;
                m = iz == 0 || iz == M ? 1 : 2;
                kk = sqrt(kx * kx + ky * ky + kz * kz);
                b = bin_of(kk, e, nb);
                const double2 v = row[iz];
                p = kk > 0.0 ? m * (v.x * v.x + v.y * v.y) : 0.0;  // delta_0 = 0
                kk *= m;
            }
            const int b1 = __reduce_max_sync(0xffffffffu, b);
            if (b1 < 0) continue;
            const int b0 = __reduce_min_sync(0xffffffffu, b < 0 ? kMaxBins : b);
            for (int bb = b0; bb <= b1; ++bb) {
                const bool in = b == bb;
                const int cnt = __reduce_add_sync(0xffffffffu, in ? m : 0);
                if (cnt == 0) continue;
                const double sp = wsum(in ? p : 0.0), sk = wsum(in ? kk : 0.0);
                if (lane == 0) {
                    acc[w][3 * bb] += sp;
                    acc[w][3 * bb + 1] += sk;
                    acc[w][3 * bb + 2] += (double)cnt;
                }
            }
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * nb; i += blockDim.x) {
        double s = 0.0;
        for (int q = 0; q < kBinWarps; ++q) s += acc[q][i];
        part[size_t(blockIdx.x) * 3 * nb + i] = s;
    }
}

// out[b * 3 + c] = sum over groups of part[(group * nb + b) * 3 + c]
__global__ void k_bin_total(const double *__restrict__ part, int groups, int nb, double *__restrict__ out,
                            const TState *__restrict__ ts, double *__restrict__ err_out) {
    __shared__ double red[32];
    const int b = blockIdx.x;
    if (b == 0 && threadIdx.x == 0) *err_out = (double)ts->err;
    for (int c = 0; c < 3; ++c) {
        double s = 0.0;
        for (int g = threadIdx.x; g < groups; g += blockDim.x) s += part[(size_t(g) * nb + b) * 3 + c];
        const double t = block_sum(s, red);
        if (threadIdx.x == 0) out[b * 3 + c] = t;
    }
}

template <typename F> std::string with_n(int n, F &&f) {
    switch (n) {
        case 16: return f(std::integral_constant<int, 16>{});
        case 32: return f(std::integral_constant<int, 32>{});
        case 48: return f(std::integral_constant<int, 48>{});
        case 64: return f(std::integral_constant<int, 64>{});
        case 96: return f(std::integral_constant<int, 96>{});
        case 128: return f(std::integral_constant<int, 128>{});
        case 256: return f(std::integral_constant<int, 256>{});
        case 512: return f(std::integral_constant<int, 512>{});
        case 1024: return f(std::integral_constant<int, 1024>{});
        default: return "unsupported grid";
    }
}

// shared-memory attribute set at each call (cheap, and per device)
template <typename Kern> cudaError_t big_smem(Kern k, size_t bytes) {
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

// workspace: [0, 5 N^2/8) z partial sums, [.., + N^2) axis partial sums, bin parts, totals
size_t off_axis(int N) { return size_t(5) * N * N / 8; }
size_t off_bins(int N) { return off_axis(N) + size_t(N) * N; }
size_t off_out(int N) { return off_bins(N) + size_t(kBinBlocks) * 3 * kMaxBins; }

}  // namespace

size_t diag_work_doubles(int N) { return off_out(N) + 3 * kMaxBins + 8; }

std::string field_means(const EngineView &v, double S, double2 *field, double *work, double xmax, double out[4],
                        cudaStream_t s) {
    const int N = v.N;
    const double n3 = double(N) * N * N;
    double *tot = work + off_out(N);
    const void *tw = nullptr, *twh = nullptr;
    std::string e = twiddle_tables(N, 0, &tw, &twh);
    if (!e.empty()) return e;
    e = with_n(N, [&](auto n) -> std::string {
        using TL = DTile<decltype(n)::value>;
        static_assert(TL::L >= 8, "partial sums");
        const int blocks = N * N / TL::L;
        auto go = [&](auto kern, const auto *psi, const auto *phi) -> std::string {
            DG_TRY(big_smem(kern, TL::SMEM));
            kern<<<blocks, TL::NT, TL::SMEM, s>>>(psi, phi, v.ts, field, work, (const double2 *)tw);
            k_sum_cols<<<1, 1024, 0, s>>>(work, blocks, 5, 4, tot, v.ts, tot + 6);
            DG_TRY(cudaGetLastError());
            return "";
        };
        if (v.precision == 0) return go(k_energy_z<double, decltype(n)::value>, (const double2 *)v.psi, (const double *)v.phi);
        return go(k_energy_z<float, decltype(n)::value>, (const float2 *)v.psi, (const float *)v.phi);
    });
    for (int axis = 1; e.empty() && axis >= 0; --axis) {
        int np = 0;
        e = axis_k2(field, N, axis, work + off_axis(N), &np, &v.ts->err, s);
        if (e.empty()) k_sum_cols<<<1, 1024, 0, s>>>(work + off_axis(N), np, 1, 1, tot + 4 + axis, v.ts, tot + 6);
    }
    if (!e.empty()) return e;
    double h[7];
    DG_TRY(cudaMemcpyAsync(h, tot, sizeof(h), cudaMemcpyDeviceToHost, s));
    DG_TRY(cudaStreamSynchronize(s));
    if ((int)h[6] & 2) return kGaveUp;
    const double S2 = S * S, kf = 3.14159265358979323846 / xmax;  // k = pi kappa / xmax
    out[0] = h[0] / n3 * S2;
    // Parseval per axis: sum_x |d psi/dz|^2 = sum over lines of sum_k k^2 |.|^2 / N
    out[1] = (h[3] + h[4] + h[5]) / N / n3 * kf * kf * S2;
    out[2] = h[2] / n3 * S2;
    out[3] = h[1] / n3 * S2 * S2;
    return "";
}

std::string power_spectrum(const EngineView &v, double S, double2 *field, double *work, double L, int nbins,
                           const double *edges, double *k_out, double *pk_out, long long *modes_out, double *mean_rho,
                           cudaStream_t s) {
    const int N = v.N;
    if (nbins < 1 || nbins > kMaxBins) return "nbins must be 1.." + std::to_string(kMaxBins);
    const double n3 = double(N) * N * N;
    BinEdges ed{};
    if (edges) {
        for (int i = 0; i <= nbins; ++i) {
            ed.e[i] = edges[i];
            if (i > 0 && !(edges[i] > edges[i - 1])) return "bin edges must increase";
        }
    } else {
        // log-spaced |kappa| edges from 1 to N/2
        const double top = std::log10(N / 2.0);
        for (int i = 0; i <= nbins; ++i) ed.e[i] = std::pow(10.0, i * (top / nbins));
        ed.e[0] = 1.0;
        ed.e[nbins] = N / 2.0;
    }
    double *tot = work + off_out(N);
    const void *tw = nullptr, *twh = nullptr;
    std::string e = twiddle_tables(N, 0, &tw, &twh);
    if (!e.empty()) return e;
    e = with_n(N, [&](auto n) -> std::string {
        using TL = DTile<decltype(n)::value>;
        const int blocks = N * N / TL::L;
        auto go = [&](auto kern, const auto *psi) -> std::string {
            DG_TRY(big_smem(kern, TL::SMEM));
            kern<<<blocks, TL::NT, TL::SMEM, s>>>(psi, field, work, (const double2 *)tw, (const double2 *)twh);
            k_sum_cols<<<1, 1024, 0, s>>>(work, blocks, 1, 1, tot + 3 * kMaxBins, v.ts, tot + 3 * kMaxBins + 1);
            DG_TRY(cudaGetLastError());
            return "";
        };
        if (v.precision == 0) return go(k_rho_half_z<double, decltype(n)::value>, (const double2 *)v.psi);
        return go(k_rho_half_z<float, decltype(n)::value>, (const float2 *)v.psi);
    });
    if (e.empty()) e = fft_half_axis(field, N, 1, v.ts, s);
    if (e.empty()) e = fft_half_axis(field, N, 0, v.ts, s);
    if (!e.empty()) return e;
    k_bin_half<<<kBinBlocks, kBinThreads, 0, s>>>(field, N, half_pitch<double>(N), nbins, ed, work + off_bins(N));
    k_bin_total<<<nbins, 256, 0, s>>>(work + off_bins(N), kBinBlocks, nbins, tot, v.ts, tot + 3 * kMaxBins + 1);
    DG_TRY(cudaGetLastError());
    std::vector<double> h(3 * kMaxBins + 2);
    DG_TRY(cudaMemcpyAsync(h.data(), tot, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, s));
    DG_TRY(cudaStreamSynchronize(s));
    if ((int)h[3 * kMaxBins + 1] & 2) return kGaveUp;
    const double mean = h[3 * kMaxBins] / n3;
    if (mean_rho) *mean_rho = mean * S * S;
    // delta_k = rho_k / mean for kappa != 0 (the bins exclude kappa = 0)
    const double twopi = 6.283185307179586476925286766559;
    const double norm = (L * L * L) / (n3 * n3) / (mean * mean);
    for (int b = 0; b < nbins; ++b) {
        const double cnt = h[3 * b + 2];
        if (modes_out) modes_out[b] = (long long)cnt;
        if (pk_out) pk_out[b] = cnt > 0 ? h[3 * b] / cnt * norm : 0.0;
        if (k_out) k_out[b] = cnt > 0 ? h[3 * b + 1] / cnt * twopi / L : 0.0;
    }
    return "";
}

}  // namespace ifdm
