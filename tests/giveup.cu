// The ring-fed transforms when one load never completes: bounded waits give up,
// and what was given up is reported.  The loads of one tile are left out (in
// bounds, nothing faults); the spin limit is a compile-time one.
//   giveup -> one line per kernel and error word: name, err word, elements that
//   differ from the run with every load, NaN among them, expected number of NaN
#include "tma.cuh"

#include <cudaTypedefs.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

namespace ifdm {
__device__ unsigned long long g_skip_src;  // source of the row copy that is left out
__device__ int g_skip_c0;                  // first coordinate of the tile copies that are left out, -1: none
__device__ __forceinline__ void lossy_bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    if ((unsigned long long)src != g_skip_src) bulk_load(dst, src, bytes, bar);
}
__device__ __forceinline__ void lossy_2d(void *dst, const CUtensorMap *m, int c0, int c1, uint64_t *bar) {
    if (c0 != g_skip_c0) tma_load_2d(dst, m, c0, c1, bar);
}
__device__ __forceinline__ void lossy_3d(void *dst, const CUtensorMap *m, int c0, int c1, int c2, uint64_t *bar) {
    if (c0 != g_skip_c0) tma_load_3d(dst, m, c0, c1, c2, bar);
}
}  // namespace ifdm
#define bulk_load lossy_bulk_load
#define tma_load_2d lossy_2d
#define tma_load_3d lossy_3d
#include "step_kernels.cuh"
#include "tma_passes.cuh"
#include "zpass_tma.cuh"

using namespace ifdm;

#define TRY(x)                                                                  \
    do {                                                                        \
        auto e_ = (x);                                                          \
        if ((int)e_ != 0) {                                                     \
            std::printf("%s failed: %d\n", #x, (int)e_);                        \
            std::exit(1);                                                       \
        }                                                                       \
    } while (0)

constexpr int N = 256;  // one plane: 256 lines

static CUtensorMap field_map(void *base, bool f64, int axis, int L) {
    static PFN_cuTensorMapEncodeTiled enc = nullptr;
    if (!enc) {
        cudaDriverEntryPointQueryResult q;
        TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", (void **)&enc, cudaEnableDefault, &q));
    }
    const cuuint64_t es = f64 ? 8 : 4;
    CUtensorMap m;
    const cuuint64_t d[3] = {2 * N, N, 1}, st[2] = {2 * N * es, 2 * N * N * es};
    const cuuint32_t b[3] = {cuuint32_t(2 * L), N, 1}, one[3] = {1, 1, 1};
    TRY(enc(&m, f64 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, axis == 1 ? 3 : 2, base, d, st, b, one,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
    return m;
}

// launch(data, ts): the transform along axis 2 (z), 1 (y) or 0 (x) of one plane on 3 blocks.  Tile 4 (block 1's
// second of L lines) is lost; block 1 gives up it and its later tiles.
template <typename R, typename F> static void check(const char *name, int L, int axis, TState *ts, F launch) {
    using G = cx<R>;
    std::vector<G> x(size_t(N) * N), full(x.size()), got(x.size());
    for (size_t i = 0; i < x.size(); ++i) {
        x[i].x = (R)std::sin(0.37 * double(i));
        x[i].y = (R)std::cos(0.73 * double(i));
    }
    G *d = nullptr;
    TRY(cudaMalloc(&d, x.size() * sizeof(G)));
    const unsigned long long none = 0, src = (unsigned long long)(d + size_t(4) * L * N);
    const int off = -1, c0 = 2 * 4 * L;
    for (int word = 0; word < 2; ++word) {
        TRY(cudaMemset(ts, 0, sizeof(TState)));
        for (int lose = 0; lose < 2; ++lose) {
            TRY(cudaMemcpyToSymbol(g_skip_src, lose && axis == 2 ? &src : &none, sizeof(src)));
            TRY(cudaMemcpyToSymbol(g_skip_c0, lose && axis != 2 ? &c0 : &off, sizeof(int)));
            TRY(cudaMemcpy(d, x.data(), x.size() * sizeof(G), cudaMemcpyHostToDevice));
            launch(d, word ? ts : nullptr);
            TRY(cudaDeviceSynchronize());
            TRY(cudaMemcpy((lose ? got : full).data(), d, x.size() * sizeof(G), cudaMemcpyDeviceToHost));
        }
        TState t;
        TRY(cudaMemcpy(&t, ts, sizeof t, cudaMemcpyDeviceToHost));
        size_t differ = 0, nan = 0, lost = 0;
        for (int i = 4; i < N / L; i += 3) lost += size_t(L) * N;  // block 1's tiles from the lost one on
        for (size_t i = 0; i < x.size(); ++i) {
            const bool bad = std::isnan(got[i].x) && std::isnan(got[i].y);
            nan += bad;
            differ += bad || std::memcmp(&got[i], &full[i], sizeof(G)) != 0;
        }
        std::printf("%s %d %d %zu %zu %zu\n", name, word, t.err, differ, nan, lost);
    }
    TRY(cudaFree(d));
}

template <typename Kern> static Kern big(Kern k, size_t smem) {
    TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return k;
}

int main() {
    std::vector<double2> t64(N);
    std::vector<float2> t32(2 * N);
    for (int m = 0; m < N; ++m) {
        const double q = -2 * M_PI * m / N;
        t64[m] = make_double2(std::cos(q), std::sin(q));
        t32[2 * m] = make_float2((float)t64[m].x, (float)t64[m].y);
        t32[2 * m + 1] = make_float2((float)(t64[m].x - t32[2 * m].x), (float)(t64[m].y - t32[2 * m].y));
    }
    double2 *w64 = nullptr;
    float2 *w32 = nullptr;
    TState *ts = nullptr;
    TRY(cudaMalloc(&w64, N * sizeof(double2)));
    TRY(cudaMalloc(&w32, 2 * N * sizeof(float2)));
    TRY(cudaMalloc(&ts, sizeof(TState)));
    TRY(cudaMemcpy(w64, t64.data(), N * sizeof(double2), cudaMemcpyHostToDevice));
    TRY(cudaMemcpy(w32, t32.data(), 2 * N * sizeof(float2), cudaMemcpyHostToDevice));
    {
        using Z = ZT<N, double, double>;
        const size_t sm = 2 * Z::SLOT5 + 64 + tw_bytes<double2>(N);
        auto k = big(k_fft_z_tma<N, 2, 3, double, double, -1>, sm);
        check<double>("z-fp64", Z::L, 2, ts, [&](double2 *d, TState *t) {
            k<<<3, Z::NT, sm>>>(d, w64, t ? &t->err : nullptr, N / Z::L, 0u);
        });
    }
    {
        using Z = ZT<N>;
        const size_t sm = 2 * Z::SLOT5 + 64 + tw_bytes<float2>(N);
        auto k = big(k_fft_z_pair<N, 2, 3, -1>, sm);
        check<float>("z-fp32", Z::L, 2, ts, [&](float2 *d, TState *t) {
            k<<<3, Z::NT / 2, sm>>>(d, w32, t ? &t->err : nullptr, N / Z::L);
        });
    }
    auto plain = [&](auto axis) {
        constexpr int A = decltype(axis)::value;
        using T = TmaTile<double, double, N, A>;
        auto k = big(k_yx_tma<double, double, N, A, 0, -1>, T::SMEM);
        auto kf = big(k_yx_tma<double, double, N, A, 0, -1, true>, T::SMEM);
        check<double>(A == 1 ? "y-fp64" : "x-fp64", T::L, A == 1 ? 1 : 0, ts, [&](double2 *d, TState *t) {
            (t ? k : kf)<<<3, T::NT, T::SMEM>>>(field_map(d, true, A, T::L), d, A == 1 ? N : 1, A == 1 ? N : 1, N / T::L, t, 2, nullptr, w64);
        });
        using P = TmaPair<N, 2, 3>;
        auto kp = big(k_yx_tma_pair<N, A, 0, -1, 2, 3>, P::SMEM);
        auto kpf = big(k_yx_tma_pair<N, A, 0, -1, 2, 3, 8, true>, P::SMEM);
        check<float>(A == 1 ? "y-fp32" : "x-fp32", P::L, A == 1 ? 1 : 0, ts, [&](float2 *d, TState *t) {
            (t ? kp : kpf)<<<3, P::NT, P::SMEM>>>(field_map(d, false, A, P::L), d, A == 1 ? N : 1, A == 1 ? N : 1, N / P::L, t, nullptr, w32);
        });
    };
    plain(std::integral_constant<int, 1>{});
    plain(std::integral_constant<int, 2>{});
    std::printf("done\n");
    return 0;
}
