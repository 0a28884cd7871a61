// batch_launch.cuh -- host-side launchers of the batch kernels of one precision.
//
// Each precision's kernels are instantiated in their own translation unit
// (batch_fp64.cu, batch_fp32.cu, batch_mixed.cu) so they compile in parallel;
// the engine reaches them through the BatchKernels function table.
#pragma once

#include "batch_kernels.cuh"
#include "box_launch.cuh"

#include <string>

namespace ifdm {

struct BatchKernels {
    // items per phase and dynamic shared memory of an N-box; false if N is not a batch size
    bool (*items)(int N, int *items, size_t *smem);
    // tiled boxes: set the kernels' shared-memory attributes; *fit = persistent CTAs per SM that fit
    std::string (*setup)(int N, size_t smem, int *fit);
    cudaError_t (*persistent)(int N, int grid, size_t smem, cudaStream_t s, const BatchArgs &a);
    cudaError_t (*phase)(int N, int ph, int tiles, int nboxes, size_t smem, cudaStream_t s, const BatchBox *boxes);
    // the per-phase kernels of the boxes whose plane fits a CTA (box_kernels.cuh), radix plan V
    std::string (*box_setup)(int N, int V);
    cudaError_t (*box_phase)(int N, int V, int ph, int nboxes, cudaStream_t s, const BoxRun *boxes);
};
constexpr int kBoxPhases = 6;  // timestep, A .. E

const BatchKernels &batch_kernels(int precision);  // 0 FP64, 1 FP32, 2 mixed

template <typename R, typename K, int N> struct BatchLaunch {
    static std::string setup(size_t smem, int *fit) {
        const int sm = (int)smem;
        cudaError_t e = cudaFuncSetAttribute(k_batch<R, K, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
        const void *ph[kBatchPhases] = {
            (const void *)k_batch_phase<R, K, N, 0>, (const void *)k_batch_phase<R, K, N, 1>,
            (const void *)k_batch_phase<R, K, N, 2>, (const void *)k_batch_phase<R, K, N, 3>,
            (const void *)k_batch_phase<R, K, N, 4>, (const void *)k_batch_phase<R, K, N, 5>,
            (const void *)k_batch_phase<R, K, N, 6>, (const void *)k_batch_phase<R, K, N, 7>,
            (const void *)k_batch_phase<R, K, N, 8>, (const void *)k_batch_phase<R, K, N, 9>};
        for (int p = 0; p < kBatchPhases && e == cudaSuccess; ++p)
            e = cudaFuncSetAttribute(ph[p], cudaFuncAttributeMaxDynamicSharedMemorySize, sm);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(fit, k_batch<R, K, N>, kBatchThreads, smem);
        return e == cudaSuccess ? "" : std::string("batch kernel setup: ") + cudaGetErrorString(e);
    }
    static cudaError_t persistent(int grid, size_t smem, cudaStream_t s, const BatchArgs &a) {
        k_batch<R, K, N><<<grid, kBatchThreads, smem, s>>>(a);
        return cudaGetLastError();
    }
    static cudaError_t phase(int ph, int tiles, int nboxes, size_t smem, cudaStream_t s, const BatchBox *b) {
        const dim3 g((unsigned)tiles, (unsigned)nboxes);
        switch (ph) {
            case 0: k_batch_phase<R, K, N, 0><<<g, kBatchThreads, smem, s>>>(b); break;
            case 1: k_batch_phase<R, K, N, 1><<<g, kBatchThreads, smem, s>>>(b); break;
            case 2: k_batch_phase<R, K, N, 2><<<g, kBatchThreads, smem, s>>>(b); break;
            case 3: k_batch_phase<R, K, N, 3><<<g, kBatchThreads, smem, s>>>(b); break;
            case 4: k_batch_phase<R, K, N, 4><<<g, kBatchThreads, smem, s>>>(b); break;
            case 5: k_batch_phase<R, K, N, 5><<<g, kBatchThreads, smem, s>>>(b); break;
            case 6: k_batch_phase<R, K, N, 6><<<g, kBatchThreads, smem, s>>>(b); break;
            case 7: k_batch_phase<R, K, N, 7><<<g, kBatchThreads, smem, s>>>(b); break;
            case 8: k_batch_phase<R, K, N, 8><<<g, kBatchThreads, smem, s>>>(b); break;
            case 9: k_batch_phase<R, K, N, 9><<<g, kBatchThreads, smem, s>>>(b); break;
            default: return cudaErrorInvalidValue;
        }
        return cudaGetLastError();
    }
};

// Sizes whose plane does not fit a CTA (128 in FP64 arithmetic) run the tiles of the ten passes.
template <typename R, typename K, typename F> static bool with_tiled(int N, F &&f) {
    if constexpr (!box_fits<R, K, 128>()) {
        if (N == 128) {
            f(BatchLaunch<R, K, 128>{});
            return true;
        }
    }
    return false;
}
// f(BoxOps) of an (N, V) box that fits
template <typename R, typename K, typename F> static bool with_box_nv(int N, int V, F &&f) {
    if (V) {
        switch (N) {
            case 32: f(BoxOps<R, K, 32, 1>{}); return true;
            case 48: f(BoxOps<R, K, 48, 1>{}); return true;
            case 64: f(BoxOps<R, K, 64, 1>{}); return true;
            case 96: f(BoxOps<R, K, 96, 1>{}); return true;
            default: break;
        }
    }
    return BoxTable<R, K>::with_n(N, f);
}

template <typename R, typename K> struct BatchTable {
    static bool items(int N, int *it, size_t *smem) {
        for (int p = 0; p < kBatchPhases; ++p) it[p] = 0;
        *smem = 0;
        if (with_box_nv<R, K>(N, 0, [](auto) {})) {
            for (int p = 0; p < kBoxPhases; ++p) it[p] = p ? N : 1;
            return true;
        }
        return with_tiled<R, K>(N, [&](auto l) {
            for (int p = 0; p < kBatchPhases; ++p) it[p] = batch_items<R, K, 128>(p);
            *smem = batch_smem<R, K, 128>();
        });
    }
    template <typename RR, typename KK, int N, int V> static std::string set_phases(BoxOps<RR, KK, N, V>) {
        using O = BoxOps<RR, KK, N, V>;
        const void *ph[kBoxPhases] = {(const void *)k_box_phase<RR, KK, N, V, 0>, (const void *)k_box_phase<RR, KK, N, V, 1>,
                                      (const void *)k_box_phase<RR, KK, N, V, 2>, (const void *)k_box_phase<RR, KK, N, V, 3>,
                                      (const void *)k_box_phase<RR, KK, N, V, 4>, (const void *)k_box_phase<RR, KK, N, V, 5>};
        for (const void *f : ph) {
            cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)O::SMEM);
            if (e != cudaSuccess) return std::string("batch kernel setup: ") + cudaGetErrorString(e);
        }
        return "";
    }
    static std::string box_setup(int N, int V) {
        std::string e = "batch: res " + std::to_string(N) + " has no plane kernels";
        with_box_nv<R, K>(N, V, [&](auto o) { e = set_phases(o); });
        return e;
    }
    template <typename RR, typename KK, int N, int V>
    static cudaError_t one_phase(BoxOps<RR, KK, N, V>, int ph, int nb, cudaStream_t s, const BoxRun *b) {
        using O = BoxOps<RR, KK, N, V>;
        const dim3 g(ph ? unsigned(N) : 1u, unsigned(nb));
        switch (ph) {
            case 0: k_box_phase<RR, KK, N, V, 0><<<g, O::NT, O::SMEM, s>>>(b); break;
            case 1: k_box_phase<RR, KK, N, V, 1><<<g, O::NT, O::SMEM, s>>>(b); break;
            case 2: k_box_phase<RR, KK, N, V, 2><<<g, O::NT, O::SMEM, s>>>(b); break;
            case 3: k_box_phase<RR, KK, N, V, 3><<<g, O::NT, O::SMEM, s>>>(b); break;
            case 4: k_box_phase<RR, KK, N, V, 4><<<g, O::NT, O::SMEM, s>>>(b); break;
            case 5: k_box_phase<RR, KK, N, V, 5><<<g, O::NT, O::SMEM, s>>>(b); break;
            default: return cudaErrorInvalidValue;
        }
        return cudaGetLastError();
    }
    static cudaError_t box_phase(int N, int V, int ph, int nb, cudaStream_t s, const BoxRun *b) {
        cudaError_t e = cudaErrorInvalidValue;
        with_box_nv<R, K>(N, V, [&](auto o) { e = one_phase(o, ph, nb, s, b); });
        return e;
    }
    static std::string setup(int N, size_t smem, int *fit) {
        std::string e = "batch: res " + std::to_string(N) + " is not a batch size";
        with_tiled<R, K>(N, [&](auto L) { e = decltype(L)::setup(smem, fit); });
        return e;
    }
    static cudaError_t persistent(int N, int grid, size_t smem, cudaStream_t s, const BatchArgs &a) {
        cudaError_t e = cudaErrorInvalidValue;
        with_tiled<R, K>(N, [&](auto L) { e = decltype(L)::persistent(grid, smem, s, a); });
        return e;
    }
    static cudaError_t phase(int N, int ph, int tiles, int nboxes, size_t smem, cudaStream_t s,
                             const BatchBox *b) {
        cudaError_t e = cudaErrorInvalidValue;
        with_tiled<R, K>(N, [&](auto L) { e = decltype(L)::phase(ph, tiles, nboxes, smem, s, b); });
        return e;
    }
    static const BatchKernels &table() {
        static const BatchKernels t{&items, &setup, &persistent, &phase, &box_setup, &box_phase};
        return t;
    }
};

}  // namespace ifdm
