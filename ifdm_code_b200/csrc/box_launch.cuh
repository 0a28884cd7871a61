// box_launch.cuh -- host-side launchers of the one-launch box kernels of one
// precision (box_kernels.cuh), instantiated in box_fp64.cu, box_fp32.cu and
// box_mixed.cu so they compile in parallel; the engines reach them through
// the BoxKernels function table.
#pragma once

#include "box_kernels.cuh"

#include <string>

namespace ifdm {

constexpr int kBoxLaunchSteps = 512;  // most steps per launch (tens of milliseconds at 128^3)

// `boxes` groups of `group` CTAs each; a group is a cluster or (one box) the
// whole grid of a cooperative launch.
struct BoxLaunch {
    int group = 0, boxes = 1;
    bool cluster = false;
    cudaStream_t stream = nullptr;
};

struct BoxKernels {
    bool (*fits)(int N);  // a plane of an N-box fits a CTA
    // set the kernels' attributes on the current device
    std::string (*setup)(int N, int V);
    // groups of `group` CTAs that are resident at once (a cluster, or a cooperative grid)
    int (*resident)(int N, int group, bool cluster);
    cudaError_t (*run)(int N, int V, const BoxLaunch &l, const BoxRun &one, const BoxRun *many, int nsteps);
    cudaError_t (*load)(int N, const BoxLaunch &l, const BoxRun &one);
    cudaError_t (*sweep)(int N, const BoxLaunch &l, const BoxSweep &one);
};

const BoxKernels &box_kernels(int precision);  // 0 FP64, 1 FP32, 2 mixed

template <typename R, typename K> struct BoxTable {
    template <typename Fn> static bool with_n(int N, Fn &&f) {
        switch (N) {
            case 16: f(BoxOps<R, K, 16, 0>{}); return true;
            case 32: f(BoxOps<R, K, 32, 0>{}); return true;
            case 48: f(BoxOps<R, K, 48, 0>{}); return true;
            case 64: f(BoxOps<R, K, 64, 0>{}); return true;
            case 96: f(BoxOps<R, K, 96, 0>{}); return true;
            case 128:
                if constexpr (box_fits<R, K, 128>()) {
                    f(BoxOps<R, K, 128, 0>{});
                    return true;
                } else {
                    return false;
                }
            default: return false;
        }
    }
    // f(kernel, threads, shared memory) of the run kernel with plan V
    template <typename Fn> static bool with_run(int N, int V, Fn &&f) {
        if (!V) return with_n(N, [&](auto o) { pass_run<0>(o, f); });
        switch (N) {
            case 32: pass_run<1>(BoxOps<R, K, 32, 1>{}, f); return true;
            case 48: pass_run<1>(BoxOps<R, K, 48, 1>{}, f); return true;
            case 64: pass_run<1>(BoxOps<R, K, 64, 1>{}, f); return true;
            case 96: pass_run<1>(BoxOps<R, K, 96, 1>{}, f); return true;
            default: return with_n(N, [&](auto o) { pass_run<0>(o, f); });
        }
    }
    template <int V, typename RR, typename KK, int N, int V2, typename Fn>
    static void pass_run(BoxOps<RR, KK, N, V2>, Fn &&f) {
        using O = BoxOps<RR, KK, N, V2>;
        f(k_box_run<RR, KK, N, V2>, int(O::NT), size_t(O::SMEM));
    }
    template <typename RR, typename KK, int N, int V2, typename Fn> static void pass_load(BoxOps<RR, KK, N, V2>, Fn &&f) {
        using O = BoxOps<RR, KK, N, V2>;
        f(k_box_load<RR, KK, N, V2>, int(O::NT), size_t(O::SMEM));
    }
    template <typename RR, typename KK, int N, int V2, typename Fn> static void pass_sweep(BoxOps<RR, KK, N, V2>, Fn &&f) {
        using O = BoxOps<RR, KK, N, V2>;
        f(k_box_sweep<RR, KK, N, V2>, int(O::NT), size_t(O::SMEM));
    }

    template <typename Kern> static cudaError_t attributes(Kern k, size_t smem) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        // clusters of 16 CTAs
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        return e;
    }
    static void config(const BoxLaunch &l, int nt, size_t smem, cudaLaunchConfig_t *c, cudaLaunchAttribute *at) {
        *c = cudaLaunchConfig_t{};
        c->gridDim = dim3(unsigned(l.group * l.boxes));
        c->blockDim = dim3(unsigned(nt));
        c->dynamicSmemBytes = smem;
        c->stream = l.stream;
        if (l.cluster) {
            at->id = cudaLaunchAttributeClusterDimension;
            at->val.clusterDim.x = unsigned(l.group);
            at->val.clusterDim.y = at->val.clusterDim.z = 1;
        } else {
            at->id = cudaLaunchAttributeCooperative;
            at->val.cooperative = 1;
        }
        c->attrs = at;
        c->numAttrs = 1;
    }

    static bool fits(int N) {
        return with_n(N, [](auto) {});
    }
    static std::string setup(int N, int V) {
        cudaError_t e = cudaErrorInvalidValue;
        with_run(N, V, [&](auto k, int, size_t smem) { e = attributes(k, smem); });
        if (e == cudaSuccess && !V)
            with_n(N, [&](auto o) {
                pass_load(o, [&](auto k, int, size_t smem) { e = attributes(k, smem); });
                if (e == cudaSuccess) pass_sweep(o, [&](auto k, int, size_t smem) { e = attributes(k, smem); });
            });
        return e == cudaSuccess ? "" : std::string("box kernel setup: ") + cudaGetErrorString(e);
    }
    static int resident(int N, int group, bool cluster) {
        int best = 1 << 30;
        auto one = [&](auto k, int nt, size_t smem) {
            int n = 0;
            if (cluster) {
                BoxLaunch l;
                l.group = group;
                l.cluster = true;
                cudaLaunchConfig_t c;
                cudaLaunchAttribute at;
                config(l, nt, smem, &c, &at);
                if (cudaOccupancyMaxActiveClusters(&n, k, &c) != cudaSuccess) n = 0;
            } else {
                int dev = 0, sms = 0, per = 0, coop = 0;
                if (cudaGetDevice(&dev) != cudaSuccess ||
                    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
                    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, nt, smem) != cudaSuccess)
                    per = sms = 0;
                n = per * sms / group;
            }
            if (n < best) best = n;
        };
        cudaGetLastError();
        if (!with_n(N, [&](auto o) {
                pass_run<0>(o, one);
                pass_load(o, one);
                pass_sweep(o, one);
            }))
            return 0;
        cudaGetLastError();
        return best;
    }
    static cudaError_t run(int N, int V, const BoxLaunch &l, const BoxRun &one, const BoxRun *many, int nsteps) {
        cudaError_t e = cudaErrorInvalidValue;
        with_run(N, V, [&](auto k, int nt, size_t smem) {
            cudaLaunchConfig_t c;
            cudaLaunchAttribute at;
            config(l, nt, smem, &c, &at);
            e = cudaLaunchKernelEx(&c, k, one, many, nsteps, l.group, int(l.cluster));
        });
        return e;
    }
    static cudaError_t load(int N, const BoxLaunch &l, const BoxRun &one) {
        cudaError_t e = cudaErrorInvalidValue;
        with_n(N, [&](auto o) {
            pass_load(o, [&](auto k, int nt, size_t smem) {
                cudaLaunchConfig_t c;
                cudaLaunchAttribute at;
                config(l, nt, smem, &c, &at);
                e = cudaLaunchKernelEx(&c, k, one, l.group, int(l.cluster));
            });
        });
        return e;
    }
    static cudaError_t sweep(int N, const BoxLaunch &l, const BoxSweep &one) {
        cudaError_t e = cudaErrorInvalidValue;
        with_n(N, [&](auto o) {
            pass_sweep(o, [&](auto k, int nt, size_t smem) {
                cudaLaunchConfig_t c;
                cudaLaunchAttribute at;
                config(l, nt, smem, &c, &at);
                e = cudaLaunchKernelEx(&c, k, one, l.group, int(l.cluster));
            });
        });
        return e;
    }
    static const BoxKernels &table() {
        static const BoxKernels t{&fits, &setup, &resident, &run, &load, &sweep};
        return t;
    }
};

}  // namespace ifdm
