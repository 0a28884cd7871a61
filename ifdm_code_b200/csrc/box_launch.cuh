// box_launch.cuh -- host-side launchers of the one-launch box kernels of one
// grid size and precision (box_kernels.cuh).  box_size.cu is compiled once for
// each: they compile in parallel, and a process loads the modules of the sizes it
// uses (all sizes of a precision in one module took 13-17 ms at its first box).
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
    // set the kernels' attributes on the current device; V: radix plan of the run kernel
    std::string (*setup)(int V);
    // groups of `group` CTAs that are resident at once (a cluster, or a cooperative grid)
    int (*resident)(int group, bool cluster);
    cudaError_t (*run)(int V, const BoxLaunch &l, const BoxRun &one, const BoxRun *many, int nsteps);
    cudaError_t (*load)(const BoxLaunch &l, const BoxRun &one);
    cudaError_t (*sweep)(const BoxLaunch &l, const BoxSweep &one);
};

// precision 0 FP64, 1 FP32, 2 mixed; null where a plane of an N-box does not fit a CTA
const BoxKernels *box_kernels(int precision, int N);

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
};

template <typename R, typename K, int N> struct BoxSize {
    using O = BoxOps<R, K, N, 0>;
    // another radix plan (V = 1)
    static constexpr bool kTwoPlans = N != 16 && N != 128;

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

    static std::string setup(int V) {
        cudaError_t e = cudaSuccess;
        if constexpr (kTwoPlans) {
            if (V) e = attributes(k_box_run<R, K, N, 1>, BoxOps<R, K, N, 1>::SMEM);
        }
        if (!V || !kTwoPlans) {
            e = attributes(k_box_run<R, K, N, 0>, O::SMEM);
            if (e == cudaSuccess) e = attributes(k_box_load<R, K, N, 0>, O::SMEM);
            if (e == cudaSuccess) e = attributes(k_box_sweep<R, K, N, 0>, O::SMEM);
        }
        return e == cudaSuccess ? "" : std::string("box kernel setup: ") + cudaGetErrorString(e);
    }
    template <typename Kern> static int resident_of(Kern k, int group, bool cluster) {
        int n = 0;
        if (cluster) {
            BoxLaunch l;
            l.group = group;
            l.cluster = true;
            cudaLaunchConfig_t c;
            cudaLaunchAttribute at;
            config(l, O::NT, O::SMEM, &c, &at);
            if (cudaOccupancyMaxActiveClusters(&n, k, &c) != cudaSuccess) n = 0;
        } else {
            int dev = 0, sms = 0, per = 0, coop = 0;
            if (cudaGetDevice(&dev) != cudaSuccess ||
                cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
                cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k, O::NT, O::SMEM) != cudaSuccess)
                per = sms = 0;
            n = per * sms / group;
        }
        return n;
    }
    static int resident(int group, bool cluster) {
        cudaGetLastError();
        const int n[3] = {resident_of(k_box_run<R, K, N, 0>, group, cluster), resident_of(k_box_load<R, K, N, 0>, group, cluster),
                          resident_of(k_box_sweep<R, K, N, 0>, group, cluster)};
        cudaGetLastError();
        return n[0] < n[1] ? (n[0] < n[2] ? n[0] : n[2]) : (n[1] < n[2] ? n[1] : n[2]);
    }
    template <int V> static cudaError_t run_plan(const BoxLaunch &l, const BoxRun &one, const BoxRun *many, int nsteps) {
        using P = BoxOps<R, K, N, V>;
        cudaLaunchConfig_t c;
        cudaLaunchAttribute at;
        config(l, P::NT, P::SMEM, &c, &at);
        return cudaLaunchKernelEx(&c, k_box_run<R, K, N, V>, one, many, nsteps, l.group, int(l.cluster));
    }
    static cudaError_t run(int V, const BoxLaunch &l, const BoxRun &one, const BoxRun *many, int nsteps) {
        if constexpr (kTwoPlans) {
            if (V) return run_plan<1>(l, one, many, nsteps);
        }
        return run_plan<0>(l, one, many, nsteps);
    }
    static cudaError_t load(const BoxLaunch &l, const BoxRun &one) {
        cudaLaunchConfig_t c;
        cudaLaunchAttribute at;
        config(l, O::NT, O::SMEM, &c, &at);
        return cudaLaunchKernelEx(&c, k_box_load<R, K, N, 0>, one, l.group, int(l.cluster));
    }
    static cudaError_t sweep(const BoxLaunch &l, const BoxSweep &one) {
        cudaLaunchConfig_t c;
        cudaLaunchAttribute at;
        config(l, O::NT, O::SMEM, &c, &at);
        return cudaLaunchKernelEx(&c, k_box_sweep<R, K, N, 0>, one, l.group, int(l.cluster));
    }
    static const BoxKernels &table() {
        static const BoxKernels t{&setup, &resident, &run, &load, &sweep};
        return t;
    }
};

}  // namespace ifdm
