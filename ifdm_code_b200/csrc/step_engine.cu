// step_engine.cu -- buffers, twiddle tables and launch sequence of the fused
// leap-frog step (kernels in step_kernels.cuh / timestep.cuh).
#include "physics.hpp"
#include "step_engine.hpp"
#include "timestep.cuh"
#include "tma_passes.cuh"
#include "zpass_pipe.cuh"
#include "zpass_tma.cuh"
#include "adjoint_kernels.cuh"
#include "box_launch.cuh"

#include <cudaTypedefs.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <algorithm>
#include <array>
#include <map>
#include <mutex>
#include <set>

namespace ifdm {

// guards this file's process-wide caches (kernel attributes per device, the
// twiddle tables, the tensor-map encoder): contexts may be driven from
// several host threads at once (the batched adjoint does)
static std::mutex &setup_mutex() {
    static std::mutex m;
    return m;
}

const char *const kPassNames[kNumPasses] = {
    "T_timestep", "P1_kick_fft_z", "P2_fft_y", "P3_fft_x_drift_ifft_x", "P4_ifft_y",
    "P5_ifft_z_density_r2c_z", "P6_fft_y_half", "P7_fft_x_poisson_ifft_x", "P8_ifft_y_half", "P9_c2r_z_phi"};

#define CUDA_TRY(expr)                                                                   \
    do {                                                                                 \
        cudaError_t e_ = (expr);                                                         \
        if (e_ != cudaSuccess) return std::string(#expr) + ": " + cudaGetErrorString(e_); \
    } while (0)

bool supported_n(int n) {
    switch (n) {
        case 16: case 32: case 48: case 64: case 96: case 128: case 256: case 512: case 1024: return true;
        default: return false;
    }
}

bool supported_n(int n, int precision) {
    if (precision == 2 && n >= 1024) return false;  // mixed: FP64 exchange tiles exceed shared memory
    return supported_n(n);
}

// map of one axis pass over a caller's field: axis 1 [planes][N][N], axis 0 [N][planes][N]; L lines a tile
static std::string make_field_map(CUtensorMap *m, void *base, bool f64, int N, int planes, int axis, int L);
static std::string make_axis_maps(CUtensorMap *my, CUtensorMap *mx, void *base, bool f64, int N, int W, int Ly,
                                  int Lx, int boxr);

// ---------------------------------------------------------------- per-N ops --
template <typename R_, typename K_, int N> struct Box {
    using R = R_;
    using K = K_;
    using TL = Tile<R, K, N>;   // y/x passes (strided lines)
    using TZ = TileZ<R, K, N>;  // z passes (contiguous rows)
    using C = cx<K>;
    using G = cx<R>;
    static constexpr int NH = N / 2 + 1;
    static constexpr int NHP = half_pitch<R>(N);
    static constexpr size_t SM = TL::SMEM;
    static constexpr size_t SMZ = TZ::SMEM;
    static constexpr size_t SMZ9 = TZ::SMEM9;
    // every launch covers its array exactly: no partial tiles
    static_assert((N * N) % TL::L == 0 && (N * N) % TZ::L == 0, "z/y/x tiles must divide N^2 lines");
    static_assert((N * NHP) % TL::L == 0, "half-spectrum tiles must divide N*NHP lines");
    static_assert(NHP >= NH, "half-spectrum pitch");
    static_assert(TL::NT <= 1024 && TZ::NT <= 1024, "block size");
    static_assert(SM <= 227 * 1024 && SMZ9 <= 227 * 1024, "shared memory per block");

    template <typename Kern> static cudaError_t prep(Kern kern, size_t smem) {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }

    static std::string configure() {
        // once per device (kernel attributes are per device), under the lock
        // that guards every process-wide cache of this file
        std::lock_guard<std::mutex> lk(setup_mutex());
        static std::set<int> done_on;
        int dev = 0;
        CUDA_TRY(cudaGetDevice(&dev));
        if (done_on.count(dev)) return "";
        CUDA_TRY(prep(k_kick_fft_z<R, K, N>, SMZ));
        CUDA_TRY(prep(k_fft_yx<R, K, N, -1, 1>, SM));
        CUDA_TRY(prep(k_fft_yx<R, K, N, +1, 1>, SM));
        CUDA_TRY(prep(k_fft_yx<R, K, N, -1, 2>, SM));
        CUDA_TRY(prep(k_fft_yx<R, K, N, +1, 2>, SM));
        CUDA_TRY(prep(k_fft_x_drift<R, K, N>, SM));
        CUDA_TRY(prep(k_density_r2c_z<R, K, N, true>, SMZ));
        CUDA_TRY(prep(k_density_r2c_z<R, K, N, false>, SMZ));
        CUDA_TRY(prep(k_fft_x_poisson<R, K, N>, SM));
        CUDA_TRY(prep(k_c2r_z_phi<R, K, N>, SMZ9));
        CUDA_TRY(prep(k_fft_z<R, K, N, -1>, SMZ));
        CUDA_TRY(prep(k_fft_z<R, K, N, +1>, SMZ));
        CUDA_TRY(prep(k_source_r2c_z<R, K, N>, SMZ));
        CUDA_TRY(prep(k_fft_x_poisson_slab<R, K, N>, SM));
        if constexpr (std::is_same<R, double>::value && N < 256) {
            CUDA_TRY(prep(k_line_k2<N, 1>, SM));
            CUDA_TRY(prep(k_line_k2<N, 2>, SM));
        }
        int sms = 0;
        CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        if constexpr (kZPipe) {
            using ZP = ZPipe<R, N>;
            CUDA_TRY(prep(k_density_r2c_z_pipe<R, N>, ZP::SMEM5));
            int b5 = 0;
            CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b5, k_density_r2c_z_pipe<R, N>, ZP::NT, ZP::SMEM5));
            zgrid = sms * (b5 > 0 ? b5 : 1);
        }
        if constexpr (kZT) {
            using Z = ZT<N, R, K>;
            CUDA_TRY(prep(k_kick_fft_z_tma<N, ZST1, ZB1, R, K>, ZSM1));
            CUDA_TRY(prep(k_density_r2c_z_tma<N, ZST5, ZB5, R, K>, ZSM5));
            CUDA_TRY(prep(k_c2r_z_tma<N, ZST9, ZB9, R, K>, ZSM9));
            int b1 = 0, b5 = 0, b9 = 0;
            CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1, k_kick_fft_z_tma<N, ZST1, ZB1, R, K>, Z::NT, ZSM1));
            CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b5, k_density_r2c_z_tma<N, ZST5, ZB5, R, K>, Z::NT, ZSM5));
            CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b9, k_c2r_z_tma<N, ZST9, ZB9, R, K>, Z::NT, ZSM9));
            zt1grid = sms * (b1 > 0 ? b1 : 1);
            zt5grid = sms * (b5 > 0 ? b5 : 1);
            zt9grid = sms * (b9 > 0 ? b9 : 1);
            if constexpr (!kPairZ) {
                CUDA_TRY(prep(k_fft_z_tma<N, ZST5, ZB5, R, K, -1>, ZSM5));
                CUDA_TRY(prep(k_fft_z_tma<N, ZST5, ZB5, R, K, +1>, ZSM5));
            } else {
                CUDA_TRY(prep(k_fft_z_pair<N, ZST5P, ZB5P, -1>, ZSM5P));
                CUDA_TRY(prep(k_fft_z_pair<N, ZST5P, ZB5P, +1>, ZSM5P));
                CUDA_TRY(prep(k_kick_fft_z_pair<N, ZST1P, ZB1P>, ZSM1P));
                CUDA_TRY(prep(k_density_r2c_z_pair<N, ZST5P, ZB5P>, ZSM5P));
                CUDA_TRY(prep(k_c2r_z_pair<N, ZST9P, ZB9P>, ZSM9P));
                int b1p = 0, b5p = 0, b9p = 0;
                CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b1p, k_kick_fft_z_pair<N, ZST1P, ZB1P>,
                                                                       Z::NT / 2, ZSM1P));
                CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b5p, k_density_r2c_z_pair<N, ZST5P, ZB5P>,
                                                                       Z::NT / 2, ZSM5P));
                CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b9p, k_c2r_z_pair<N, ZST9P, ZB9P>,
                                                                       Z::NT / 2, ZSM9P));
                zt1pgrid = sms * (b1p > 0 ? b1p : 1);
                zt5pgrid = sms * (b5p > 0 ? b5p : 1);
                zt9pgrid = sms * (b9p > 0 ? b9p : 1);
            }
        }
        if constexpr (kTma) {
            CUDA_TRY(prep(k_yx_tma<R, K, N, 1, 0, -1>, TT::SMEM));
            CUDA_TRY(prep(k_yx_tma<R, K, N, 1, 0, +1>, TT::SMEM));
            CUDA_TRY(prep(k_yx_tma<R, K, N, 2, 1, 0>, TX::SMEM));
            CUDA_TRY(prep(k_yx_tma<R, K, N, 2, 2, 0>, TX::SMEM));
            if constexpr (kFftTma && !kPair) {  // the callers' fields (axis_pass)
                CUDA_TRY(prep(k_yx_tma<R, K, N, 1, 0, -1, true>, TT::SMEM));
                CUDA_TRY(prep(k_yx_tma<R, K, N, 1, 0, +1, true>, TT::SMEM));
                CUDA_TRY(prep(k_yx_tma<R, K, N, 2, 0, -1, true>, TX::SMEM));
                CUDA_TRY(prep(k_yx_tma<R, K, N, 2, 0, +1, true>, TX::SMEM));
            }
            if constexpr (kFftTma && std::is_same<R, double>::value) {  // the diagnostics
                CUDA_TRY(prep(k_yx_tma<R, K, N, 2, 0, -1>, TX::SMEM));
                CUDA_TRY(prep(k_line_k2_tma<N, 1>, TT::SMEM));
                CUDA_TRY(prep(k_line_k2_tma<N, 2>, TX::SMEM));
            }
            // persistent grids: every block resident at once (one wave)
            int by = 0, bx = 0;
            CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&by, k_yx_tma<R, K, N, 1, 0, -1>, TT::NT, TT::SMEM));
            CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bx, k_yx_tma<R, K, N, 2, 1, 0>, TX::NT, TX::SMEM));
            ygrid = sms * (by > 0 ? by : 1);
            xgrid = sms * (bx > 0 ? bx : 1);
            if constexpr (kPair) {
                CUDA_TRY(prep(k_yx_tma_pair<N, 1, 0, -1, PSTY, PBY>, TPY::SMEM));
                CUDA_TRY(prep(k_yx_tma_pair<N, 1, 0, +1, PSTY, PBY>, TPY::SMEM));
                CUDA_TRY(prep(k_yx_tma_pair<N, 2, 1, 0, PSTX, PBX>, TPX::SMEM));
                CUDA_TRY(prep(k_yx_tma_pair<N, 2, 2, 0, PSTX, PBX>, TPX::SMEM));
                CUDA_TRY(prep(k_yx_tma_pair<N, 1, 0, -1, PSTY, PBY, 8, true>, TPY::SMEM));
                CUDA_TRY(prep(k_yx_tma_pair<N, 1, 0, +1, PSTY, PBY, 8, true>, TPY::SMEM));
                CUDA_TRY(prep(k_yx_tma_pair<N, 2, 0, -1, PSTX, PBF, PLF, true>, TPF::SMEM));
                CUDA_TRY(prep(k_yx_tma_pair<N, 2, 0, +1, PSTX, PBF, PLF, true>, TPF::SMEM));
                int pf = 0;
                CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&pf, k_yx_tma_pair<N, 2, 0, -1, PSTX, PBF, PLF, true>,
                                                                       TPF::NT, TPF::SMEM));
                pfgrid = sms * (pf > 0 ? pf : 1);
                int py = 0, px = 0;
                CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&py, k_yx_tma_pair<N, 1, 0, -1, PSTY, PBY>,
                                                                       TPY::NT, TPY::SMEM));
                CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&px, k_yx_tma_pair<N, 2, 1, 0, PSTX, PBX>,
                                                                       TPX::NT, TPX::SMEM));
                pygrid = sms * (py > 0 ? py : 1);
                pxgrid = sms * (px > 0 ? px : 1);
            }
        }
        done_on.insert(dev);
        return "";
    }

    // TMA-pipelined y/x passes for N >= 128.  The cp.async-pipelined P5 is
    // used in FP32 only: measured at 512^3 it cut FP32 P5 from 1.42 to 1.02 ms
    // but slowed the FP64 z passes (one 2-slot block per SM hides less latency
    // than three plain blocks), and pipelined P1/P9 gained nothing.
    static constexpr bool kTma = N >= 128;
    static constexpr bool kFftTma = N >= 256;  // the callers' own fields (axis_pass)
    static constexpr bool kZPipe = N >= 128 && N <= 512 && std::is_same<R, float>::value && std::is_same<K, float>::value;
    // z passes fed by bulk copies (zpass_tma.cuh) for N >= 256 and, in FP64
    // arithmetic, 128 (8 FP32 or 4 FP64 rows per tile; FP32 at 128 runs the
    // box kernels); ring depth and resident blocks per SM of P1, P5 and P9.
    // D3: one slot (two in P5) and three blocks at 512, six at 256, twelve at
    // 128: the blocks hide each other's loads (FP64 512^3 step 7.45 -> 7.35 ms
    // against two or three slots at two blocks; 256^3 873 -> 862 us)
    static constexpr bool kZT = (N >= 256 && (std::is_same<R, K>::value || N <= 512)) || (N == 128 && sizeof(K) == 8);
    static constexpr bool D3 = sizeof(C) == 16 && N >= 128 && N <= 512;
    static constexpr int ZST1 = D3 ? 1 : 2, ZST5 = D3 ? 2 : 3, ZST9 = D3 ? 1 : 3;
    static constexpr int ZB1 = N >= 1024 ? 1 : (D3 ? 3 * 512 / N : 2), ZB5 = ZB1, ZB9 = ZB1;
    using ZG = ZT<(kZT ? N : 256), R, K>;
    // ring slots, the mbarriers (64 bytes) and the staged twiddle table
    static constexpr size_t ZSM1 = kZT ? ZST1 * ZG::SLOT1 + 64 + ZG::WORK + tw_bytes<C>(N) : 0;
    static constexpr size_t ZSM5 = kZT ? ZST5 * ZG::SLOT5 + 64 + ZG::WORK + tw_bytes<C>(N) : 0;
    static constexpr size_t ZSM9 = kZT ? ZST9 * ZG::SLOT9 + 64 + ZG::WORK + tw_bytes<C>(N) : 0;
    static inline int zt1grid = 0, zt5grid = 0, zt9grid = 0;  // persistent grids of the bulk-copy z passes
    // the paired z passes (two rows per thread, 256 threads at 512, 512 at
    // 1024; kPairZ below): ring slots, resident blocks per SM, shared memory
    // and persistent grids (at 512, P1 and P9 with one slot at three blocks
    // per SM measured 0.641 -> 0.593 ms and 0.273 -> 0.244 ms against two or
    // three slots at two blocks: the blocks overlap each other's loads; the y
    // passes at one slot and four blocks measured slower, 0.392 -> 0.43 ms;
    // at 1024 the slots leave room for one block)
    static constexpr int ZB = N >= 1024 ? 1 : (N == 256 ? 6 : 3);
    static constexpr int ZST1P = 1, ZB1P = ZB, ZST5P = 2, ZB5P = ZB, ZST9P = 1, ZB9P = ZB;
    static constexpr size_t ZSM1P = kZT ? ZST1P * ZG::SLOT1 + 64 + tw_bytes<C>(N) : 0;
    static constexpr size_t ZSM5P = kZT ? ZST5P * ZG::SLOT5 + 64 + tw_bytes<C>(N) : 0;
    static constexpr size_t ZSM9P = kZT ? ZST9P * ZG::SLOT9 + 64 + tw_bytes<C>(N) : 0;
    static inline int zt1pgrid = 0, zt5pgrid = 0, zt9pgrid = 0;
    using TT = TmaTile<R, K, N, 1>;
    using TX = TmaTile<R, K, N, 2>;
    // FP32 passes at N = 512 with two lines per thread: the y/x passes
    // (k_yx_tma_pair, the same tiles and maps as TT/TX; ring slots and resident
    // blocks per SM of the y and x passes below) and the z passes
    // (k_*_z_pair, ZST*P/ZB*P above).  IFDM_NO_PAIR selects the one-line kernels.
    // (512 and 1024; at 1024 a tile takes 512 threads, one block per SM:
    // measured at 1024^3, step 57.5 -> 44.6 ms, P3 14.8 -> 8.4 ms, P5 9.0 ->
    // 6.7 ms)
    static constexpr bool kPair = N >= 256 && std::is_same<R, float>::value && std::is_same<K, float>::value;
    static constexpr bool kPairZ = kPair;  // the z passes
    static constexpr int PSTY = 2, PBY = N >= 1024 ? 1 : (N == 256 ? 5 : 3), PSTX = 2, PBX = PBY;
    using TPY = TmaPair<(kPair ? N : 512), PSTY, PBY>;
    using TPX = TmaPair<(kPair ? N : 512), PSTX, PBX>;
    // one x transform of a caller's field at 512: 16 lines, 128-byte rows, one
    // block an SM (512^3 complex64 x pass: 8 lines at three blocks 563 us, 404
    // so; the two-transform passes are bound by their arithmetic and lost,
    // 752 -> 819 us with the drift)
    static constexpr int PLF = N == 512 ? 16 : 8, PBF = N == 512 ? 1 : PBX;
    using TPF = TmaPair<(kPair ? N : 512), PSTX, PBF, PLF>;
    static_assert(!kPair || (TT::L == TPY::L && TX::L == TPX::L), "pair kernels share the tensor maps");
    static inline int pygrid = 0, pxgrid = 0, pfgrid = 0;
    static inline int zgrid = 0;             // persistent grid of the pipelined P5
    static inline int ygrid = 0, xgrid = 0;  // persistent grids of the TMA y and x passes

    // lines per TMA tile of the y and x passes (the inner box extent of their maps)
    static void tma_lines(int &ly, int &lx) {
        ly = TT::L;
        lx = TX::L;
    }

    static unsigned zblocks() { return unsigned(size_t(N) * N / TL::L); }  // y-pass tiles
    static unsigned zrows() { return unsigned(size_t(N) * N / TZ::L); }    // z-pass tiles
    static unsigned hblocks() { return unsigned(size_t(N) * NHP / TL::L); }

    // one pass by index 1..9; tm: TMA maps (psi y, psi x, rho y, rho x) or null
    static void pass(int p, cudaStream_t s, G *psi, R *phi, G *rhok, TState *ts, const C *drift, const C *tw,
                     const C *twh, long wr, int wt, const CUtensorMap *tm = nullptr) {
        const unsigned nt = TL::NT;
        if constexpr (kZT) {
            if (tm && (p == 1 || p == 5 || p == 9)) {
                using Z = ZT<N, R, K>;
                const int nz = int(size_t(N) * N / Z::L);
                if constexpr (kPairZ) {
                    if (std::getenv("IFDM_NO_PAIR") == nullptr) {
                        const unsigned q = Z::NT / 2;
                        if (p == 1)
                            k_kick_fft_z_pair<N, ZST1P, ZB1P><<<zt1pgrid, q, ZSM1P, s>>>(psi, phi, ts, tw, nz);
                        else if (p == 5)
                            k_density_r2c_z_pair<N, ZST5P, ZB5P><<<zt5pgrid, q, ZSM5P, s>>>(psi, rhok, ts, tw, nz);
                        else
                            k_c2r_z_pair<N, ZST9P, ZB9P><<<zt9pgrid, q, ZSM9P, s>>>(rhok, phi, ts, wr, wt, tw, nz / 2);
                        return;
                    }
                }
                if (p == 1)
                    k_kick_fft_z_tma<N, ZST1, ZB1, R, K><<<zt1grid, Z::NT, ZSM1, s>>>(psi, phi, ts, tw, nz);
                else if (p == 5)
                    k_density_r2c_z_tma<N, ZST5, ZB5, R, K><<<zt5grid, Z::NT, ZSM5, s>>>(psi, rhok, ts, tw, nz);
                else
                    k_c2r_z_tma<N, ZST9, ZB9, R, K><<<zt9grid, Z::NT, ZSM9, s>>>(rhok, phi, ts, wr, wt, tw, nz / 2);
                return;
            }
        }
        if constexpr (kZPipe) {
            if (tm && p == 5 && std::getenv("IFDM_NO_ZPIPE") == nullptr) {
                using ZP = ZPipe<R, N>;
                const int nz = int(size_t(N) * N / ZP::L);
                k_density_r2c_z_pipe<R, N><<<zgrid, ZP::NT, ZP::SMEM5, s>>>(psi, rhok, ts, tw, twh, nz);
                return;
            }
        }
        if constexpr (kTma) {
            if (tm && (p == 2 || p == 3 || p == 4 || p == 6 || p == 7 || p == 8)) {
                // y tiles (TT) and x tiles (TX) may differ in lines per tile
                const int tcy = int(size_t(N) * N / TT::L), thy = int(size_t(N) * NHP / TT::L);
                const int tcx = int(size_t(N) * N / TX::L), thx = int(size_t(N) * NHP / TX::L);
                const unsigned gy = unsigned(ygrid), gx = unsigned(xgrid), ny = TT::NT, nx = TX::NT;
                const size_t sy = TT::SMEM, sx = TX::SMEM;
                if constexpr (kPair) {
                    if (std::getenv("IFDM_NO_PAIR") == nullptr) {
                        const unsigned py = unsigned(pygrid), px = unsigned(pxgrid), qy = TPY::NT, qx = TPX::NT;
                        const size_t my = TPY::SMEM, mx = TPX::SMEM;
                        switch (p) {
                            case 2: k_yx_tma_pair<N, 1, 0, -1, PSTY, PBY><<<py, qy, my, s>>>(tm[0], psi, N, N, tcy, ts, drift, tw); break;
                            case 3: k_yx_tma_pair<N, 2, 1, 0, PSTX, PBX><<<px, qx, mx, s>>>(tm[1], psi, N, N, tcx, ts, drift, tw); break;
                            case 4: k_yx_tma_pair<N, 1, 0, +1, PSTY, PBY><<<py, qy, my, s>>>(tm[0], psi, N, N, tcy, ts, drift, tw); break;
                            case 6: k_yx_tma_pair<N, 1, 0, -1, PSTY, PBY><<<py, qy, my, s>>>(tm[2], rhok, NHP, NH, thy, ts, drift, tw); break;
                            case 7: k_yx_tma_pair<N, 2, 2, 0, PSTX, PBX><<<px, qx, mx, s>>>(tm[3], rhok, NHP, NH, thx, ts, drift, tw); break;
                            case 8: k_yx_tma_pair<N, 1, 0, +1, PSTY, PBY><<<py, qy, my, s>>>(tm[2], rhok, NHP, NH, thy, ts, drift, tw); break;
                        }
                        return;
                    }
                }
                switch (p) {
                    case 2: k_yx_tma<R, K, N, 1, 0, -1><<<gy, ny, sy, s>>>(tm[0], psi, N, N, tcy, ts, 2, drift, tw); break;
                    case 3: k_yx_tma<R, K, N, 2, 1, 0><<<gx, nx, sx, s>>>(tm[1], psi, N, N, tcx, ts, 3, drift, tw); break;
                    case 4: k_yx_tma<R, K, N, 1, 0, +1><<<gy, ny, sy, s>>>(tm[0], psi, N, N, tcy, ts, 4, drift, tw); break;
                    case 6: k_yx_tma<R, K, N, 1, 0, -1><<<gy, ny, sy, s>>>(tm[2], rhok, NHP, NH, thy, ts, 6, drift, tw); break;
                    case 7: k_yx_tma<R, K, N, 2, 2, 0><<<gx, nx, sx, s>>>(tm[3], rhok, NHP, NH, thx, ts, 7, drift, tw); break;
                    case 8: k_yx_tma<R, K, N, 1, 0, +1><<<gy, ny, sy, s>>>(tm[2], rhok, NHP, NH, thy, ts, 8, drift, tw); break;
                }
                return;
            }
        }
        switch (p) {
            case 1: k_kick_fft_z<R, K, N><<<zrows(), TZ::NT, SMZ, s>>>(psi, phi, ts, tw); break;
            case 2: k_fft_yx<R, K, N, -1, 1><<<zblocks(), nt, SM, s>>>(psi, N, N, ts, 2, tw); break;
            case 3: k_fft_x_drift<R, K, N><<<zblocks(), nt, SM, s>>>(psi, drift, ts, tw); break;
            case 4: k_fft_yx<R, K, N, +1, 1><<<zblocks(), nt, SM, s>>>(psi, N, N, ts, 4, tw); break;
            case 5:
                k_density_r2c_z<R, K, N, true><<<zrows(), TZ::NT, SMZ, s>>>(psi, rhok, ts, nullptr, tw, twh);
                break;
            case 6: k_fft_yx<R, K, N, -1, 1><<<hblocks(), nt, SM, s>>>(rhok, NHP, NH, ts, 6, tw); break;
            case 7: k_fft_x_poisson<R, K, N><<<hblocks(), nt, SM, s>>>(rhok, ts, tw); break;
            case 8: k_fft_yx<R, K, N, +1, 1><<<hblocks(), nt, SM, s>>>(rhok, NHP, NH, ts, 8, tw); break;
            case 9: k_c2r_z_phi<R, K, N><<<zrows(), TZ::NT, SMZ9, s>>>(rhok, phi, ts, wr, wt, tw, twh); break;
            default: break;
        }
    }

    static void initial_density(cudaStream_t s, G *psi, G *rhok, TState *ts, double *part, const C *tw,
                                const C *twh) {
        k_density_r2c_z<R, K, N, false><<<zrows(), TZ::NT, SMZ, s>>>(psi, rhok, ts, part, tw, twh);
        k_reduce_init<<<1, 256, 0, s>>>(ts, part, (int)zrows(), double(N) * N * N);
    }

    // One transform along z of `rows` rows: the ring-fed kernels where the base
    // is 16-byte aligned (bulk copies), else the plain one.
    static void z_pass(cudaStream_t s, G *data, size_t rows, int sign, const C *tw, uint32_t salt, bool ring, int *err) {
        if constexpr (kZT) {
            if (ring) {
                using Z = ZT<N, R, K>;
                const int nz = int(rows / Z::L);
                if constexpr (kPairZ) {
                    if (sign < 0) k_fft_z_pair<N, ZST5P, ZB5P, -1><<<zt5pgrid, Z::NT / 2, ZSM5P, s>>>(data, tw, err, nz);
                    else k_fft_z_pair<N, ZST5P, ZB5P, +1><<<zt5pgrid, Z::NT / 2, ZSM5P, s>>>(data, tw, err, nz);
                } else {
                    if (sign < 0) k_fft_z_tma<N, ZST5, ZB5, R, K, -1><<<zt5grid, Z::NT, ZSM5, s>>>(data, tw, err, nz, salt);
                    else k_fft_z_tma<N, ZST5, ZB5, R, K, +1><<<zt5grid, Z::NT, ZSM5, s>>>(data, tw, err, nz, salt);
                }
                return;
            }
        }
        const unsigned gz = unsigned(rows / TZ::L);
        if (sign < 0) k_fft_z<R, K, N, -1><<<gz, TZ::NT, SMZ, s>>>(data, tw, salt);
        else k_fft_z<R, K, N, +1><<<gz, TZ::NT, SMZ, s>>>(data, tw, salt);
    }

    // g <- U^H g: forward FFT, drift with the conjugate tables, inverse FFT
    static void adj_drift(cudaStream_t s, G *g, TState *ts_adj, const C *drift_conj, const C *tw,
                          const CUtensorMap *tm, uint32_t salt) {
        z_pass(s, g, size_t(N) * N, -1, tw, salt, tm != nullptr, &ts_adj->err);
        pass(2, s, g, nullptr, nullptr, ts_adj, drift_conj, tw, nullptr, 0, 0, tm);
        pass(3, s, g, nullptr, nullptr, ts_adj, drift_conj, tw, nullptr, 0, 0, tm);
        pass(4, s, g, nullptr, nullptr, ts_adj, drift_conj, tw, nullptr, 0, 0, tm);
        z_pass(s, g, size_t(N) * N, +1, tw, salt ^ 0x68e31da4u, tm != nullptr, &ts_adj->err);
    }
    // pw = phi_s[w]: real source -> half spectrum -> -1/kappa^2 -> real
    static void poisson_of(cudaStream_t s, const R *w, R *pw, G *rhok, TState *ts_adj, const C *tw, const C *twh,
                           const CUtensorMap *tm) {
        k_source_r2c_z<R, K, N><<<zrows(), TZ::NT, SMZ, s>>>(w, rhok, ts_adj, tw, twh);
        for (int p = 6; p <= 9; ++p) pass(p, s, nullptr, pw, rhok, ts_adj, nullptr, tw, twh, 0, 0, tm);
    }

    // Forward pass along axis 1 (y) or 0 (x) of a half spectrum [N][N][NHP]
    // (diagnostics; FP64); a wait that gives up sets ts->err
    static std::string half_axis(G *data, int axis, const C *tw, TState *ts, cudaStream_t s) {
        if constexpr (kFftTma && std::is_same<R, double>::value) {
            CUtensorMap my, mx;
            std::string e = make_axis_maps(&my, &mx, data, true, N, NHP, TT::L, TX::L, N < 256 ? N : 256);
            if (!e.empty()) return e;
            if (axis == 1)
                k_yx_tma<R, K, N, 1, 0, -1><<<ygrid, TT::NT, TT::SMEM, s>>>(my, data, NHP, NH, int(size_t(N) * NHP / TT::L), ts, 6, nullptr, tw);
            else
                k_yx_tma<R, K, N, 2, 0, -1><<<xgrid, TX::NT, TX::SMEM, s>>>(mx, data, NHP, NH, int(size_t(N) * NHP / TX::L), ts, 7, nullptr, tw);
        } else if (axis == 1) {
            k_fft_yx<R, K, N, -1, 1><<<hblocks(), TL::NT, SM, s>>>(data, NHP, NH, nullptr, 0, tw);
        } else {
            k_fft_yx<R, K, N, -1, 2><<<hblocks(), TL::NT, SM, s>>>(data, NHP, NH, nullptr, 0, tw);
        }
        return "";
    }
    // sum of kappa^2 |.|^2 over the forward transforms along axis 1 or 0 of a
    // field [N][N][N] (diagnostics; FP64): one partial sum a block, *nparts of them
    static std::string line_k2(const G *data, int axis, double *part, int *nparts, const C *tw, int *err, cudaStream_t s) {
        if constexpr (std::is_same<R, double>::value) {
            if constexpr (kFftTma) {
                CUtensorMap my, mx;
                std::string e = make_axis_maps(&my, &mx, const_cast<G *>(data), true, N, N, TT::L, TX::L, N < 256 ? N : 256);
                if (!e.empty()) return e;
                const int nt = int(size_t(N) * N / (axis == 1 ? TT::L : TX::L));
                *nparts = axis == 1 ? ygrid : xgrid;
                if (axis == 1) k_line_k2_tma<N, 1><<<ygrid, TT::NT, TT::SMEM, s>>>(my, nt, tw, part, err);
                else k_line_k2_tma<N, 2><<<xgrid, TX::NT, TX::SMEM, s>>>(mx, nt, tw, part, err);
            } else {
                *nparts = int(zblocks());
                if (axis == 1) k_line_k2<N, 1><<<zblocks(), TL::NT, SM, s>>>(data, tw, part);
                else k_line_k2<N, 2><<<zblocks(), TL::NT, SM, s>>>(data, tw, part);
            }
            return "";
        }
        return "line_k2 needs FP64";
    }
    // One axis of a slab's local FFT step (plain passes): axis 2 = z on the
    // x-slab [planes][N][N], axis 1 = y on the x-slab, axis 0 = x on the
    // transposed y-slab [N][planes][N] (op 1: forward, -1/(kappa^2 N^3) with
    // global y offset y0, inverse).
    static std::string fft_slab(G *data, int planes, int axis, int sign, int op, int y0, const C *tw, cudaStream_t s) {
        const size_t nl = size_t(planes) * N;
        if (nl % TL::L || nl % TZ::L) return "planes * n must be a multiple of the tile lines";
        const unsigned gl = unsigned(nl / TL::L), nt = TL::NT;
        if (axis == 2) {
            z_pass(s, data, nl, sign, tw, 0x2545f491u, false, nullptr);
        } else if (axis == 1) {
            if (sign < 0) k_fft_yx<R, K, N, -1, 1><<<gl, nt, SM, s>>>(data, N, N, nullptr, 0, tw);
            else k_fft_yx<R, K, N, +1, 1><<<gl, nt, SM, s>>>(data, N, N, nullptr, 0, tw);
        } else if (op == 1) {
            k_fft_x_poisson_slab<R, K, N><<<gl, nt, SM, s>>>(data, planes, y0, tw);
        } else {
            if (sign < 0) k_fft_yx<R, K, N, -1, 2><<<gl, nt, SM, s>>>(data, planes, planes, nullptr, 0, tw);
            else k_fft_yx<R, K, N, +1, 2><<<gl, nt, SM, s>>>(data, planes, planes, nullptr, 0, tw);
        }
        return "";
    }

    // One axis (2 = z, 1 = y, 0 = x) of the callers' field of planes * N lines
    // (see fft_slab for the layouts) with the pipelined kernels of the steps;
    // base 16-byte aligned (bulk copies), N >= 256.  One axis pass of 256^3
    // complex128 measured 172 us plain.  Below 256 the field is in L2 and the
    // passes are as long as their launches either way.
    static std::string axis_pass(G *data, int planes, int axis, int sign, const C *tw, cudaStream_t s) {
        if constexpr (kFftTma) {
            const size_t lines = size_t(planes) * N;
            if (axis == 2) {
                z_pass(s, data, lines, sign, tw, 0x2545f491u, true, nullptr);
                return "";
            }
            CUtensorMap m;
            std::string e = make_field_map(&m, data, std::is_same<R, double>::value, N, planes, axis, axis == 1 ? TT::L : (kPair ? TPF::L : TX::L));
            if (!e.empty()) return e;
            if constexpr (kPair) {
                const int nt = int(lines / (axis == 1 ? TPY::L : TPF::L));
                if (axis == 1) {
                    if (sign < 0) k_yx_tma_pair<N, 1, 0, -1, PSTY, PBY, 8, true><<<pygrid, TPY::NT, TPY::SMEM, s>>>(m, data, N, N, nt, nullptr, nullptr, tw);
                    else k_yx_tma_pair<N, 1, 0, +1, PSTY, PBY, 8, true><<<pygrid, TPY::NT, TPY::SMEM, s>>>(m, data, N, N, nt, nullptr, nullptr, tw);
                } else {
                    if (sign < 0) k_yx_tma_pair<N, 2, 0, -1, PSTX, PBF, PLF, true><<<pfgrid, TPF::NT, TPF::SMEM, s>>>(m, data, planes, planes, nt, nullptr, nullptr, tw);
                    else k_yx_tma_pair<N, 2, 0, +1, PSTX, PBF, PLF, true><<<pfgrid, TPF::NT, TPF::SMEM, s>>>(m, data, planes, planes, nt, nullptr, nullptr, tw);
                }
            } else if (axis == 1) {
                const int nt = int(lines / TT::L);
                if (sign < 0) k_yx_tma<R, K, N, 1, 0, -1, true><<<ygrid, TT::NT, TT::SMEM, s>>>(m, data, N, N, nt, nullptr, 2, nullptr, tw);
                else k_yx_tma<R, K, N, 1, 0, +1, true><<<ygrid, TT::NT, TT::SMEM, s>>>(m, data, N, N, nt, nullptr, 2, nullptr, tw);
            } else {
                const int nt = int(lines / TX::L);
                if (sign < 0) k_yx_tma<R, K, N, 2, 0, -1, true><<<xgrid, TX::NT, TX::SMEM, s>>>(m, data, planes, planes, nt, nullptr, 3, nullptr, tw);
                else k_yx_tma<R, K, N, 2, 0, +1, true><<<xgrid, TX::NT, TX::SMEM, s>>>(m, data, planes, planes, nt, nullptr, 3, nullptr, tw);
            }
            return "";
        }
        return fft_slab(data, planes, axis, sign, 0, 0, tw, s);
    }
};

// Runtime (N, precision) -> Box<R, K, N>
template <typename R, typename K, typename F> static std::string with_box(int n, F &&f) {
    switch (n) {
        case 16: return f(Box<R, K, 16>{});
        case 32: return f(Box<R, K, 32>{});
        case 48: return f(Box<R, K, 48>{});
        case 64: return f(Box<R, K, 64>{});
        case 96: return f(Box<R, K, 96>{});
        case 128: return f(Box<R, K, 128>{});
        case 256: return f(Box<R, K, 256>{});
        case 512: return f(Box<R, K, 512>{});
        case 1024:
            // the mixed mode's FP64 exchange tiles do not fit shared memory at 1024
            if constexpr (std::is_same<R, K>::value) return f(Box<R, K, 1024>{});
            else return "grid size 1024 is not supported in mixed precision";
        default: return "unsupported grid size " + std::to_string(n);
    }
}
template <typename F> static std::string with_box2(int n, int prec, F &&f) {
    switch (prec) {
        case 0: return with_box<double, double>(n, f);
        case 1: return with_box<float, float>(n, f);
        case 2: return with_box<float, double>(n, f);
        default: return "unknown precision " + std::to_string(prec);
    }
}
// cuTensorMapEncodeTiled through the runtime's driver entry point (no libcuda link)
static std::string encode_map(CUtensorMap *m, void *base, bool f64, int rank, const cuuint64_t *dims,
                              const cuuint64_t *strides, const cuuint32_t *box) {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    {
        std::lock_guard<std::mutex> lk(setup_mutex());
        if (!fn) {
            cudaDriverEntryPointQueryResult q;
            CUDA_TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", (void **)&fn, cudaEnableDefault, &q));
            if (q != cudaDriverEntryPointSuccess || !fn) {
                fn = nullptr;
                return "cuTensorMapEncodeTiled unavailable";
            }
        }
    }
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(m, f64 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, (cuuint32_t)rank,
                    base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? "" : "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")";
}

// y-pass map: [x][y][W complex] as (2W reals, N, N); x-pass map: (2*N*W reals, N).
// Boxes: Ly (Lx) lines by boxr rows.
static std::string make_axis_maps(CUtensorMap *my, CUtensorMap *mx, void *base, bool f64, int N, int W, int Ly,
                                  int Lx, int boxr) {
    const cuuint64_t es = f64 ? 8 : 4;
    const cuuint64_t dy[3] = {cuuint64_t(2) * W, cuuint64_t(N), cuuint64_t(N)};
    const cuuint64_t sy[2] = {cuuint64_t(2) * W * es, cuuint64_t(2) * W * N * es};
    const cuuint32_t by[3] = {cuuint32_t(2 * Ly), cuuint32_t(boxr), 1};
    std::string e = encode_map(my, base, f64, 3, dy, sy, by);
    if (!e.empty()) return e;
    const cuuint64_t dx[2] = {cuuint64_t(2) * N * W, cuuint64_t(N)};
    const cuuint64_t sx[1] = {cuuint64_t(2) * W * N * es};
    const cuuint32_t bx[2] = {cuuint32_t(2 * Lx), cuuint32_t(boxr)};
    return encode_map(mx, base, f64, 2, dx, sx, bx);
}

static std::string make_field_map(CUtensorMap *m, void *base, bool f64, int N, int planes, int axis, int L) {
    const cuuint64_t es = f64 ? 8 : 4;
    const cuuint32_t boxr = cuuint32_t(N < 256 ? N : 256);
    if (axis == 1) {
        const cuuint64_t d[3] = {cuuint64_t(2) * N, cuuint64_t(N), cuuint64_t(planes)};
        const cuuint64_t st[2] = {cuuint64_t(2) * N * es, cuuint64_t(2) * N * N * es};
        const cuuint32_t b[3] = {cuuint32_t(2 * L), boxr, 1};
        return encode_map(m, base, f64, 3, d, st, b);
    }
    const cuuint64_t d[2] = {cuuint64_t(2) * N * planes, cuuint64_t(N)};
    const cuuint64_t st[1] = {cuuint64_t(2) * N * planes * es};
    const cuuint32_t b[2] = {cuuint32_t(2 * L), boxr};
    return encode_map(m, base, f64, 2, d, st, b);
}

// arithmetic type of a precision mode: 0 double, 1 float
static int compute_kind(int prec) { return prec == 1 ? 1 : 0; }
static size_t storage_bytes(int prec) { return prec == 0 ? 8 : 4; }

// twiddles exp(-2 pi i m / n), m < n, from long double; FP32 tables pair each
// rounded twiddle with its rounding remainder (exact - rounded): entries 2m, 2m+1
template <typename C> static std::vector<C> twiddles(int n) {
    using T = decltype(C{}.x);
    const int per = sizeof(T) == 4 ? 2 : 1;
    std::vector<C> t(size_t(per) * n);
    const long double twopi = 6.283185307179586476925286766559005768L;
    for (int m = 0; m < n; ++m) {
        const long double ang = -twopi * (long double)m / (long double)n;
        const long double c = cosl(ang), s = sinl(ang);
        C &h = t[size_t(per) * m];
        h.x = (T)c;
        h.y = (T)s;
        if (per == 2) {
            t[2 * size_t(m) + 1].x = (T)(c - (long double)h.x);
            t[2 * size_t(m) + 1].y = (T)(s - (long double)h.y);
        }
    }
    return t;
}

// cached per-(n, precision) tables on the current device
static std::string get_twiddles(int n, int prec, void **out) {
    struct Entry { int dev, n, prec; void *p; };
    std::lock_guard<std::mutex> lk(setup_mutex());
    static std::vector<Entry> cache;
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    for (auto &e : cache)
        if (e.dev == dev && e.n == n && e.prec == prec) { *out = e.p; return ""; }
    void *p = nullptr;
    if (prec == 0) {
        auto t = twiddles<double2>(n);
        CUDA_TRY(cudaMalloc(&p, sizeof(double2) * n));
        CUDA_TRY(cudaMemcpy(p, t.data(), sizeof(double2) * n, cudaMemcpyHostToDevice));
    } else {
        auto t = twiddles<float2>(n);
        CUDA_TRY(cudaMalloc(&p, sizeof(float2) * t.size()));
        CUDA_TRY(cudaMemcpy(p, t.data(), sizeof(float2) * t.size(), cudaMemcpyHostToDevice));
    }
    // a copy from pageable memory may return before it has landed, and the
    // kernels run on streams that do not order themselves against its stream
    CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));
    cache.push_back({dev, n, prec, p});
    *out = p;
    return "";
}

#define BOX_SIZES(X, name) X(name, 16) X(name, 32) X(name, 48) X(name, 64) X(name, 96)
#define BOX_DECLARE(name, n) const BoxKernels &box_kernels_##name##_##n();
#define BOX_CASE(name, n) \
    case n: return &box_kernels_##name##_##n();
BOX_SIZES(BOX_DECLARE, fp64)
BOX_SIZES(BOX_DECLARE, fp32)
BOX_DECLARE(fp32, 128)
BOX_SIZES(BOX_DECLARE, mixed)
static_assert(box_fits<float, float, 128>() && !box_fits<double, double, 128>() && !box_fits<float, double, 128>(), "sizes");

const BoxKernels *box_kernels(int precision, int N) {
    if (precision == 0) {
        switch (N) { BOX_SIZES(BOX_CASE, fp64) }
    } else if (precision == 1) {
        switch (N) { BOX_SIZES(BOX_CASE, fp32) BOX_CASE(fp32, 128) }
    } else {
        switch (N) { BOX_SIZES(BOX_CASE, mixed) }
    }
    return nullptr;
}

// ------------------------------------------------------------ StepEngine --
StepEngine::~StepEngine() {
    leave_full_boxes();
    cudaFree(box_scr_);
    cudaFree(psi_);
    cudaFree(phi_);
    cudaFree(rhok_);
    cudaFree(drift64_);
    cudaFree(drift32_);
    cudaFree(ts_);
    cudaFree(gmax_);
    cudaFree(part_);
    cudaFree(log_);
    cudaFree(ckpt_psi_);
    cudaFree(ckpt_phi_);
    cudaFree(seg_psi_);
    cudaFree(seg_phi_);
    cudaFree(g_);
    cudaFree(w_);
    cudaFree(pw_);
    cudaFree(ts_adj_);
    cudaFree(drift64_adj_);
    cudaFree(drift32_adj_);
    if (ev_read_) cudaEventDestroy(ev_read_);
    if (copy_stream_) cudaStreamSynchronize(copy_stream_);
    for (int s = 0; s < 2; ++s) {
        cudaFree(stage_[s]);
        if (ev_copied_[s]) cudaEventDestroy(ev_copied_[s]);
        if (ev_free_[s]) cudaEventDestroy(ev_free_[s]);
    }
    if (copy_stream_) cudaStreamDestroy(copy_stream_);
}

std::string StepEngine::ensure_staging() {
    if (stage_[0]) return "";
    CUDA_TRY(cudaStreamCreateWithFlags(&copy_stream_, cudaStreamNonBlocking));
    for (int s = 0; s < 2; ++s) {
        CUDA_TRY(cudaMalloc(&stage_[s], kStageElems * sizeof(double2)));
        CUDA_TRY(cudaEventCreateWithFlags(&ev_copied_[s], cudaEventDisableTiming));
        CUDA_TRY(cudaEventCreateWithFlags(&ev_free_[s], cudaEventDisableTiming));
    }
    return "";
}

std::string StepEngine::init(const EngineConfig &cfg, cudaStream_t stream) {
    cfg_ = cfg;
    stream_ = stream;
    const int N = cfg.N;
    if (!supported_n(N, cfg.precision)) return "unsupported grid size " + std::to_string(N);
    const size_t n3 = n3_();
    const size_t rs = storage_bytes(cfg.precision), cs = 2 * rs;
    const int nhp = cfg.precision == 0 ? half_pitch<double>(N) : half_pitch<float>(N);
    CUDA_TRY(cudaMalloc(&psi_, n3 * cs));
    CUDA_TRY(cudaMalloc(&phi_, n3 * rs));
    CUDA_TRY(cudaMalloc(&rhok_, size_t(N) * N * nhp * cs));
    CUDA_TRY(cudaMemsetAsync(rhok_, 0, size_t(N) * N * nhp * cs, stream_));
    CUDA_TRY(cudaMalloc(&drift64_, sizeof(double2) * N));
    CUDA_TRY(cudaMalloc(&drift32_, sizeof(float2) * N));
    CUDA_TRY(cudaMalloc(&ts_, sizeof(TState)));
    CUDA_TRY(cudaMemsetAsync(ts_, 0, sizeof(TState), stream_));
    CUDA_TRY(cudaEventCreateWithFlags(&ev_read_, cudaEventDisableTiming));
    std::string e = get_twiddles(N, compute_kind(cfg.precision), &tw_);
    if (!e.empty()) return e;
    e = get_twiddles(N / 2, compute_kind(cfg.precision), &twh_);
    if (!e.empty()) return e;
    e = with_box2(N, cfg.precision, [](auto box) { return decltype(box)::configure(); });
    if (!e.empty()) return e;
    // TMA descriptors for the pipelined y/x passes
    use_tma_ = N >= 128 && std::getenv("IFDM_NO_TMA") == nullptr;
    if (use_tma_) {
        const bool f64 = cfg.precision == 0;
        with_box2(N, cfg.precision, [&](auto box) -> std::string {
            decltype(box)::tma_lines(tma_ly_, tma_lx_);
            return "";
        });
        const int boxr = N < 256 ? N : 256;
        e = make_axis_maps(&map_psi_y_, &map_psi_x_, psi_, f64, N, N, tma_ly_, tma_lx_, boxr);
        if (e.empty()) e = make_axis_maps(&map_rho_y_, &map_rho_x_, rhok_, f64, N, nhp, tma_ly_, tma_lx_, boxr);
        if (!e.empty()) return e;
    }
    // max|phi| scan window of the reference: first N^3 doubles of the padded
    // [N][N][2(N/2+1)] array (the vector holds only N^3 elements,
    // src/struct3D.h:110,117; scanned at src/CosmoBEC_MPI.cpp:26)
    const long P = 2 * (N / 2 + 1);
    const long tot = long(N) * N * N;
    win_rows_ = tot / P;
    win_tail_ = int(tot - win_rows_ * P);
    return init_box();
}

// Whole runs in one launch where a plane of the box fits a CTA.
// IFDM_NO_FUSE keeps the one-launch-per-pass kernels.
std::string StepEngine::init_box() {
    const int N = cfg_.N;
    const BoxKernels *bk = box_kernels(cfg_.precision, N);
    if (!bk) return "";
    // one CTA per plane; a cluster where that is a cluster (its barrier takes
    // 1000-2000 cycles against 3000 of the counter in global memory), else a cooperative grid
    box_group_ = N;
    box_cluster_ = N <= 16;
    int resident = 0;
    {
        // attributes and the occupancy query once per device, size and precision
        std::lock_guard<std::mutex> lk(setup_mutex());
        static std::map<std::array<int, 3>, int> known;
        int dev = 0;
        CUDA_TRY(cudaGetDevice(&dev));
        const std::array<int, 3> key{dev, N, cfg_.precision};
        auto it = known.find(key);
        if (it == known.end()) {
            std::string e = bk->setup(0);
            if (!e.empty()) return e;
            it = known.emplace(key, bk->resident(box_group_, box_cluster_)).first;
        }
        resident = it->second;
    }
    int sms = 0;
    CUDA_TRY(cudaGetDevice(&dev_));
    CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev_));
    box_half_ = resident == 1 && !box_cluster_ && sms / (N / 2) >= 3;
    box_ = resident >= 1 && std::getenv("IFDM_NO_FUSE") == nullptr;
    if (box_ && box_half_) {
        std::string e = join_full_boxes();
        if (!e.empty()) return e;
    }
    box_half_ = box_half_ && box_;
    CUDA_TRY(cudaMalloc(&box_scr_, sizeof(BoxScratch)));
    CUDA_TRY(cudaMemsetAsync(box_scr_, 0, sizeof(BoxScratch), stream_));
    return "";
}

// Boxes of 96^3 hold a CTA on each of 96 SMs, so a second group does not fit
// beside one and the boxes would take turns with 52 of 148 SMs idle.  Groups of
// N/2 with two planes a CTA let three boxes run side by side, which costs one box
// time (a step's phases double, its barriers do not): taken while a batch works
// on several, or while another such box has work in flight.  One step of four
// contexts stepped in turn, us, whole / half groups: FP32 218 / 127, mixed 320 /
// 199, FP64 290 / 224 (a launch per pass: 182, 285, 297).  FP32 128^3 keeps whole
// groups: two halves of it gain nothing (329 / 336).  The results do not depend
// on the group.
namespace {
struct FullBoxes {
    std::mutex m;
    std::vector<StepEngine *> all;
};
FullBoxes &full_boxes() {
    static FullBoxes f;
    return f;
}
}  // namespace

std::string StepEngine::join_full_boxes() {
    CUDA_TRY(cudaEventCreateWithFlags(&ev_run_, cudaEventDisableTiming));
    std::lock_guard<std::mutex> lk(full_boxes().m);
    full_boxes().all.push_back(this);
    return "";
}
void StepEngine::leave_full_boxes() {
    if (!ev_run_) return;
    {
        std::lock_guard<std::mutex> lk(full_boxes().m);
        auto &v = full_boxes().all;
        v.erase(std::remove(v.begin(), v.end(), this), v.end());
    }
    cudaEventDestroy(ev_run_);
}
void StepEngine::pick_group() {
    if (!box_half_) return;
    bool other = shared_;
    if (!other) {
        // a query is refused while another thread captures a graph, unless in relaxed mode
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        {
            std::lock_guard<std::mutex> lk(full_boxes().m);
            for (StepEngine *o : full_boxes().all) {
                if (o == this || o->dev_ != dev_) continue;
                const cudaError_t e = cudaEventQuery(o->ev_run_);
                other = e == cudaErrorNotReady;
                if (e != cudaSuccess) cudaGetLastError();
                if (other) break;
            }
        }
        cudaThreadExchangeStreamCaptureMode(&mode);
    }
    box_group_ = other ? cfg_.N / 2 : cfg_.N;
}
std::string StepEngine::mark_run() {
    if (box_half_) CUDA_TRY(cudaEventRecord(ev_run_, stream_));
    return "";
}

// timestep: 1 each step's own (appended to log when given), 0 the one *ts_
// holds (one step), 2 replay log[0 ..]; save: keep the state before each step in
// the segment buffers.
std::string StepEngine::box_run(int nsteps, int timestep, double dt_scale, void *log, bool save) {
    BoxRun a{};
    a.psi = psi_;
    a.phi = phi_;
    a.rhok = rhok_;
    a.tw = tw_;
    a.ts = ts_;
    a.scr = (BoxScratch *)box_scr_;
    a.ph = phys_;
    a.ph.dt_scale = dt_scale;
    a.win_rows = win_rows_;
    a.win_tail = win_tail_;
    a.timestep = timestep;
    BoxLaunch l;
    l.group = box_group_;
    l.cluster = box_cluster_;
    l.stream = stream_;
    const size_t n3 = n3_(), rs = storage_bytes(cfg_.precision);
    for (int n = 0; n < nsteps; n += kBoxLaunchSteps) {
        const int cnt = std::min(kBoxLaunchSteps, nsteps - n);
        a.log = log ? (StepLog *)log + n : nullptr;
        a.seg_psi = save ? (char *)seg_psi_ + size_t(n) * n3 * 2 * rs : nullptr;
        a.seg_phi = save ? (char *)seg_phi_ + size_t(n) * n3 * rs : nullptr;
        CUDA_TRY(box_kernels(cfg_.precision, cfg_.N)->run(0, l, a, nullptr, cnt));
    }
    return "";
}

size_t StepEngine::n3_() const { return size_t(cfg_.N) * cfg_.N * cfg_.N; }

void StepEngine::set_physics(double rhoc) {
    using namespace phys;
    cfg_.rhoc = rhoc;
    const double m = cfg_.mfdm, ms = cfg_.mfdm_solar;
    const double S2 = rhoc / ms;
    S_ = std::sqrt(S2);
    Phi0_ = 4.0 * M_PI * bigG * rhoc * (cfg_.xmax / M_PI) * (cfg_.xmax / M_PI);
    Phys &ph = phys_;
    ph.A_KE = 4. / (3. * M_PI) * (m / pow(c, 2)) / hbar * pow(cfg_.dx, 2);
    ph.B_PE = 2. * M_PI * hbar / (m / pow(c, 2));
    ph.C_QI = cfg_.g != 0 ? 2. * M_PI * hbar / fabs(cfg_.g) : 0.0;
    ph.g = cfg_.g;
    ph.H0 = H_0;
    ph.Om = Omega_m0;
    ph.kP = m / pow(c, 2) / hbar * Phi0_;
    ph.kQ = cfg_.g / hbar * S2;
    ph.kin = 0.5 * hbar / (m / pow(c, 2)) * (M_PI / cfg_.xmax) * (M_PI / cfg_.xmax);
    ph.Phi0 = Phi0_;
    ph.S2 = S2;
    ph.dt_scale = 1.0;
    ph.N = cfg_.N;
    ph.dither = (cfg_.precision == 1 && std::getenv("IFDM_NO_DITHER") == nullptr) ? 1 : 0;
    ph.limit = 64;
}

std::string StepEngine::reset_state(double a) {
    TState t;
    std::memset(&t, 0, sizeof t);
    t.a = a;
    CUDA_TRY(cudaMemcpyAsync(ts_, &t, sizeof t, cudaMemcpyHostToDevice, stream_));
    CUDA_TRY(cudaStreamSynchronize(stream_));
    return "";
}

std::string StepEngine::load_psi(const double *psi, bool on_device, double a, double rhoc) {
    set_physics(rhoc);
    const size_t n3 = n3_();
    const double invS = 1.0 / S_;
    const int prec = cfg_.precision;
    if (!box_) {
        std::string e = reset_state(a);
        if (!e.empty()) return e;
    }
    if (on_device) {
        const int nb = (int)std::min<size_t>(1184, (n3 + 255) / 256);
        if (prec == 0) k_psi_in<double><<<nb, 256, 0, stream_>>>((const double2 *)psi, (double2 *)psi_, invS, n3);
        else k_psi_in<float><<<nb, 256, 0, stream_>>>((const double2 *)psi, (float2 *)psi_, invS, n3);

        CUDA_TRY(cudaGetLastError());
        CUDA_TRY(cudaEventRecord(ev_read_, stream_));
    } else {
        // chunk i: host -> slot i%2 on the copy stream, then the conversion on
        // the compute stream; the copy of chunk i+1 runs during conversion i,
        // and a slot is refilled only after its previous conversion finished
        std::string e2 = ensure_staging();
        if (!e2.empty()) return e2;
        int i = 0;
        for (size_t off = 0; off < n3; off += kStageElems, ++i) {
            const int s = i & 1;
            const size_t cnt = std::min(kStageElems, n3 - off);
            CUDA_TRY(cudaStreamWaitEvent(copy_stream_, ev_free_[s], 0));
            CUDA_TRY(cudaMemcpyAsync(stage_[s], psi + 2 * off, cnt * sizeof(double2), cudaMemcpyHostToDevice,
                                     copy_stream_));
            CUDA_TRY(cudaEventRecord(ev_copied_[s], copy_stream_));
            CUDA_TRY(cudaStreamWaitEvent(stream_, ev_copied_[s], 0));
            if (prec == 0)
                k_psi_in<double><<<1184, 256, 0, stream_>>>(stage_[s], (double2 *)psi_ + off, invS, cnt);
            else
                k_psi_in<float><<<1184, 256, 0, stream_>>>(stage_[s], (float2 *)psi_ + off, invS, cnt);
            CUDA_TRY(cudaGetLastError());
            CUDA_TRY(cudaEventRecord(ev_free_[s], stream_));
        }
        // the caller may reuse its buffer once every copy has landed
        CUDA_TRY(cudaStreamSynchronize(copy_stream_));
    }
    if (box_) {
        BoxRun a0{};
        a0.psi = psi_;
        a0.phi = phi_;
        a0.rhok = rhok_;
        a0.tw = tw_;
        a0.ts = ts_;
        a0.scr = (BoxScratch *)box_scr_;
        a0.win_rows = win_rows_;
        a0.win_tail = win_tail_;
        a0.a0 = a;
        BoxLaunch l;
        l.group = box_group_;
        l.cluster = box_cluster_;
        l.stream = stream_;
        CUDA_TRY(cudaMemsetAsync(box_scr_, 0, sizeof(BoxScratch), stream_));
        CUDA_TRY(box_kernels(prec, cfg_.N)->load(l, a0));
    } else {
        std::string e = launch_initial_density();
        if (!e.empty()) return e;
    }
    // stream_ may still hold earlier steps: the caller's tensor is free for
    // reuse on any stream only once the kernel that reads it has run.  That is a
    // short one of its own, so that the passes above are not waited for (24
    // boxes set and stepped as a batch: 6.16 ms without a wait, 6.80 with one
    // for the whole load)
    if (on_device) CUDA_TRY(cudaEventSynchronize(ev_read_));
    return "";
}

std::string StepEngine::psi_to_host(double *host_out, int which) {
    std::string e = ensure_staging();
    if (!e.empty()) return e;
    const size_t n3 = n3_();
    int i = 0;
    for (size_t off = 0; off < n3; off += kStageElems, ++i) {
        const int s = i & 1;
        const size_t cnt = std::min(kStageElems, n3 - off);
        // slot s is rewritten only after its previous copy to the host finished
        CUDA_TRY(cudaStreamWaitEvent(stream_, ev_free_[s], 0));
        if (cfg_.precision == 0)
            k_psi_out<double><<<1184, 256, 0, stream_>>>((const double2 *)psi_ + off, (const double *)phi_ + off, ts_,
                                                         which, S_, stage_[s], cnt);
        else
            k_psi_out<float><<<1184, 256, 0, stream_>>>((const float2 *)psi_ + off, (const float *)phi_ + off, ts_,
                                                        which, S_, stage_[s], cnt);
        CUDA_TRY(cudaGetLastError());
        CUDA_TRY(cudaEventRecord(ev_copied_[s], stream_));
        CUDA_TRY(cudaStreamWaitEvent(copy_stream_, ev_copied_[s], 0));
        CUDA_TRY(cudaMemcpyAsync(host_out + 2 * off, stage_[s], cnt * sizeof(double2), cudaMemcpyDeviceToHost,
                                 copy_stream_));
        CUDA_TRY(cudaEventRecord(ev_free_[s], copy_stream_));
    }
    CUDA_TRY(cudaStreamSynchronize(copy_stream_));
    return "";
}

std::string StepEngine::launch_initial_density() {
    return with_box2(cfg_.N, cfg_.precision, [&](auto box) -> std::string {
        using B = decltype(box);
        using C = typename B::C;
        using G = typename B::G;
        using R = typename B::R;
        G *psi = (G *)psi_, *rhok = (G *)rhok_;
        R *phi = (R *)phi_;
        const C *tw = (const C *)tw_, *twh = (const C *)twh_;
        if (!part_) CUDA_TRY(cudaMalloc(&part_, sizeof(double) * 3 * B::zrows()));
        B::initial_density(stream_, psi, rhok, ts_, part_, tw, twh);
        const CUtensorMap tm[4] = {map_psi_y_, map_psi_x_, map_rho_y_, map_rho_x_};
        for (int p = 6; p <= 9; ++p)
            B::pass(p, stream_, psi, phi, rhok, ts_, nullptr, tw, twh, win_rows_, win_tail_, use_tma_ ? tm : nullptr);
        CUDA_TRY(cudaGetLastError());
        return "";
    });
}

std::string StepEngine::launch_timestep(double dt_scale) {
    Phys ph = phys_;
    ph.dt_scale = dt_scale;
    const int nt = std::max(32, std::min(kTimestepThreads, cfg_.N));
    k_timestep<<<1, nt, 0, stream_>>>(ts_, ph, drift64_, drift32_);
    CUDA_TRY(cudaGetLastError());
    return "";
}

std::string StepEngine::launch_passes(cudaEvent_t *ev) {
    return with_box2(cfg_.N, cfg_.precision, [&](auto box) -> std::string {
        using B = decltype(box);
        using C = typename B::C;
        using G = typename B::G;
        using R = typename B::R;
        G *psi = (G *)psi_, *rhok = (G *)rhok_;
        R *phi = (R *)phi_;
        const C *tw = (const C *)tw_, *twh = (const C *)twh_;
        const C *drift = compute_kind(cfg_.precision) == 0 ? (const C *)(void *)drift64_ : (const C *)(void *)drift32_;
        const CUtensorMap tm[4] = {map_psi_y_, map_psi_x_, map_rho_y_, map_rho_x_};
        for (int p = 1; p <= 9; ++p) {
            B::pass(p, stream_, psi, phi, rhok, ts_, drift, tw, twh, win_rows_, win_tail_, use_tma_ ? tm : nullptr);
            if (ev) CUDA_TRY(cudaEventRecord(ev[p], stream_));
        }
        CUDA_TRY(cudaGetLastError());
        return "";
    });
}

std::string StepEngine::timestep_only(double dt_scale) { return launch_timestep(dt_scale); }
std::string StepEngine::passes_only() {
    if (!box_) return launch_passes(nullptr);
    pick_group();
    std::string e = box_run(1, 0, 1.0, nullptr, false);
    return e.empty() ? mark_run() : e;
}

std::string StepEngine::step(int nsteps, double dt_scale) {
    if (box_) {
        pick_group();
        std::string e = box_run(nsteps, 1, dt_scale, nullptr, false);
        return e.empty() ? mark_run() : e;
    }
    for (int i = 0; i < nsteps; ++i) {
        std::string e = launch_timestep(dt_scale);
        if (!e.empty()) return e;
        e = launch_passes(nullptr);
        if (!e.empty()) return e;
    }
    return "";
}

std::string StepEngine::profile(int nsteps, double dt_scale, std::vector<double> &ms) {
    cudaEvent_t ev[kNumPasses + 1];
    for (auto &e : ev) CUDA_TRY(cudaEventCreate(&e));
    ms.assign(kNumPasses, 0.0);
    for (int i = 0; i < nsteps; ++i) {
        CUDA_TRY(cudaEventRecord(ev[0], stream_));
        std::string e = launch_timestep(dt_scale);
        if (!e.empty()) return e;
        CUDA_TRY(cudaEventRecord(ev[1], stream_));
        // passes record ev[p] after pass p; shift so ev[p+1] follows pass p
        cudaEvent_t pe[kNumPasses];
        for (int p = 1; p <= 9; ++p) pe[p] = ev[p + 1];
        e = launch_passes(pe);
        if (!e.empty()) return e;
        CUDA_TRY(cudaEventSynchronize(ev[kNumPasses]));
        for (int p = 0; p < kNumPasses; ++p) {
            float t = 0.f;
            CUDA_TRY(cudaEventElapsedTime(&t, ev[p], ev[p + 1]));
            ms[p] += t;
        }
    }
    for (auto &v : ms) v /= nsteps;
    for (auto &e : ev) cudaEventDestroy(e);
    return "";
}

std::vector<double> StepEngine::pass_bytes() const {
    const double n3 = (double)n3_();
    const double N = cfg_.N;
    const double nh = N * N * (N / 2 + 1);
    const double rs = (double)storage_bytes(cfg_.precision), cs = 2 * rs;
    return {0.0,
            n3 * (2 * cs + rs),         // P1 psi in/out + phi in
            2 * cs * n3,                // P2
            2 * cs * n3,                // P3
            2 * cs * n3,                // P4
            2 * cs * n3 + cs * nh,      // P5 psi in/out + half spectrum out
            2 * cs * nh,                // P6
            2 * cs * nh,                // P7
            2 * cs * nh,                // P8
            cs * nh + rs * n3};         // P9 half spectrum in + phi out
}

std::string StepEngine::psi_out(double *dev_out, int which) {
    const size_t n3 = n3_();
    if (cfg_.precision == 0)
        k_psi_out<double><<<1184, 256, 0, stream_>>>((const double2 *)psi_, (const double *)phi_, ts_, which, S_,
                                                     (double2 *)dev_out, n3);
    else
        k_psi_out<float><<<1184, 256, 0, stream_>>>((const float2 *)psi_, (const float *)phi_, ts_, which, S_,
                                                    (double2 *)dev_out, n3);
    CUDA_TRY(cudaGetLastError());
    return "";
}

std::string StepEngine::phi_out(double *dev_out) {
    const size_t n3 = n3_();
    if (cfg_.precision == 0)
        k_phi_out<double><<<1184, 256, 0, stream_>>>((const double *)phi_, Phi0_, dev_out, n3);
    else
        k_phi_out<float><<<1184, 256, 0, stream_>>>((const float *)phi_, Phi0_, dev_out, n3);
    CUDA_TRY(cudaGetLastError());
    return "";
}

std::string StepEngine::read_state(TState &out) {
    CUDA_TRY(cudaMemcpyAsync(&out, ts_, sizeof(TState), cudaMemcpyDeviceToHost, stream_));
    CUDA_TRY(cudaStreamSynchronize(stream_));
    return "";
}

// ------------------------------------------------------------------ adjoint --
std::string StepEngine::adjoint_error(int &err) {
    int e[2] = {0, 0};
    CUDA_TRY(cudaMemcpyAsync(&e[0], &ts_->err, sizeof(int), cudaMemcpyDeviceToHost, stream_));
    if (!box_) CUDA_TRY(cudaMemcpyAsync(&e[1], &ts_adj_->err, sizeof(int), cudaMemcpyDeviceToHost, stream_));
    CUDA_TRY(cudaStreamSynchronize(stream_));
    err = e[0] | e[1];
    return "";
}

std::string StepEngine::ensure_adjoint_buffers(int nsteps, int ckpt) {
    const size_t n3 = n3_();
    const size_t rs = storage_bytes(cfg_.precision), cs = 2 * rs;
    const int nck = (nsteps + ckpt - 1) / ckpt;
    if (nsteps > log_cap_) {
        cudaFree(log_);
        log_ = nullptr;
        CUDA_TRY(cudaMalloc(&log_, sizeof(StepLog) * nsteps));
        log_cap_ = nsteps;
    }
    if (nck > nckpt_cap_) {
        cudaFree(ckpt_psi_);
        cudaFree(ckpt_phi_);
        ckpt_psi_ = ckpt_phi_ = nullptr;
        CUDA_TRY(cudaMalloc(&ckpt_psi_, n3 * cs * nck));
        CUDA_TRY(cudaMalloc(&ckpt_phi_, n3 * rs * nck));
        nckpt_cap_ = nck;
    }
    if (ckpt > seg_cap_) {
        cudaFree(seg_psi_);
        cudaFree(seg_phi_);
        seg_psi_ = seg_phi_ = nullptr;
        CUDA_TRY(cudaMalloc(&seg_psi_, n3 * cs * ckpt));
        CUDA_TRY(cudaMalloc(&seg_phi_, n3 * rs * ckpt));
        seg_cap_ = ckpt;
    }
    if (!g_) {
        CUDA_TRY(cudaMalloc(&g_, n3 * cs));
        CUDA_TRY(cudaMalloc(&w_, n3 * rs));
        CUDA_TRY(cudaMalloc(&pw_, n3 * rs));
        CUDA_TRY(cudaMalloc(&ts_adj_, sizeof(TState)));
        CUDA_TRY(cudaMemsetAsync(ts_adj_, 0, sizeof(TState), stream_));
        CUDA_TRY(cudaMalloc(&gmax_, sizeof(unsigned long long)));
        CUDA_TRY(cudaMalloc(&drift64_adj_, sizeof(double2) * cfg_.N));
        CUDA_TRY(cudaMalloc(&drift32_adj_, sizeof(float2) * cfg_.N));
        if (use_tma_) {
            const int N = cfg_.N, boxr = N < 256 ? N : 256;
            std::string e = make_axis_maps(&map_g_y_, &map_g_x_, g_, cfg_.precision == 0, N, N, tma_ly_, tma_lx_, boxr);
            if (!e.empty()) return e;
        }
    }
    return "";
}

std::string StepEngine::record(int nsteps, double dt_scale, int ckpt) {
    if (nsteps <= 0 || ckpt <= 0) return "record: nsteps and checkpoint interval must be positive";
    std::string e = ensure_adjoint_buffers(nsteps, ckpt);
    if (!e.empty()) return e;
    const size_t n3 = n3_();
    const size_t rs = storage_bytes(cfg_.precision), cs = 2 * rs;
    ckpt_every_ = ckpt;
    recorded_ = 0;
    StepLog *lg = static_cast<StepLog *>(log_);
    pick_group();
    for (int n = 0; n < nsteps; ++n) {
        if (n % ckpt == 0) {
            const size_t k = size_t(n / ckpt);
            CUDA_TRY(cudaMemcpyAsync((char *)ckpt_psi_ + k * n3 * cs, psi_, n3 * cs, cudaMemcpyDeviceToDevice, stream_));
            CUDA_TRY(cudaMemcpyAsync((char *)ckpt_phi_ + k * n3 * rs, phi_, n3 * rs, cudaMemcpyDeviceToDevice, stream_));
        }
        if (box_) {  // up to the next checkpoint
            const int cnt = std::min(ckpt - n % ckpt, nsteps - n);
            e = box_run(cnt, 1, dt_scale, lg + n, false);
            if (!e.empty()) return e;
            n += cnt - 1;
            continue;
        }
        e = launch_timestep(dt_scale);
        if (!e.empty()) return e;
        k_log_step<<<1, 1, 0, stream_>>>(ts_, lg + n);
        e = launch_passes(nullptr);
        if (!e.empty()) return e;
    }
    recorded_ = nsteps;
    return mark_run();
}

// one kick adjoint on g_: w, pw = phi_s[w], combine
std::string StepEngine::adjoint_kick(void *psi, void *phi, double a, double aP, double b, double alpha,
                                     long long tag) {
    const size_t n3 = n3_();
    return with_box2(cfg_.N, cfg_.precision, [&](auto box) -> std::string {
        using B = decltype(box);
        using C = typename B::C;
        using G = typename B::G;
        using R = typename B::R;
        using K = typename B::K;
        const C *tw = (const C *)tw_, *twh = (const C *)twh_;
        const CUtensorMap tm[4] = {map_g_y_, map_g_x_, map_rho_y_, map_rho_x_};
        k_adj_w<R, K><<<1184, 256, 0, stream_>>>((const G *)g_, (const G *)psi, (const R *)phi, a, b, alpha, (R *)w_,
                                                 n3);
        B::poisson_of(stream_, (const R *)w_, (R *)pw_, (G *)rhok_, ts_adj_, tw, twh, use_tma_ ? tm : nullptr);
        k_adj_combine<R, K><<<1184, 256, 0, stream_>>>((G *)g_, (const G *)psi, (const R *)phi, (const R *)pw_,
                                                       (const R *)w_, a, aP, b, alpha, n3,
                                                       (uint32_t)(tag * 0x9e3779b9ull) ^ 0x7f4a7c15u);
        CUDA_TRY(cudaGetLastError());
        return "";
    });
}

std::string StepEngine::adjoint(const double *g_final_dev, double *g0_dev) {
    if (recorded_ <= 0) return "adjoint: no recorded steps";
    if (!box_) CUDA_TRY(cudaMemsetAsync(ts_adj_, 0, sizeof(TState), stream_));
    const size_t n3 = n3_();
    const size_t rs = storage_bytes(cfg_.precision), cs = 2 * rs;
    const int M = recorded_, K = ckpt_every_;
    std::vector<StepLog> lg(M);
    CUDA_TRY(cudaMemcpyAsync(lg.data(), log_, sizeof(StepLog) * M, cudaMemcpyDeviceToHost, stream_));
    TState fin{};
    CUDA_TRY(cudaMemcpyAsync(&fin, ts_, sizeof(TState), cudaMemcpyDeviceToHost, stream_));
    CUDA_TRY(cudaStreamSynchronize(stream_));
    // natural units -> gradient with respect to the stored (scaled) field:
    // g_s = S g.  S ~ 1e50, so in FP32 storage S g overflows for any
    // cotangent of order one; the sweep is linear in g, so FP32 and mixed
    // carry lambda S g with a power of two lambda that brings max|lambda S g|
    // into [1, 2) (a power of two changes no rounding) and divide it out at
    // the end.  FP64 keeps lambda = 1.
    double lambda = 1.0;
    if (cfg_.precision != 0) {
        CUDA_TRY(cudaMemsetAsync(gmax_, 0, sizeof(unsigned long long), stream_));
        k_absmax<<<1184, 256, 0, stream_>>>(g_final_dev, 2 * n3, gmax_);
        CUDA_TRY(cudaGetLastError());
        unsigned long long bits = 0;
        CUDA_TRY(cudaMemcpyAsync(&bits, gmax_, sizeof(bits), cudaMemcpyDeviceToHost, stream_));
        CUDA_TRY(cudaStreamSynchronize(stream_));
        double gmax = 0.0;
        std::memcpy(&gmax, &bits, sizeof(gmax));
        const double top = gmax * S_;
        if (top > 0.0 && std::isfinite(top)) lambda = std::ldexp(1.0, -std::ilogb(top));
    }
    if (cfg_.precision == 0)
        k_scale_in<double><<<1184, 256, 0, stream_>>>((const double2 *)g_final_dev, (double2 *)g_, S_, n3);
    else
        k_scale_in<float><<<1184, 256, 0, stream_>>>((const double2 *)g_final_dev, (float2 *)g_, S_ * lambda, n3);
    CUDA_TRY(cudaGetLastError());
    if (box_) {
        pick_group();
        std::string eb = adjoint_box(fin);
        if (eb.empty()) eb = mark_run();
        if (!eb.empty()) return eb;
        return adjoint_finish(g0_dev, lambda);
    }
    // the output map: psi_out = S psi exp(-i (pendP phi + pendQ |psi|^2 - gphase))
    std::string e = adjoint_kick(psi_, phi_, fin.pendP, fin.pendP, fin.pendQ, -fin.gphase, 1ll << 40);
    if (!e.empty()) return e;
    for (int seg = (M - 1) / K; seg >= 0; --seg) {
        const int start = seg * K, end = std::min(M, start + K);
        // replay the segment from its checkpoint, keeping every (psi_n, phi_n)
        CUDA_TRY(cudaMemcpyAsync(psi_, (char *)ckpt_psi_ + size_t(seg) * n3 * cs, n3 * cs, cudaMemcpyDeviceToDevice,
                                 stream_));
        CUDA_TRY(cudaMemcpyAsync(phi_, (char *)ckpt_phi_ + size_t(seg) * n3 * rs, n3 * rs, cudaMemcpyDeviceToDevice,
                                 stream_));
        for (int n = start; n < end; ++n) {
            CUDA_TRY(cudaMemcpyAsync((char *)seg_psi_ + size_t(n - start) * n3 * cs, psi_, n3 * cs,
                                     cudaMemcpyDeviceToDevice, stream_));
            CUDA_TRY(cudaMemcpyAsync((char *)seg_phi_ + size_t(n - start) * n3 * rs, phi_, n3 * rs,
                                     cudaMemcpyDeviceToDevice, stream_));
            if (n + 1 < end) {  // the last state of the segment is not needed
                k_replay_step<<<1, 256, 0, stream_>>>(ts_, (const StepLog *)log_ + n, cfg_.N, 0, -1, drift64_, drift32_);
                e = launch_passes(nullptr);
                if (!e.empty()) return e;
            }
        }
        for (int n = end - 1; n >= start; --n) {
            k_replay_step<<<1, 256, 0, stream_>>>(ts_adj_, (const StepLog *)log_ + n, cfg_.N, 1, (1ll << 32) + n,
                                                  drift64_adj_, drift32_adj_);
            e = with_box2(cfg_.N, cfg_.precision, [&](auto box) -> std::string {
                using B = decltype(box);
                using C = typename B::C;
                using G = typename B::G;
                const C *tw = (const C *)tw_;
                const C *dconj = compute_kind(cfg_.precision) == 0 ? (const C *)(void *)drift64_adj_
                                                                   : (const C *)(void *)drift32_adj_;
                const CUtensorMap tm[4] = {map_g_y_, map_g_x_, map_rho_y_, map_rho_x_};
                B::adj_drift(stream_, (G *)g_, ts_adj_, dconj, tw, use_tma_ ? tm : nullptr,
                             (uint32_t)(n * 0x85ebca6bull) ^ 0xc2b2ae35u);
                CUDA_TRY(cudaGetLastError());
                return "";
            });
            if (!e.empty()) return e;
            const StepLog &L = lg[n];
            e = adjoint_kick((char *)seg_psi_ + size_t(n - start) * n3 * cs,
                             (char *)seg_phi_ + size_t(n - start) * n3 * rs, L.coefP, L.coefP, L.coefQ, L.alpha, n);
            if (!e.empty()) return e;
        }
    }
    return adjoint_finish(g0_dev, lambda);
}

// gradient with respect to the natural-unit psi_0 = S psi_s: g0 = g_s / S
std::string StepEngine::adjoint_finish(double *g0_dev, double lambda) {
    const size_t n3 = n3_();
    if (cfg_.precision == 0)
        k_scale_out<double><<<1184, 256, 0, stream_>>>((const double2 *)g_, (double2 *)g0_dev, 1.0 / S_, n3);
    else
        k_scale_out<float><<<1184, 256, 0, stream_>>>((const float2 *)g_, (double2 *)g0_dev, 1.0 / (S_ * lambda),
                                                      n3);
    CUDA_TRY(cudaGetLastError());
    recorded_ = 0;  // the replay consumed the state; record again before another adjoint
    return "";
}

// The sweep over the recorded steps with the one-launch kernels: per segment
// the checkpoint's copy, one replay launch that keeps the states before its
// steps, and one backward launch.  The last state of a segment stays in
// psi_, phi_.
std::string StepEngine::adjoint_box(const TState &fin) {
    const size_t n3 = n3_();
    const size_t rs = storage_bytes(cfg_.precision), cs = 2 * rs;
    const int M = recorded_, K = ckpt_every_;
    BoxSweep a{};
    a.g = g_;
    a.rhok = rhok_;
    a.tw = tw_;
    a.scr = (BoxScratch *)box_scr_;
    a.err = &ts_->err;
    a.log = (const StepLog *)log_;
    a.seg_psi = seg_psi_;
    a.seg_phi = seg_phi_;
    a.last_psi = psi_;
    a.last_phi = phi_;
    BoxLaunch l;
    l.group = box_group_;
    l.cluster = box_cluster_;
    l.stream = stream_;
    const BoxKernels &bk = *box_kernels(cfg_.precision, cfg_.N);
    // the output map: psi_out = S psi exp(-i (pendP phi + pendQ |psi|^2 - gphase))
    a.start = a.end = M;
    a.a = fin.pendP;
    a.b = fin.pendQ;
    a.alpha = -fin.gphase;
    CUDA_TRY(bk.sweep(l, a));
    for (int seg = (M - 1) / K; seg >= 0; --seg) {
        const int start = seg * K, end = std::min(M, start + K);
        CUDA_TRY(cudaMemcpyAsync(psi_, (char *)ckpt_psi_ + size_t(seg) * n3 * cs, n3 * cs, cudaMemcpyDeviceToDevice,
                                 stream_));
        CUDA_TRY(cudaMemcpyAsync(phi_, (char *)ckpt_phi_ + size_t(seg) * n3 * rs, n3 * rs, cudaMemcpyDeviceToDevice,
                                 stream_));
        if (end - start > 1) {
            std::string e = box_run(end - start - 1, 2, 1.0, (StepLog *)log_ + start, true);
            if (!e.empty()) return e;
        }
        a.start = start;
        a.end = end;
        CUDA_TRY(bk.sweep(l, a));
    }
    return "";
}

// bulk copies need a 16-byte base; a complex64 view may start at 8
static bool field_aligned(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

std::string fft_slab(void *data, int n, int planes, int axis, int precision, int sign, int op, int y0,
                     cudaStream_t stream) {
    if (!supported_n(n, precision)) return "unsupported grid size " + std::to_string(n);
    void *tw = nullptr;
    std::string e = get_twiddles(n, compute_kind(precision), &tw);
    if (!e.empty()) return e;
    return with_box2(n, precision, [&](auto box) -> std::string {
        using B = decltype(box);
        using C = typename B::C;
        using G = typename B::G;
        std::string e2 = B::configure();
        if (!e2.empty()) return e2;
        if (op == 0 && field_aligned(data) && planes * n % 16 == 0)
            e2 = B::axis_pass((G *)data, planes, axis, sign, (const C *)tw, stream);
        else e2 = B::fft_slab((G *)data, planes, axis, sign, op, y0, (const C *)tw, stream);
        if (!e2.empty()) return e2;
        CUDA_TRY(cudaGetLastError());
        return "";
    });
}

// FP64 pieces of the diagnostics: the N-point table, a half-spectrum axis
// pass, the kappa^2 sums along an axis (Box::half_axis, Box::line_k2)
template <typename F> static std::string with_fp64(int n, F &&f) {
    if (!supported_n(n)) return "unsupported grid size " + std::to_string(n);
    void *tw = nullptr;
    std::string e = get_twiddles(n, 0, &tw);
    if (!e.empty()) return e;
    return with_box<double, double>(n, [&](auto box) -> std::string {
        using B = decltype(box);
        std::string e2 = B::configure();
        if (!e2.empty()) return e2;
        e2 = f(box, (const double2 *)tw);
        if (!e2.empty()) return e2;
        CUDA_TRY(cudaGetLastError());
        return "";
    });
}
std::string fft_half_axis(void *data, int n, int axis, TState *ts, cudaStream_t stream) {
    return with_fp64(n, [&](auto box, const double2 *tw) {
        return decltype(box)::half_axis((double2 *)data, axis, tw, ts, stream);
    });
}
std::string axis_k2(const void *data, int n, int axis, double *part, int *nparts, int *err, cudaStream_t stream) {
    return with_fp64(n, [&](auto box, const double2 *tw) {
        return decltype(box)::line_k2((const double2 *)data, axis, part, nparts, tw, err, stream);
    });
}
std::string twiddle_tables(int n, int precision, const void **tw, const void **twh) {
    void *a = nullptr, *b = nullptr;
    std::string e = get_twiddles(n, compute_kind(precision), &a);
    if (e.empty()) e = get_twiddles(n / 2, compute_kind(precision), &b);
    *tw = a;
    *twh = b;
    return e;
}

std::string fft3d(void *data, int n, int precision, int sign, cudaStream_t stream) {
    if (!supported_n(n, precision)) return "unsupported grid size " + std::to_string(n);
    void *tw = nullptr;
    std::string e = get_twiddles(n, compute_kind(precision), &tw);
    if (!e.empty()) return e;
    return with_box2(n, precision, [&](auto box) -> std::string {
        using B = decltype(box);
        using C = typename B::C;
        using G = typename B::G;
        std::string e2 = B::configure();
        if (!e2.empty()) return e2;
        for (int axis = 2; axis >= 0; --axis) {  // z, y, x
            e2 = field_aligned(data) ? B::axis_pass((G *)data, n, axis, sign, (const C *)tw, stream)
                                     : B::fft_slab((G *)data, n, axis, sign, 0, 0, (const C *)tw, stream);
            if (!e2.empty()) return e2;
        }
        CUDA_TRY(cudaGetLastError());
        return "";
    });
}

}  // namespace ifdm
