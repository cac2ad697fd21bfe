// itlbm_step.cu -- the fused time step, the initial state and population export/import.
//
// State layout in HBM (per case, per buffer): tile-major (CaseDev in itlbm_internal.h).  Each 32 x 8
// tile is one contiguous block of 2 colours x 19 directions planes of 256 nodes, so every plane of a
// node is at a compile-time offset (q x 256 elements) from the node's address.
//   FP64 plain:  plane (0, i) = f_R,i and (1, i) = f_B,i
//   FP32 shifted: plane (0, i) = e_i = f_i - w_i rho0 and (1, i) = d_i = f_R,i - f_B,i
// A buffer holds the populations at the top of a step -- the reference's inif_R / inif_B after the
// swap (Imm_OPS.cpp:368-371) -- so initial states need no shift.  The step reads buffer `src`,
// collides every node and pushes each post-collision population to its neighbour x + c_i in buffer
// `dst`, as propag_site does (SimBoltz_Functions/LBM_functions.cpp:1220-1247).  The post-collision
// values the diagnostics need are therefore dst(x + c_i, i).
//
// One CTA of 256 threads handles a tile of 256 nodes (512 in the fold, two rows per thread) of one
// case (the work table says which; its shape -- 32 x 8, or 16 x 16 / 8 x 32 at the edge of a box
// whose width is not a multiple of 32 -- is that of the kernel).  It stages rho^N for the tile plus a
// halo of 1 (P1, P3, F3) or 2 (F1, F2) nodes in shared memory -- the halo nodes are
// re-read from L2, where the neighbouring tiles keep them -- then evaluates the mediator gradient,
// the force of class F on a ring-1 region of auxiliary fields, and collides.  No mediator
// populations or force fields ever reach HBM.
#include "itlbm_node.cuh"

#include <climits>

namespace itlbm {

namespace {

// Global loads and stores of the step, with cache hints chosen by measurement (build-time switches;
// the differences measured on B200 were within 1 %: promotion on the own-node loads is kept, the
// streaming stores cost the FP64 step 3 %):
//   ITLBM_LD_HINT  0: plain read-only loads; 1: L2 256-byte sector promotion on the own-node loads;
//                  2: on the halo-ring loads too
//   ITLBM_ST_HINT  0: plain stores; 1: streaming (evict-first) stores
#ifndef ITLBM_LD_HINT
#define ITLBM_LD_HINT 1
#endif
#ifndef ITLBM_ST_HINT
#define ITLBM_ST_HINT 0
#endif
template <bool PROMOTE>
__device__ __forceinline__ float ldg(const float *p) {
    if constexpr (PROMOTE) {
        float v;
        asm("ld.global.nc.L2::256B.f32 %0, [%1];" : "=f"(v) : "l"(p));
        return v;
    } else {
        return __ldg(p);
    }
}
template <bool PROMOTE>
__device__ __forceinline__ double ldg(const double *p) {
    if constexpr (PROMOTE) {
        double v;
        asm("ld.global.nc.L2::256B.f64 %0, [%1];" : "=d"(v) : "l"(p));
        return v;
    } else {
        return __ldg(p);
    }
}
constexpr bool LD_OWN = ITLBM_LD_HINT >= 1, LD_RING = ITLBM_LD_HINT >= 2;
__device__ __forceinline__ void stg(float *p, float v) {
#if ITLBM_ST_HINT == 1
    __stcs(p, v);
#else
    *p = v;
#endif
}
__device__ __forceinline__ void stg(double *p, double v) {
#if ITLBM_ST_HINT == 1
    __stcs(p, v);
#else
    *p = v;
#endif
}

__device__ __forceinline__ int wrapi(int a, int n) {
    int r = a % n;
    return r < 0 ? r + n : r;
}
// a in [-HMAX, n + HMAX) -> a mod n by compare and add; only boxes narrower than the halo take the
// division
__device__ __forceinline__ int wrap_near(int a, int n) {
    int r = a < 0 ? a + n : (a >= n ? a - n : a);
    if ((unsigned)r >= (unsigned)n) r = wrapi(r, n);
    return r;
}

// Shared memory of a W x Hh tile.
template <class S, int W, int Hh>
struct SmemT {
    static constexpr int PX = W + 2 * HMAX, PY = Hh + 2 * HMAX;  // staged phase tile
    static constexpr int QX = W + 2, QY = Hh + 2;                // ring-1 region of the F1/F2 auxiliaries
    S phi[PY][PX];        // rho^N of tile + halo (HMAX), position (px, py) = global (x0-2+px, y0-2+py)
    S g[QY][QX][3];       // ring-1 gradient (F1, F2)
    S aux[QY][QX][AUXS];  // ring-1 normal (F1) or stress (F2), 6 values at an odd stride
};

// ring position r -> staged-tile coordinates (px, py) for a halo of H (1 or 2) around the W x Hh
// interior; consecutive r run along x in the top and bottom bands, so loads of consecutive r
// coalesce.  The divisions by the band width B are a multiply by ceil(2^16 / B) and a shift, exact
// for r < 2^16 / B (r stays below the band length, at most 2 x 36, here).
template <int W, int Hh>
__device__ __forceinline__ void ring_pos(int r, int H, int &px, int &py) {
    constexpr int W1 = W + 2, W2 = W + 4;
    constexpr int M1 = (65536 + W1 - 1) / W1, M2 = (65536 + W2 - 1) / W2;
    static_assert(2 * W2 < 65536 / W2, "ring index range: the multiply-shift division is exact");
    const int B = W + 2 * H, M = H == 1 ? M1 : M2;
    const int nTop = H * B;
    if (r < 2 * nTop) {
        const int band = r < nTop ? 0 : 1;
        r -= band * nTop;
        const int q = (r * M) >> 16;
        py = band ? HMAX + Hh + q : HMAX - H + q;
        px = HMAX - H + (r - q * B);
    } else {
        r -= 2 * nTop;
        const int q = H == 1 ? (r >> 1) : (r >> 2);  // r / (2 H)
        const int k = r - q * 2 * H;
        py = HMAX + q;
        px = k < H ? HMAX - H + k : HMAX + W + (k - H);
    }
}

// One tile of one case.
//   phase A  each thread loads its node: FP64 keeps f_i = f_R,i + f_B,i and the colour sums (all
//            colisao_comum needs, Operadores_tensao.cpp:343-360), FP32 keeps e_i and the sums;
//            the halo ring is loaded as (ring node, colour) items spread over all threads, each an
//            ordered sum of 19 values, and the two colours' lanes form the ring node's rho^N;
//   phase B  F1 / F2: gradient and normal or stress on the ring-1 region;
//   phase C  mediator gradient, force, collision, recolouring, push to x + c_i.
// FOLD (FP32 only): the nine in-plane classes per colour instead of the 19 populations.
template <class S, bool FOLD, int W, int Hh, int R>
__device__ __forceinline__ void step_tile(const CaseDev &c, int tile, int k, int aux_k,
                                          SmemT<S, W, Hh> &sm) {
    constexpr int NP = FOLD ? NK : NV;  // storage planes per colour
    constexpr int QX = SmemT<S, W, Hh>::QX, QY = SmemT<S, W, Hh>::QY;
    constexpr int HT = Hh / R;          // rows of one pass of the CTA's threads
    static_assert(HT * W == STEP_THREADS, "a pass of the threads covers W x HT nodes");
    const int tid = threadIdx.x;
    const int lx = tid % W, ly = tid / W;  // the thread's nodes are rows ly + jr HT, jr < R
    const int nx = c.nx, ny = c.ny, tiles_x = c.tiles_x;
    constexpr int TE = 2 * NP * PLANE;  // elements per tile block
    // the address of node (x, y) in a buffer; plane q of the node is at [q * PLANE] from it
    auto node = [tiles_x](auto *buf, int x_, int y_) { return buf + node_off(tiles_x, TE, x_, y_); };
    const int x0 = (int)((unsigned)tile & 0xFFFFu) * 8, y0 = (int)((unsigned)tile >> 16) * 8;
    const int xe = min(x0 + W, nx), ye = min(y0 + Hh, ny);  // end of the valid interior
    const int H = c.halo;
    const int cur = (c.parity0 + k) & 1;
    const S *__restrict__ src = (const S *)c.buf[cur];
    S *__restrict__ dst = (S *)c.buf[cur ^ 1];
    const int tipo = c.tipo;
    const float rho0f = c.pf.rho0;  // FP32: the reference density in float (phase_of)

    // ---- phase A ----------------------------------------------------------------------------
    const int x = x0 + lx;
    S f[R][NP], sa[R], sb[R];
    double sbd[R];
#pragma unroll
    for (int jr = 0; jr < R; jr++) {
        const int lyj = ly + jr * HT, y = y0 + lyj;
        const bool valid = (x < xe) && (y < ye);
        sa[jr] = S(0);
        sb[jr] = S(0);
        sbd[jr] = 0.0;
        if (x < xe + H && y < ye + H) {
            const int xw = valid ? x : wrap_near(x, nx), yw = valid ? y : wrap_near(y, ny);
            const S *own = node(src, xw, yw);
            S a[NP], b[NP];
#pragma unroll
            for (int i = 0; i < NP; i++) a[i] = ldg<LD_OWN>(own + i * PLANE);
#pragma unroll
            for (int i = 0; i < NP; i++) b[i] = ldg<LD_OWN>(own + (NP + i) * PLANE);
#pragma unroll
            for (int i = 0; i < NP; i++) sa[jr] = sa[jr] + a[i];
#pragma unroll
            for (int i = 0; i < NP; i++) sb[jr] = sb[jr] + b[i];
            if constexpr (std::is_same<S, float>::value) {
                // FP32: rho^N from the FP32 sums (as for the halo nodes); the colour difference is
                // also summed in FP64 for the rest population's complement (see the split below)
#pragma unroll
                for (int i = 0; i < NP; i++) sbd[jr] += (double)b[i];
            }
            if constexpr (std::is_same<S, double>::value) {
#pragma unroll
                for (int i = 0; i < NP; i++) f[jr][i] = a[i] + b[i];
            } else {
#pragma unroll
                for (int i = 0; i < NP; i++) f[jr][i] = a[i];
            }
            sm.phi[lyj + HMAX][lx + HMAX] = phase_of(sa[jr], sb[jr], rho0f);
        }
    }
    // halo ring: item it = (ring node it / 2, colour it % 2), the two colours of a node on adjacent
    // lanes, which exchange their sums by a shuffle; the loop runs in whole warps (the bound is a
    // multiple of 32) so that every lane of a warp takes part in the shuffle
    const int nring = (W + 2 * H) * (Hh + 2 * H) - W * Hh;
    for (int it = tid; it < ((2 * nring + 31) & ~31); it += STEP_THREADS) {
        const int colour = it & 1, r = it >> 1;
        int px = 0, py = 0;
        if (r < nring) ring_pos<W, Hh>(r, H, px, py);
        const int gx = x0 - HMAX + px, gy = y0 - HMAX + py;
        const bool act = r < nring && gx < xe + H && gy < ye + H;
        S acc = S(0);
        if (act) {
            const S *rn = node(src, wrap_near(gx, nx), wrap_near(gy, ny)) + colour * NP * PLANE;
            S v[NP];
#pragma unroll
            for (int i = 0; i < NP; i++) v[i] = ldg<LD_RING>(rn + i * PLANE);
#pragma unroll
            for (int i = 0; i < NP; i++) acc = acc + v[i];
        }
        const S other = __shfl_xor_sync(0xffffffffu, acc, 1);
        if (act && colour == 0) sm.phi[py][px] = phase_of(acc, other, rho0f);
    }
    __syncthreads();

    // ---- phase B: ring-1 gradient and normal / stress (F1, F2) -------------------------------
    const bool ring_aux = (tipo == ITLBM_OP_F1 || tipo == ITLBM_OP_F2);
    if (ring_aux) {
        for (int q = tid; q < QX * QY; q += STEP_THREADS) {
            const int qx = q % QX, qy = q / QX;
            const int gx = x0 - 1 + qx, gy = y0 - 1 + qy;
            if (gx < xe + 1 && gy < ye + 1) {
                ring_aux_node(c, tipo, [&](int dx, int dy) { return sm.phi[qy + 1 + dy][qx + 1 + dx]; },
                              sm.g[qy][qx], sm.aux[qy][qx]);
            }
        }
        __syncthreads();
    }

    // ---- phase C: mediator gradient, force, collision, push ----------------------------------
#pragma unroll
    for (int jr = 0; jr < R; jr++) {
      const int lyj = ly + jr * HT, y = y0 + lyj;
      if ((x < xe) && (y < ye)) {
        CaseDev::F32Par pf{};  // FP32: the case's parameters in float
        if constexpr (std::is_same<S, float>::value) pf = load_pf(c);
        const int px = lx + HMAX, py = lyj + HMAX;
        S gmx, gmy, gmz, Fx, Fy, Fz;
        auto phi_at = [&](int dx, int dy) { return sm.phi[py + dy][px + dx]; };
        auto aux_at = [&](int dx, int dy) { return sm.aux[lyj + 1 + dy][lx + 1 + dx]; };
        node_force<S>(c, tipo, pf, phi_at, aux_at, sm.g[lyj + 1][lx + 1], gmx, gmy, gmz, Fx, Fy, Fz);
        // the destination node x + c_i (periodic) of D3Q19 direction i, or of class i of the fold
        const int xp = (x + 1 == nx) ? 0 : x + 1, xm = (x == 0) ? nx - 1 : x - 1;
        const int yp = (y + 1 == ny) ? 0 : y + 1, ym = (y == 0) ? ny - 1 : y - 1;
        auto dst_node = [&](int i) {
            const int ex = FOLD ? kx(i) : cx(i), ey = FOLD ? ky(i) : cy(i);
            return node(dst, ex == 0 ? x : (ex > 0 ? xp : xm), ey == 0 ? y : (ey > 0 ? yp : ym));
        };
        const bool force = tipo >= ITLBM_OP_F1;
        Recolour<S, FOLD> rc;
        if constexpr (std::is_same<S, double>::value) gradient_size(gmx, gmy, gmz, rc);
        node_moments<S, FOLD>(pf, f[jr], sa[jr], sb[jr], rc);
        if (force) {
            node_relax<true, S, FOLD>(c, pf, f[jr], sa[jr], sb[jr], Fx, Fy, Fz, rc);
            if (!rc.skip) node_finish<true, S, FOLD>(c, pf, f[jr], sa[jr], gmx, gmy, gmz, rc);
        } else {
            node_relax<false, S, FOLD>(c, pf, f[jr], sa[jr], sb[jr], Fx, Fy, Fz, rc);
            if (!rc.skip) node_finish<false, S, FOLD>(c, pf, f[jr], sa[jr], gmx, gmy, gmz, rc);
        }
        if (!rc.skip)
            node_split<S, FOLD>(pf, f[jr], sbd[jr], rc, [&](auto Q, S v) {
                constexpr int q = decltype(Q)::value;
                stg(dst_node(q % NP) + q * PLANE, v);
            });
        if (rc.skip) {  // rho <= 1e-30: the site is streamed unchanged (Operadores_tensao.cpp:347)
            const S *own = node(src, x, y);
            sfor<0, NP>([&](auto I) {
                constexpr int i = decltype(I)::value;
                S *n = dst_node(i);
                n[i * PLANE] = own[i * PLANE];
                n[(NP + i) * PLANE] = own[(NP + i) * PLANE];
            });
        }

        if (c.aux != nullptr && (k == aux_k || (c.aux_at_end && k == c.chunk_len - 1))) {
            keep_aux(c, x, y, Fx, Fy, Fz, gmx, gmy, gmz);
        }
      }
    }
    __syncthreads();
}

// Resident CTAs per SM the register allocation is sized for: 2 x 256 threads for FP64, 4 x 256
// threads for FP32 (the kernel is latency-bound at lower occupancy; see the ncu summaries).
#ifndef ITLBM_F64_BLOCKS
#define ITLBM_F64_BLOCKS 2
#endif
#ifndef ITLBM_F32_BLOCKS
#define ITLBM_F32_BLOCKS 4
#endif
#ifndef ITLBM_FOLD_BLOCKS  // the fold at 5 or 6 CTAs per SM (48 or 40 registers, with spills) measured
#define ITLBM_FOLD_BLOCKS 4   // 17 % and 8 % slower on the 600-case batch
#endif
#ifdef ITLBM_STEP_F64
#define ITLBM_STEP_MIN_BLOCKS(fold) (ITLBM_F64_BLOCKS * 256 / STEP_THREADS)
#else
#define ITLBM_STEP_MIN_BLOCKS(fold) (((fold) ? ITLBM_FOLD_BLOCKS : ITLBM_F32_BLOCKS) * 256 / STEP_THREADS)
#endif

template <class S, bool FOLD, int W>
__global__ void __launch_bounds__(STEP_THREADS, ITLBM_STEP_MIN_BLOCKS(FOLD)) k_step(const CaseDev *__restrict__ cases,
                                                       const TileRef *__restrict__ tiles,
                                                       int ntiles, const int *__restrict__ ntiles_dev,
                                                       int k, int aux_k) {
    constexpr int R = FOLD ? ITLBM_FOLD_ROWS : (std::is_same<S, float>::value ? ITLBM_F32_ROWS : 1);  // rows per thread
    constexpr int Hh = R * STEP_THREADS / W;
    __shared__ SmemT<S, W, Hh> sm;
    // The next step's launch may begin while this one runs (its CTAs take the places that the last ones
    // leave); each waits here until the step before it is complete, and only then lets the step after it begin:
    // CTAs that wait for more than one step pile up on the SMs with free places, and when they run, several of one
    // step share an SM (B200, us per step with the two calls the other way round and this way: FP32 P3 160 x 160
    // 8.7 and 5.4, FP32 F2 256 x 256 10.9 and 8.1, fold F2 256 x 256 11.4 and 7.2, FP64 P3 160 x 160 9.7 and 7.2).
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
    const int nt = ntiles_dev ? *ntiles_dev : ntiles;
    for (int t = blockIdx.x; t < nt; t += gridDim.x) {
        const TileRef tr = tiles[t];
        const CaseDev &c = cases[tr.case_id];
        if (k >= c.chunk_len) continue;
        step_tile<S, FOLD, W, Hh, R>(c, tr.tile, k, aux_k, sm);
    }
}

template <class S, bool FOLD>
cudaError_t launch_shape(const CaseDev *cases_dev, const TileRef *tiles, int ntiles, const int *ntiles_dev,
                         int grid, int k, int aux_k, int shape, bool early, cudaStream_t s) {
    if (grid <= 0) return cudaSuccess;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(STEP_THREADS);
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    // On a stream the early begin hides what lies between two launches; measured on B200, us per step: FP64 P3
    // 300 x 300 16.6 -> 14.0, FP32 P3 512 x 512 18.4 -> 16.8, 2048 x 2048 235.6 -> 232.2, fold 125.1 -> 120.9.  In a
    // graph there is less to hide and an early edge costs more: FP32 100 x 100 5.3 -> 8.0, eight of them 7.8 -> 9.8,
    // 512 x 512 16.7 -> 17.4, fold 600 x 600 12.9 -> 13.6; larger launches differ by less than 1 %.
    cfg.numAttrs = early ? 1 : 0;
    switch (shape) {
        case SHAPE_32x8: return cudaLaunchKernelEx(&cfg, k_step<S, FOLD, 32>, cases_dev, tiles, ntiles, ntiles_dev, k, aux_k);
        case SHAPE_16x16: return cudaLaunchKernelEx(&cfg, k_step<S, FOLD, 16>, cases_dev, tiles, ntiles, ntiles_dev, k, aux_k);
        case SHAPE_8x32: return cudaLaunchKernelEx(&cfg, k_step<S, FOLD, 8>, cases_dev, tiles, ntiles, ntiles_dev, k, aux_k);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace

// This file is compiled twice: with ITLBM_STEP_F64 (and --fmad=false, so that every FP64 operation
// rounds exactly as the reference's own code compiled with strict IEEE semantics) and without it.
#ifdef ITLBM_STEP_F64
cudaError_t launch_step_f64(const CaseDev *cases_dev, const TileRef *tiles, int ntiles,
                            const int *ntiles_dev, int grid, int k, int aux_k, int shape, bool early, cudaStream_t s) {
    return launch_shape<double, false>(cases_dev, tiles, ntiles, ntiles_dev, grid, k, aux_k, shape, early, s);
}
// The occupancy queries also load every shape's kernel (with lazy module loading a kernel is loaded
// at its first launch, which would otherwise fall inside the batch's first timed tuning window).
int step_occupancy_f64() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_step<double, false, 32>, STEP_THREADS, 0);
    cudaFuncAttributes a;
    cudaFuncGetAttributes(&a, k_step<double, false, 16>);
    cudaFuncGetAttributes(&a, k_step<double, false, 8>);
    return n;
}
#else
cudaError_t launch_step_f32(const CaseDev *cases_dev, const TileRef *tiles, int ntiles,
                            const int *ntiles_dev, int grid, int k, int aux_k, int shape, bool early, cudaStream_t s) {
    return launch_shape<float, false>(cases_dev, tiles, ntiles, ntiles_dev, grid, k, aux_k, shape, early, s);
}
int step_occupancy_f32() {
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_step<float, false, 32>, STEP_THREADS, 0);
    cudaFuncAttributes a;
    cudaFuncGetAttributes(&a, k_step<float, false, 16>);
    cudaFuncGetAttributes(&a, k_step<float, false, 8>);
    cudaFuncGetAttributes(&a, k_step<float, true, 32>);
    cudaFuncGetAttributes(&a, k_step<float, true, 16>);
    cudaFuncGetAttributes(&a, k_step<float, true, 8>);
    return n;
}
cudaError_t launch_step_fold(const CaseDev *cases_dev, const TileRef *tiles, int ntiles,
                             const int *ntiles_dev, int grid, int k, int aux_k, int shape, bool early, cudaStream_t s) {
    return launch_shape<float, true>(cases_dev, tiles, ntiles, ntiles_dev, grid, k, aux_k, shape, early, s);
}
#endif

}  // namespace itlbm
