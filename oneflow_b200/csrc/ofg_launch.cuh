// Launch sequences of the tasks, templated on the face arithmetic type.
// Included by one translation unit per precision (ofg_k64.cu is compiled
// without FMA contraction so that the FP64 path rounds like the reference).
#pragma once
#include <algorithm>

#include "ofg_ctx.h"
#include "ofg_chain.cuh"
#include "ofg_kernels.cuh"
#include "ofg_turb.cuh"

namespace ofg {

// step < 0: the device-side outer-step counter's next step
static __global__ void k_cfl(double *scal, long long *ext, double step, Ramp ramp) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    start_step(scal, ext, step < 0 ? scal[S_STEP] + 1.0 : step, ramp);
}

// before n fused iterations: the counters follow the host's, and the first outer step starts (not the multi-stage
// scheme's, whose iterations start their own)
static __global__ void k_begin(double *scal, long long *ext, double done, bool start, Ramp ramp) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    scal[S_STEP] = scal[S_HISTN] = scal[S_THISTN] = done;
    if (start) start_step(scal, ext, done + 1.0, ramp);
}

static __global__ void k_clear_extremes(long long *ext) {
    if (threadIdx.x == 0) clear_extremes(ext);
}

static __global__ void k_norm_hist(double *scal, double *hist, int cap) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    int n = int(scal[S_HISTN]);
    if (n < cap)
        for (int e = 0; e < NEQ; ++e) hist[(size_t)n * NEQ + e] = scal[S_NORM + e];
    scal[S_HISTN] = double(n + 1);
}

template <typename R>
KArgs<R> make_args(ofg_ctx *c, bool onCurrent) {
    KArgs<R> A;
    A.P = c->dp;
    A.nCells = c->nCells; A.nBFaces = c->nBFaces; A.nFaces = c->nFaces; A.nT = c->nT;
    A.nb_off = c->d_nb_off; A.nbl = reinterpret_cast<const int2 *>(c->d_nbl);
    A.lo_off = c->d_lo_off; A.lol = reinterpret_cast<const int2 *>(c->d_lol);
    A.up_off = c->d_up_off; A.upl = reinterpret_cast<const int2 *>(c->d_upl);
    A.bcType = c->d_bct; A.key = c->d_key; A.walldist = c->d_wdist;
    A.fgeo = static_cast<const R *>(c->d_fgeo); A.cgeo = static_cast<const R *>(c->d_cgeo);
    A.fgeoD = sizeof(R) == 8 ? static_cast<const double *>(c->d_fgeo) : c->d_fgeoD;
    A.fofs = c->d_fofs; A.lr = reinterpret_cast<const int2 *>(c->d_lr); A.fout = c->d_fout;
    int nx = onCurrent ? c->cur : c->cur ^ 1;
    A.q = c->d_q[c->cur];
    A.qn = c->d_q[nx];
    if (sizeof(R) == 4) {
        A.qs = reinterpret_cast<const R *>(c->d_qs[c->cur]);
        A.qsn = reinterpret_cast<R *>(c->d_qs[nx]);
    } else {
        A.qs = reinterpret_cast<const R *>(A.q);
        A.qsn = reinterpret_cast<R *>(A.qn);
    }
    A.res = c->d_res; A.dq = static_cast<R *>(c->d_dq); A.dt = c->d_dt; A.invsr = c->d_invsr; A.vissr = c->d_vissr;
    A.rad = c->d_rad;
    A.bcq = c->d_bcq; A.gl = static_cast<R *>(c->d_gl[c->gl]); A.mm = static_cast<R *>(c->d_mm);
    A.scal = c->d_scal; A.ext = c->d_ext; A.fixlist = c->d_fix; A.fixcap = c->fixcap;
    A.npart = c->d_npart; A.tpart = c->d_tpart; A.red = c->d_red; A.redCount = c->d_redCount;
    A.nut = c->d_nut; A.dnut = c->d_dnut; A.resT = c->d_resT; A.impsrT = c->d_impsrT;
    A.matL = c->d_matL; A.matR = c->d_matR; A.gnut = static_cast<R *>(c->d_gnut);
    return A;
}

inline int nblk(long long n, int b) { return int((n + b - 1) / b); }

#define OFG_LAUNCH(kern, grid, block, stream, ...)                         \
    do {                                                                   \
        kern<<<(grid), (block), 0, (stream)>>>(__VA_ARGS__);               \
        ++c->launches;                                                     \
    } while (0)

// gradients and limiter of the current state (UPDATE_RESIDUALS' first half);
// started: the outer step's start has cleared the limiter extremes, and no
// gradient pass since has widened them
template <typename R>
void launch_gradlim(ofg_ctx *c, const KArgs<R> &A, cudaStream_t s, bool started = false) {
    const int N = c->nCells;
    bool needGrad = c->p.ilim != -1 || c->p.vismodel > 0;
    if (!needGrad) return;
    int nvar = c->p.vismodel > 0 ? 6 : 5;
    bool venkatGlobal = c->p.ilim == 2 && !c->p.venkat_kh3;
    int limMode = (c->p.ilim == 1 || c->p.ilim == 2) ? (venkatGlobal ? 2 : 1) : 0;
    int nb = nblk(N, 128);
    if (limMode == 2 && !started) OFG_LAUNCH(k_clear_extremes, 1, 32, s, A.ext);
    if constexpr (sizeof(R) == 4) {
        const int gb = c->tune.grad_block == 64 ? 64 : 128;   // the limiter's block extremes are exact either way
        nb = nblk(N, gb);
        switch (c->tune.grad_min_blocks) {
        case 4: OFG_LAUNCH((k_gradlim<R, 4>), nb, gb, s, A, nvar, limMode); break;
        case 8: OFG_LAUNCH((k_gradlim<R, 8>), nb, gb, s, A, nvar, limMode); break;
        default: OFG_LAUNCH((k_gradlim<R, 6>), nb, gb, s, A, nvar, limMode); break;
        }
    } else {
        OFG_LAUNCH(k_gradlim<R>, nb, 128, s, A, nvar, limMode);
    }
    if (limMode == 2) OFG_LAUNCH(k_limiter_global<R>, nblk(N, 128), 128, s, A);
}

// Whether the FP64 residual pass runs with four lanes a cell: as long as its
// blocks (32 cells, two to an SM) all run at once.  Measured, us an iteration
// with a thread a cell / four lanes: Euler triangles, 1,200 cells 27.5 / 27.5,
// 6,144 31.5 / 29.6, 8,192 30.7 / 29.6, 10,240 31.7 / 35.7; laminar quadrilaterals,
// 1,200 43.9 / 37.8, 8,000 44.2 / 40.5, 10,000 45.2 / 47.4; tetrahedra (SA), 5,880
// 99.8 / 95.5, 8,976 99.9 / 95.8, 10,800 100.3 / 103.7.
inline bool quad_residual(int cells) { return cells <= 9000; }

// The flux / time-step pass of MODE (as k_residual): the FP64 path's
// per-cell gather, or the mixed path's face pass followed by the per-cell sum
// of the face results (part: 1 the first kernel only, 2 the second only, 3 both).
template <typename R, int MODE>
void launch_flux(ofg_ctx *c, const KArgs<R> &A, cudaStream_t s, int part = 3) {
    const int N = c->nCells;
    const bool vv = c->p.ivischeme >= 2;   // the TEST / NEW1 / NEW2 viscous face gradients
    if constexpr (sizeof(R) == 8) {
        if (!(part & 1)) return;
        if (vv) OFG_LAUNCH((k_residual<R, MODE, true>), nblk(N, 128), 128, s, A);
        else if (!c->crowded && quad_residual(N)) OFG_LAUNCH((k_residual_quad<R, MODE>), 4 * nblk(N, 128), 128, s, A);
        else OFG_LAUNCH((k_residual<R, MODE>), nblk(N, 128), 128, s, A);
    } else {
        if (part & 1) {
            const int F = c->nFaces, bs = c->tune.face_block;
            if (vv) {
                OFG_LAUNCH((k_face_pass<MODE, true>), nblk(F, 128), 128, s, A);
            } else if constexpr (MODE == 0) {   // the iteration's pass: the tuned shape
                switch (c->tune.face_min_blocks) {
                case 2: OFG_LAUNCH((k_face_pass<0, false, 2>), nblk(F, bs), bs, s, A); break;
                case 4: OFG_LAUNCH((k_face_pass<0, false, 4>), nblk(F, bs), bs, s, A); break;
                case 5: OFG_LAUNCH((k_face_pass<0, false, 5>), nblk(F, bs), bs, s, A); break;
                default: OFG_LAUNCH((k_face_pass<0, false, 3>), nblk(F, bs), bs, s, A); break;
                }
            } else {
                OFG_LAUNCH((k_face_pass<MODE>), nblk(F, 128), 128, s, A);
            }
        }
        if (part & 2) OFG_LAUNCH((k_face_sum<MODE>), nblk(N, 128), 128, s, A);
    }
}

// Blocks of a chained sweep's cluster, by the mean cells of a level.  A block
// takes 32 kChainWarps = 192 cells of a level at once, two cells a thread
// pipe-bound; a cluster pays about 0.4 us a level for its signals.  Measured,
// us a sweep: 119 levels of 29 cells (FP64) 83 with one block, 107 with 4;
// 385 of 170 (FP64) 565, 434, 450 with 1, 4, 8 blocks; 228 of 631 (FP64) 2,790,
// 1,330, 1,120, 1,210 with 1, 4, 8, 16.
inline int chain_blocks(const ofg_ctx *c) {
    const int mean = c->nCells / std::max(1, c->chain[0].nlev);
    return mean <= 96 ? 1 : mean <= 400 ? 4 : 8;
}

// Whether this context's sweeps run chained (one launch per sweep)
inline bool chained(const ofg_ctx *c) { return c->tune.sweep_persistent && c->chain[0].lev && c->chain[1].lev; }

inline ChainPlan chain_plan(const ofg_ctx *c, bool lower) {
    const ChainBuf &b = c->chain[lower ? 0 : 1];
    return ChainPlan{reinterpret_cast<const int4 *>(b.lev), lower ? c->d_lowOrder : c->d_upOrder, b.ref,
                     reinterpret_cast<const int4 *>(b.edge), b.nlev, b.far, b.slots, c->chainStatus};
}

// Whether an FP64 sweep level runs with four lanes a cell: as long as that
// still leaves the SMs room.  Measured, us an iteration with a thread a cell /
// four lanes: levels of 288 cells 33.3 / 29.2, 2,048 35.3 / 31.4, 8,192 35.3 / 32.1,
// 18,432 37.4 / 35.3, 14,400 tetrahedra (SA) 203 / 193; of 32,768 46.1 / 51.2.
// (The mixed path's approximate quotients and roots leave no such chain.)
inline bool quad_level(int cells) { return cells <= 20000; }

// Whether the fused iteration runs the NS lower sweep's first level with the
// diagonal (k_timestep_clip): a launch fewer, but its blocks then write
// increments colour by colour.  Measured, us an iteration
// without / with: 4,096 cells 38.3 / 36.2, 113,886 84.9 / 82.2, 312,000 (FP64)
// 624.2 / 622.4, 600,000 469.9 / 470.8, 768,640 631.6 / 634.2.
inline bool first_level_early(const ofg_ctx *c) { return !chained(c) && c->nCells <= 400000; }

template <typename K, typename... Args>
int launch_chain(ofg_ctx *c, K one, K many, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = chain_blocks(c);
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    K kern = at.val.clusterDim.x > 1 ? many : one;
    cfg.gridDim = dim3(at.val.clusterDim.x);
    cfg.blockDim = dim3(kChainThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    if (e == cudaSuccess && at.val.clusterDim.x > 8)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, kern, args...);
    if (e != cudaSuccess) return c->fail(OFG_E_CUDA, std::string("chained sweep: ") + cudaGetErrorString(e));
    ++c->launches;
    return OFG_OK;
}

template <typename R, bool LOWER>
int launch_chain_ns(ofg_ctx *c, const KArgs<R> &A, cudaStream_t s) {
    const ChainPlan P = chain_plan(c, LOWER);
    R *coef = static_cast<R *>(c->d_chainCoef);
    OFG_LAUNCH((k_chain_coef<R, LOWER>), nblk(std::max<long long>(P.slots, A.nCells), 128), 128, s, A, P, coef,
               c->d_chainCell);
    return launch_chain(c, k_chain_ns<R, LOWER, false>, k_chain_ns<R, LOWER, true>,
                        kChainRing * ChainNs<R, LOWER, true>::kBytes, s, A, P, (const R *)coef,
                        (const double *)c->d_chainCell);
}

template <typename R, bool LOWER>
int launch_chain_sa(ofg_ctx *c, const KArgs<R> &A, cudaStream_t s) {
    const ChainPlan P = chain_plan(c, LOWER);
    double *mat = static_cast<double *>(c->d_chainCoef);
    OFG_LAUNCH((k_chain_mat<R, LOWER>), nblk(std::max<long long>(P.slots, A.nCells), 128), 128, s, A, P, mat,
               c->d_chainCell);
    return launch_chain(c, k_chain_sa<R, LOWER, false>, k_chain_sa<R, LOWER, true>,
                        kChainRing * ChainSa<R, LOWER, true>::kBytes, s, A, P, (const double *)mat,
                        (const double *)c->d_chainCell);
}

template <typename R>
int launch_task(ofg_ctx *c, int task, cudaStream_t s) {
    const int N = c->nCells;
    const Ramp ramp{c->p.cflst, c->p.cfled, c->p.ncfl};
    switch (task) {
    case T_CFL: {
        OFG_LAUNCH(k_cfl, 1, 32, s, c->d_scal, c->d_ext, double(c->outerSteps), ramp);
        break;
    }
    case T_ADVANCE: {
        OFG_LAUNCH(k_cfl, 1, 32, s, c->d_scal, c->d_ext, -1.0, ramp);
        break;
    }
    case T_BEGIN: {
        OFG_LAUNCH(k_begin, 1, 32, s, c->d_scal, c->d_ext, double(c->outerSteps), c->p.time_integral != 1, ramp);
        break;
    }
    case T_TIMESTEP: {   // CALC_TIME_STEP alone (after T_CFL, which resets the minimum)
        KArgs<R> A = make_args<R>(c, false);
        launch_flux<R, 1>(c, A, s);
        OFG_LAUNCH(k_timestep_clip<R>, nblk(N, 256), 256, s, A);
        break;
    }
    case T_RESIDUAL: {   // UPDATE_RESIDUALS alone
        KArgs<R> A = make_args<R>(c, false);
        launch_gradlim<R>(c, A, s);
        launch_flux<R, 2>(c, A, s);
        break;
    }
    case T_TS_RES:       // CALC_TIME_STEP + LOAD_RESIDUALS + UPDATE_RESIDUALS in one gather
    case T_P_GRADLIM:    // (its parts, launched separately by the profiler and the fused iteration)
    case T_GRADLIM0:
    case T_P_FLUX:
    case T_P_FSUM:
    case T_P_CLIP: {
        KArgs<R> A = make_args<R>(c, false);
        if (task == T_TS_RES || task == T_P_GRADLIM || task == T_GRADLIM0) launch_gradlim<R>(c, A, s, task == T_GRADLIM0);
        if (task == T_TS_RES) launch_flux<R, 0>(c, A, s);
        if (task == T_P_FLUX) launch_flux<R, 0>(c, A, s, 1);
        if (task == T_P_FSUM) launch_flux<R, 0>(c, A, s, 2);
        if (task == T_TS_RES || task == T_P_CLIP) OFG_LAUNCH(k_timestep_clip<R>, nblk(N, 256), 256, s, A);
        break;
    }
    case T_CLIP0: {
        KArgs<R> A = make_args<R>(c, false);
        if (first_level_early(c)) OFG_LAUNCH((k_timestep_clip<R, true>), nblk(N, 256), 256, s, A);
        else OFG_LAUNCH(k_timestep_clip<R>, nblk(N, 256), 256, s, A);
        break;
    }
    case T_CALC_LHS: {   // CALC_LHS of the multi-stage scheme (same 128-cell blocks as the norm partials)
        KArgs<R> A = make_args<R>(c, false);
        OFG_LAUNCH(k_calc_lhs<R>, nblk(N, 128), 128, s, A, c->lhsCoef);
        break;
    }
    case T_LOWER:
    case T_LOWER1: {
        KArgs<R> A = make_args<R>(c, false);
        int nl = int(c->lowOff.size()) - 1;
        if (chained(c)) return launch_chain_ns<R, true>(c, A, s);
        for (int l = task == T_LOWER1 && first_level_early(c) ? 1 : 0; l < nl; ++l) {
            int st = c->lowOff[l], cnt = c->lowOff[l + 1] - st;
            const int *ord = (const int *)c->d_lowOrder;
            if constexpr (sizeof(R) == 4) {
                const int bs = c->tune.sweep_block;
                switch (c->tune.sweep_min_blocks) {
                case 6: OFG_LAUNCH((k_lusgs_lower<R, 6>), nblk(cnt, bs), bs, s, A, ord, st, cnt); break;
                case 10: OFG_LAUNCH((k_lusgs_lower<R, 10>), nblk(cnt, bs), bs, s, A, ord, st, cnt); break;
                default: OFG_LAUNCH((k_lusgs_lower<R, 8>), nblk(cnt, bs), bs, s, A, ord, st, cnt); break;
                }
            } else {
                if (!c->crowded && quad_level(cnt)) OFG_LAUNCH((k_lusgs_quad<R, true>), nblk(4LL * cnt, 128), 128, s, A, ord, st, cnt);
                else OFG_LAUNCH(k_lusgs_lower<R>, nblk(cnt, 128), 128, s, A, ord, st, cnt);
            }
        }
        break;
    }
    case T_UPPER: {
        // level 0 of the upper sweep holds the cells without later
        // neighbours: their increment gains -(+0)/rad, which leaves it
        // unchanged bit for bit (add_neg_quot), so that level is not launched
        KArgs<R> A = make_args<R>(c, false);
        int nl = int(c->upOff.size()) - 1;
        if (chained(c)) return launch_chain_ns<R, false>(c, A, s);
        for (int l = 1; l < nl; ++l) {
            int st = c->upOff[l], cnt = c->upOff[l + 1] - st;
            const int *ord = (const int *)c->d_upOrder;
            if constexpr (sizeof(R) == 4) {
                const int bs = c->tune.sweep_block;
                switch (c->tune.sweep_min_blocks) {
                case 6: OFG_LAUNCH((k_lusgs_upper<R, 6>), nblk(cnt, bs), bs, s, A, ord, st, cnt); break;
                case 10: OFG_LAUNCH((k_lusgs_upper<R, 10>), nblk(cnt, bs), bs, s, A, ord, st, cnt); break;
                default: OFG_LAUNCH((k_lusgs_upper<R, 8>), nblk(cnt, bs), bs, s, A, ord, st, cnt); break;
                }
            } else {
                if (!c->crowded && quad_level(cnt)) OFG_LAUNCH((k_lusgs_quad<R, false>), nblk(4LL * cnt, 128), 128, s, A, ord, st, cnt);
                else OFG_LAUNCH(k_lusgs_upper<R>, nblk(cnt, 128), 128, s, A, ord, st, cnt);
            }
        }
        break;
    }
    case T_UPDATE:
    case T_UPDATE_NEXT: {
        KArgs<R> A = make_args<R>(c, false);
        OFG_LAUNCH(k_update<R>, nblk(N, 256), 256, s, A);
        if (task == T_UPDATE_NEXT) OFG_LAUNCH((k_solution_fix<R, true>), 1, 32, s, A, ramp);
        else OFG_LAUNCH(k_solution_fix<R>, 1, 32, s, A, ramp);
        break;
    }
    case T_BOUNDARY_NEXT: {
        KArgs<R> A = make_args<R>(c, false);
        if (c->nBFaces > 0) OFG_LAUNCH(k_boundary<R>, nblk(c->nBFaces, 256), 256, s, A, (const int *)c->d_lcb);
        break;
    }
    case T_BOUNDARY_CUR: {
        KArgs<R> A = make_args<R>(c, true);
        OFG_LAUNCH(k_interior_tvisl<R>, nblk(N, 256), 256, s, A);
        if (c->nBFaces > 0) OFG_LAUNCH(k_boundary<R>, nblk(c->nBFaces, 256), 256, s, A, (const int *)c->d_lcb);
        break;
    }
    case T_PACK_STATE: {
        KArgs<R> A = make_args<R>(c, true);
        OFG_LAUNCH(k_pack_state<R>, nblk(c->nT, 256), 256, s, A, (const double *)c->d_stage);
        break;
    }
    case T_UNPACK_STATE: {
        KArgs<R> A = make_args<R>(c, true);
        OFG_LAUNCH(k_unpack_state<R>, nblk(c->nT, 256), 256, s, A, c->d_stage);
        break;
    }
    case T_GRAD_ONLY: {   // gradients of the current buffer (no limiter), for a path that keeps none
        KArgs<R> A = make_args<R>(c, true);
        OFG_LAUNCH(k_gradlim<R>, nblk(N, 128), 128, s, A, 5, 0);
        break;
    }
    case T_FORCES: {
        KArgs<R> A = make_args<R>(c, true);
        if (c->nWall == 0) break;
        int nb = nblk(c->nWall, 256);
        if (nb > 64) nb = 64;   // the block sums fit the reduction buffer
        OFG_LAUNCH(k_forces<R>, nb, 256, s, A, reinterpret_cast<const int2 *>(c->d_wall), (const double *)c->d_wallG,
                   c->nWall, c->d_scal + S_FORCE);
        break;
    }
    case T_NORM:         // norms of the last residual, appended to the history
    case T_NORM_ONLY: {  // the same without the history entry
        KArgs<R> A = make_args<R>(c, false);
        OFG_LAUNCH(k_norm_final<R>, kRedBlocks, 256, s, A, nblk(N, 128));
        if (task == T_NORM) OFG_LAUNCH(k_norm_hist, 1, 32, s, c->d_scal, c->d_hist, c->histCap);
        break;
    }
    case T_TURB_RHS:
    case T_P_TURB_GRAD:  // (its parts, launched separately by the profiler)
    case T_P_TURB_FLUX: {
        KArgs<R> A = make_args<R>(c, true);
        if (task != T_P_TURB_FLUX) {
            if (c->nBFaces > 0) OFG_LAUNCH(k_turb_bc<R>, nblk(c->nBFaces, 256), 256, s, A, (const int *)c->d_lcb, 0);
            OFG_LAUNCH(k_turb_grad<R>, nblk(N, 128), 128, s, A);
        }
        if (task != T_P_TURB_GRAD) OFG_LAUNCH(k_turb_rhs<R>, nblk(N, 128), 128, s, A);
        break;
    }
    case T_TURB_LOWER: {
        KArgs<R> A = make_args<R>(c, true);
        int nl = int(c->lowOff.size()) - 1;
        if (chained(c)) return launch_chain_sa<R, true>(c, A, s);
        for (int l = 0; l < nl; ++l) {
            int st = c->lowOff[l], cnt = c->lowOff[l + 1] - st;
            OFG_LAUNCH(k_turb_lower<R>, nblk(cnt, 128), 128, s, A, (const int *)c->d_lowOrder, st, cnt);
        }
        break;
    }
    case T_TURB_UPPER: {   // level 0 skipped, as in T_UPPER
        KArgs<R> A = make_args<R>(c, true);
        int nl = int(c->upOff.size()) - 1;
        if (chained(c)) return launch_chain_sa<R, false>(c, A, s);
        for (int l = 1; l < nl; ++l) {
            int st = c->upOff[l], cnt = c->upOff[l + 1] - st;
            OFG_LAUNCH(k_turb_upper<R>, nblk(cnt, 128), 128, s, A, (const int *)c->d_upOrder, st, cnt);
        }
        break;
    }
    case T_TURB_UPDATE: {
        KArgs<R> A = make_args<R>(c, true);
        OFG_LAUNCH(k_turb_update<R>, nblk(N, 256), 256, s, A, 1);
        break;
    }
    case T_TURB_BOUNDARY: {
        KArgs<R> A = make_args<R>(c, true);
        if (c->nBFaces > 0) OFG_LAUNCH(k_turb_bc<R>, nblk(c->nBFaces, 256), 256, s, A, (const int *)c->d_lcb, 1);
        break;
    }
    case T_TURB_BOUNDARY_CUR: {
        KArgs<R> A = make_args<R>(c, true);
        OFG_LAUNCH(k_turb_vist<R>, nblk(N, 256), 256, s, A);
        if (c->nBFaces > 0) OFG_LAUNCH(k_turb_bc<R>, nblk(c->nBFaces, 256), 256, s, A, (const int *)c->d_lcb, 1);
        break;
    }
    case T_TURB_NORM:
    case T_TURB_NORM_ONLY: {
        KArgs<R> A = make_args<R>(c, true);
        OFG_LAUNCH(k_turb_norm_final<R>, kRedBlocks, 256, s, A, nblk(N, 128),
                   task == T_TURB_NORM ? c->d_thist : (double *)nullptr, c->histCap);
        break;
    }
    default:
        return c->fail(OFG_E_ARG, "unknown task");
    }
    return OFG_OK;
}

}  // namespace ofg
