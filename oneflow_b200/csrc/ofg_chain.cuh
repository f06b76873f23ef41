// The chained LU-SGS sweeps: one launch per sweep, for meshes whose sweep
// order makes many small levels (the reference's own cell order: hundreds of
// levels of tens to hundreds of cells).  A launch per level costs about 6 us
// there (measured: 385 levels of 170 cells, 3.15 ms per sweep), nearly all of it
// latency: the launch, four dependent loads per face, and a serial chain of
// FP64 divisions and roots that does not depend on the increments at all.
//
// k_chain_coef forms everything of an edge (cell, neighbour) that does not
// depend on the increments for all edges at once, level after level in slots
// [level][j-th edge][cell of the level], so that the sweep's loads are
// contiguous.  k_chain_ns / k_chain_sa then run every level in one cluster of
// blocks.  The warps of a block form kChainGroups groups; group g takes the
// levels g, g + kChainGroups, ... and loads a level's coefficients while the
// levels before it run.  A level's increments go to a ring in the shared
// memory of every block of the cluster (neighbours further back than the ring
// are read from global memory), and its warps arrive on an mbarrier of every
// block that the next level's group waits on: the only latency between
// levels is that arrival, the ring reads and the increment's own arithmetic.
// Per-cell arithmetic and its order are those of the level launches: the same
// bits.  Every wait is bounded; one that runs out raises *status.
//
// Measured, us a sweep (level launches / chained): 385 levels of 170 cells,
// FP64, 3,130 / 400; 119 of 29 cells 785-950 / 80.  What bounds a level now
// (0.66 us alone, 1.03 us in a cluster of 4) is the arithmetic of its cells: about
// 160 FP64 instructions a cell at 2.4 cycles a warp, their 9-cycle latencies
// and the signal (0.06 us in a block, 0.25 us in a cluster).  Two groups of six
// warps: the loads of a level (0.5 us) end before its wait does, and 168
// registers a thread hold two edges without spills (four groups of four warps
// spilled: 1.3 us a level).
#pragma once
#include "ofg_kernels.cuh"

namespace ofg {

constexpr unsigned kChainWaitLimit = 1u << 20; // try_wait rounds before a wait gives up
constexpr int kChainPre = 2;                   // edges of a cell loaded ahead of the wait

// One sweep's schedule (device arrays)
struct ChainPlan {
    const int4 *lev;       // per level {first position, cells, first slot, slots per cell}
    const int *order;      // [nCells] cell at each position of the level order
    const int *ref;        // [slots] ring slot of the neighbour, ~cell when it is further back, kChainNone
    const int4 *edge;      // [slots] {face | side << 31, neighbour, cell, -}; y < 0 on an empty slot
    int nlev;
    int far;               // 1: some neighbour lies further back than the ring; 2: and within a few levels
    long long slots;
    unsigned *status;      // pinned host word: nonzero once a wait ran out
};

// Everything the NS sweep reads besides the increments, in the sweep's own
// order: the edges' coefficients coef[kEdgeCoefs][slots]; and the cells'
// right-hand side (LOWER: the residual; upper: the lower sweep's increment),
// diagonal and its reciprocal cells[kChainCell][nCells].
template <typename R, bool LOWER>
__global__ void __launch_bounds__(128) k_chain_coef(KArgs<R> A, ChainPlan P, R *coef, double *cells) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s < A.nCells) {
        const int c = __ldg(P.order + s);
        const double d = A.rad[c];
#pragma unroll
        for (int e = 0; e < NEQ; ++e)
            cells[(size_t)e * A.nCells + s] = LOWER ? A.res[(size_t)c * NEQ + e] : double(A.dq[(size_t)c * DQR + e]);
        cells[(size_t)NEQ * A.nCells + s] = d;
        cells[(size_t)(NEQ + 1) * A.nCells + s] = 1.0 / d;
    }
    if (s >= P.slots) return;
    const int4 e4 = __ldg(P.edge + s);
    if (e4.y < 0) return;
    const int2 e2 = make_int2(e4.x, e4.y);
    const int c = e4.z, f = nb_face(e2), nb = e4.y;
    R qc[REC], qn[REC], fg[FGR];
    ld8(A.qs + (size_t)c * REC, qc);
    ld8(A.qs + (size_t)nb * REC, qn);
    ld8(A.fgeo + (size_t)f * FGR, fg);
    R volb = A.P.visSRModel == 1 ? A.cgeo[(size_t)nb * CGR + 3] : R(1);
    R xn = fg[0], yn = fg[1], zn = fg[2];
    if (nb_right(e2)) { xn = -xn; yn = -yn; zn = -zn; }   // GCom::SetGeometry
    EdgeCoef<R> E;
    edge_coef(A.P, qc, qn, xn, yn, zn, fg[3], fg[7], volb, E);
    const R *v = &E.lmd1;
#pragma unroll
    for (int k = 0; k < kEdgeCoefs; ++k) coef[(size_t)k * P.slots + s] = v[k];
}

// The same for the SA sweep: the edges' face matrices mat[slots], and
// right-hand side, diagonal and reciprocal cells[3][nCells].
template <typename R, bool LOWER>
__global__ void __launch_bounds__(128) k_chain_mat(KArgs<R> A, ChainPlan P, double *mat, double *cells) {
    const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (s < A.nCells) {
        const int c = __ldg(P.order + s);
        const double d = A.impsrT[c];
        cells[s] = LOWER ? A.resT[c] : A.dnut[c];
        cells[(size_t)A.nCells + s] = d;
        cells[2 * (size_t)A.nCells + s] = 1.0 / d;
    }
    if (s >= P.slots) return;
    const int4 e4 = __ldg(P.edge + s);
    const int2 e2 = make_int2(e4.x, e4.y);
    if (e2.y >= 0) mat[s] = (nb_right(e2) ? A.matL : A.matR)[nb_face(e2)];
}

// Read-only loads that stay where they are written, ahead of the wait (plain
// ones may be moved down to their first use)
__device__ __forceinline__ double chain_ld(const double *p) {
    double v;
    asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float chain_ld(const float *p) {
    float v;
    asm volatile("ld.global.nc.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int chain_ld(const int *p) {
    int v;
    asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// ---- the cluster's barriers ------------------------------------------------
__device__ __forceinline__ uint32_t chain_smem(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t chain_peer(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ uint32_t chain_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t chain_size() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void chain_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// a block's own mbarrier (one block: block scope)
__device__ __forceinline__ void chain_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// a cluster: the same without an order of its own (the data come with the
// bytes; global copies are ordered by a fence ahead of it where they are read)
__device__ __forceinline__ void chain_arrive_relaxed(uint32_t bar) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void chain_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.relaxed.cluster.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
// a 16-byte store to a block of the cluster that counts on that block's mbarrier
__device__ __forceinline__ void chain_send(uint32_t addr, double a, double b, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(addr),
                 "d"(a), "d"(b), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void chain_send(uint32_t addr, float a, float b, float c, float d, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                     addr),
                 "f"(a), "f"(b), "f"(c), "f"(d), "r"(bar)
                 : "memory");
}
template <bool CL>
__device__ __forceinline__ bool chain_wait(uint32_t bar, uint32_t parity) {
    for (unsigned i = 0; i < kChainWaitLimit; ++i) {
        uint32_t done;
        if constexpr (CL)
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(bar), "r"(parity)
                : "memory");
        else
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.acquire.cta.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(bar), "r"(parity)
                : "memory");
        if (done) return true;
    }
    return false;
}

// The schedule common to the NS and SA sweeps.  Body: load(t, m) reads what
// does not depend on the increments (for the thread's first cell of a level
// before the wait), solve(t, m) forms the cell's increment, send(t, m, bar, n)
// puts it in the ring of every block, store() writes its global copy.
//
// Every warp of a level's group arrives once on its block's mbarrier of that
// level, whether it has cells of the level or not.  One block: after its cells. A
// cluster: as soon as it has seen the level before, since the increments travel
// by st.async, which counts their bytes on the receiving block's mbarrier; and
// every block sends one more 16-byte word to every block for every level. So
// - no phase of an mbarrier completes before every warp of the block has seen the
//   level before it, and with it the mbarrier's own last phase: a warp that
//   lags meets the parity it waits for, and the next phase's bytes and arrivals
//   never meet the one before;
// - no block runs two levels ahead of what another has seen: its word of a
//   level follows all its warps' arrivals in the level before.
// (With the first warp's arrival alone, a warp without cells in two levels could
// miss both and wait for a phase that waits for it.)
template <bool CL, typename Body>
__device__ __forceinline__ void chain_run(const ChainPlan &P, uint64_t *bars, double2 *word, Body &body) {
    // a level's increments and words stay below what an mbarrier can count
    static_assert(kChainLevel * Body::kBytes + 16 * kChainMaxBlocks < (1u << 20), "a level's bytes");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n = CL ? chain_size() : 1, rank = CL ? chain_rank() : 0;
    const int g = warp / kChainWarps, w = warp % kChainWarps, cw = w * n + rank;
    const int step = 32 * kChainWarps * n;
    const uint32_t bar0 = chain_smem(bars);
    if (threadIdx.x == 0) {
        for (int k = 0; k < kChainGroups; ++k)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar0 + 8 * k), "r"(kChainArrivals) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (CL) chain_cluster_sync();
    for (int l = g; l < P.nlev; l += kChainGroups) {
        const int4 m = __ldg(P.lev + l);
        const uint32_t bar = bar0 + 8 * (l % kChainGroups);
        int t = cw * 32 + lane;
        body.load(t, m);
        // a cluster: the mbarrier's own last phase first, so that every warp has acquired every level
        bool ok = !CL || l < kChainGroups || chain_wait<CL>(bar, (l / kChainGroups - 1) & 1);
        if (ok) ok = l == 0 || chain_wait<CL>(bar0 + 8 * ((l - 1) % kChainGroups), ((l - 1) / kChainGroups) & 1);
        if (!__all_sync(0xffffffffu, ok)) {            // the whole warp leaves together
            *reinterpret_cast<volatile unsigned *>(P.status) = 1u;   // pinned host memory
            break;
        }
        if (CL) {
            if (P.far) {   // this warp's earlier global copies
                __syncwarp();
                asm volatile("fence.acq_rel.cluster;" ::: "memory");
            }
            if (w == 0) {
                if (lane == 0) chain_expect(bar, uint32_t(m.y) * Body::kBytes + 16u * n);
                if (lane < n) chain_send(chain_peer(chain_smem(word + rank), lane), 0.0, 0.0, chain_peer(bar, lane));
            } else if (lane == 0) {
                chain_arrive_relaxed(bar);
            }
        }
        // a cell's global copy goes out after its signal, off the path between
        // levels; first where a level may read it that starts before this
        // warp's next arrival is known to every block
        auto put = [&](int at) {
            if (P.far == 2) {
                body.store();
                if (CL) asm volatile("fence.acq_rel.cluster;" ::: "memory");
            }
            body.send(at, m, bar, n);
            if (P.far != 2 && (CL || at + step < m.y)) body.store();
        };
        const bool mine = t < m.y;
        if (mine) {
            body.solve(t, m);
            put(t);
        }
#pragma unroll 1
        for (t += step; t < m.y; t += step) {
            body.load(t, m);
            body.solve(t, m);
            put(t);
        }
        if (!CL) {
            __syncwarp();
            if (lane == 0) chain_arrive(bar);
            if (P.far != 2 && mine) body.store();   // the last cell's
        }
    }
    if (CL) {
        // no block leaves while increments of the last level, which nobody
        // waited for, may still be on their way to its ring: a block sees
        // its own in, then all blocks leave together
        if (warp == 0 && !chain_wait<CL>(bar0 + 8 * ((P.nlev - 1) % kChainGroups), ((P.nlev - 1) / kChainGroups) & 1))
            *reinterpret_cast<volatile unsigned *>(P.status) = 1u;
        __syncwarp();
        chain_cluster_sync();
    }
}

// One sweep of the NS increments.  LOWER: dq = (res - rhs0) / rad; else the
// cell's own lower-sweep increment minus rhs0 / rad (cells without later
// neighbours keep theirs: add_neg_quot).
template <typename R, bool LOWER, bool CL>
struct ChainNs {
    const KArgs<R> &A;
    const ChainPlan &P;
    const R *coef;
    const double *cells;
    R *ring;                 // [kChainRing][kStride]
    uint32_t ringAddr;
    static constexpr int kStride = sizeof(R) == 8 ? 6 : 8;   // whole 16-byte words
    static constexpr uint32_t kBytes = kStride * sizeof(R);
    int c, ref[kChainPre];
    Divisor rad;
    double own[NEQ];         // the cell's right-hand side, then its increment
    EdgeCoef<R> E[kChainPre];

    __device__ __forceinline__ void load_edge(int t, const int4 &m, int j, int &rf, EdgeCoef<R> &e) const {
        const long long s = (long long)m.z + (long long)j * m.y + t;
        rf = chain_ld(P.ref + s);
        R *v = &e.lmd1;
#pragma unroll
        for (int k = 0; k < kEdgeCoefs; ++k) v[k] = chain_ld(coef + (size_t)k * P.slots + s);
    }
    __device__ __forceinline__ void load(int t, const int4 &m) {
        if (t >= m.y) return;
        c = chain_ld(P.order + m.x + t);
#pragma unroll
        for (int j = 0; j < kChainPre; ++j) {
            ref[j] = kChainNone;
            if (j < m.w) load_edge(t, m, j, ref[j], E[j]);
        }
#pragma unroll
        for (int e = 0; e < NEQ; ++e) own[e] = chain_ld(cells + (size_t)e * A.nCells + m.x + t);
        rad.d = chain_ld(cells + (size_t)NEQ * A.nCells + m.x + t);
        rad.r = chain_ld(cells + (size_t)(NEQ + 1) * A.nCells + m.x + t);
    }
    // the neighbour's increment: the ring's, or through L2 where it is further
    // back (another block may have written it); an empty slot gets any value
    __device__ __forceinline__ void fetch(int rf, R *d) const {
        const R *r = ring + max(rf, 0) * kStride;
#pragma unroll
        for (int k = 0; k < NEQ; ++k) d[k] = r[k];
        if (P.far && rf < 0 && rf != kChainNone) {
#pragma unroll
            for (int k = 0; k < NEQ; ++k) d[k] = __ldcg(A.dq + (size_t)(~rf) * DQR + k);
        }
    }
    __device__ __forceinline__ void apply(int rf, const EdgeCoef<R> &e, const R *d, double *rhs0) const {
        double t[NEQ];   // without a branch: the edges' chains overlap
#pragma unroll
        for (int k = 0; k < NEQ; ++k) t[k] = rhs0[k];
        edge_apply(A.P, e, d, t);
#pragma unroll
        for (int k = 0; k < NEQ; ++k) rhs0[k] = rf == kChainNone ? rhs0[k] : t[k];
    }
    __device__ __forceinline__ void solve(int t, const int4 &m) {
        double rhs0[NEQ] = {0.0, 0.0, 0.0, 0.0, 0.0};
        R d[kChainPre][NEQ];
#pragma unroll
        for (int j = 0; j < kChainPre; ++j) fetch(ref[j], d[j]);
#pragma unroll
        for (int j = 0; j < kChainPre; ++j) apply(ref[j], E[j], d[j], rhs0);
#pragma unroll 1
        for (int j = kChainPre; j < m.w; ++j) {
            int rf;
            EdgeCoef<R> e;
            load_edge(t, m, j, rf, e);
            fetch(rf, d[0]);
            apply(rf, e, d[0], rhs0);
        }
        if (LOWER) {
#pragma unroll
            for (int e = 0; e < NEQ; ++e) rhs0[e] = own[e] - rhs0[e];
            div_by<NEQ>(rhs0, rad, own);
        } else if (m.w > 0) {   // without later neighbours the upper sweep leaves a cell as it is
            add_neg_quot<NEQ>(own, rhs0, rad);
        }
    }
    __device__ __forceinline__ void send(int t, const int4 &m, uint32_t bar, int n) const {
        R o[NEQ];
#pragma unroll
        for (int e = 0; e < NEQ; ++e) o[e] = R(own[e]);
        const int p = (m.x + t) & (kChainRing - 1);
        if constexpr (!CL) {
            R *to = ring + p * kStride;
#pragma unroll
            for (int e = 0; e < NEQ; ++e) to[e] = o[e];
        } else {
            for (int r = 0; r < n; ++r) {
                const uint32_t a = chain_peer(ringAddr + p * kBytes, r), b = chain_peer(bar, r);
                if constexpr (sizeof(R) == 8) {
                    chain_send(a, o[0], o[1], b);
                    chain_send(a + 16, o[2], o[3], b);
                    chain_send(a + 32, o[4], 0.0, b);
                } else {
                    chain_send(a, o[0], o[1], o[2], o[3], b);
                    chain_send(a + 16, o[4], 0.0f, 0.0f, 0.0f, b);
                }
            }
        }
    }
    __device__ __forceinline__ void store() const {
        const R o[DQR] = {R(own[0]), R(own[1]), R(own[2]), R(own[3]), R(own[4]), R(0), R(0), R(0)};
        st8(A.dq + (size_t)c * DQR, o);
    }
};

template <typename R, bool LOWER, bool CL>
__global__ void __launch_bounds__(kChainThreads, 1) k_chain_ns(KArgs<R> A, ChainPlan P, const R *coef, const double *cells) {
    extern __shared__ __align__(16) unsigned char chain_sm[];
    __shared__ uint64_t bars[kChainGroups];
    __shared__ double2 word[kChainMaxBlocks];
    ChainNs<R, LOWER, CL> body{A, P, coef, cells, reinterpret_cast<R *>(chain_sm), chain_smem(chain_sm)};
    chain_run<CL>(P, bars, word, body);
}

// One sweep of the SA increments (FP64 on both paths): the face matrices come
// straight from the arrays the right-hand side wrote.
template <typename R, bool LOWER, bool CL>
struct ChainSa {
    const KArgs<R> &A;
    const ChainPlan &P;
    const double *mats, *cells;
    double2 *ring;           // [kChainRing]: 16-byte words, as st.async sends them
    uint32_t ringAddr;
    static constexpr uint32_t kBytes = 16;
    int c, ref[kChainPre];
    Divisor diag;
    double own, mat[kChainPre];

    __device__ __forceinline__ void load_edge(int t, const int4 &m, int j, int &rf, double &a) const {
        const long long s = (long long)m.z + (long long)j * m.y + t;
        rf = chain_ld(P.ref + s);
        a = chain_ld(mats + s);
    }
    __device__ __forceinline__ void load(int t, const int4 &m) {
        if (t >= m.y) return;
        c = chain_ld(P.order + m.x + t);
#pragma unroll
        for (int j = 0; j < kChainPre; ++j) {
            ref[j] = kChainNone;
            if (j < m.w) load_edge(t, m, j, ref[j], mat[j]);
        }
        own = chain_ld(cells + m.x + t);
        diag.d = chain_ld(cells + (size_t)A.nCells + m.x + t);
        diag.r = chain_ld(cells + 2 * (size_t)A.nCells + m.x + t);
    }
    __device__ __forceinline__ void apply(int rf, double a, double &rhs0) const {
        double d = ring[max(rf, 0)].x;
        if (P.far && rf < 0 && rf != kChainNone) d = __ldcg(A.dnut + (~rf));
        const double t = rhs0 + a * d;
        rhs0 = rf == kChainNone ? rhs0 : t;
    }
    __device__ __forceinline__ void solve(int t, const int4 &m) {
        double rhs0 = 0.0;
#pragma unroll
        for (int j = 0; j < kChainPre; ++j) apply(ref[j], mat[j], rhs0);
#pragma unroll 1
        for (int j = kChainPre; j < m.w; ++j) {
            int rf;
            double a;
            load_edge(t, m, j, rf, a);
            apply(rf, a, rhs0);
        }
        if (LOWER) {
            const double y = own - rhs0;
            div_by<1>(&y, diag, &own);
        } else if (m.w > 0) {
            add_neg_quot<1>(&own, &rhs0, diag);
        }
    }
    __device__ __forceinline__ void send(int t, const int4 &m, uint32_t bar, int n) const {
        const int p = (m.x + t) & (kChainRing - 1);
        if constexpr (!CL) ring[p].x = own;
        else
            for (int r = 0; r < n; ++r) chain_send(chain_peer(ringAddr + p * kBytes, r), own, 0.0, chain_peer(bar, r));
    }
    __device__ __forceinline__ void store() const { A.dnut[c] = own; }
};

template <typename R, bool LOWER, bool CL>
__global__ void __launch_bounds__(kChainThreads, 1) k_chain_sa(KArgs<R> A, ChainPlan P, const double *mats, const double *cells) {
    extern __shared__ __align__(16) unsigned char chain_sm[];
    __shared__ uint64_t bars[kChainGroups];
    __shared__ double2 word[kChainMaxBlocks];
    ChainSa<R, LOWER, CL> body{A, P, mats, cells, reinterpret_cast<double2 *>(chain_sm), chain_smem(chain_sm)};
    chain_run<CL>(P, bars, word, body);
}

}  // namespace ofg
