// The coordinate MLP's fused passes: networks whose layers fit one pair of
// SMs (every padded width at most 256, the outputs at most 128).
//
// k_mlp_pass takes a tile of 128 rows through every layer, and in training
// back again, without leaving the chip: a cluster of two blocks holds the
// tile's activations in shared memory, each block computes half of a layer's
// columns (tcgen05.mma, FP32 accumulator in tensor memory), applies bias and
// GELU from the accumulator and writes its BF16 half into both blocks' tiles.
// A layer's weights are stored in the order the tensor core reads them (8 x 8
// core matrices), so that a block fetches its half with one cp.async.bulk, one
// layer ahead.  Training keeps each layer's input (BF16) and GELU' (FP32)
// for the way back, in tile images that k_mlp_dw copies the same way.
//
// The same products in the same order as layer-by-layer GEMMs (k_gemm): the
// same bits.  Every wait is bounded; one that runs out sets g_gemm_status and
// the block goes on without waiting or fetching, to the end, where it waits (again
// within the limit) for what it has in flight.
//
// Measured on the 22 -> 6 x 256 -> 4 network.  Prediction of 294,912 rows: 1.25 ms
// with one tile a pair and cluster barriers (a stage of 10,500 cycles: 2,400
// MMA, 6,500 GELU, 1,200 barriers), 0.79 ms with two tiles in flight and
// mbarriers.  A training step of 8,192 rows: k_mlp_pass 72 us, k_mlp_dw 31,
// k_mlp_update 19 (with a launch per layer and pass over FP32 arrays 550 us).
// What bounds the passes is the instruction issue of erff and expf (about 47
// instructions a hidden value forth, 74 in training): 5,100 of the 6,500 cycles;
// the MMAs, 64 cycles each for 8 KB of operands, run behind it.
#pragma once

constexpr int kMlpLayers = 24;                  // layers a fused network may have
constexpr int kMlpWidth = 256, kMlpOut = 128;   // largest padded widths
constexpr int FT = 512;                         // epilogue threads: four warps for each quarter of a tile's rows
constexpr int FS = FT / 128;                    // shares of a result's columns, one per such warp
constexpr int DT = 256;                         // threads of k_mlp_dw
constexpr int TILE_ROWS = 128;
constexpr int ACT_BYTES = TILE_ROWS * kMlpWidth * 2;        // one tile's activations
constexpr int WGT_BYTES = kMlpWidth * kMlpWidth;            // half a layer's weights
constexpr int SMEM_PASS = ACT_BYTES + 2 * WGT_BYTES + 64;   // two of one kind, one of the other; barriers, slot
constexpr int DW_STAGE = 2 * ACT_BYTES / 2;                 // k_mlp_dw: 128 features of both operands' tile images
constexpr int SMEM_DW = DW_STAGE + 32;

// Layer l: [rows x K[l]] -> [rows x N[l]].  Activations and gradients of a
// layer lie as tile images [tile][feature / 8][row][8]; GELU' as
// [tile][column / 16][4][row][4].
struct MlpNet {
    int L, nin, nout;
    int K[kMlpLayers], N[kMlpLayers];
    int woff[kMlpLayers], boff[kMlpLayers];        // into the weights / biases
    long long hoff[kMlpLayers], zoff[kMlpLayers];  // of a layer's input and output-gradient images, one tile's elements
    const bf16 *wf, *wk;                           // weights packed for the way forth and back
    const float *b;
    bf16 *H, *dZ;                                  // training only
    float *G, *rowErr;
    long long tiles;
};

// columns of the first block of a pair: half of them in whole 16s; an output layer's all
__host__ __device__ inline int mlp_half(int n, bool last) { return last ? n : ((n >> 4) + 1) / 2 * 16; }
// element (k, n) of a layer's K x N weights in the two packings
__host__ __device__ inline int mlp_fwd_index(int K, int N, bool last, int k, int n) {
    const int h = mlp_half(N, last), second = n >= h, w = second ? N - h : h, m = n - (second ? h : 0);
    return (second ? K * h : 0) + ((k >> 3) * (w >> 3) + (m >> 3)) * 64 + (k & 7) * 8 + (m & 7);
}
__host__ __device__ inline int mlp_bwd_index(int N, int k, int n) {
    return ((k >> 3) * (N >> 3) + (n >> 3)) * 64 + (k & 7) * 8 + (n & 7);
}

// shared-memory matrix descriptor with K and M / N strides of the core matrices
__device__ __forceinline__ uint64_t mlp_desc(uint32_t addr, uint32_t kstride, uint32_t mnstride) {
    return uint64_t((addr >> 4) & 0x3FFF) | (uint64_t(kstride >> 4) << 16) | (uint64_t(mnstride >> 4) << 32) |
           (uint64_t(1) << 46);
}
__device__ __forceinline__ void mlp_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mlp_bulk(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// generic writes to shared memory of the pair, before the tensor cores read them
__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async.shared::cluster;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t peer_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_peer(uint32_t addr, uint4 v) {
    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z),
                 "r"(v.w)
                 : "memory");
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ uint4 pack8(const float *v) {
    return make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
}

__device__ __forceinline__ void mbar_init_n(uint32_t bar, uint32_t n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(n) : "memory");
}
__device__ __forceinline__ void arrive_cluster(uint32_t bar) {   // an mbarrier of either block
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_wait_cluster(uint32_t bar, uint32_t parity) {
    for (unsigned i = 0; i < WAIT_LIMIT; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}
// arrives on the mbarrier at this place in both blocks once the MMAs issued before are done
__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
        "h"(static_cast<uint16_t>(3))
        : "memory");
}

// After a wait that ran out, within the limit again: the thread's copies in flight
// on the mbarriers full ..., whatever their phase, then its MMAs
__device__ __noinline__ void mlp_drain(uint32_t full, int buffers) {
    for (int k = 0; k < 2 * buffers + 2; ++k) {
        if (k == 2 * buffers) mma_commit(full);
        mbar_wait_cluster(full + 8 * (k / 2 % buffers), k & 1);
    }
}

// where a pass's rows come from
struct MlpRows {
    const float *x, *y;     // samples; y: targets (training), else null
    int64_t n;              // samples
    int rows;               // of this pass
    bool hashed;            // row r of step `step` is sample hash(seed, step, r) mod n; else sample r
    uint64_t seed, step;
    float *out;             // predictions [n][nout]
};

// A block of the pair: sixteen warps that turn accumulators into the next
// layer's operand, and one that fetches weights and issues the MMAs.  Per
// tile in flight two mbarriers: `acc`, both blocks' MMAs of a stage are done
// (each commits to both), so that either tile may be overwritten; `act`, every
// warp of both blocks has written the next operand.  Prediction keeps two tiles
// in flight, the MMAs of one behind the GELUs of the other (grid: any number of
// pairs, pair p takes tiles p, p + pairs, ...); training, one tile a pair, forth
// and back, with the weights of two stages resident instead.
template <bool TRAIN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(FT + 32, 1) k_mlp_pass(MlpNet P, MlpRows R) {
    constexpr int NT = TRAIN ? 1 : 2, WB = 3 - NT;   // tiles in flight, weight buffers
    extern __shared__ __align__(1024) unsigned char sm[];
    const uint32_t act0 = smem_u32(sm), wgt = act0 + NT * ACT_BYTES, bars = wgt + WB * WGT_BYTES;
    const uint32_t full = bars, acc = bars + 8 * WB, act = acc + 8 * NT, slot = act + 8 * NT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();
    if (tid == 0) {
        for (int k = 0; k < WB; ++k) mbar_init(full + 8 * k);
        for (int k = 0; k < NT; ++k) {
            mbar_init_n(acc + 8 * k, 2);
            mbar_init_n(act + 8 * k, 2 * (FT / 32));
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(128 * NT)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_arrive();
    cluster_wait();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(sm + (slot - act0));
    bool ok = true;
    auto wait = [&](uint32_t bar, uint32_t parity) {
        if (ok && !mbar_wait_cluster(bar, parity)) {
            ok = false;
            atomicOr(&g_gemm_status, 1u);
        }
    };
    const int L = P.L, stages = TRAIN ? 2 * L - 1 : L;
    const int tiles = (R.rows + TILE_ROWS - 1) / TILE_ROWS, pairs = gridDim.x >> 1, pair = blockIdx.x >> 1;
    // stage s of a tile: layer s forth, then layers L-1 .. 1 back; this block's columns of its result
    struct Stage { bool fwd, last; int l, kk, nn, h, n0, nt; };
    auto stage = [&](int s) {
        Stage q;
        q.fwd = s < L;
        q.l = q.fwd ? s : 2 * L - 1 - s;
        q.kk = q.fwd ? P.K[q.l] : P.N[q.l];
        q.nn = q.fwd ? P.N[q.l] : P.K[q.l];
        q.last = q.fwd && q.l + 1 == L;
        q.h = mlp_half(q.nn, q.last);
        q.n0 = rank ? q.h : 0;
        q.nt = rank ? q.nn - q.h : q.h;
        return q;
    };
    if (warp == FT / 32) {
        if (lane == 0) {
            auto fetch = [&](int s, int buf) {
                const Stage q = stage(s);
                const bf16 *src = q.fwd ? P.wf + P.woff[q.l] + (rank ? q.kk * q.h : 0)
                                        : P.wk + P.woff[q.l] + (rank ? q.h * q.kk : 0);
                const uint32_t bytes = uint32_t(q.nt) * q.kk * 2;
                mlp_expect(full + 8 * buf, bytes);
                if (bytes) mlp_bulk(wgt + buf * WGT_BYTES, src, bytes, full + 8 * buf);
            };
            uint32_t done = 0, seen[NT] = {};   // stages of all rounds; phases of each tile's barriers
            if (pair < tiles)
                for (int k = 0; k < WB; ++k)
                    if (k < stages) fetch(k, k);
            for (int t0 = pair; t0 < tiles; t0 += NT * pairs)
                for (int s = 0; s < stages; ++s, ++done) {
                    const Stage q = stage(s);
                    const int buf = done % WB;
                    const uint32_t bk = q.fwd ? uint32_t(q.nt) * 16 : 128, bn = q.fwd ? 128 : uint32_t(q.kk) * 16;
                    const uint32_t idesc = instr_desc(q.nt, 0u, q.fwd ? 1u : 0u), b0 = wgt + buf * WGT_BYTES;
                    wait(full + 8 * buf, (done / WB) & 1);
                    int behind = 0;
#pragma unroll
                    for (int t = 0; t < NT; ++t) {
                        if (t0 + t * pairs >= tiles) break;
                        wait(act + 8 * t, seen[t] & 1);
                        ++seen[t];
                        behind = t;
                        if (!ok) continue;
                        tc_fence_after();
                        if (q.nt > 0)
                            for (int j = 0; j < q.kk / 16; ++j)
                                mma_bf16(tmem + 128 * t, mlp_desc(act0 + t * ACT_BYTES + j * 4096, 2048, 128),
                                         mlp_desc(b0 + j * 2 * bk, bk, bn), idesc, j != 0);
                        mma_commit_pair(acc + 8 * t);
                    }
                    // the buffer's next weights, once its last MMAs are done
                    const int next = s + WB;
                    const bool more = next < stages || (!TRAIN && t0 + NT * pairs < tiles);
                    if (more) {
                        wait(acc + 8 * behind, (seen[behind] - 1) & 1);
                        if (__builtin_expect(ok, 1)) fetch(next % stages, buf);
                    }
                }
            if (__builtin_expect(!ok, 0)) mlp_drain(full, WB);
        }
        __syncwarp();
    } else {
        const int row = (warp & 3) * 32 + lane, share = warp >> 2;   // this thread's row of a tile, its share of columns
        const uint32_t peer = peer_addr(act0, rank ^ 1);
        uint32_t seen[NT] = {};
        // the operand is written: to both blocks
        auto signal = [&](int t) {
            fence_async();
            tc_fence_before();
            __syncwarp();
            if (lane < 2) arrive_cluster(peer_addr(act + 8 * t, lane));
        };
        auto sample = [&](int r) {
            if (!R.hashed) return int64_t(r);
            return int64_t(mix64(R.seed ^ mix64(R.step * 0x9e3779b97f4a7c15ULL + uint64_t(r))) % uint64_t(R.n));
        };
        for (int t0 = pair; t0 < tiles; t0 += NT * pairs) {
            // the tiles' inputs (each block its own copy), and in training their image
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const int tile = t0 + t * pairs, r = tile * TILE_ROWS + row;
                if (tile >= tiles) break;
                const bool in = r < R.rows;
                const int64_t s = in ? sample(r) : 0;
                const int K0 = P.K[0];
                for (int kb = share; kb < K0 / 8; kb += FS) {
                    float v[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const int c = kb * 8 + j;
                        v[j] = in && c < P.nin ? __ldg(R.x + s * P.nin + c) : 0.0f;
                    }
                    const uint4 w = pack8(v);
                    *reinterpret_cast<uint4 *>(sm + t * ACT_BYTES + kb * 2048 + row * 16) = w;
                    if (TRAIN && rank == 0)
                        *reinterpret_cast<uint4 *>(P.H + P.hoff[0] * P.tiles + ((size_t)tile * K0 / 8 + kb) * 1024 +
                                                   row * 8) = w;
                }
                signal(t);
            }
            for (int s = 0; s < stages; ++s) {
                const Stage q = stage(s);
                const int l = q.l;
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    const int tile = t0 + t * pairs, r = tile * TILE_ROWS + row;
                    if (tile >= tiles) break;
                    const uint32_t tq = tmem + 128 * t + (uint32_t((warp & 3) * 32) << 16);
                    const bool more = s + 1 < stages;
                    // 8 columns of the result, from c on, into both blocks' operand
                    auto put = [&](int c, uint4 w) {
                        const uint32_t off = t * ACT_BYTES + uint32_t(c >> 3) * 2048 + row * 16;
                        *reinterpret_cast<uint4 *>(sm + off) = w;
                        st_peer(peer + off, w);
                    };
                    auto image_at = [&](bf16 *image, int c) {
                        return reinterpret_cast<uint4 *>(image + ((size_t)tile * q.nn / 8 + (c >> 3)) * 1024 + row * 8);
                    };
                    if (q.last) {
                        // outputs, and in training the gradient of the squared error; the
                        // rows' own warps take every column, in order
                        wait(acc + 8 * t, seen[t]++ & 1);
                        tc_fence_after();
                        if (share == 0 && q.nt > 0) {
                            const int64_t smp = TRAIN && r < R.rows ? sample(r) : 0;
                            float e = 0.0f;
                            for (int c = 0; c < q.nt; c += 16) {
                                uint32_t a[16];
                                __syncwarp();
                                tmem_ld16(tq + uint32_t(c), a);
                                float g[16];
#pragma unroll
                                for (int j = 0; j < 16; ++j) {
                                    const int cc = c + j;
                                    const float y = __uint_as_float(a[j]) + __ldg(P.b + P.boff[l] + cc);
                                    g[j] = 0.0f;
                                    if (TRAIN) {
                                        if (cc < P.nout && r < R.rows) {
                                            const float d = y - __ldg(R.y + smp * P.nout + cc);
                                            e += d * d;
                                            g[j] = 2.0f * d / float(R.rows * P.nout);
                                        }
                                    } else if (cc < P.nout && r < R.rows) {
                                        R.out[(int64_t)r * P.nout + cc] = y;
                                    }
                                }
                                if (TRAIN) {
                                    bf16 *image = P.dZ + P.zoff[l] * P.tiles;
                                    const uint4 w0 = pack8(g), w1 = pack8(g + 8);
                                    put(c, w0);
                                    put(c + 8, w1);
                                    *image_at(image, c) = w0;
                                    *image_at(image, c + 8) = w1;
                                }
                            }
                            if (TRAIN && r < R.rows) P.rowErr[r] = e;
                        }
                        if (more) signal(t);
                        continue;
                    }
                    // hidden columns: at most UN units of 16 a warp; what goes to
                    // global memory goes after the signal
                    constexpr int UN = kMlpWidth / 2 / 16 / FS;
                    float4 g[TRAIN ? UN : 1][4];
                    uint4 w[UN][2];
                    float4 *G = nullptr;
                    auto gat = [&](int u) {
                        return ((size_t)tile * q.nn / 16 + (q.n0 / 16 + u)) * 4 * TILE_ROWS + row;
                    };
                    if (TRAIN) {
                        G = reinterpret_cast<float4 *>(P.G + P.zoff[q.fwd ? l : l - 1] * P.tiles);
                        if (!q.fwd) {   // this thread wrote them on the way forth
#pragma unroll
                            for (int i = 0; i < UN; ++i)
                                if (share + i * FS < q.nt / 16)
#pragma unroll
                                    for (int j = 0; j < 4; ++j) g[i][j] = G[gat(share + i * FS) + j * TILE_ROWS];
                        }
                    }
                    wait(acc + 8 * t, seen[t]++ & 1);
                    tc_fence_after();
#pragma unroll
                    for (int i = 0; i < UN; ++i) {
                        const int u = share + i * FS;
                        if (u >= q.nt / 16) break;
                        uint32_t a[16];
                        __syncwarp();
                        tmem_ld16(tq + uint32_t(u * 16), a);
                        const int c = q.n0 + u * 16;
                        float v[16];
                        if (q.fwd) {
                            float bias[16], gr[16];
#pragma unroll
                            for (int j = 0; j < 16; j += 4)
                                *reinterpret_cast<float4 *>(bias + j) =
                                    __ldg(reinterpret_cast<const float4 *>(P.b + P.boff[l] + c + j));
#pragma unroll
                            for (int j = 0; j < 16; ++j) {
                                const float z = __uint_as_float(a[j]) + bias[j];
                                const float f = erff(z * 0.70710678118654752f);
                                v[j] = gelu_of(z, f);
                                if (TRAIN) gr[j] = gelu_grad_of(z, f);
                            }
                            if (TRAIN) {
#pragma unroll
                                for (int j = 0; j < 4; ++j)
                                    g[i][j] = make_float4(gr[4 * j], gr[4 * j + 1], gr[4 * j + 2], gr[4 * j + 3]);
                            }
                        } else if (TRAIN) {
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                v[4 * j] = __uint_as_float(a[4 * j]) * g[i][j].x;
                                v[4 * j + 1] = __uint_as_float(a[4 * j + 1]) * g[i][j].y;
                                v[4 * j + 2] = __uint_as_float(a[4 * j + 2]) * g[i][j].z;
                                v[4 * j + 3] = __uint_as_float(a[4 * j + 3]) * g[i][j].w;
                            }
                        }
                        w[i][0] = pack8(v);
                        w[i][1] = pack8(v + 8);
                        if (more) {
                            put(c, w[i][0]);
                            put(c + 8, w[i][1]);
                        }
                    }
                    if (more) signal(t);
                    if (TRAIN) {
                        bf16 *image = q.fwd ? P.H + P.hoff[l + 1] * P.tiles : P.dZ + P.zoff[l - 1] * P.tiles;
#pragma unroll
                        for (int i = 0; i < UN; ++i) {
                            const int u = share + i * FS;
                            if (u >= q.nt / 16) break;
                            *image_at(image, q.n0 + u * 16) = w[i][0];
                            *image_at(image, q.n0 + u * 16 + 8) = w[i][1];
                            if (q.fwd) {
#pragma unroll
                                for (int j = 0; j < 4; ++j) G[gat(u) + j * TILE_ROWS] = g[i][j];
                            }
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_arrive();   // no block leaves while the other may still write to it
    cluster_wait();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128 * NT) : "memory");
    }
}

// Weight gradients of every layer, dW = H^T dZ, split over the rows in parts of
// `chunk` (their sums left in part[part][K x N] at offset parts x woff), and the
// bias gradients (column sums of dZ) of every layer.  Blocks: each layer's
// 128 x 128 tiles x parts, then each layer's groups of 8 columns.
struct DwGrid {
    int parts, chunk, rows;
    int first[kMlpLayers + 1];    // first block of each layer's tiles
    int bias[kMlpLayers + 1];     // first block of each layer's column groups
};

__global__ void __launch_bounds__(DT, 3) k_mlp_dw(MlpNet P, DwGrid D, float *part, float *gb) {
    extern __shared__ __align__(1024) unsigned char sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int l = 0;
    if (int(blockIdx.x) >= D.first[P.L]) {
        // column sums, 8 columns a block: a thread's rows in ascending order, then the tree of 256
        while (int(blockIdx.x) >= D.bias[l + 1]) ++l;
        const int cb = blockIdx.x - D.bias[l], N = P.N[l];
        const bf16 *z = P.dZ + P.zoff[l] * P.tiles;
        float a[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = 0.0f;
        for (int r = tid; r < D.rows; r += DT) {
            const uint4 w = *reinterpret_cast<const uint4 *>(z + ((size_t)(r >> 7) * N / 8 + cb) * 1024 + (r & 127) * 8);
            const bf16 *v = reinterpret_cast<const bf16 *>(&w);
#pragma unroll
            for (int j = 0; j < 8; ++j) a[j] += __bfloat162float(v[j]);
        }
        float(*s)[DT] = reinterpret_cast<float(*)[DT]>(sm);
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j][tid] = a[j];
        __syncthreads();
        for (int w = DT / 2; w > 0; w >>= 1) {
            if (tid < w) {
#pragma unroll
                for (int j = 0; j < 8; ++j) s[j][tid] += s[j][tid + w];
            }
            __syncthreads();
        }
        if (tid < 8) gb[P.boff[l] + cb * 8 + tid] = s[tid][0];
        return;
    }
    while (int(blockIdx.x) >= D.first[l + 1]) ++l;
    const int K = P.K[l], N = P.N[l], ct = (N + BN - 1) / BN;
    const int b = blockIdx.x - D.first[l], p = b % D.parts, t = b / D.parts;
    const int m0 = t / ct * BM, n0 = t % ct * BN, mt = min(BM, K - m0), nt = min(BN, N - n0);
    const int k0 = p * D.chunk, k1 = min(D.rows, k0 + D.chunk);
    const uint32_t base = smem_u32(sm), full = base + DW_STAGE, all = full + 8, slot = all + 8;
    if (tid == 0) {
        mbar_init(full);
        mbar_init(all);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(128)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(sm + (slot - base));
    // the part's rows of one tile image after the other; three blocks an SM
    // overlap one another's copies, MMAs and results
    const int t0 = k0 >> 7, segs = ((k1 - 1) >> 7) - t0 + 1;
    bool ok = true;
    if (warp == 0) {
        const uint32_t idesc = instr_desc(nt, 1u, 1u);
        for (int i = 0; i < segs; ++i) {
            const int a = max(k0, (t0 + i) << 7), n = min(k1, (t0 + i + 1) << 7) - a, ra = a & 127;
            const bf16 *A = P.H + P.hoff[l] * P.tiles + ((size_t)(t0 + i) * K / 8 + m0 / 8) * 1024 + ra * 8;
            const bf16 *B = P.dZ + P.zoff[l] * P.tiles + ((size_t)(t0 + i) * N / 8 + n0 / 8) * 1024 + ra * 8;
            if (lane == 0) mlp_expect(full, uint32_t(mt + nt) / 8 * n * 16);
            __syncwarp();
            if (n == 128) {   // a whole image: one copy an operand
                if (lane == 0) mlp_bulk(base, A, mt * 256, full);
                if (lane == 16) mlp_bulk(base + DW_STAGE / 2, B, nt * 256, full);
            } else {          // one copy for each 8 features
                const int f = lane & 15;
                if (lane < 16 && f < mt / 8) mlp_bulk(base + f * 2048, A + f * 1024, n * 16, full);
                if (lane >= 16 && f < nt / 8) mlp_bulk(base + DW_STAGE / 2 + f * 2048, B + f * 1024, n * 16, full);
            }
            ok = __all_sync(0xffffffffu, mbar_wait(full, i & 1));
            if (!ok) {
                mbar_wait(full, i & 1);   // the copies in flight, once more
                break;
            }
            if (lane == 0) {
                tc_fence_after();
                for (int j = 0; j < n / 16; ++j)
                    mma_bf16(tmem, mlp_desc(base + j * 256, 128, 2048),
                             mlp_desc(base + DW_STAGE / 2 + j * 256, 128, 2048), idesc, (i | j) != 0);
                mma_commit(all);
            }
            __syncwarp();
            ok = __all_sync(0xffffffffu, mbar_wait(all, i & 1));   // before the next copies, and the results
            if (!ok) {
                mbar_wait(all, i & 1);
                break;
            }
        }
        if (!ok && lane == 0) atomicOr(&g_gemm_status, 1u);
    }
    __syncthreads();
    __syncwarp();
    tc_fence_after();
    const int m = (warp & 3) * 32 + lane;
    float *out = part + (size_t)D.parts * P.woff[l] + (size_t)p * K * N;
    for (int u = warp >> 2; u < nt / 16; u += 2) {
        uint32_t v[16];
        __syncwarp();
        tmem_ld16(tmem + (uint32_t((warp & 3) * 32) << 16) + uint32_t(u * 16), v);
        if (m < mt) {
            float4 *o = reinterpret_cast<float4 *>(out + (size_t)(m0 + m) * N + n0 + u * 16);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                o[j] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]),
                                   __uint_as_float(v[4 * j + 3]));
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(128) : "memory");
    }
}

// The parts of every weight gradient summed in order; then, for a training
// step, Adam on weights and biases with both packings refreshed, and (one
// block more) the minibatch loss.  gw / gb: the gradients kept (ofg_mlp_loss_grad).
struct AdamStep {
    float lr, b1, b2, eps, c1, c2;
    float *w, *mw, *vw, *b, *mb, *vb;
    bf16 *wf, *wk;
    const unsigned char *wmask, *bmask;
    float *loss;
    double scale;
    int rows;
};

__global__ void __launch_bounds__(256) k_mlp_update(MlpNet P, int nw, int nb, int parts, const float *part, float *gw,
                                                    const float *gb, AdamStep S) {
    const int wblocks = (nw / 4 + 255) / 256, bblocks = (nb + 255) / 256;
    if (int(blockIdx.x) == wblocks + bblocks) {
        batch_loss(S.rows, S.scale, P.rowErr, S.loss);
        return;
    }
    if (int(blockIdx.x) >= wblocks) {
        const int i = (blockIdx.x - wblocks) * 256 + threadIdx.x;
        if (i < nb && S.bmask[i]) adam_step(S.b, S.mb, S.vb, gb[i], i, S.lr, S.b1, S.b2, S.eps, S.c1, S.c2);
        return;
    }
    const int i = 4 * (blockIdx.x * 256 + threadIdx.x);   // four weights of one row
    if (i >= nw) return;
    int l = 0;
    while (l + 1 < P.L && i >= P.woff[l + 1]) ++l;
    const int N = P.N[l], K = P.K[l], j = i - P.woff[l];
    const size_t n = (size_t)K * N;
    const float *q = part + (size_t)parts * P.woff[l] + j;
    float a[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 8
    for (int p = 0; p < parts; ++p) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(q + p * n));
        a[0] += v.x; a[1] += v.y; a[2] += v.z; a[3] += v.w;
    }
    if (gw) {
        *reinterpret_cast<float4 *>(gw + i) = make_float4(a[0], a[1], a[2], a[3]);
        return;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (!S.wmask[i + k]) continue;
        const bf16 w = __float2bfloat16(adam_step(S.w, S.mw, S.vw, a[k], i + k, S.lr, S.b1, S.b2, S.eps, S.c1, S.c2));
        S.wf[P.woff[l] + mlp_fwd_index(K, N, l + 1 == P.L, j / N, j % N + k)] = w;
        S.wk[P.woff[l] + mlp_bwd_index(N, j / N, j % N + k)] = w;
    }
}

// both packings of FP32 weights
__global__ void __launch_bounds__(256) k_mlp_pack(MlpNet P, int nw, const float *w, bf16 *wf, bf16 *wk) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= nw) return;
    int l = 0;
    while (l + 1 < P.L && i >= P.woff[l + 1]) ++l;
    const int N = P.N[l], j = i - P.woff[l];
    const bf16 v = __float2bfloat16(w[i]);
    wf[P.woff[l] + mlp_fwd_index(P.K[l], N, l + 1 == P.L, j / N, j % N)] = v;
    wk[P.woff[l] + mlp_bwd_index(N, j / N, j % N)] = v;
}
