// out[M,N] = act(A[M,K] · W[N,K]ᵀ + bias[N]) + add0[M,N] + add1[M,N]
//
// The plain matrix product: 32-bit FMA on CUDA cores, every element type, every
// size.  It is the whole 32-bit path (no tensor-core mode of reduced precision
// is ever used there) and the product every faster kernel is checked against.
// A row's result does not depend on what else is in the batch: whatever M, N or the
// tile an element falls in, it sums over k in one order (the reference's product is a
// per-row dot, simd.go:188-196).
//
// Two kernels.  32-bit operands with whole 16-byte rows run gemm_f32_kernel (below);
// everything else (16-bit or mixed operands of odd K, unaligned rows) runs
// gemm_simt_kernel, tiles of 64 x 64 with k in ascending order.
#include <cooperative_groups.h>

#include "common.cuh"
#include "tma.cuh"
namespace cg = cooperative_groups;

#define SG_BM 64
#define SG_BN 64
#define SG_BK 16

struct GemmArgs {
    const void* a;        // [M, K]
    const void* w;        // [N, K]
    const float* bias;    // [N] or null
    const float* add0;    // [M, N] or null, 32-bit
    const float* add1;    // [M, N] or null, 32-bit
    void* out;            // [M, N]
    int M, N, K, act;
    // (the rest of the record as the other products read it; only the activation's numbers are used here)
    const void* a2_unused;
    const void* w2_unused;
    const float* bias2_unused;
    int K2_unused;
    const void* wB_unused;
    const float* biasB_unused;
    void* outB_unused;
    int NB_unused, actB_unused;
    const int* group_of_tile_unused;
    int groups_unused;
    float act_p0, act_p1;       // the numbers of an activation that has some (GL_ACT_XIELU)
};

template <typename TA, typename TW, typename TO>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(GemmArgs g) {
    __shared__ float As[SG_BK][SG_BM + 4];
    __shared__ float Ws[SG_BK][SG_BN + 4];
    const TA* A = (const TA*)g.a;
    const TW* W = (const TW*)g.w;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * SG_BM, n0 = blockIdx.x * SG_BN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < g.K; k0 += SG_BK) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = tid + i * 256, r = e >> 4, c = e & 15;
            const int k = k0 + c;
            float va = 0.f, vw = 0.f;
            if (k < g.K) {
                if (m0 + r < g.M) va = gl_load(A + (size_t)(m0 + r) * g.K + k);
                if (n0 + r < g.N) vw = gl_load(W + (size_t)(n0 + r) * g.K + k);
            }
            As[c][r] = va;
            Ws[c][r] = vw;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < SG_BK; ++kk) {
            float av[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) av[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
    TO* O = (TO*)g.out;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= g.M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= g.N) continue;
            float v = acc[i][j];
            if (g.bias) v += g.bias[n];
            v = gl_activate<true>(v, g.act, g.act_p0, g.act_p1);
            const size_t o = (size_t)m * g.N + n;
            if (g.add0) v += g.add0[o];
            if (g.add1) v += g.add1[o];
            gl_store(O + o, v);
        }
    }
}

template <typename TA, typename TW, typename TO>
static int launch_simt(const GemmArgs& g, cudaStream_t stream) {
    dim3 grid((g.N + SG_BN - 1) / SG_BN, (g.M + SG_BM - 1) / SG_BM);
    if (grid.y > 65535) return GL_ERR_SHAPE;
    gemm_simt_kernel<TA, TW, TO><<<grid, 256, 0, stream>>>(g);
    return gl_check_launch();
}

template <typename TA, typename TW>
static int dispatch_out(const GemmArgs& g, int out_dtype, cudaStream_t stream) {
    if (out_dtype == GL_F32) return launch_simt<TA, TW, float>(g, stream);
    if (out_dtype == GL_BF16) return launch_simt<TA, TW, __nv_bfloat16>(g, stream);
    return GL_ERR_DTYPE;
}

// ---------------------------------------------------------------------------
// 32-bit operands.  With many rows the FMA rate bounds it, with few rows the weights'
// way from memory.  Tiles of both operands arrive by TMA (128-byte swizzled rows of 32
// k, several stages ahead; the weights' first ones before the kernel waits for the one
// before it).  Both operands hold k in consecutive words, so the packed FMA takes two k at
// once (even k in one half of the accumulator, odd k in the other) and nothing has to be
// transposed or duplicated; a thread's 8 x 8 elements need 16 shared-memory loads of 16
// bytes for 128 packed FMA, which keeps the load path as busy as the FMA units.
//
// The order of a sum: K is cut into FG_SEGS parts of whole k-blocks; in a part the even
// and the odd k are summed in ascending order and the two added, and the eight parts meet
// in pairs, ((q0 + q1) + (q2 + q3)) + ((q4 + q5) + (q6 + q7)).  A cluster of 1, 2, 4 or 8
// blocks shares a tile's parts, so the cut fills the SMs where tiles are few or their last
// wave is nearly empty, and the result is the same number whichever way it was cut.
//
// Measured with Phi-1.5's products, weights from memory, against gemm_simt_kernel: 632 rows x 8192 x 2048
// 0.98 -> 0.53 ms (40 TFLOP/s), x 2048 x 8192 1.18 -> 0.53 ms; 4 rows x 8192 x 2048 347 -> 24 us (2.9 TB/s),
// x 2048 x 8192 1317 -> 27 us, x 51200 x 2048 840 -> 93 us (4.5 TB/s).
#define FG_BK 32
#define FG_SEGS 8

__device__ __forceinline__ void fg_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float fg_halves(unsigned long long v) {
    return __uint_as_float((unsigned)v) + __uint_as_float((unsigned)(v >> 32));
}

// WM x WN warps of LM x (32 / LM) lanes with TM x TN elements a lane
template <int WM_, int WN_, int LM_, int TM_, int TN_, int STAGES_>
struct FgShape {
    static constexpr int WM = WM_, WN = WN_, LM = LM_, LN = 32 / LM_, TM = TM_, TN = TN_, STAGES = STAGES_;
    static constexpr int BM = WM * LM * TM, BN = WN * LN * TN, THREADS = WM * WN * 32;
    static constexpr int A_ROWS = BM < 8 ? 8 : BM, A_BYTES = A_ROWS * 128, STAGE = A_BYTES + BN * 128, TILE = BM * BN * 4;
    // sums of its own parts that a block puts by, one per level of pairs: 3, 2, 1 or none
    static constexpr size_t smem(int S) { return (size_t)STAGES * STAGE + (S == 1 ? 3 : S == 2 ? 2 : S == 4 ? 1 : 0) * TILE + 1024; }
    static_assert(A_ROWS % 8 == 0 && BN % 8 == 0 && STAGES * STAGE >= TILE, "swizzled tiles, and room for the last exchange");
};

template <typename SH, typename TO>
__global__ void __launch_bounds__(SH::THREADS)
gemm_f32_kernel(GemmArgs g, const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w) {
    extern __shared__ unsigned char smem_raw[];
    constexpr int LM = SH::LM, LN = SH::LN, TM = SH::TM, TN = SH::TN, STAGES = SH::STAGES, BM = SH::BM, BN = SH::BN;
    constexpr int ROWS = TN >= 8 ? 1 : (8 / TN < TM ? 8 / TN : TM);         // rows taken together: eight products before one that waits for an earlier one
    cg::cluster_group cluster = cg::this_cluster();
    const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = (int)blockIdx.y * BM, n0 = ((int)blockIdx.x / S) * BN;     // (columns on the grid's long side)
    unsigned char* smem = smem_raw + ((1024u - (gl_smem_u32(smem_raw) & 1023u)) & 1023u);
    const unsigned base = gl_smem_u32(smem);
    __shared__ alignas(8) unsigned long long bars[2 * STAGES];
    const unsigned bar_full = gl_smem_u32(bars), bar_empty = bar_full + 8 * STAGES;
    const int k_blocks = (g.K + FG_BK - 1) / FG_BK, seg_blocks = (k_blocks + FG_SEGS - 1) / FG_SEGS;
    const int segs = FG_SEGS / S;                                             // parts this block sums
    const int kb0 = min(rank * segs * seg_blocks, k_blocks), kb1 = min(kb0 + segs * seg_blocks, k_blocks);

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(bar_full + 8 * s, 1); mbar_init(bar_empty + 8 * s, SH::THREADS / 32); }
        mbar_fence_init();
    }
    __syncthreads();
    gl_grid_launch_dependents();
    auto load_w = [&](int it) {
        const unsigned bar = bar_full + 8 * (it % STAGES);
        mbar_expect_tx(bar, SH::STAGE);                                       // the rows' tile counts too
        tma_load_2d(base + (it % STAGES) * SH::STAGE + SH::A_BYTES, &map_w, (kb0 + it) * FG_BK, n0, bar);
    };
    auto load_a = [&](int it) {
        tma_load_2d(base + (it % STAGES) * SH::STAGE, &map_a, (kb0 + it) * FG_BK, m0, bar_full + 8 * (it % STAGES));
    };
    const int iters = kb1 - kb0;
    // the bias of the column this thread finishes: asked for before the wait, not behind the sums
    constexpr int BATCH = 8;
    static_assert(BN <= SH::THREADS && SH::THREADS % BN == 0, "a thread finishes one column");
    const int my_n = n0 + rank * (BN / S) + (tid & (BN / S - 1));
    const float my_bias = g.bias && my_n < g.N ? g.bias[my_n] : 0.f;
    if (tid == 0)
        for (int it = 0; it < STAGES && it < iters; ++it) load_w(it);
    gl_grid_wait();
    if (tid == 0)
        for (int it = 0; it < STAGES && it < iters; ++it) load_a(it);

    // lanes next to each other take rows next to each other: the swizzle then spreads a load over all banks
    const int lm = lane / LN, ln = lane % LN;
    const int mrow = (warp / SH::WN) * (LM * TM) + lm, nrow = (warp % SH::WN) * (LN * TN) + ln;
    const unsigned a_off = mrow * 128, w_off = SH::A_BYTES + nrow * 128;
    unsigned long long acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0;
    // a part put by: element (m, n) of the tile, columns swizzled so that the rows of a warp do not meet in a bank
    auto at = [&](int i, int j) { const int m = mrow + LM * i, n = nrow + LN * j; return m * BN + (n ^ ((m & 3) << 3)); };
    float* put = (float*)(smem + STAGES * SH::STAGE);
    // the part in the accumulators, joined with the sums put by on the levels of pairs in ``levels``, to level ``to``
    auto put_by = [&](int levels, float* to) {
        float q[TM][TN];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) { q[i][j] = fg_halves(acc[i][j]); acc[i][j] = 0; }
        for (int l = 0; levels >> l; ++l)
            if ((levels >> l) & 1) {
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) q[i][j] = put[at(i, j) + l * (BM * BN)] + q[i][j];
            }
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int j = 0; j < TN; ++j) to[at(i, j)] = q[i][j];
    };
    // (parts behind the end of K are zeros: nothing changes where they are left out)
    const int last = iters > 0 ? (iters - 1) / seg_blocks : 0;

    int it = 0;
    bool ok = true;
    for (int seg = 0; seg <= last; ++seg) {
        const int stop = min((seg + 1) * seg_blocks, iters);
        for (; it < stop && ok; ++it) {
            if (tid == 0 && it > 0 && it - 1 + STAGES < iters) {              // refill the stage all have left behind
                ok = mbar_wait(bar_empty + 8 * ((it - 1) % STAGES), ((it - 1) / STAGES) & 1);
                if (ok) { load_w(it - 1 + STAGES); load_a(it - 1 + STAGES); }
            }
            ok = ok && mbar_wait(bar_full + 8 * (it % STAGES), (it / STAGES) & 1);
            ok = __all_sync(0xffffffffu, ok);
            const unsigned char *sa = smem + (it % STAGES) * SH::STAGE + a_off, *sw = smem + (it % STAGES) * SH::STAGE + w_off;
#pragma unroll
            for (int c = 0; c < FG_BK / 4; ++c) {
                ulonglong2 w[TN];
#pragma unroll
                for (int j = 0; j < TN; ++j) w[j] = *(const ulonglong2*)(sw + j * (LN * 128) + ((c ^ ((nrow + LN * j) & 7)) << 4));
#pragma unroll
                for (int i0 = 0; i0 < TM; i0 += ROWS) {
                    ulonglong2 a[ROWS];
#pragma unroll
                    for (int i = 0; i < ROWS; ++i) a[i] = *(const ulonglong2*)(sa + (i0 + i) * (LM * 128) + ((c ^ ((mrow + LM * (i0 + i)) & 7)) << 4));
#pragma unroll
                    for (int i = 0; i < ROWS; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) fg_fma2(acc[i0 + i][j], a[i].x, w[j].x);
#pragma unroll
                    for (int i = 0; i < ROWS; ++i)
#pragma unroll
                        for (int j = 0; j < TN; ++j) fg_fma2(acc[i0 + i][j], a[i].y, w[j].y);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_empty + 8 * (it % STAGES));
        }
        if (seg < last) put_by(seg & ~(seg + 1), put + (__ffs(seg + 1) - 1) * (BM * BN));      // what pairs with it so far
    }
    // a wait that ran out: the copies still on their way must not land in memory that is used for something else by then
    if (tid == 0 && !ok)
        for (int i = it - 1; i < min(iters, it - 1 + STAGES); ++i) mbar_wait(bar_full + 8 * (i % STAGES), (i / STAGES) & 1);
    // the block's sum over its parts, where the cluster can read it
    float* tile = S == FG_SEGS ? (float*)smem : put;
    __syncthreads();                                                          // (the stages are free now)
    put_by(last, tile);
    cluster.sync();
    // each block finishes its share of the tile's columns
    const int log_cols = __ffs(BN / S) - 1, cols = 1 << log_cols, total = min(BM, g.M - m0) << log_cols;
    const float* part[FG_SEGS];
#pragma unroll
    for (int s = 0; s < FG_SEGS; ++s) part[s] = s < S ? cluster.map_shared_rank(tile, s) : nullptr;
    TO* O = (TO*)g.out;
    for (int e0 = tid; e0 < total; e0 += BATCH * SH::THREADS) {
        float v[BATCH], a0[BATCH], a1[BATCH];
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {                                     // everything asked for before anything is stored
            const int e = e0 + u * SH::THREADS, m = e >> log_cols, nl = rank * cols + (e & (cols - 1)), n = n0 + nl;
            v[u] = a0[u] = a1[u] = 0.f;
            if (e < total && n < g.N) {
                const int x = m * BN + (nl ^ ((m & 3) << 3));
                const size_t o = (size_t)(m0 + m) * g.N + n;
                if (g.add0) a0[u] = g.add0[o];
                if (g.add1) a1[u] = g.add1[o];
                float q[FG_SEGS];
#pragma unroll
                for (int s = 0; s < FG_SEGS; ++s) q[s] = s < S ? part[s][x] : 0.f;
                v[u] = q[0];
                if (S > 1) v[u] += q[1];
                if (S > 2) v[u] += q[2] + q[3];
                if (S > 4) v[u] += (q[4] + q[5]) + (q[6] + q[7]);
            }
        }
#pragma unroll
        for (int u = 0; u < BATCH; ++u) {
            const int e = e0 + u * SH::THREADS, m = e >> log_cols, n = n0 + rank * cols + (e & (cols - 1));
            if (e < total && n < g.N) {
                float r = v[u];
                if (g.bias) r += my_bias;
                r = gl_activate<true>(r, g.act, g.act_p0, g.act_p1);
                if (g.add0) r += a0[u];
                if (g.add1) r += a1[u];
                gl_store(O + (size_t)(m0 + m) * g.N + n, r);
            }
        }
    }
    cluster.sync();                                                           // nobody leaves while a peer may read its tile
}

template <typename SH, typename TO>
static int launch_f32(const GemmArgs& g, cudaStream_t stream) {
    // clusters of S blocks that run at once, on each device (a kernel's shared memory is allowed device by device)
    struct AtOnce { int n[FG_SEGS + 1] = {}; };
    static std::unordered_map<int, AtOnce> devices;
    static std::mutex mu;
    const long tiles_n = ((long)g.N + SH::BN - 1) / SH::BN, tiles_m = ((long)g.M + SH::BM - 1) / SH::BM;
    if (tiles_m > 65535) return GL_ERR_SHAPE;
    int dev = 0, at_once[FG_SEGS + 1];
    if (cudaGetDevice(&dev) != cudaSuccess) return GL_ERR_LAUNCH;
    {
        std::lock_guard<std::mutex> lock(mu);
        AtOnce& known = devices[dev];
        if (!known.n[1]) {
            if (cudaFuncSetAttribute(gemm_f32_kernel<SH, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SH::smem(1)) != cudaSuccess) {
                cudaGetLastError();
                return GL_ERR_SMEM;
            }
            for (int S = FG_SEGS; S >= 1; S /= 2) {
                cudaLaunchConfig_t cfg = {};
                cfg.gridDim = dim3(S, 1, 1);
                cfg.blockDim = dim3(SH::THREADS, 1, 1);
                cfg.dynamicSmemBytes = SH::smem(S);
                cudaLaunchAttribute attr[1];
                attr[0].id = cudaLaunchAttributeClusterDimension;
                attr[0].val.clusterDim.x = S;
                attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
                cfg.attrs = attr;
                cfg.numAttrs = 1;
                int n = 0;
                if (cudaOccupancyMaxActiveClusters(&n, gemm_f32_kernel<SH, TO>, &cfg) != cudaSuccess || n < 1) { cudaGetLastError(); n = 1; }
                known.n[S] = n;
            }
        }
        memcpy(at_once, known.n, sizeof(at_once));
    }
    CUtensorMap map_a, map_w;
    int rc = gl_cached_map(&map_a, g.a, (uint64_t)g.M, (uint64_t)g.K, SH::A_ROWS, FG_BK, 4);
    if (rc != GL_OK) return rc;
    rc = gl_cached_map(&map_w, g.w, (uint64_t)g.N, (uint64_t)g.K, SH::BN, FG_BK, 4);
    if (rc != GL_OK) return rc;
    // Blocks a tile: the waves of clusters, each as long as a block's k-blocks; meeting in a cluster costs about as
    // much as FG_MEET of them (a barrier over the SMs and the peers' shared memory), so short products are not cut.
    const long k_blocks = (g.K + FG_BK - 1) / FG_BK, seg_blocks = (k_blocks + FG_SEGS - 1) / FG_SEGS;
    const long n_tiles = tiles_n * tiles_m, FG_MEET = SH::THREADS > 32 ? 2 : 4;
    int S = 1;
    long best = -1;
    for (int s = 1; s <= FG_SEGS; s *= 2) {
        const long mine = s == FG_SEGS ? seg_blocks : (FG_SEGS / s) * seg_blocks;
        const long waves = (n_tiles + at_once[s] - 1) / at_once[s];
        const long cost = waves * ((mine < k_blocks ? mine : k_blocks) + (s > 1 ? FG_MEET : 0));
        if (best < 0 || cost < best) { best = cost; S = s; }
    }
    if (gl_launch(gemm_f32_kernel<SH, TO>, dim3((unsigned)(S * tiles_n), (unsigned)tiles_m), dim3(SH::THREADS), SH::smem(S), stream, S, g, map_a, map_w) != 0)
        return GL_ERR_LAUNCH;
    return GL_OK;
}

// The same sums with the loop of gemm_simt_kernel: blocks of 256 threads, several an SM, no copies ahead, 64 x 64 results.
// For short K with many tiles, where a block of gemm_f32_kernel (one an SM, its shared memory being mostly stages and sums
// put by) spends more on starting and finishing a tile than on its few k-blocks.  Even and odd k, parts and pairs of parts as
// there, so a row is the same number from either.  Sums of one and of two parts wait in shared memory (in registers they
// would cost one of four blocks an SM); with more than four parts (TOP) those of four wait in registers and three blocks fit
// (four, with the registers spilled or three quarters of them in shared memory, took 3 to 13 % longer).
template <typename TO, bool TOP>
__global__ void __launch_bounds__(256, TOP ? 3 : 4)
gemm_f32_short_kernel(GemmArgs g) {
    extern __shared__ float put[];                     // [levels that wait here][16][256], a thread's own place
    __shared__ float As[SG_BK][SG_BM + 4];
    __shared__ float Ws[SG_BK][SG_BN + 4];
    const float *A = (const float*)g.a, *W = (const float*)g.w;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * SG_BM, n0 = blockIdx.x * SG_BN;
    const int k_blocks = (g.K + FG_BK - 1) / FG_BK, part = (k_blocks + FG_SEGS - 1) / FG_SEGS * FG_BK;
    float acc[2][4][4], top[TOP ? 16 : 1];
    auto clear = [&]() {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[0][i][j] = acc[1][i][j] = 0.f;
    };
    // the finished part, joined with the sums that wait on the levels of pairs in ``levels``
    auto joined = [&](int levels, int i, int j) {
        float q = acc[0][i][j] + acc[1][i][j];
        const int at = (i * 4 + j) * 256 + tid;
        if (levels & 1) q = put[at] + q;
        if (levels & 2) q = put[16 * 256 + at] + q;
        if (TOP && (levels & 4)) q = top[TOP ? i * 4 + j : 0] + q;
        return q;
    };
    clear();
    int seg = 0;
    for (int k_at = 0;; k_at += part, ++seg) {
        const int stop = min(k_at + part, g.K);
        for (int k0 = k_at; k0 < stop; k0 += SG_BK) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int e = tid + i * 256, r = e >> 4, c = e & 15;
                const int k = k0 + c;
                float va = 0.f, vw = 0.f;
                if (k < g.K) {
                    if (m0 + r < g.M) va = A[(size_t)(m0 + r) * g.K + k];
                    if (n0 + r < g.N) vw = W[(size_t)(n0 + r) * g.K + k];
                }
                As[c][r] = va;
                Ws[c][r] = vw;
            }
            __syncthreads();
#pragma unroll
            for (int kk = 0; kk < SG_BK; ++kk) {
                float av[4], wv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) av[i] = As[kk][ty * 4 + i];
#pragma unroll
                for (int j = 0; j < 4; ++j) wv[j] = Ws[kk][tx * 4 + j];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[kk & 1][i][j] = fmaf(av[i], wv[j], acc[kk & 1][i][j]);
            }
            __syncthreads();
        }
        if (stop == g.K) break;
        const int levels = seg & ~(seg + 1);           // what pairs with the part so far: it waits on the next level
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float q = joined(levels, i, j);
                if (levels == 0) put[(i * 4 + j) * 256 + tid] = q;
                else if (levels == 1) put[(16 + i * 4 + j) * 256 + tid] = q;
                else if (TOP) top[TOP ? i * 4 + j : 0] = q;
            }
        clear();
    }
    TO* O = (TO*)g.out;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= g.M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= g.N) continue;
            float v = joined(seg, i, j);
            if (g.bias) v += g.bias[n];
            v = gl_activate<true>(v, g.act, g.act_p0, g.act_p1);
            const size_t o = (size_t)m * g.N + n;
            if (g.add0) v += g.add0[o];
            if (g.add1) v += g.add1[o];
            gl_store(O + o, v);
        }
    }
}

template <typename TO>
static int launch_f32_short(const GemmArgs& g, cudaStream_t stream) {
    const int k_blocks = (g.K + FG_BK - 1) / FG_BK, seg_blocks = (k_blocks + FG_SEGS - 1) / FG_SEGS, parts = (k_blocks + seg_blocks - 1) / seg_blocks;
    const dim3 grid((g.N + SG_BN - 1) / SG_BN, (g.M + SG_BM - 1) / SG_BM);
    if (grid.y > 65535) return GL_ERR_SHAPE;
    const size_t smem = (size_t)(parts > 2 ? 2 : parts > 1 ? 1 : 0) * 16 * 256 * sizeof(float);
    if (parts > 4) gemm_f32_short_kernel<TO, true><<<grid, 256, smem, stream>>>(g);
    else gemm_f32_short_kernel<TO, false><<<grid, 256, smem, stream>>>(g);
    return gl_check_launch();
}

static int fg_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 148;
}

// Rows of a tile: as few as hold all rows, since up to about 20 rows the weights' stream is the longer of the two and
// beyond that every padded row costs FMA time.  The few rows' blocks are a warp each, so that enough of them fit an SM to
// keep both the weights' stream and the FMA units busy.  From 33 rows on tiles of 64 x 128, whose shared-memory loads
// are half as many a product as those of 32 x 64 (632 rows x 8192 x 2048: 40 against 22 TFLOP/s), unless the product is
// too small to occupy the SMs with them: then a tile's own start and finish count (80 rows x 256 x 64: 24 us against 16).
// Short K with many tiles: gemm_f32_short_kernel.  us with the TMA tiles / with it: 2,048 rows x 8192 x 32 230 / 78, x 64
// 263 / 119, x 128 326 / 205, x 192 391 / 326, x 256 456 / 422, x 384 547 / 584; 632 x 2048 x 128 28 / 26; 200 x 4096 x 128
// 20 / 22; 200 x 8192 x 256 64 / 80 (512 tiles of 64 x 64).  Below 64 also with few tiles: there is a k-block or two to fetch
// ahead (64 x 2048 x 32 9.3 / 7.9, x 64 10.5 / 11.8).
template <typename TO>
static int dispatch_f32(const GemmArgs& g, cudaStream_t stream) {
    if (g.M <= 4) return launch_f32<FgShape<1, 1, 1, 4, 1, 5>, TO>(g, stream);
    if (g.M <= 8) return launch_f32<FgShape<1, 1, 1, 8, 1, 5>, TO>(g, stream);
    if (g.M <= 16) return launch_f32<FgShape<1, 1, 2, 8, 2, 4>, TO>(g, stream);
    const long short_tiles = (long)((g.M + SG_BM - 1) / SG_BM) * ((g.N + SG_BN - 1) / SG_BN);
    if (g.K < 64 || (g.K <= 128 && short_tiles >= 256) || (g.K <= 256 && short_tiles >= 1024)) return launch_f32_short<TO>(g, stream);
    const long big_tiles = (long)((g.M + 63) / 64) * ((g.N + 127) / 128), k_blocks = (g.K + FG_BK - 1) / FG_BK;
    if (g.M <= 32 || big_tiles * k_blocks < 8 * fg_sms()) return launch_f32<FgShape<1, 2, 4, 8, 4, 4>, TO>(g, stream);
    return launch_f32<FgShape<2, 2, 4, 8, 8, 3>, TO>(g, stream);
}

GL_API int gl_gemm_simt(const GemmArgs* args, int a_dtype, int w_dtype, int out_dtype, cudaStream_t stream) {
    const GemmArgs& g = *args;
    if (g.M <= 0 || g.N <= 0) return GL_OK;
    if (g.K <= 0) return GL_ERR_SHAPE;
    if (a_dtype == GL_F32 && w_dtype == GL_F32 && g.K % 4 == 0 && (((uintptr_t)g.a | (uintptr_t)g.w) & 15) == 0) {
        if (out_dtype == GL_F32) return dispatch_f32<float>(g, stream);
        if (out_dtype == GL_BF16) return dispatch_f32<__nv_bfloat16>(g, stream);
    }
    if (a_dtype == GL_F32 && w_dtype == GL_F32) return dispatch_out<float, float>(g, out_dtype, stream);
    if (a_dtype == GL_BF16 && w_dtype == GL_BF16) return dispatch_out<__nv_bfloat16, __nv_bfloat16>(g, out_dtype, stream);
    if (a_dtype == GL_BF16 && w_dtype == GL_F32) return dispatch_out<__nv_bfloat16, float>(g, out_dtype, stream);
    if (a_dtype == GL_F32 && w_dtype == GL_BF16) return dispatch_out<float, __nv_bfloat16>(g, out_dtype, stream);
    return GL_ERR_DTYPE;
}
