// Mixers that carry a fixed-size state from token to token instead of a growing cache:
// matrix memories with outer-product updates (an exponentially gated one with a normaliser and a
// running maximum, and one whose per-channel forget gate also sets what is written) and the short
// causal convolution (the selective state-space scan behind it is in selective_scan.cu, the memories'
// walk over long runs in memory_chunks.cu).
//
// A step brings, for every sequence of the batch, a run of one or more tokens; the state of a
// sequence lives in its row of a 32-bit table (row = the sequence's slot), is read when the run
// starts and written back when it ends, so a prompt gives the same result whole, in pieces or token
// by token.  Everything that enters a recurrence (gates, decays, step sizes, the state itself) is
// 32-bit; the projections that feed it arrive in the activation type.
//
// The scans walk a run's tokens in order.  Work is spread over what is independent: sequences,
// heads and the columns of a memory (or the channels of the scan); a thread keeps its part of the
// state in registers for the whole run, and the tokens' inputs are staged in shared memory a few
// tokens at a time.
#include "common.cuh"
#include "recurrent_common.cuh"

#define MS_THREADS 256     // the matrix memories' blocks

// ---------------------------------------------------------------------------
// Matrix memories.  Per head a state S [D, V]; a token's output is S^T q.
//   kind 0, gated with a normaliser: log gates gi = cap tanh(i/cap), gf = logsigmoid(cap tanh(f/cap));
//       m' = max(gf + m, gi);  S' = e^(gf+m-m') S + e^(gi-m') k v^T;  n' likewise with k alone;
//       o = S'^T q / (max(|n'.q|, e^(-m')) + 1e-6).     m starts at 0 (a zeroed state row).
//   kind 1, forget gate with a lower bound: f = l + (1-l) sigmoid(fpre) per row;
//       S' = diag(f) S + (1-f) v^T;  o = S'^T q,  q = silu(qpre).
//   kind 2, gated delta rule: q and k (shared by H / KVH heads) brought to unit length, x / sqrt(sum x^2 + 1e-6),
//       q times q_scale; beta = sigmoid(b), g = e^(-e^(A_log) softplus(a + dt_bias)) per head, from a second
//       tensor of projections (``gates``: b at column i_off + h, a at f_off + h);
//       S <- g S;  u = beta (v - S^T k);  S' = S + k u^T;  o = S'^T q.
//   kind 3, plain decay: S' = keep S + take k v^T;  o = S'^T q + skip_h v.  q and k (shared by H / KVH heads) may be
//       rotated by the token's position first (the first 2 rot_half dims of a head, dim i paired with i + rot_half,
//       cosines and sines [T, rot_half] of the step's tokens) and are then scaled by q_scale and k_scale.  The
//       decay is fixed per head (keep = lower[h], take = 1: retention) or follows a step size from a second tensor
//       of projections (``gates``, column f_off + h): dt = softplus(x + dt_bias[h]), keep = e^(-e^(A_log[h]) dt),
//       take = dt (a state-space layer with a scalar decay per head, whose B, x, C are this memory's k, v, q).
// State row: S [H, D, V], then for kind 0 n [H, D] and m [H].  Every block of a head's columns reads n and m
// when it starts, and blocks of one head may run one after the other, so the new n and m go to a scratch
// [B, H, D + 1] first and a second kernel moves them into the rows once all blocks are done.
// ---------------------------------------------------------------------------
struct MemoryScanArgs {
    const void* proj;         // [T, ld] activation type: the joined projections of the step's tokens
    float* out;               // [T, H*V] 32-bit
    float* state;             // [slots, state_stride]
    const float* lower;       // kind 1: [H*D] lower bounds of the forget gate
    const int* seq_slot;      // [B]
    const int* seq_qstart;    // [B]
    const int* seq_qlen;      // [B]
    int ld, q_off, k_off, v_off, i_off, f_off;
    int B, H, D, V, state_stride, kind;
    float cap, q_scale;
    float* nm_next;           // kind 0: [B, H, D + 1] scratch for the new normaliser and maximum
    // kind 2:
    const void* gates;        // [T, gates_ld] activation type: the projections behind beta and the decay
    const float* a_log;       // [H]
    const float* dt_bias;     // [H]
    int gates_ld, KVH;        // KVH: heads of q and k (each shared by H / KVH heads of v)
    int rows_per_thread;      // 0: chosen by the grid's size; else 32, 8, 4, 2 or 1 (for measurements)
    // kind 3:
    const float* cosv;        // [T, rot_half] or null: q and k are rotated by the token's position
    const float* sinv;
    int rot_half;
    float k_scale;            // multiplies k after the rotation
    const float* d_skip;      // [H] or null: o += d_skip[h] * v
};

// FULL: D == R * DPT and D a multiple of 4, so a thread's rows are DPT / 4 groups of four consecutive ones read
// as float4 and no row needs a bounds check.
// Blocks an SM, stated: left to itself the compiler gives some of these kernels half as many registers or twice as many
// depending on what else the file holds.  Chosen by time, each kind with 1 to 64 sequences of 1, 37 and 120 tokens and seven
// sizes from 16 x 16 x 16 to 32 x 128 x 128: the bounded forget's eight whole rows want a fourth block for their last wave (4 x
// 120 tokens of 32 x 128 x 128: 304 us with three, 230), the delta rule few blocks and all the registers its longer token takes,
// one or two rows of it in 32 bits excepted (1 x 37 tokens of 16 x 64 x 64 in bfloat16: 25.6 us with three, 20.5), the gated kind's
// eight rows three (one token of 16 sequences took 13 % longer with two).  The plain decay's four rows keep four (4 x 100 tokens of
// 8 x 128 x 256 in 32 bits 120 us, 155 with three), though where the grid is smaller than the machine they lose to more
// registers (4 x 100 of 4 x 128 x 128: 56 us, 51 in an earlier build).
__host__ __device__ constexpr int ms_blocks(int bytes, int dpt, int kind, bool full) {
    if (dpt >= 32) return 1;
    if (kind == 2) return bytes == 2 || dpt >= 4 ? 2 : 3;
    if (kind == 1 && full) return 4;
    return dpt >= 8 ? 3 : 4;
}
template <typename TA, int DPT, int KIND, bool FULL>
__global__ void __launch_bounds__(MS_THREADS, ms_blocks(sizeof(TA), DPT, KIND, FULL))
memory_scan_kernel(MemoryScanArgs a, int R, int CH) {
    extern __shared__ __align__(16) float smem[];
    // (launched in order, not early: placed beside the kernel before, the blocks of a scan sat several to an SM
    // for its whole length, and a prompt of 2,048 tokens took 25 ms instead of 16)
    gl_grid_wait();
    const int D = a.D, V = a.V, H = a.H;
    const int CT = MS_THREADS / R;                    // columns of a block
    const int b = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * CT;
    const int r = threadIdx.x % R, c = threadIdx.x / R;
    const int col = col0 + c;
    const bool live = col < V;
    const int qlen = a.seq_qlen[b], qstart = a.seq_qstart[b];
    float* qs = smem;                                 // [CHUNK][D]
    float* ks = qs + CH * D;                    // [CHUNK][D]   kind 0: k;  kind 1: f
    float* vs = ks + CH * D;                    // [CHUNK][CT]
    float* gs = vs + CH * CT;                   // [CHUNK][4]   kind 0: gi, gf, then keep, take; [.][3] reused
    float* es = gs + CH * 4;                    // [CHUNK]      kind 0: e^(-m')

    const int kh = (KIND == 2 || KIND == 3) ? h / (H / a.KVH) : h;   // the head of q and k this head reads
    float* srow = a.state + (size_t)a.seq_slot[b] * a.state_stride;
    float* S_g = srow + (size_t)h * D * V;
    const float* n_g = srow + (size_t)H * D * V + (size_t)h * D;
    const float* m_g = srow + (size_t)H * D * V + (size_t)H * D + h;
    float S[DPT], n[DPT];
#pragma unroll
    for (int i = 0; i < DPT; ++i) {
        const int d = FULL ? ((((i >> 2) * R + r) << 2) + (i & 3)) : r + R * i;
        S[i] = (live && d < D) ? S_g[(size_t)d * V + col] : 0.f;
        n[i] = (KIND == 0 && d < D) ? n_g[d] : 0.f;
    }
    float m = KIND == 0 ? *m_g : 0.f;                 // only thread 0 keeps it current
    float* out_col = a.out + (size_t)qstart * H * V + (size_t)h * V + (live ? col : 0);
    float pending = 0.f;                              // kind 2: a token's read-out before its lanes are summed

    // The delta rule's inputs in bfloat16, rows of whole 16-byte units: a chunk's q, k, v and gate inputs are
    // asked for as 16-byte pieces while the chunk before is still being walked (they wait in registers), so that
    // a chunk's trip to memory does not stand between two walks.  (Fetched two bytes at a time behind the walk,
    // the staging of 32 tokens took longer than walking them.)
    constexpr int PIECES = 3;                         // CH * D <= 5120: at most 640 pieces of 8 for 256 threads
    const bool fast = KIND == 2 && sizeof(TA) == 2 && (a.ld % 8 == 0) && (a.q_off % 8 == 0) && (a.k_off % 8 == 0) &&
                      (a.v_off % 8 == 0) && (D % 8 == 0) && (V % 8 == 0) && (((uintptr_t)a.proj & 15) == 0) &&
                      CH * D <= PIECES * 8 * MS_THREADS;
    uint4 rq[PIECES], rk[PIECES], rv = make_uint4(0, 0, 0, 0);
    float rb = 0.f, ra = 0.f;
    auto fetch = [&](int s0) {
        const int ns = min(CH, qlen - s0), d8n = D / 8;
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const int e = threadIdx.x + i * MS_THREADS;
            if (e < ns * d8n) {
                const int s = e / d8n, d8 = (e - s * d8n) * 8;
                const TA* row = (const TA*)a.proj + (size_t)(qstart + s0 + s) * a.ld;
                rq[i] = *(const uint4*)(row + a.q_off + kh * D + d8);
                rk[i] = *(const uint4*)(row + a.k_off + kh * D + d8);
            }
        }
        const int c8n = CT / 8;
        if ((int)threadIdx.x < ns * c8n) {
            const int s = threadIdx.x / c8n, j8 = (threadIdx.x - s * c8n) * 8;
            const TA* row = (const TA*)a.proj + (size_t)(qstart + s0 + s) * a.ld;
            rv = col0 + j8 < V ? *(const uint4*)(row + a.v_off + h * V + col0 + j8) : make_uint4(0, 0, 0, 0);
        }
        if ((int)threadIdx.x < ns) {
            const TA* row = (const TA*)a.gates + (size_t)(qstart + s0 + threadIdx.x) * a.gates_ld;
            rb = gl_load(row + a.i_off + h);
            ra = gl_load(row + a.f_off + h);
        }
    };
    auto spread = [](const uint4& r, float* dst) {
        const __nv_bfloat162* p2 = (const __nv_bfloat162*)&r;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(p2[i]);
            dst[2 * i] = f.x;
            dst[2 * i + 1] = f.y;
        }
    };
    auto stash = [&](int ns) {
        const int d8n = D / 8, c8n = CT / 8;
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const int e = threadIdx.x + i * MS_THREADS;
            if (e < ns * d8n) {
                spread(rq[i], qs + e * 8);
                spread(rk[i], ks + e * 8);
            }
        }
        if ((int)threadIdx.x < ns * c8n) spread(rv, vs + threadIdx.x * 8);
        if ((int)threadIdx.x < ns) {
            gs[threadIdx.x * 4 + 0] = rc_sigmoid(rb);
            gs[threadIdx.x * 4 + 1] = rc_decay(-expf(a.a_log[h]) * rc_softplus(ra + a.dt_bias[h]));
        }
    };
    if (fast && qlen > 0) fetch(0);

    for (int s0 = 0; s0 < qlen; s0 += CH) {
        const int ns = min(CH, qlen - s0);
        __syncthreads();
        if (fast) stash(ns);
#pragma unroll 4
        for (int e = threadIdx.x; !fast && e < ns * D; e += MS_THREADS) {
            const int s = e / D, d = e - s * D;
            const TA* row = (const TA*)a.proj + (size_t)(qstart + s0 + s) * a.ld;
            const float qp = gl_load(row + a.q_off + kh * D + d);
            if (KIND == 0) {
                qs[e] = qp * a.q_scale;
                ks[e] = gl_load(row + a.k_off + h * D + d);
            } else if (KIND == 2) {
                qs[e] = qp;
                ks[e] = gl_load(row + a.k_off + kh * D + d);
            } else if (KIND == 3) {
                float qv = qp, kv = gl_load(row + a.k_off + kh * D + d);
                if (a.cosv && d < 2 * a.rot_half) {
                    // the pair (u, v) = (dim i, dim i + rot_half) becomes (u c - v s, v c + u s)
                    const bool first = d < a.rot_half;
                    const int i = first ? d : d - a.rot_half, other = first ? d + a.rot_half : d - a.rot_half;
                    const float c = a.cosv[(size_t)(qstart + s0 + s) * a.rot_half + i];
                    const float sn = a.sinv[(size_t)(qstart + s0 + s) * a.rot_half + i];
                    const float qo = gl_load(row + a.q_off + kh * D + other), ko = gl_load(row + a.k_off + kh * D + other);
                    qv = first ? qv * c - qo * sn : qv * c + qo * sn;
                    kv = first ? kv * c - ko * sn : kv * c + ko * sn;
                }
                qs[e] = qv * a.q_scale;
                ks[e] = kv * a.k_scale;
            } else {
                qs[e] = rc_silu(qp);
                const float l = a.lower[h * D + d];
                ks[e] = l + (1.0f - l) * rc_sigmoid(gl_load(row + a.f_off + h * D + d));
            }
        }
        for (int e = threadIdx.x; !fast && e < ns * CT; e += MS_THREADS) {
            const int s = e / CT, j = e - s * CT;
            const TA* row = (const TA*)a.proj + (size_t)(qstart + s0 + s) * a.ld;
            vs[e] = col0 + j < V ? gl_load(row + a.v_off + h * V + col0 + j) : 0.f;
        }
        if (KIND == 2) {
            if (!fast && threadIdx.x < ns) {
                const TA* row = (const TA*)a.gates + (size_t)(qstart + s0 + threadIdx.x) * a.gates_ld;
                gs[threadIdx.x * 4 + 0] = rc_sigmoid(gl_load(row + a.i_off + h));
                gs[threadIdx.x * 4 + 1] = rc_decay(-expf(a.a_log[h]) * rc_softplus(gl_load(row + a.f_off + h) + a.dt_bias[h]));
            }
            __syncthreads();
            // unit length: a warp a token
            for (int s = threadIdx.x >> 5; s < ns; s += MS_THREADS / 32) {
                float sq = 0.f, sk = 0.f;
                for (int d = threadIdx.x & 31; d < D; d += 32) {
                    sq = fmaf(qs[s * D + d], qs[s * D + d], sq);
                    sk = fmaf(ks[s * D + d], ks[s * D + d], sk);
                }
                const float fq = a.q_scale / sqrtf(gl_warp_sum(sq) + 1e-6f), fk = 1.0f / sqrtf(gl_warp_sum(sk) + 1e-6f);
                for (int d = threadIdx.x & 31; d < D; d += 32) {
                    qs[s * D + d] *= fq;
                    ks[s * D + d] *= fk;
                }
            }
            if (fast && s0 + CH < qlen) fetch(s0 + CH);       // the next chunk's inputs travel while this one is walked
        }
        if (KIND == 3 && threadIdx.x < ns) {
            float take = 1.0f, keep = a.lower ? a.lower[h] : 1.0f;
            if (a.gates) {
                const TA* row = (const TA*)a.gates + (size_t)(qstart + s0 + threadIdx.x) * a.gates_ld;
                take = rc_softplus(gl_load(row + a.f_off + h) + a.dt_bias[h]);
                keep = rc_decay(-expf(a.a_log[h]) * take);
            }
            gs[threadIdx.x * 4 + 0] = take;
            gs[threadIdx.x * 4 + 1] = keep;
        }
        if (KIND == 0) {
            if (threadIdx.x < ns) {
                const TA* row = (const TA*)a.proj + (size_t)(qstart + s0 + threadIdx.x) * a.ld;
                gs[threadIdx.x * 4 + 0] = a.cap * tanhf(gl_load(row + a.i_off + h) / a.cap);
                gs[threadIdx.x * 4 + 1] = rc_log_sigmoid(a.cap * tanhf(gl_load(row + a.f_off + h) / a.cap));
            }
            __syncthreads();
            // the maximum is the only thing that goes from token to token here: one thread walks it, and the
            // tokens' factors are then taken side by side
            if (threadIdx.x == 0) {
                for (int s = 0; s < ns; ++s) {
                    const float m_new = fmaxf(gs[s * 4 + 1] + m, gs[s * 4 + 0]);
                    gs[s * 4 + 2] = m;
                    gs[s * 4 + 3] = m_new;
                    m = m_new;
                }
            }
            __syncthreads();
            if (threadIdx.x < ns) {
                const int s = threadIdx.x;
                const float gi = gs[s * 4 + 0], gf = gs[s * 4 + 1], m_old = gs[s * 4 + 2], m_new = gs[s * 4 + 3];
                gs[s * 4 + 2] = rc_decay(gf + m_old - m_new);
                gs[s * 4 + 3] = expf(gi - m_new);
                es[s] = expf(-m_new);
            }
        }
        __syncthreads();
#pragma unroll 4
        for (int s = 0; s < ns; ++s) {
            const float* q = qs + s * D;
            const float* k = ks + s * D;
            const float v = vs[s * CT + c];
            float num = 0.f, nq = 0.f;
            float qr[DPT], kr[DPT];
            if constexpr (FULL && DPT >= 4) {
#pragma unroll
                for (int i = 0; i < DPT; i += 4) {
                    // (a thread's rows are groups of four, R groups apart: the lanes of a column read consecutive
                    // 16-byte pieces, which the banks serve in one go)
                    const float4 q4 = *(const float4*)(q + (((i >> 2) * R + r) << 2)), k4 = *(const float4*)(k + (((i >> 2) * R + r) << 2));
                    qr[i] = q4.x; qr[i + 1] = q4.y; qr[i + 2] = q4.z; qr[i + 3] = q4.w;
                    kr[i] = k4.x; kr[i + 1] = k4.y; kr[i + 2] = k4.z; kr[i + 3] = k4.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < DPT; ++i) {
                    const int d = r + R * i;
                    qr[i] = d < D ? q[d] : 0.f;
                    kr[i] = d < D ? k[d] : (KIND == 1 ? 1.f : 0.f);      // a row that does not exist keeps its zero
                }
            }
            if (KIND == 0) {
                const float keep = gs[s * 4 + 2], take = gs[s * 4 + 3];
                const float tv = take * v;
#pragma unroll
                for (int i = 0; i < DPT; ++i) {
                    S[i] = fmaf(keep, S[i], kr[i] * tv);
                    n[i] = fmaf(keep, n[i], take * kr[i]);
                    num = fmaf(S[i], qr[i], num);
                    nq = fmaf(n[i], qr[i], nq);
                }
            } else if (KIND == 2) {
                const float beta = gs[s * 4 + 0], decay = gs[s * 4 + 1];
                // (sums in up to four parts: one chain of DPT dependent multiply-adds would set the token's pace)
                constexpr int PARTS = DPT >= 4 ? 4 : 1;
                float part[PARTS];
#pragma unroll
                for (int j = 0; j < PARTS; ++j) part[j] = 0.f;
#pragma unroll
                for (int i = 0; i < DPT; ++i) {
                    S[i] *= decay;
                    part[i % PARTS] = fmaf(S[i], kr[i], part[i % PARTS]);
                }
                float kS = PARTS == 4 ? (part[0] + part[1]) + (part[2] + part[3]) : part[0];
                // Two sums over a column's lanes a token: S^T k, which the update waits for, and the read-out, which
                // nothing waits for.  A warp issues in order, so the read-out's butterfly would hold up the next
                // token; it travels with the next token's first butterfly instead, and is stored a token late.
                float late = pending;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const float other = __shfl_xor_sync(0xffffffffu, kS, o);
                    const float other_late = __shfl_xor_sync(0xffffffffu, late, o);
                    if (o < R) { kS += other; late += other_late; }
                }
                if (s > 0 && r == 0 && live) out_col[(size_t)(s0 + s - 1) * H * V] = late;
                const float u = beta * (v - kS);
#pragma unroll
                for (int j = 0; j < PARTS; ++j) part[j] = 0.f;
#pragma unroll
                for (int i = 0; i < DPT; ++i) {
                    S[i] = fmaf(kr[i], u, S[i]);
                    part[i % PARTS] = fmaf(S[i], qr[i], part[i % PARTS]);
                }
                pending = PARTS == 4 ? (part[0] + part[1]) + (part[2] + part[3]) : part[0];
            } else if (KIND == 3) {
                const float keep = gs[s * 4 + 1];
                const float tv = gs[s * 4 + 0] * v;
#pragma unroll
                for (int i = 0; i < DPT; ++i) {
                    S[i] = fmaf(keep, S[i], kr[i] * tv);
                    num = fmaf(S[i], qr[i], num);
                }
            } else {
#pragma unroll
                for (int i = 0; i < DPT; ++i) {
                    const float f = kr[i];
                    S[i] = fmaf(f, S[i], (1.0f - f) * v);
                    num = fmaf(S[i], qr[i], num);
                }
            }
            if constexpr (KIND != 2) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {                // (R is a power of two; unrolled, the steps beyond it only pass)
                const float other = __shfl_xor_sync(0xffffffffu, num, o);
                if (o < R) num += other;
                if (KIND == 0) {
                    const float other_n = __shfl_xor_sync(0xffffffffu, nq, o);
                    if (o < R) nq += other_n;
                }
            }
            if (r == 0 && live) {
                float o = num;
                if (KIND == 0) o = num / (fmaxf(fabsf(nq), es[s]) + 1e-6f);
                if (KIND == 3 && a.d_skip) o = fmaf(a.d_skip[h], v, o);
                out_col[(size_t)(s0 + s) * H * V] = o;
            }
            }
        }
        if constexpr (KIND == 2) {                        // the chunk's last token's read-out
            float late = pending;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const float other_late = __shfl_xor_sync(0xffffffffu, late, o);
                if (o < R) late += other_late;
            }
            if (r == 0 && live) out_col[(size_t)(s0 + ns - 1) * H * V] = late;
        }
    }
#pragma unroll
    for (int i = 0; i < DPT; ++i) {
        const int d = FULL ? ((((i >> 2) * R + r) << 2) + (i & 3)) : r + R * i;
        if (d < D) {
            if (live) S_g[(size_t)d * V + col] = S[i];
            if (KIND == 0 && blockIdx.x == 0 && c == 0) a.nm_next[((size_t)b * H + h) * (D + 1) + d] = n[i];
        }
    }
    if (KIND == 0 && blockIdx.x == 0 && threadIdx.x == 0) a.nm_next[((size_t)b * H + h) * (D + 1) + D] = m;
}

__global__ void __launch_bounds__(128)
memory_commit_kernel(MemoryScanArgs a) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const int b = blockIdx.y, h = blockIdx.x, H = a.H, D = a.D;
    float* srow = a.state + (size_t)a.seq_slot[b] * a.state_stride + (size_t)H * D * a.V;
    const float* src = a.nm_next + ((size_t)b * H + h) * (D + 1);
    for (int d = threadIdx.x; d < D; d += blockDim.x) srow[(size_t)h * D + d] = src[d];
    if (threadIdx.x == 0) srow[(size_t)H * D + h] = src[D];
}

template <typename TA, int DPT>
static int launch_memory_scan(const MemoryScanArgs& a, cudaStream_t stream) {
    int R = 1;
    while (R * DPT < a.D) R <<= 1;
    if (R > 32) return GL_ERR_SHAPE;
    const int CT = MS_THREADS / R;
    // tokens staged at a time: as many as 40 KB hold, at most 32 (a chunk costs a round trip to memory and
    // three block-wide waits, which a few tokens do not pay for)
    const int per_token = (2 * a.D + CT + 5) * (int)sizeof(float);
    int CH = (40 * 1024) / per_token;
    CH = CH > 32 ? 32 : CH;
    if (CH < 1) return GL_ERR_SMEM;
    const size_t smem = (size_t)CH * per_token;
    const dim3 grid((a.V + CT - 1) / CT, a.H, a.B);
    const bool full = DPT >= 4 && a.D == R * DPT;
    if (a.kind == 0) {
        if (full) return gl_launch_in_order(memory_scan_kernel<TA, DPT, 0, true>, grid, dim3(MS_THREADS), smem, stream, a, R, CH);
        return gl_launch_in_order(memory_scan_kernel<TA, DPT, 0, false>, grid, dim3(MS_THREADS), smem, stream, a, R, CH);
    }
    if (a.kind == 2) {
        if (full) return gl_launch_in_order(memory_scan_kernel<TA, DPT, 2, true>, grid, dim3(MS_THREADS), smem, stream, a, R, CH);
        return gl_launch_in_order(memory_scan_kernel<TA, DPT, 2, false>, grid, dim3(MS_THREADS), smem, stream, a, R, CH);
    }
    if (a.kind == 3) {
        if (full) return gl_launch_in_order(memory_scan_kernel<TA, DPT, 3, true>, grid, dim3(MS_THREADS), smem, stream, a, R, CH);
        return gl_launch_in_order(memory_scan_kernel<TA, DPT, 3, false>, grid, dim3(MS_THREADS), smem, stream, a, R, CH);
    }
    if (full) return gl_launch_in_order(memory_scan_kernel<TA, DPT, 1, true>, grid, dim3(MS_THREADS), smem, stream, a, R, CH);
    return gl_launch_in_order(memory_scan_kernel<TA, DPT, 1, false>, grid, dim3(MS_THREADS), smem, stream, a, R, CH);
}

static int memory_scan_blocks(const MemoryScanArgs& a, int dpt) {
    int R = 1;
    while (R * dpt < a.D) R <<= 1;
    if (R > 32) return -1;
    const int CT = MS_THREADS / R;
    return ((a.V + CT - 1) / CT) * a.H * a.B;
}

template <typename TA>
static int dispatch_memory_scan(const MemoryScanArgs& a, cudaStream_t stream) {
    // A thread walks the run's tokens one after the other, so the time of a long run is set by how little
    // each thread does per token and by how many warps an SM has to switch between: rows of a column are
    // spread over more lanes (fewer rows a thread) until the grid gives every SM several blocks.  With many
    // sequences of one token the widest threads do, and fewer blocks re-read the tokens' q and k.
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    // (the delta rule's token is a longer chain of dependent steps, which more rows a thread shorten: measured,
    // a grid of about one block an SM is its best, four an SM the other kinds')
    const int want = a.kind == 2 ? sms * 85 / 100 : 4 * sms;
    const int dpts[5] = {32, 8, 4, 2, 1};
    int pick = -1;
    for (int i = 0; i < 5; ++i) {
        const int blocks = memory_scan_blocks(a, dpts[i]);
        if (blocks < 0) continue;
        pick = dpts[i];                                  // the last that exists if none gives enough blocks
        if (blocks >= want) break;
    }
    if (a.rows_per_thread > 0 && memory_scan_blocks(a, a.rows_per_thread) > 0) pick = a.rows_per_thread;
    int rc;
    switch (pick) {
        case 32: rc = launch_memory_scan<TA, 32>(a, stream); break;
        case 8: rc = launch_memory_scan<TA, 8>(a, stream); break;
        case 4: rc = launch_memory_scan<TA, 4>(a, stream); break;
        case 2: rc = launch_memory_scan<TA, 2>(a, stream); break;
        case 1: rc = launch_memory_scan<TA, 1>(a, stream); break;
        default: return GL_ERR_SHAPE;
    }
    if (rc != 0 || a.kind != 0) return rc;
    return gl_launch(memory_commit_kernel, dim3(a.H, a.B), dim3(128), 0, stream, 1, a) == 0 ? GL_OK : GL_ERR_LAUNCH;
}

GL_API int gl_memory_scan(const MemoryScanArgs* args, int act_dtype, cudaStream_t stream) {
    const MemoryScanArgs& a = *args;
    if (a.B <= 0) return GL_OK;
    if (a.H <= 0 || a.D <= 0 || a.V <= 0 || a.D > 512 || a.B > 65535 || a.H > 65535) return GL_ERR_SHAPE;
    if (a.kind < 0 || a.kind > 3) return GL_ERR_SHAPE;
    if (a.kind == 2 && (!a.gates || !a.a_log || !a.dt_bias || a.KVH <= 0 || a.H % a.KVH)) return GL_ERR_SHAPE;
    if (a.kind == 3) {
        if (a.KVH <= 0 || a.H % a.KVH) return GL_ERR_SHAPE;
        if (a.gates ? (!a.a_log || !a.dt_bias) : !a.lower) return GL_ERR_SHAPE;
        if (a.cosv && (!a.sinv || a.rot_half <= 0 || 2 * a.rot_half > a.D)) return GL_ERR_SHAPE;
    }
    if (a.kind == 0 && (!(a.cap > 0.f) || !a.nm_next)) return GL_ERR_SHAPE;
    if (a.state_stride < (long long)a.H * a.D * a.V + (a.kind == 0 ? (long long)a.H * (a.D + 1) : 0)) return GL_ERR_SHAPE;
    if (act_dtype == GL_F32) return dispatch_memory_scan<float>(a, stream);
    if (act_dtype == GL_BF16) return dispatch_memory_scan<__nv_bfloat16>(a, stream);
    return GL_ERR_DTYPE;
}

// ---------------------------------------------------------------------------
// Per-head unit norm of a memory's output, a weight and an optional gate:
//   out[t, h, j] = o[t, h, j] / sqrt(mean_j o[t, h, :]^2 + eps) * w * sigmoid(gate[t, h*V + j])
// w is [H*V] (w_per_head = 1) or [V] shared by the heads (null: no weight); gate (activation type, row pitch
// gate_ld, first column gate_off) may be absent; gate_silu multiplies by silu(gate) instead of the sigmoid.
// gate_first: gating first, then the norm of the gated values: out = g / sqrt(mean_j g^2 + eps) * w with g = o * act(gate).
// One warp per (token, head).
// ---------------------------------------------------------------------------
template <typename TA>
__global__ void __launch_bounds__(128)
head_norm_gate_kernel(const float* o, const float* __restrict__ w, const TA* gate, TA* __restrict__ out,
                      long long items, int H, int V, int w_per_head, int gate_ld, int gate_off, float eps, int gate_silu,
                      int gate_first) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const int lane = threadIdx.x & 31;
    const long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (item >= items) return;
    const long long t = item / H;
    const int h = (int)(item - t * H);
    const float* src = o + (size_t)item * V;
    const TA* grow = gate ? gate + (size_t)t * gate_ld + gate_off + h * V : nullptr;
    const bool early = gate && gate_first;
    float q = 0.f;
    for (int j = lane; j < V; j += 32) {
        float v = src[j];
        if (early) { const float z = gl_load(grow + j); v *= gate_silu ? rc_silu(z) : rc_sigmoid(z); }
        q += v * v;
    }
    const float inv = 1.0f / sqrtf(gl_warp_sum(q) / (float)V + eps);
    for (int j = lane; j < V; j += 32) {
        float y = src[j];
        if (early) { const float z = gl_load(grow + j); y *= gate_silu ? rc_silu(z) : rc_sigmoid(z); }
        y *= inv;
        if (w) y *= w[w_per_head ? h * V + j : j];
        if (gate && !early) {
            const float z = gl_load(grow + j);
            y *= gate_silu ? rc_silu(z) : rc_sigmoid(z);
        }
        gl_store(out + (size_t)item * V + j, y);
    }
}

// The same for heads of whole 16-byte pieces: L lanes an item (a head of a token), NV4 pieces a lane in registers, every load of
// an item in flight at once, the weights' ahead of the wait.  Element by element, an item's trips to memory came one after the
// other, twice over: 8 items of 512 5.2 -> 2.2 us, 68,096 of 64 24.5 -> 11.1 us, 16,376 of 512 22.0 -> 15.6 us.
__device__ __forceinline__ float4 hn_piece(const float* p) { return __ldcg((const float4*)p); }
__device__ __forceinline__ float4 hn_piece(const __nv_bfloat16* p) {
    const uint2 raw = __ldcg((const uint2*)p);
    const __nv_bfloat162* h = (const __nv_bfloat162*)&raw;
    const float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void hn_put(float* p, const float4& y) { *(float4*)p = y; }
__device__ __forceinline__ void hn_put(__nv_bfloat16* p, const float4& y) {
    __nv_bfloat162 p0 = __floats2bfloat162_rn(y.x, y.y), p1 = __floats2bfloat162_rn(y.z, y.w);
    uint2 pk;
    pk.x = *(unsigned*)&p0; pk.y = *(unsigned*)&p1;
    *(uint2*)p = pk;
}

template <typename TA, int L, int NV4>
__global__ void __launch_bounds__(128)
head_norm_gate_pieces_kernel(const float* o, const float* __restrict__ w, const TA* gate, TA* __restrict__ out,
                             long long items, int H, int V, int w_per_head, int gate_ld, int gate_off, float eps, int gate_silu,
                             int gate_first) {
    gl_grid_launch_dependents();
    const int lane = threadIdx.x % L;
    const long long mine = (long long)blockIdx.x * (128 / L) + threadIdx.x / L;
    const bool live = mine < items;
    const long long item = live ? mine : items - 1;              // (a warp's lanes all stay for the sums)
    const long long t = item / H;
    const int h = (int)(item - t * H);
    float4 g[NV4], v[NV4], z[NV4];
#pragma unroll
    for (int i = 0; i < NV4; ++i) {
        const int j = (lane + i * L) * 4;
        g[i] = w && j < V ? *(const float4*)(w + (w_per_head ? h * V + j : j)) : make_float4(1.f, 1.f, 1.f, 1.f);
    }
    gl_grid_wait();
    const float* src = o + (size_t)item * V;
    const TA* grow = gate ? gate + (size_t)t * gate_ld + gate_off + h * V : nullptr;
#pragma unroll
    for (int i = 0; i < NV4; ++i) {
        const int j = (lane + i * L) * 4;
        v[i] = j < V ? hn_piece(src + j) : make_float4(0.f, 0.f, 0.f, 0.f);
        z[i] = grow && j < V ? hn_piece(grow + j) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (grow) {
#pragma unroll
        for (int i = 0; i < NV4; ++i) {
            if (gate_silu) z[i] = make_float4(rc_silu(z[i].x), rc_silu(z[i].y), rc_silu(z[i].z), rc_silu(z[i].w));
            else z[i] = make_float4(rc_sigmoid(z[i].x), rc_sigmoid(z[i].y), rc_sigmoid(z[i].z), rc_sigmoid(z[i].w));
            if (gate_first) { v[i].x *= z[i].x; v[i].y *= z[i].y; v[i].z *= z[i].z; v[i].w *= z[i].w; }
        }
    }
    float q = 0.f;
#pragma unroll
    for (int i = 0; i < NV4; ++i) q += (v[i].x * v[i].x + v[i].y * v[i].y) + (v[i].z * v[i].z + v[i].w * v[i].w);
#pragma unroll
    for (int s = L / 2; s > 0; s >>= 1) q += __shfl_xor_sync(0xffffffffu, q, s);
    const float inv = 1.0f / sqrtf(q / (float)V + eps);
#pragma unroll
    for (int i = 0; i < NV4; ++i) {
        const int j = (lane + i * L) * 4;
        float4 y = make_float4(v[i].x * inv * g[i].x, v[i].y * inv * g[i].y, v[i].z * inv * g[i].z, v[i].w * inv * g[i].w);
        if (grow && !gate_first) { y.x *= z[i].x; y.y *= z[i].y; y.z *= z[i].z; y.w *= z[i].w; }
        if (live && j < V) hn_put(out + (size_t)item * V + j, y);
    }
}

template <typename TA>
static int launch_head_norm_gate(const float* o, const float* w, const TA* gate, TA* out, long long items, int H, int V,
                                 int w_per_head, int gate_ld, int gate_off, float eps, int gate_silu, int gate_first,
                                 cudaStream_t stream) {
    // pieces of four elements: 16 bytes of 32-bit rows, 4 * sizeof(TA) of the gate and the result
    const bool pieces = V % 4 == 0 && V <= 1024 && !(((uintptr_t)o | (uintptr_t)w) & 15)
                        && !(((uintptr_t)gate | (uintptr_t)out) & (4 * sizeof(TA) - 1)) && (!gate || (gate_ld % 4 == 0 && gate_off % 4 == 0));
#define HN_PIECES(L, NV4) gl_launch(head_norm_gate_pieces_kernel<TA, L, NV4>, dim3((unsigned)((items + 128 / L - 1) / (128 / L))), dim3(128), 0, stream, 1, \
                                    o, w, gate, out, items, H, V, w_per_head, gate_ld, gate_off, eps, gate_silu, gate_first)
    if (pieces) {
        if (V <= 32) return HN_PIECES(8, 1);
        if (V <= 64) return HN_PIECES(16, 1);
        if (V <= 128) return HN_PIECES(32, 1);
        if (V <= 256) return HN_PIECES(32, 2);
        if (V <= 512) return HN_PIECES(32, 4);
        return HN_PIECES(32, 8);
    }
#undef HN_PIECES
    return gl_launch(head_norm_gate_kernel<TA>, dim3((unsigned)((items + 3) / 4)), dim3(128), 0, stream, 1, o, w, gate, out,
                     items, H, V, w_per_head, gate_ld, gate_off, eps, gate_silu, gate_first);
}

GL_API int gl_head_norm_gate(const float* o, const float* w, const void* gate, void* out, int T, int H, int V,
                             int w_per_head, int gate_ld, int gate_off, float eps, int act_dtype, int gate_silu,
                             int gate_first, cudaStream_t stream) {
    if (T <= 0) return GL_OK;
    if (H <= 0 || V <= 0) return GL_ERR_SHAPE;
    const long long items = (long long)T * H;
    if (act_dtype == GL_F32)
        return launch_head_norm_gate(o, w, (const float*)gate, (float*)out, items, H, V, w_per_head, gate_ld, gate_off, eps, gate_silu,
                                     gate_first, stream);
    if (act_dtype == GL_BF16)
        return launch_head_norm_gate(o, w, (const __nv_bfloat16*)gate, (__nv_bfloat16*)out, items, H, V, w_per_head, gate_ld, gate_off, eps,
                                     gate_silu, gate_first, stream);
    return GL_ERR_DTYPE;
}

// ---------------------------------------------------------------------------
// Short causal convolution per channel with bias and silu (or without an activation).  The filter's last tap is the current
// token's; inputs before the run come from the sequence's state row (the last taps-1 inputs, oldest
// first, zero at a sequence's start).  A second kernel then moves the run's last inputs into the row.
// ---------------------------------------------------------------------------
struct ConvArgs {
    const void* x;            // [T, ld] activation type; the convolved channels start at column x_off
    void* out;                // [T, C] activation type
    const float* w;           // [C, taps]
    const float* bias;        // [C] or null
    float* state;             // [slots, state_stride]; the tail [C, taps-1] starts at tail_off
    const int* tok_seq;       // [T]
    const int* seq_slot;
    const int* seq_qstart;
    const int* seq_qlen;
    int T, B, C, taps, ld, x_off, state_stride, tail_off;
    int silu;                 // 0: the sum as it is
};

template <typename TA>
__global__ void __launch_bounds__(256)
conv_silu_kernel(ConvArgs a) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)a.T * a.C) return;
    const int t = (int)(i / a.C), c = (int)(i - (long long)t * a.C);
    const int b = a.tok_seq[t];
    const int idx = t - a.seq_qstart[b];
    const int back = a.taps - 1;
    const float* tail = a.state + (size_t)a.seq_slot[b] * a.state_stride + a.tail_off + (size_t)c * back;
    float acc = a.bias ? a.bias[c] : 0.f;
    for (int j = 0; j < a.taps; ++j) {
        const int rel = idx - back + j;               // place in the run; negative: before it
        const float v = rel >= 0 ? gl_load((const TA*)a.x + (size_t)(t - back + j) * a.ld + a.x_off + c) : tail[rel + back];
        acc = fmaf(a.w[(size_t)c * a.taps + j], v, acc);
    }
    gl_store((TA*)a.out + (size_t)t * a.C + c, a.silu ? rc_silu(acc) : acc);
}

// The same with 16 bytes of channels a thread (4 or 8 of them): columns, pitch and offset are whole pieces, and
// the thread's TAPS x channels weights are one run of memory that it fetches 16 bytes at a time.  The sums run in
// the order of the kernel above.
template <typename TA, int TAPS>
__global__ void __launch_bounds__(256)
conv_silu_wide_kernel(ConvArgs a) {
    constexpr int VEC = 16 / (int)sizeof(TA);
    gl_grid_launch_dependents();
    gl_grid_wait();
    const int CV = a.C / VEC;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)a.T * CV) return;
    const int t = (int)(i / CV), c0 = (int)(i - (long long)t * CV) * VEC;
    const int b = a.tok_seq[t];
    const int idx = t - a.seq_qstart[b];
    constexpr int back = TAPS - 1;
    const float* tail = a.state + (size_t)a.seq_slot[b] * a.state_stride + a.tail_off;
    __align__(16) float acc[VEC], v[VEC], w[VEC * TAPS];
#pragma unroll
    for (int q = 0; q < VEC * TAPS / 4; ++q)
        reinterpret_cast<float4*>(w)[q] = reinterpret_cast<const float4*>(a.w + (size_t)c0 * TAPS)[q];
#pragma unroll
    for (int k = 0; k < VEC; ++k) acc[k] = a.bias ? a.bias[c0 + k] : 0.f;
#pragma unroll
    for (int j = 0; j < TAPS; ++j) {
        const int rel = idx - back + j;               // place in the run; negative: before it
        if (rel >= 0) {
            mc_load16((const TA*)a.x + (size_t)(t - back + j) * a.ld + a.x_off + c0, v);
        } else {
#pragma unroll
            for (int k = 0; k < VEC; ++k) v[k] = tail[(size_t)(c0 + k) * back + rel + back];
        }
#pragma unroll
        for (int k = 0; k < VEC; ++k) acc[k] = fmaf(w[k * TAPS + j], v[k], acc[k]);
    }
    if (a.silu) {
#pragma unroll
        for (int k = 0; k < VEC; ++k) acc[k] = rc_silu(acc[k]);
    }
    mc_store16((TA*)a.out + (size_t)t * a.C + c0, acc);
}

// The same for runs of tokens: a thread takes 16 bytes of channels of four consecutive tokens, so that the weights and
// the rows the four windows share are fetched once.  (Four tokens that are not of one sequence go one by one.)
template <typename TA, int TAPS>
__global__ void __launch_bounds__(256)
conv_silu_tokens_kernel(ConvArgs a) {
    constexpr int VEC = 16 / (int)sizeof(TA), NT = 4, back = TAPS - 1;
    gl_grid_launch_dependents();
    gl_grid_wait();
    const int CV = a.C / VEC;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int t0 = (int)(i / CV) * NT, c0 = (int)(i - (long long)(t0 / NT) * CV) * VEC;
    if (t0 >= a.T) return;
    __align__(16) float w[VEC * TAPS], bias[VEC];
#pragma unroll
    for (int q = 0; q < VEC * TAPS / 4; ++q)
        reinterpret_cast<float4*>(w)[q] = reinterpret_cast<const float4*>(a.w + (size_t)c0 * TAPS)[q];
#pragma unroll
    for (int k = 0; k < VEC; ++k) bias[k] = a.bias ? a.bias[c0 + k] : 0.f;
    const int n = min(NT, a.T - t0);
    const int b_first = a.tok_seq[t0];
    const bool together = n == NT && b_first == a.tok_seq[t0 + NT - 1];
    const int idx0 = t0 - a.seq_qstart[b_first];
    const TA* x = (const TA*)a.x + a.x_off + c0;
    if (together && idx0 >= back) {
        __align__(16) float v[TAPS][VEC];             // rows t - back .. t, in a ring
#pragma unroll
        for (int j = 0; j < back; ++j) mc_load16(x + (size_t)(t0 - back + j) * a.ld, v[j]);
#pragma unroll
        for (int s = 0; s < NT; ++s) {
            mc_load16(x + (size_t)(t0 + s) * a.ld, v[(s + back) % TAPS]);
            __align__(16) float acc[VEC];
#pragma unroll
            for (int k = 0; k < VEC; ++k) acc[k] = bias[k];
#pragma unroll
            for (int j = 0; j < TAPS; ++j)
#pragma unroll
                for (int k = 0; k < VEC; ++k) acc[k] = fmaf(w[k * TAPS + j], v[(s + j) % TAPS][k], acc[k]);
            if (a.silu) {
#pragma unroll
                for (int k = 0; k < VEC; ++k) acc[k] = rc_silu(acc[k]);
            }
            mc_store16((TA*)a.out + (size_t)(t0 + s) * a.C + c0, acc);
        }
        return;
    }
    for (int s = 0; s < n; ++s) {
        const int t = t0 + s, b = a.tok_seq[t], idx = t - a.seq_qstart[b];
        const float* tail = a.state + (size_t)a.seq_slot[b] * a.state_stride + a.tail_off;
        __align__(16) float acc[VEC], v[VEC];
#pragma unroll
        for (int k = 0; k < VEC; ++k) acc[k] = bias[k];
#pragma unroll
        for (int j = 0; j < TAPS; ++j) {
            const int rel = idx - back + j;
            if (rel >= 0) {
                mc_load16(x + (size_t)(t - back + j) * a.ld, v);
            } else {
#pragma unroll
                for (int k = 0; k < VEC; ++k) v[k] = tail[(size_t)(c0 + k) * back + rel + back];
            }
#pragma unroll
            for (int k = 0; k < VEC; ++k) acc[k] = fmaf(w[k * TAPS + j], v[k], acc[k]);
        }
        if (a.silu) {
#pragma unroll
            for (int k = 0; k < VEC; ++k) acc[k] = rc_silu(acc[k]);
        }
        mc_store16((TA*)a.out + (size_t)t * a.C + c0, acc);
    }
}

template <typename TA>
static int launch_conv_silu_tokens(const ConvArgs& a, cudaStream_t stream) {
    const long long n = (long long)((a.T + 3) / 4) * (a.C / (16 / (int)sizeof(TA)));
    const dim3 grid((unsigned)((n + 255) / 256));
    switch (a.taps) {
        case 2: return gl_launch(conv_silu_tokens_kernel<TA, 2>, grid, dim3(256), 0, stream, 1, a);
        case 3: return gl_launch(conv_silu_tokens_kernel<TA, 3>, grid, dim3(256), 0, stream, 1, a);
        default: return gl_launch(conv_silu_tokens_kernel<TA, 4>, grid, dim3(256), 0, stream, 1, a);
    }
}

template <typename TA>
static int launch_conv_silu_wide(const ConvArgs& a, dim3 grid, cudaStream_t stream) {
    // (enough tokens that a quarter of the threads still fills the SMs)
    if (a.taps > 1 && (long long)a.T * (a.C / (16 / (int)sizeof(TA))) >= 4 * 148 * 512) return launch_conv_silu_tokens<TA>(a, stream);
    switch (a.taps) {
        case 1: return gl_launch(conv_silu_wide_kernel<TA, 1>, grid, dim3(256), 0, stream, 1, a);
        case 2: return gl_launch(conv_silu_wide_kernel<TA, 2>, grid, dim3(256), 0, stream, 1, a);
        case 3: return gl_launch(conv_silu_wide_kernel<TA, 3>, grid, dim3(256), 0, stream, 1, a);
        default: return gl_launch(conv_silu_wide_kernel<TA, 4>, grid, dim3(256), 0, stream, 1, a);
    }
}

template <typename TA>
__global__ void __launch_bounds__(256)
conv_tail_kernel(ConvArgs a) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)a.B * a.C) return;
    const int b = (int)(i / a.C), c = (int)(i - (long long)b * a.C);
    const int back = a.taps - 1, qlen = a.seq_qlen[b], qstart = a.seq_qstart[b];
    float* tail = a.state + (size_t)a.seq_slot[b] * a.state_stride + a.tail_off + (size_t)c * back;
    for (int k = 0; k < back; ++k) {                  // ascending: a place is read before a lower one is written
        const int rel = qlen - back + k;
        tail[k] = rel >= 0 ? gl_load((const TA*)a.x + (size_t)(qstart + rel) * a.ld + a.x_off + c) : tail[qlen + k];
    }
}

// One token a sequence: a thread owns a (sequence, channel), so it may read the tail, write the output and
// shift the tail in one go.
template <typename TA>
__global__ void __launch_bounds__(256)
conv_silu_step_kernel(ConvArgs a) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)a.B * a.C) return;
    const int b = (int)(i / a.C), c = (int)(i - (long long)b * a.C);
    const int back = a.taps - 1, t = a.seq_qstart[b];
    float* tail = a.state + (size_t)a.seq_slot[b] * a.state_stride + a.tail_off + (size_t)c * back;
    const float x = gl_load((const TA*)a.x + (size_t)t * a.ld + a.x_off + c);
    float acc = a.bias ? a.bias[c] : 0.f;
    for (int j = 0; j < back; ++j) {
        const float v = tail[j];
        acc = fmaf(a.w[(size_t)c * a.taps + j], v, acc);
        if (j > 0) tail[j - 1] = v;                   // (read before the place below it is written)
    }
    acc = fmaf(a.w[(size_t)c * a.taps + back], x, acc);
    if (back > 0) tail[back - 1] = x;
    gl_store((TA*)a.out + (size_t)t * a.C + c, a.silu ? rc_silu(acc) : acc);
}

GL_API int gl_conv_silu(const ConvArgs* args, int act_dtype, cudaStream_t stream) {
    const ConvArgs& a = *args;
    if (a.T <= 0 || a.B <= 0) return GL_OK;
    if (a.C <= 0 || a.taps <= 0) return GL_ERR_SHAPE;
    const long long n = (long long)a.T * a.C, nb = (long long)a.B * a.C;
    const dim3 g1((unsigned)((n + 255) / 256)), g2((unsigned)((nb + 255) / 256));
    int rc;
    if (a.T == a.B) {                                 // every sequence brings exactly one token
        if (act_dtype == GL_F32) return gl_launch(conv_silu_step_kernel<float>, g2, dim3(256), 0, stream, 1, a);
        if (act_dtype == GL_BF16) return gl_launch(conv_silu_step_kernel<__nv_bfloat16>, g2, dim3(256), 0, stream, 1, a);
        return GL_ERR_DTYPE;
    }
    // rows of whole, aligned 16-byte pieces: a thread takes a piece of channels
    const int vec = act_dtype == GL_F32 ? 4 : 8;
    const bool wide = a.taps <= 4 && ((size_t)a.w & 15) == 0 && a.C % vec == 0 && a.ld % vec == 0 && a.x_off % vec == 0 && ((size_t)a.x & 15) == 0 && ((size_t)a.out & 15) == 0;
    const dim3 gw((unsigned)((n / vec + 255) / 256));
    if (act_dtype == GL_F32) {
        rc = wide ? launch_conv_silu_wide<float>(a, gw, stream)
                  : gl_launch(conv_silu_kernel<float>, g1, dim3(256), 0, stream, 1, a);
        if (rc == 0 && a.taps > 1) rc = gl_launch(conv_tail_kernel<float>, g2, dim3(256), 0, stream, 1, a);
        return rc;
    }
    if (act_dtype == GL_BF16) {
        rc = wide ? launch_conv_silu_wide<__nv_bfloat16>(a, gw, stream)
                  : gl_launch(conv_silu_kernel<__nv_bfloat16>, g1, dim3(256), 0, stream, 1, a);
        if (rc == 0 && a.taps > 1) rc = gl_launch(conv_tail_kernel<__nv_bfloat16>, g2, dim3(256), 0, stream, 1, a);
        return rc;
    }
    return GL_ERR_DTYPE;
}
