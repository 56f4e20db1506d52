// The matrix memories (recurrent.cu) for long runs: chunks of tokens side by side, a lane a column.
//
// Written with a decay a_t[d] and an input b_t[d] per row (gated kind: a = keep_t for every row, b = take_t
// k_t[d]; bounded forget: a = f_t[d], b = 1 - f_t[d]) a memory is S' = diag(a) S + b v^T, column by column.
// A thread owns one column and keeps all of its rows in registers: a token costs it two multiply-adds a row
// and nothing is exchanged between lanes.  The gated kind's normaliser n is one more column whose value is
// always 1 (its "output" is n.q), so it needs no code of its own.  That mapping has only heads x columns / 32
// warps of work, so a run is cut into chunks that are walked side by side, twice:
//   walk 1: every chunk from a zero state; its last state goes to chunk_state;
//   carry:  S_start[k+1] = diag(P_k) S_start[k] + last_k, P_k[d] the product of the chunk's decays;
//   walk 2: every chunk from its start, with the raw outputs S^T q (the gated kind's division by
//           max(|n.q|, e^-m) + 1e-6 follows as a pass of its own over all tokens at once).
// The gated kind's gates come from a pass of their own: the log gates of all tokens side by side, then the
// running maximum token by token (a thread a head), which leaves keep, take and e^-m per token.
// The plain decay (kind 3) is the gated kind without a normaliser: keep and take per (token, head) come from a pass
// of their own (a fixed decay, or a step size: the formulas of memory_scan_kernel), a = keep for every row,
// b = k after its rotation and scale, and the token's value is multiplied by take before it enters, so that a
// chunk's arithmetic is the token-by-token kernel's.  q and k heads may be shared by several heads; the skip
// term d_skip[h] v is added to the read-out.
#include "common.cuh"
#include "recurrent_common.cuh"

struct MemoryChunkArgs {
    const void* proj;         // [T, ld] activation type
    float* out;               // [T, H*V] raw S^T q
    float* nq;                // gated: [T, H] n.q
    float* gates;             // gated: [T, H, 4]: log input gate, log forget gate -> keep, take, e^-m, log keep
    float* state;             // [slots, state_stride]: S [H, D, V], gated: n [H, D], m [H]
    const float* lower;       // bounded forget: [H*D]
    float* chunk_state;       // [B, n_chunks, H, D, cols]
    float* chunk_decay;       // [B, n_chunks, H, D]
    const int* tok_seq;       // [T]
    const int* seq_slot;
    const int* seq_qstart;
    const int* seq_qlen;
    int T, ld, q_off, k_off, v_off, i_off, f_off;
    int B, H, D, V, cols, state_stride, kind, chunk_len, n_chunks;
    float cap, q_scale;
    // kind 3:
    const void* gates_in;     // [T, gates_ld] activation type or null: the step sizes' projections (column f_off + h)
    const float* a_log;       // [H]
    const float* dt_bias;     // [H]
    const float* cosv;        // [T, rot_half] or null
    const float* sinv;
    const float* d_skip;      // [H] or null
    int gates_ld, KVH, rot_half;
    float k_scale;
};

#define MC_THREADS 128
#define MC_TOKENS 16

// log gates of every token: gates[t, h, 0] = cap tanh(i / cap), gates[t, h, 1] = logsigmoid(cap tanh(f / cap))
template <typename TA>
__global__ void __launch_bounds__(256)
memory_log_gates_kernel(MemoryChunkArgs a) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)a.T * a.H) return;
    const int t = (int)(i / a.H), h = (int)(i - (long long)t * a.H);
    const TA* row = (const TA*)a.proj + (size_t)t * a.ld;
    a.gates[i * 4 + 0] = a.cap * tanhf(gl_load(row + a.i_off + h) / a.cap);
    a.gates[i * 4 + 1] = rc_log_sigmoid(a.cap * tanhf(gl_load(row + a.f_off + h) / a.cap));
}

// the running maximum, token by token, a warp a (sequence, head): 32 tokens' log gates are fetched at once, the
// maximum walks them in registers (every lane follows it, lane j keeps token j's), and the lanes then take
// keep, take and e^-m of their tokens side by side
__global__ void __launch_bounds__(32)
memory_gate_walk_kernel(MemoryChunkArgs a) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const int b = blockIdx.x / a.H, h = blockIdx.x - b * a.H, lane = threadIdx.x;
    float* m_g = a.state + (size_t)a.seq_slot[b] * a.state_stride + (size_t)a.H * a.D * a.V + (size_t)a.H * a.D + h;
    float m = *m_g;
    const int qstart = a.seq_qstart[b], qlen = a.seq_qlen[b];
    for (int s0 = 0; s0 < qlen; s0 += 32) {
        const bool ok = s0 + lane < qlen;
        float* g = a.gates + ((size_t)(qstart + s0 + (ok ? lane : 0)) * a.H + h) * 4;
        const float gi = ok ? g[0] : -INFINITY, gf = ok ? g[1] : 0.f;      // a token that is not there leaves m as it is
        float m_old = 0.f, m_mine = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            const float m_new = fmaxf(__shfl_sync(0xffffffffu, gf, j) + m, __shfl_sync(0xffffffffu, gi, j));
            if (lane == j) { m_old = m; m_mine = m_new; }
            m = m_new;
        }
        if (ok) {
            g[0] = rc_decay(gf + m_old - m_mine);
            g[3] = gf + m_old - m_mine;
            g[1] = expf(gi - m_mine);
            g[2] = expf(-m_mine);
        }
    }
    if (lane == 0) *m_g = m;
}

// the plain decay's keep and take of every token: gates[t, h, 0] = keep, gates[t, h, 1] = take, gates[t, h, 3] = log keep
template <typename TA>
__global__ void __launch_bounds__(256)
memory_decay_gates_kernel(MemoryChunkArgs a) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)a.T * a.H) return;
    const int t = (int)(i / a.H), h = (int)(i - (long long)t * a.H);
    float take = 1.0f, keep = a.lower ? a.lower[h] : 1.0f, log_keep = 0.f;
    if (a.gates_in) {
        take = rc_softplus(gl_load((const TA*)a.gates_in + (size_t)t * a.gates_ld + a.f_off + h) + a.dt_bias[h]);
        log_keep = -expf(a.a_log[h]) * take;
        keep = rc_decay(log_keep);
    } else if (a.lower) {
        log_keep = (float)log((double)keep);
    }
    a.gates[i * 4 + 0] = keep;
    a.gates[i * 4 + 1] = take;
    a.gates[i * 4 + 3] = log_keep;
}

// the product of a chunk's decays per row
template <typename TA, int KIND>
__global__ void __launch_bounds__(128)
memory_chunk_decay_kernel(MemoryChunkArgs a) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const int b = blockIdx.z / a.n_chunks, chunk = blockIdx.z - b * a.n_chunks, h = blockIdx.y;
    const int d = blockIdx.x * blockDim.x + threadIdx.x;
    const int qlen = a.seq_qlen[b], qstart = a.seq_qstart[b];
    const int t0 = chunk * a.chunk_len, t1 = min(qlen, t0 + a.chunk_len);
    if (d >= a.D || t0 >= qlen) return;
    float p = 1.0f;
    const float l = KIND == 1 ? a.lower[h * a.D + d] : 0.f;
    for (int s = t0; s < t1; ++s) {
        if (KIND == 0 || KIND == 3) p *= a.gates[((size_t)(qstart + s) * a.H + h) * 4];
        else p *= l + (1.0f - l) * rc_sigmoid(gl_load((const TA*)a.proj + (size_t)(qstart + s) * a.ld + a.f_off + h * a.D + d));
    }
    a.chunk_decay[(((size_t)b * a.n_chunks + chunk) * a.H + h) * a.D + d] = p;
}

// MODE 1: from zero, keep the last state.  MODE 2: from the chunk's start, with outputs.  NT: threads (columns) a block.
// FULL: D == DMAX, so no row needs a bounds check; a token's rows are then read four at a time and updated in
// pairs (fma.rn.f32x2), and the read-out is summed in four parts (the walk issues less than half the
// instructions a row that the checked form does, which is what bounds it).
template <typename TA, int DMAX, int KIND, int MODE, int NT, bool FULL>
__global__ void __launch_bounds__(NT)
memory_chunk_walk_kernel(MemoryChunkArgs a) {
    extern __shared__ __align__(16) float smem[];
    gl_grid_wait();
    const int D = a.D, V = a.V, H = a.H, cols = a.cols;
    const int b = blockIdx.z / a.n_chunks, chunk = blockIdx.z - b * a.n_chunks, h = blockIdx.y;
    const int col0 = blockIdx.x * NT, col = col0 + threadIdx.x;
    const bool live = col < cols;
    const int qlen = a.seq_qlen[b], qstart = a.seq_qstart[b];
    const int t0 = chunk * a.chunk_len, t1 = min(qlen, t0 + a.chunk_len);
    if (t0 >= qlen) return;
    constexpr bool SCALAR = KIND == 0 || KIND == 3;   // one decay for all rows of a (token, head)
    float* as = smem;                                 // [TOKENS][D] decay (bounded forget; the other kinds' is a scalar)
    float* bs = as + MC_TOKENS * D;                   // [TOKENS][D] input per row
    float* qs = bs + MC_TOKENS * D;                   // [TOKENS][D]
    float* vs = qs + MC_TOKENS * D;                   // [TOKENS][NT]
    float* ks = vs + MC_TOKENS * NT;                  // [TOKENS] the scalar keep
    float* ts = ks + MC_TOKENS;                       // [TOKENS] the plain decay's take
    const int kh = KIND == 3 ? h / (H / a.KVH) : h;   // the head of q and k this head reads
    constexpr int VEC = 16 / (int)sizeof(TA);
    // rows of whole, aligned 16-byte pieces can be fetched as such
    const bool wide = KIND == 3 && D % VEC == 0 && V % VEC == 0 && a.ld % VEC == 0 && a.q_off % VEC == 0
                      && a.k_off % VEC == 0 && a.v_off % VEC == 0 && ((size_t)a.proj & 15) == 0;
    float* cs = a.chunk_state + ((((size_t)b * a.n_chunks + chunk) * H + h) * D) * cols;
    float S[DMAX];
#pragma unroll
    for (int d = 0; d < DMAX; ++d) S[d] = (MODE == 2 && live && d < D) ? cs[(size_t)d * cols + col] : 0.f;
    for (int s0 = t0; s0 < t1; s0 += MC_TOKENS) {
        const int ns = min(MC_TOKENS, t1 - s0);
        __syncthreads();
        if (KIND == 3 && wide) {
            // whole 16-byte pieces of the rows first, as they are; then rotation and scale in place
            const int DV = D / VEC;
            for (int e = threadIdx.x; e < ns * DV; e += NT) {
                const int s = e / DV, d = (e - s * DV) * VEC;
                const TA* row = (const TA*)a.proj + (size_t)(qstart + s0 + s) * a.ld;
                mc_load16(row + a.k_off + kh * D + d, bs + s * D + d);
                if (MODE == 2) mc_load16(row + a.q_off + kh * D + d, qs + s * D + d);
            }
            for (int e = threadIdx.x; e < ns * (NT / VEC); e += NT) {
                const int s = e / (NT / VEC), j = (e - s * (NT / VEC)) * VEC;
                const TA* row = (const TA*)a.proj + (size_t)(qstart + s0 + s) * a.ld;
                if (col0 + j < V) mc_load16(row + a.v_off + h * V + col0 + j, vs + s * NT + j);   // (V is whole pieces)
            }
            if (a.cosv || a.k_scale != 1.0f || (MODE == 2 && a.q_scale != 1.0f)) {
                __syncthreads();
                const int half = a.cosv ? a.rot_half : 0;
                for (int e = threadIdx.x; e < ns * D; e += NT) {
                    const int s = e / D, d = e - s * D;
                    if (d < half) {
                        // the pair (u, v) = (dim d, dim d + half) becomes (u c - v s, v c + u s)
                        const size_t t = (size_t)(qstart + s0 + s);
                        const float c = a.cosv[t * half + d], sn = a.sinv[t * half + d];
                        const float ku = bs[e], kv = bs[e + half];
                        bs[e] = (ku * c - kv * sn) * a.k_scale;
                        bs[e + half] = (kv * c + ku * sn) * a.k_scale;
                        if (MODE == 2) {
                            const float qu = qs[e], qv = qs[e + half];
                            qs[e] = (qu * c - qv * sn) * a.q_scale;
                            qs[e + half] = (qv * c + qu * sn) * a.q_scale;
                        }
                    } else if (d >= 2 * half) {
                        bs[e] *= a.k_scale;
                        if (MODE == 2) qs[e] *= a.q_scale;
                    }
                }
            }
        } else {
#pragma unroll 4
            for (int e = threadIdx.x; e < ns * D; e += NT) {
                const int s = e / D, d = e - s * D;
                const size_t t = (size_t)(qstart + s0 + s);
                const TA* row = (const TA*)a.proj + t * a.ld;
                if (KIND == 0) {
                    bs[e] = a.gates[(t * H + h) * 4 + 1] * gl_load(row + a.k_off + h * D + d);
                    if (MODE == 2) qs[e] = gl_load(row + a.q_off + h * D + d) * a.q_scale;
                } else if (KIND == 3) {
                    float kv = gl_load(row + a.k_off + kh * D + d), qv = MODE == 2 ? gl_load(row + a.q_off + kh * D + d) : 0.f;
                    if (a.cosv && d < 2 * a.rot_half) {
                        // the pair (u, v) = (dim i, dim i + rot_half) becomes (u c - v s, v c + u s)
                        const bool first = d < a.rot_half;
                        const int i = first ? d : d - a.rot_half, other = first ? d + a.rot_half : d - a.rot_half;
                        const float c = a.cosv[t * a.rot_half + i], sn = a.sinv[t * a.rot_half + i];
                        const float ko = gl_load(row + a.k_off + kh * D + other);
                        kv = first ? kv * c - ko * sn : kv * c + ko * sn;
                        if (MODE == 2) {
                            const float qo = gl_load(row + a.q_off + kh * D + other);
                            qv = first ? qv * c - qo * sn : qv * c + qo * sn;
                        }
                    }
                    bs[e] = kv * a.k_scale;
                    if (MODE == 2) qs[e] = qv * a.q_scale;
                } else {
                    const float l = a.lower[h * D + d];
                    const float f = l + (1.0f - l) * rc_sigmoid(gl_load(row + a.f_off + h * D + d));
                    as[e] = f;
                    bs[e] = 1.0f - f;
                    if (MODE == 2) qs[e] = rc_silu(gl_load(row + a.q_off + h * D + d));
                }
            }
            for (int e = threadIdx.x; e < ns * NT; e += NT) {
                const int s = e / NT, j = col0 + (e - s * NT);
                const TA* row = (const TA*)a.proj + (size_t)(qstart + s0 + s) * a.ld;
                vs[e] = j < V ? gl_load(row + a.v_off + h * V + j) : 1.0f;     // the normaliser's column takes 1
            }
        }
        if (SCALAR && threadIdx.x < ns) {
            const float* g = a.gates + ((size_t)(qstart + s0 + threadIdx.x) * H + h) * 4;
            ks[threadIdx.x] = g[0];
            if (KIND == 3) ts[threadIdx.x] = g[1];
        }
        __syncthreads();
        for (int s = 0; s < ns; ++s) {
            const float v_in = vs[s * NT + threadIdx.x];
            const float v = KIND == 3 ? ts[s] * v_in : v_in;
            const float keep = SCALAR ? ks[s] : 0.f;
            const float* ar = as + s * D;
            const float* br = bs + s * D;
            const float* qr = qs + s * D;
            float num = 0.f;
            if constexpr (FULL) {
                const unsigned long long v2 = mc_pack(v, v), keep2 = mc_pack(keep, keep);
                unsigned long long n01 = mc_pack(0.f, 0.f), n23 = n01;
#pragma unroll
                for (int d = 0; d < DMAX; d += 4) {
                    const float4 b4 = *reinterpret_cast<const float4*>(br + d);
                    unsigned long long a01 = keep2, a23 = keep2;
                    if (!SCALAR) {
                        const float4 a4 = *reinterpret_cast<const float4*>(ar + d);
                        a01 = mc_pack(a4.x, a4.y);
                        a23 = mc_pack(a4.z, a4.w);
                    }
                    unsigned long long s01 = mc_pack(S[d], S[d + 1]), s23 = mc_pack(S[d + 2], S[d + 3]);
                    s01 = mc_fma2(a01, s01, mc_mul2(mc_pack(b4.x, b4.y), v2));
                    s23 = mc_fma2(a23, s23, mc_mul2(mc_pack(b4.z, b4.w), v2));
                    if (MODE == 2) {
                        const float4 q4 = *reinterpret_cast<const float4*>(qr + d);
                        n01 = mc_fma2(s01, mc_pack(q4.x, q4.y), n01);
                        n23 = mc_fma2(s23, mc_pack(q4.z, q4.w), n23);
                    }
                    const float2 r01 = mc_unpack(s01), r23 = mc_unpack(s23);
                    S[d] = r01.x; S[d + 1] = r01.y; S[d + 2] = r23.x; S[d + 3] = r23.y;
                }
                if (MODE == 2) {
                    const float2 p01 = mc_unpack(n01), p23 = mc_unpack(n23);
                    num = (p01.x + p01.y) + (p23.x + p23.y);
                }
            } else {
#pragma unroll
                for (int d = 0; d < DMAX; ++d) {
                    if (d < D) {
                        S[d] = fmaf(SCALAR ? keep : ar[d], S[d], br[d] * v);
                        if (MODE == 2) num = fmaf(S[d], qr[d], num);
                    }
                }
            }
            if (MODE == 2 && live) {
                const size_t t = (size_t)(qstart + s0 + s);
                if (KIND == 3 && a.d_skip) num = fmaf(a.d_skip[h], v_in, num);
                if (col < V) a.out[t * H * V + (size_t)h * V + col] = num;
                else a.nq[t * H + h] = num;
            }
        }
    }
    if (!live) return;
    if (MODE == 1) {
#pragma unroll
        for (int d = 0; d < DMAX; ++d)
            if (d < D) cs[(size_t)d * cols + col] = S[d];
    } else if (t1 == qlen) {                          // the run's last chunk: the state row takes its last state
        float* srow = a.state + (size_t)a.seq_slot[b] * a.state_stride;
#pragma unroll
        for (int d = 0; d < DMAX; ++d) {
            if (d < D) {
                if (col < V) srow[((size_t)h * D + d) * V + col] = S[d];
                else srow[(size_t)H * D * V + (size_t)h * D + d] = S[d];
            }
        }
    }
}

// every chunk's start state from the run's start state and the chunks' last states
__global__ void __launch_bounds__(128)
memory_chunk_carry_kernel(MemoryChunkArgs a) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const int b = blockIdx.z, h = blockIdx.y;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;        // (row, column)
    if (i >= a.D * a.cols) return;
    const int d = i / a.cols, col = i - d * a.cols;
    const float* srow = a.state + (size_t)a.seq_slot[b] * a.state_stride;
    float S = col < a.V ? srow[((size_t)h * a.D + d) * a.V + col] : srow[(size_t)a.H * a.D * a.V + (size_t)h * a.D + d];
    const int chunks = (a.seq_qlen[b] + a.chunk_len - 1) / a.chunk_len;
    // eight chunks' last states and decays are asked for at once, so that a chunk costs no trip to memory of its own
    for (int k0 = 0; k0 < chunks; k0 += 8) {
        float last[8], decay[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const size_t at = ((size_t)b * a.n_chunks + min(k0 + j, chunks - 1)) * a.H + h;
            last[j] = a.chunk_state[(at * a.D + d) * a.cols + col];
            decay[j] = a.chunk_decay[at * a.D + d];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (k0 + j < chunks) {
                const size_t at = ((size_t)b * a.n_chunks + k0 + j) * a.H + h;
                a.chunk_state[(at * a.D + d) * a.cols + col] = S;
                S = fmaf(decay[j], S, last[j]);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// The scalar-decay memories' chunks (gated kind and plain decay) as matrix products, for bfloat16 inputs.
//
// With one decay a (token, head), the tokens of a chunk meet in closed form.  L_t = keep_1 .. keep_t within the chunk,
// S_0 the state the chunk starts from:
//   o_t  = L_t S_0^T q_t + sum_{s <= t} (L_t / L_s) take_s (q_t . k_s) v_s,
//   S_C  = L_C S_0 + sum_s (L_C / L_s) take_s k_s v_s^T,
// products of 64 x 64 x D, 64 x D x V and D x 64 x V numbers a chunk and head instead of a walk over its tokens.
//
// Nothing is computed with fewer bits than in the walk.  q, k and v are bfloat16 and enter exactly; what is a 32-bit number
// (the weighted keys, the weighted scores, the state, keys and queries after a rotation) enters as a sum of three bfloat16
// numbers, 24 bits, and each of the three is multiplied.  The products accumulate in 32 bits; since the tensor cores cut off
// what an addition cannot hold instead of rounding it, a product's 16 terms (its parts, smallest first) are summed from zero and
// the sums added in registers: accumulated in place the error was three times the walk's.  L_t / L_s is e to the
// difference of sums of logarithms; the sums are taken in 64-bit, so that a token that forgets nearly everything leaves the
// later ones' decays as exact as they were.
//
// What bounds it: the phases of a block one after the other (fetch, split, products, store) with two or three blocks an SM to fill
// in: the tensor pipe is active 30 % of the time for the chunks' own states and 23 % for the read-outs, DRAM 11 and 14 %, a fifth of the
// warps' places taken.  Token by token on CUDA cores the same took six times the
// arithmetic instructions.
// With 64 heads of 128 x 64, a run of 2,047 tokens: 426 -> 166 us; 16 heads of 64 x 128 with a rotation 122 -> 78; gated, 8 heads of
// 128 x 256, runs of 64, 376, 688 and 1,000 tokens 413 -> 120.  Relative error of the results against 64 bits, walk and
// products: 3.9e-8 and 3.4e-8, fixed decays 2.2e-7 and 1.7e-7, rotated 5.4e-8 and 5.7e-8, gated 2.5e-7 and 1.3e-7.
//
// What is infinite or NaN reaches nothing before its token: a value shows in its column from its token on (a zero weight times
// infinity would be NaN in the tokens before: such values are taken out of the products and their column is NaN from there
// on, also where the walk has infinity), a gate or a key in its head from its token on, a query in its row.
#define MT_TOKENS 64                 // tokens of a chunk, at most
#define MT_COLS 64                   // columns of a block
#define MT_VP (MT_COLS + 8)          // pitches in elements: rows of 16-byte pieces on different banks
#define MT_LOG_MIN -200.f            // e^-200 is zero in 32 bits: a keep of zero keeps its logarithm finite

__device__ __forceinline__ void mt_ldm4(unsigned addr, unsigned (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mt_ldm4t(unsigned addr, unsigned (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mt_mma(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mt_add(float (&d)[4], const float (&f)[4]) {
#pragma unroll
    for (int e = 0; e < 4; ++e) d[e] += f[e];
}
// two 32-bit numbers as three pairs of bfloat16: x = p0.x + p1.x + p2.x up to the last of 24 bits
__device__ __forceinline__ void mt_split2(float x, float y, unsigned& p0, unsigned& p1, unsigned& p2) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 hf = __bfloat1622float2(h);
    x -= hf.x; y -= hf.y;
    const __nv_bfloat162 m = __floats2bfloat162_rn(x, y);
    const float2 mf = __bfloat1622float2(m);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - mf.x, y - mf.y);
    p0 = *(const unsigned*)&h; p1 = *(const unsigned*)&m; p2 = *(const unsigned*)&l;
}
__device__ __forceinline__ void mt_unpack8(const uint4& raw, float (&f)[8]) {
    const __nv_bfloat162* h = (const __nv_bfloat162*)&raw;
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 v = __bfloat1622float2(h[i]); f[2 * i] = v.x; f[2 * i + 1] = v.y; }
}
// eight 32-bit numbers into the three planes of a tile, 16 bytes a plane
__device__ __forceinline__ void mt_put8(const float (&f)[8], __nv_bfloat16* dst, int plane) {
    uint4 p[3];
    mt_split2(f[0], f[1], p[0].x, p[1].x, p[2].x);
    mt_split2(f[2], f[3], p[0].y, p[1].y, p[2].y);
    mt_split2(f[4], f[5], p[0].z, p[1].z, p[2].z);
    mt_split2(f[6], f[7], p[0].w, p[1].w, p[2].w);
#pragma unroll
    for (int i = 0; i < 3; ++i) *(uint4*)(dst + (size_t)i * plane) = p[i];
}

// the first warp: the sums of the logarithms of keep up to each of a chunk's n tokens, and take (zero behind the n-th)
__device__ __forceinline__ void mt_gates(const MemoryChunkArgs& a, int h, int t_first, int n, double* cum, float* take) {
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    double x[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int s = 2 * lane + i;
        const float* g = a.gates + ((size_t)(t_first + min(s, n - 1)) * a.H + h) * 4;
        const float l = g[3];
        x[i] = s < n ? (double)(l < MT_LOG_MIN ? MT_LOG_MIN : l) : 0.0;
        take[s] = s < n ? g[1] : 0.f;
    }
    double sum = x[0] + x[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += up;
    }
    // (from the tokens before alone: taken as the sum up to the next token less that token's, it would be NaN where that one is)
    const double before = __shfl_up_sync(0xffffffffu, sum, 1);
    cum[2 * lane] = (lane > 0 ? before : 0.0) + x[0];
    cum[2 * lane + 1] = sum;
}

// A block's share of the rows [0, n) of q or k (column ``off`` of proj on): all of a thread's pieces are asked for at once (load),
// then turned by their positions where the kind does that and handed to put(row, first dim, eight 32-bit numbers); rows
// behind the n-th are zeros.
template <int D, bool ROT, int THREADS>
struct MtRows {
    static constexpr int P = D / 8, IT = MT_TOKENS * P / THREADS;
    uint4 raw[IT], partner[ROT ? IT : 1];
    __device__ __forceinline__ void load(const MemoryChunkArgs& a, int off, int t_first, int n) {
        const int half = ROT ? a.rot_half / 8 : 0;                  // pieces of a half of the rotated dims
#pragma unroll
        for (int i = 0; i < IT; ++i) {
            const int e = threadIdx.x + i * THREADS, s = e / P, p = e - s * P;
            const __nv_bfloat16* row = (const __nv_bfloat16*)a.proj + (size_t)(t_first + s) * a.ld + off;
            raw[i] = s < n ? *(const uint4*)(row + p * 8) : make_uint4(0, 0, 0, 0);
            if constexpr (ROT) partner[i] = s < n && p < half ? *(const uint4*)(row + (p + half) * 8) : make_uint4(0, 0, 0, 0);
        }
    }
    template <typename Put>
    __device__ __forceinline__ void each(const MemoryChunkArgs& a, int t_first, int n, const Put& put) const {
        const int half = ROT ? a.rot_half / 8 : 0;
#pragma unroll
        for (int i = 0; i < IT; ++i) {
            const int e = threadIdx.x + i * THREADS, s = e / P, p = e - s * P;
            if (ROT && p >= half && p < 2 * half) continue;         // (comes with its partner)
            float u[8];
            mt_unpack8(raw[i], u);
            if (ROT && p < half) {
                float v[8], x[8], y[8];
                mt_unpack8(partner[i], v);
                const size_t at = (size_t)(t_first + min(s, n - 1)) * a.rot_half + p * 8;
                const float *cs = a.cosv + at, *sn = a.sinv + at;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    x[k] = u[k] * cs[k] - v[k] * sn[k];
                    y[k] = v[k] * cs[k] + u[k] * sn[k];
                }
                put(s, p * 8, x);
                put(s, (p + half) * 8, y);
            } else {
                put(s, p * 8, u);
            }
        }
    }
    // the pieces as they are
    __device__ __forceinline__ void copy(__nv_bfloat16* to, int pitch) const {
#pragma unroll
        for (int i = 0; i < IT; ++i) {
            const int e = threadIdx.x + i * THREADS, s = e / P, p = e - s * P;
            *(uint4*)(to + s * pitch + p * 8) = raw[i];
        }
    }
};
// the same of a block's columns of v
template <int THREADS>
struct MtValues {
    static constexpr int P = MT_COLS / 8, IT = MT_TOKENS * P / THREADS;
    uint4 raw[IT];
    __device__ __forceinline__ void load(const MemoryChunkArgs& a, int h, int col0, int t_first, int n) {
#pragma unroll
        for (int i = 0; i < IT; ++i) {
            const int e = threadIdx.x + i * THREADS, s = e / P, j = col0 + (e - s * P) * 8;
            raw[i] = s < n && j < a.V ? *(const uint4*)((const __nv_bfloat16*)a.proj + (size_t)(t_first + s) * a.ld + a.v_off + h * a.V + j)
                                      : make_uint4(0, 0, 0, 0);
        }
    }
};

// the chunk states' layout here: S [D, V], then (gated kind) n [D]
__device__ __forceinline__ float* mt_chunk_state(const MemoryChunkArgs& a, int b, int chunk, int h) {
    return a.chunk_state + (((size_t)b * a.n_chunks + chunk) * a.H + h) * a.D * a.cols;
}

template <int D>
static constexpr size_t mt_states_smem() { return (size_t)(3 * MT_TOKENS * (D + 8) + MT_TOKENS * MT_VP) * 2; }

// every chunk from a zero state: sum_s (L_C / L_s) take_s k_s v_s^T, and the product of its decays
template <int D, bool ROT, bool GATED>
__global__ void __launch_bounds__(128)
memory_chunk_states_tc_kernel(MemoryChunkArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double cum[MT_TOKENS];
    __shared__ float take[MT_TOKENS], weight[MT_TOKENS];
    constexpr int KP = D + 8, PLANE = MT_TOKENS * KP;
    __nv_bfloat16* wk = (__nv_bfloat16*)smem_raw;                   // [3][tokens][D]
    __nv_bfloat16* vs = wk + 3 * PLANE;                             // [tokens][columns]
    gl_grid_wait();
    const int b = blockIdx.z / a.n_chunks, chunk = blockIdx.z - b * a.n_chunks, h = blockIdx.y;
    const int col0 = blockIdx.x * MT_COLS, V = a.V;
    const int qlen = a.seq_qlen[b], t_first = a.seq_qstart[b] + chunk * a.chunk_len;
    const int n = min(a.chunk_len, qlen - chunk * a.chunk_len);
    if (n <= 0) return;
    const int kh = GATED ? h : h / (a.H / a.KVH);
    MtRows<D, ROT, 128> keys;
    MtValues<128> values;
    keys.load(a, a.k_off + kh * D, t_first, n);
    values.load(a, h, col0, t_first, n);
    mt_gates(a, h, t_first, n, cum, take);
#pragma unroll
    for (int i = 0; i < values.IT; ++i) {
        const int e = threadIdx.x + i * 128, s = e / values.P;
        *(uint4*)(vs + s * MT_VP + (e - s * values.P) * 8) = values.raw[i];
    }
    __syncthreads();
    if (threadIdx.x < MT_TOKENS)                                    // (the weights enter a long sum: e in 64-bit, rounded once)
        weight[threadIdx.x] = (float)(exp(cum[n - 1] - cum[threadIdx.x]) * (double)take[threadIdx.x] * (GATED ? 1.0 : (double)a.k_scale));
    __syncthreads();
    keys.each(a, t_first, n, [&](int s, int d, const float (&f)[8]) {
        float y[8];
        const float w = weight[s];
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = s < n ? w * f[i] : 0.f;
        mt_put8(y, wk + s * KP + d, PLANE);
    });
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane >> 2, tq = lane & 3;
    constexpr int MT = D / 64;                                      // tiles of 16 rows a warp
    float acc[MT][8][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.f;
    const unsigned wk0 = (unsigned)__cvta_generic_to_shared(wk), vs0 = (unsigned)__cvta_generic_to_shared(vs);
    for (int ks = 0; ks * 16 < n; ++ks) {
        unsigned bf[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            mt_ldm4t(vs0 + ((ks * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * MT_VP + j * 16 + (lane >> 4) * 8) * 2, bf[j]);
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            float f[8][4] = {};
#pragma unroll
            for (int p = 2; p >= 0; --p) {
                unsigned af[4];
                mt_ldm4t(wk0 + (p * PLANE + (ks * 16 + (lane & 7) + (lane >> 4) * 8) * KP + (warp * MT + i) * 16 + ((lane >> 3) & 1) * 8) * 2, af);
#pragma unroll
                for (int j = 0; j < 8; ++j) mt_mma(f[j], af, bf[j >> 1][(j & 1) * 2], bf[j >> 1][(j & 1) * 2 + 1]);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) mt_add(acc[i][j], f[j]);
        }
    }
    float* cs = mt_chunk_state(a, b, chunk, h);
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int d = (warp * MT + i) * 16 + grp, col = col0 + j * 8 + 2 * tq;
            if (col < V) {                                          // (V is whole pieces of 8)
                *(float2*)(cs + (size_t)d * V + col) = make_float2(acc[i][j][0], acc[i][j][1]);
                *(float2*)(cs + (size_t)(d + 8) * V + col) = make_float2(acc[i][j][2], acc[i][j][3]);
            }
        }
    if (blockIdx.x != 0) return;
    if (GATED && threadIdx.x < D) {
        float sum = 0.f;
        for (int s = 0; s < n; ++s) {
            const __nv_bfloat16* w = wk + s * KP + threadIdx.x;
            sum += __bfloat162float(w[0]) + (__bfloat162float(w[PLANE]) + __bfloat162float(w[2 * PLANE]));
        }
        cs[(size_t)D * V + threadIdx.x] = sum;
    }
    if (threadIdx.x == 0) a.chunk_decay[(((size_t)b * a.n_chunks + chunk) * a.H + h) * D] = (float)exp(cum[n - 1]);
}

// every chunk's start state from the run's start state and what the chunks add, and the run's last state
__global__ void __launch_bounds__(128)
memory_chunk_carry4_kernel(MemoryChunkArgs a) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const int b = blockIdx.z, h = blockIdx.y;
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) * 4, DV = a.D * a.V;
    if (i >= a.D * a.cols) return;
    float* srow = a.state + (size_t)a.seq_slot[b] * a.state_stride;
    float* mine = i < DV ? srow + (size_t)h * DV + i : srow + (size_t)a.H * DV + (size_t)h * a.D + (i - DV);
    float S[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) S[k] = mine[k];                     // (a slot's row begins anywhere)
    const int chunks = (a.seq_qlen[b] + a.chunk_len - 1) / a.chunk_len;
    for (int k0 = 0; k0 < chunks; k0 += 8) {
        float4 last[8];
        float decay[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = min(k0 + j, chunks - 1);
            last[j] = *(const float4*)(mt_chunk_state(a, b, c, h) + i);
            decay[j] = a.chunk_decay[(((size_t)b * a.n_chunks + c) * a.H + h) * a.D];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (k0 + j < chunks) {
                *(float4*)(mt_chunk_state(a, b, k0 + j, h) + i) = make_float4(S[0], S[1], S[2], S[3]);
                S[0] = fmaf(decay[j], S[0], last[j].x); S[1] = fmaf(decay[j], S[1], last[j].y);
                S[2] = fmaf(decay[j], S[2], last[j].z); S[3] = fmaf(decay[j], S[3], last[j].w);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) mine[k] = S[k];
}

template <int D, bool ROT>
static constexpr size_t mt_outputs_smem() {
    return (size_t)((ROT ? 6 : 2) * MT_TOKENS * (D + 8) + MT_TOKENS * MT_VP + 3 * D * MT_VP) * 2;
}

// blocks an SM, stated by shared memory: with 128 rows and a rotation one fits, and held to the registers of two it spilled (16 heads
// of 128 x 128, 2,047 tokens: 181 -> 163 us a launch of all kernels)
template <int D, bool ROT>
static constexpr int mt_outputs_blocks() { return 2 * (mt_outputs_smem<D, ROT>() + 4096) <= 227 * 1024 ? 2 : 1; }

// the read-outs of a chunk from its start state, 64 columns a block: eight warps, 16 tokens and 32 columns each (both of a row
// group's warps take its scores, which are few beside the state's products)
template <int D, bool ROT, bool GATED>
__global__ void __launch_bounds__(256, mt_outputs_blocks<D, ROT>())
memory_chunk_outputs_tc_kernel(MemoryChunkArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ double cum[MT_TOKENS];
    __shared__ float take[MT_TOKENS], n0[GATED ? D : 1];
    __shared__ int bad[MT_COLS];                                    // a column's first token whose value is not finite
    constexpr int KP = D + 8, PLANE = MT_TOKENS * KP, TQ = ROT ? 3 : 1, SPLANE = D * MT_VP;
    __nv_bfloat16* qs = (__nv_bfloat16*)smem_raw;                   // [TQ][tokens][D]
    __nv_bfloat16* ks = qs + TQ * PLANE;
    __nv_bfloat16* vs = ks + TQ * PLANE;                            // [tokens][columns]
    __nv_bfloat16* ss = vs + MT_TOKENS * MT_VP;                     // [3][D][columns]
    gl_grid_wait();
    const int b = blockIdx.z / a.n_chunks, chunk = blockIdx.z - b * a.n_chunks, h = blockIdx.y;
    const int col0 = blockIdx.x * MT_COLS, V = a.V;
    const int qlen = a.seq_qlen[b], t_first = a.seq_qstart[b] + chunk * a.chunk_len;
    const int n = min(a.chunk_len, qlen - chunk * a.chunk_len);
    if (n <= 0) return;
    const int kh = GATED ? h : h / (a.H / a.KVH);
    const float* cs = mt_chunk_state(a, b, chunk, h);
    // everything the block reads is asked for before any of it is used
    MtRows<D, ROT, 256> queries, keys;
    MtValues<256> values;
    float4 start[D * MT_COLS / 1024];
    queries.load(a, a.q_off + kh * D, t_first, n);
    keys.load(a, a.k_off + kh * D, t_first, n);
    values.load(a, h, col0, t_first, n);
#pragma unroll
    for (int i = 0; i < D * MT_COLS / 1024; ++i) {
        const int e = threadIdx.x + i * 256, d = e / (MT_COLS / 4), j = col0 + (e - d * (MT_COLS / 4)) * 4;
        start[i] = j < V ? *(const float4*)(cs + (size_t)d * V + j) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (GATED && threadIdx.x < D) n0[threadIdx.x] = cs[(size_t)D * V + threadIdx.x];
    if (threadIdx.x < MT_COLS) bad[threadIdx.x] = MT_TOKENS;
    mt_gates(a, h, t_first, n, cum, take);
    if constexpr (ROT) {
        queries.each(a, t_first, n, [&](int s, int d, const float (&f)[8]) { mt_put8(f, qs + s * KP + d, PLANE); });
        keys.each(a, t_first, n, [&](int s, int d, const float (&f)[8]) { mt_put8(f, ks + s * KP + d, PLANE); });
    } else {
        queries.copy(qs, KP);
        keys.copy(ks, KP);
    }
#pragma unroll
    for (int i = 0; i < D * MT_COLS / 1024; ++i) {
        const int e = threadIdx.x + i * 256, d = e / (MT_COLS / 4), j = (e - d * (MT_COLS / 4)) * 4;
        uint2 p[3];
        mt_split2(start[i].x, start[i].y, p[0].x, p[1].x, p[2].x);
        mt_split2(start[i].z, start[i].w, p[0].y, p[1].y, p[2].y);
#pragma unroll
        for (int k = 0; k < 3; ++k) *(uint2*)(ss + k * SPLANE + d * MT_VP + j) = p[k];
    }
    __syncthreads();                                                // (``bad`` is set before anyone lowers it)
#pragma unroll
    for (int i = 0; i < values.IT; ++i) {
        const int e = threadIdx.x + i * 256, s = e / values.P, j = (e - s * values.P) * 8;
        unsigned x[4] = {values.raw[i].x, values.raw[i].y, values.raw[i].z, values.raw[i].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if ((x[k] & 0x7f80u) == 0x7f80u) { x[k] &= 0xffff0000u; atomicMin(&bad[j + 2 * k], s); }
            if ((x[k] & 0x7f800000u) == 0x7f800000u) { x[k] &= 0xffffu; atomicMin(&bad[j + 2 * k + 1], s); }
        }
        *(uint4*)(vs + s * MT_VP + j) = make_uint4(x[0], x[1], x[2], x[3]);
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = lane >> 2, tq = lane & 3;
    const int group = warp >> 1, r0 = group * 16, c0 = (warp & 1) * 32;      // this warp's tokens and columns
    if (r0 >= n) return;
    const unsigned q0 = (unsigned)__cvta_generic_to_shared(qs), k0 = (unsigned)__cvta_generic_to_shared(ks);
    const unsigned v0 = (unsigned)__cvta_generic_to_shared(vs), s0 = (unsigned)__cvta_generic_to_shared(ss);
    float acc[4][4], g[8][4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) g[j][e] = 0.f;
    for (int kk = 0; kk < D / 16; ++kk) {
        unsigned af[TQ][4];
#pragma unroll
        for (int p = 0; p < TQ; ++p)
            mt_ldm4(q0 + (p * PLANE + (r0 + (lane & 7) + ((lane >> 3) & 1) * 8) * KP + kk * 16 + (lane >> 4) * 8) * 2, af[p]);
        // the state, smallest parts first (parts whose product is below the last of 24 bits are left out)
        float f[4][4] = {};
#pragma unroll
        for (int p = 2; p >= 0; --p) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                unsigned bf[4];
                mt_ldm4t(s0 + (p * SPLANE + (kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * MT_VP + c0 + j * 16 + (lane >> 4) * 8) * 2, bf);
#pragma unroll
                for (int q = TQ - 1; q >= 0; --q) {
                    if (p + q > 2) continue;
                    mt_mma(f[2 * j], af[q], bf[0], bf[1]);
                    mt_mma(f[2 * j + 1], af[q], bf[2], bf[3]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) mt_add(acc[j], f[j]);
        // the scores of the tokens up to this group's last
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (j > group) break;
            float u[2][4] = {};
#pragma unroll
            for (int p = TQ - 1; p >= 0; --p) {
                unsigned bf[4];
                mt_ldm4(k0 + (p * PLANE + (j * 16 + (lane & 7) + (lane >> 4) * 8) * KP + kk * 16 + ((lane >> 3) & 1) * 8) * 2, bf);
#pragma unroll
                for (int q = TQ - 1; q >= 0; --q) {
                    if (p + q > 2) continue;
                    mt_mma(u[0], af[q], bf[0], bf[1]);
                    mt_mma(u[1], af[q], bf[2], bf[3]);
                }
            }
            mt_add(g[2 * j], u[0]);
            mt_add(g[2 * j + 1], u[1]);
        }
    }
    const int ta = r0 + grp, tb = ta + 8;                            // this lane's two tokens
    const double ca = cum[ta], cb = cum[tb];
    const float la = expf((float)ca) * a.q_scale, lb = expf((float)cb) * a.q_scale;
#pragma unroll
    for (int j = 0; j < 4; ++j) { acc[j][0] *= la; acc[j][1] *= la; acc[j][2] *= lb; acc[j][3] *= lb; }
    const float sc = a.q_scale * (GATED ? 1.0f : a.k_scale);
    float na = 0.f, nb = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        if (j > 2 * group + 1) break;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int s = j * 8 + 2 * tq + e;
            const double c = cum[s];
            const float f = take[s] * sc;
            // (a choice, not a product with zero: what a later token's key is must not show)
            g[j][e] = s <= ta ? g[j][e] * (f * expf((float)(ca - c))) : 0.f;
            g[j][2 + e] = s <= tb ? g[j][2 + e] * (f * expf((float)(cb - c))) : 0.f;
            na += g[j][e];
            nb += g[j][2 + e];
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (i > group) break;
        unsigned pf[3][4];
        mt_split2(g[2 * i][0], g[2 * i][1], pf[0][0], pf[1][0], pf[2][0]);
        mt_split2(g[2 * i][2], g[2 * i][3], pf[0][1], pf[1][1], pf[2][1]);
        mt_split2(g[2 * i + 1][0], g[2 * i + 1][1], pf[0][2], pf[1][2], pf[2][2]);
        mt_split2(g[2 * i + 1][2], g[2 * i + 1][3], pf[0][3], pf[1][3], pf[2][3]);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            unsigned bf[4];
            mt_ldm4t(v0 + ((i * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * MT_VP + c0 + j * 16 + (lane >> 4) * 8) * 2, bf);
            float u[2][4] = {};
#pragma unroll
            for (int p = 2; p >= 0; --p) {
                mt_mma(u[0], pf[p], bf[0], bf[1]);
                mt_mma(u[1], pf[p], bf[2], bf[3]);
            }
            mt_add(acc[2 * j], u[0]);
            mt_add(acc[2 * j + 1], u[1]);
        }
    }
    float da = 1.f, db = 1.f;
    if (GATED) {
        // the normaliser: n.q of the start state (a quad shares a token's dims) and of the chunk's own keys
        float ua = 0.f, ub = 0.f;
        for (int d = tq; d < D; d += 4) {
            ua = fmaf(__bfloat162float(qs[ta * KP + d]), n0[d], ua);
            ub = fmaf(__bfloat162float(qs[tb * KP + d]), n0[d], ub);
        }
        na = fmaf(la, ua, na);
        nb = fmaf(lb, ub, nb);
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) { na += __shfl_xor_sync(0xffffffffu, na, o); nb += __shfl_xor_sync(0xffffffffu, nb, o); }
        const float* ga = a.gates + ((size_t)(t_first + min(ta, n - 1)) * a.H + h) * 4;
        const float* gb = a.gates + ((size_t)(t_first + min(tb, n - 1)) * a.H + h) * 4;
        da = fmaxf(fabsf(na), ga[2]) + 1e-6f;
        db = fmaxf(fabsf(nb), gb[2]) + 1e-6f;
    }
    const float skip = !GATED && a.d_skip ? a.d_skip[h] : 0.f;
    float* out = a.out + (size_t)t_first * a.H * V + (size_t)h * V + col0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int col = c0 + j * 8 + 2 * tq;
        if (col0 + col >= V) continue;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int t = r ? tb : ta;
            if (t >= n) continue;
            float2 y = make_float2(acc[j][2 * r], acc[j][2 * r + 1]);
            if (GATED) { y.x /= r ? db : da; y.y /= r ? db : da; }
            if (!GATED && a.d_skip) {
                y.x = fmaf(skip, __bfloat162float(vs[t * MT_VP + col]), y.x);
                y.y = fmaf(skip, __bfloat162float(vs[t * MT_VP + col + 1]), y.y);
            }
            if (t >= bad[col]) y.x = __int_as_float(0x7fffffff);
            if (t >= bad[col + 1]) y.y = __int_as_float(0x7fffffff);
            *(float2*)(out + (size_t)t * a.H * V + col) = y;
        }
    }
}

// Whether these sizes go on the tensor cores: a chunk's tokens and a head's rows in one block's tiles, rows of whole 16-byte
// pieces.  (Everything else walks: other head sizes, 32-bit inputs, longer chunks, rows that begin anywhere.)
static bool mt_takes(const MemoryChunkArgs& a, int act_dtype) {
    return act_dtype == GL_BF16 && (a.kind == 0 || a.kind == 3) && (a.D == 64 || a.D == 128) && a.V % 8 == 0 && a.chunk_len <= MT_TOKENS
           && a.ld % 8 == 0 && a.q_off % 8 == 0 && a.k_off % 8 == 0 && a.v_off % 8 == 0 && (!a.cosv || a.rot_half % 8 == 0)
           && !(((uintptr_t)a.proj | (uintptr_t)a.chunk_state) & 15) && !((uintptr_t)a.out & 7);
}

template <int D, bool ROT, bool GATED>
static int mt_launch(const MemoryChunkArgs& a, cudaStream_t stream) {
    constexpr size_t s1 = mt_states_smem<D>(), s2 = mt_outputs_smem<D, ROT>();
    if (cudaFuncSetAttribute(memory_chunk_states_tc_kernel<D, ROT, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s1) != cudaSuccess ||
        cudaFuncSetAttribute(memory_chunk_outputs_tc_kernel<D, ROT, GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s2) != cudaSuccess) {
        cudaGetLastError();
        return GL_ERR_SMEM;
    }
    const dim3 grid((a.V + MT_COLS - 1) / MT_COLS, a.H, a.B * a.n_chunks);
    int rc = gl_launch_in_order(memory_chunk_states_tc_kernel<D, ROT, GATED>, grid, dim3(128), s1, stream, a);
    if (rc != 0) return rc;
    rc = gl_launch(memory_chunk_carry4_kernel, dim3((a.D * a.cols / 4 + 127) / 128, a.H, a.B), dim3(128), 0, stream, 1, a);
    if (rc != 0) return rc;
    return gl_launch_in_order(memory_chunk_outputs_tc_kernel<D, ROT, GATED>, grid, dim3(256), s2, stream, a);
}

static int mt_chunks(const MemoryChunkArgs& a, cudaStream_t stream) {
    const bool rot = a.kind == 3 && a.cosv;
    if (a.kind == 0) return a.D == 64 ? mt_launch<64, false, true>(a, stream) : mt_launch<128, false, true>(a, stream);
    if (a.D == 64) return rot ? mt_launch<64, true, false>(a, stream) : mt_launch<64, false, false>(a, stream);
    return rot ? mt_launch<128, true, false>(a, stream) : mt_launch<128, false, false>(a, stream);
}
// ---------------------------------------------------------------------------

// the gated kind's outputs divided by max(|n.q|, e^-m) + 1e-6, all tokens at once
__global__ void __launch_bounds__(256)
memory_divide_kernel(MemoryChunkArgs a) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const long long n = (long long)a.T * a.H * a.V;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long th = i / a.V;
        a.out[i] = a.out[i] / (fmaxf(fabsf(a.nq[th]), a.gates[th * 4 + 2]) + 1e-6f);
    }
}

template <typename TA, int DMAX, int KIND, int NT>
static int launch_memory_chunks_nt(const MemoryChunkArgs& a, cudaStream_t stream) {
    const size_t smem = (size_t)MC_TOKENS * (3 * a.D + NT + 2) * sizeof(float);
    if (smem > 48 * 1024) return GL_ERR_SMEM;
    const dim3 walk((a.cols + NT - 1) / NT, a.H, a.B * a.n_chunks);
    int rc;
    if (KIND == 0 || KIND == 3) {
        const long long n = (long long)a.T * a.H;
        if (KIND == 0) rc = gl_launch(memory_log_gates_kernel<TA>, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, 1, a);
        else rc = gl_launch(memory_decay_gates_kernel<TA>, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, stream, 1, a);
        if (rc != 0) return rc;
    }
    if (KIND == 0) {
        rc = gl_launch(memory_gate_walk_kernel, dim3(a.B * a.H), dim3(32), 0, stream, 1, a);
        if (rc != 0) return rc;
    }
    if constexpr (sizeof(TA) == 2 && (KIND == 0 || KIND == 3)) {
        if (mt_takes(a, GL_BF16)) return mt_chunks(a, stream);
    }
    rc = gl_launch(memory_chunk_decay_kernel<TA, KIND>, dim3((a.D + 127) / 128, a.H, a.B * a.n_chunks), dim3(128), 0, stream, 1, a);
    if (rc != 0) return rc;
    const bool full = a.D == DMAX;
    rc = full ? gl_launch_in_order(memory_chunk_walk_kernel<TA, DMAX, KIND, 1, NT, true>, walk, dim3(NT), smem, stream, a)
              : gl_launch_in_order(memory_chunk_walk_kernel<TA, DMAX, KIND, 1, NT, false>, walk, dim3(NT), smem, stream, a);
    if (rc != 0) return rc;
    rc = gl_launch(memory_chunk_carry_kernel, dim3((a.D * a.cols + 127) / 128, a.H, a.B), dim3(128), 0, stream, 1, a);
    if (rc != 0) return rc;
    rc = full ? gl_launch_in_order(memory_chunk_walk_kernel<TA, DMAX, KIND, 2, NT, true>, walk, dim3(NT), smem, stream, a)
              : gl_launch_in_order(memory_chunk_walk_kernel<TA, DMAX, KIND, 2, NT, false>, walk, dim3(NT), smem, stream, a);
    if (rc != 0 || KIND != 0) return rc;
    const long long n = (long long)a.T * a.H * a.V;
    const long long want = (n + 255) / 256;
    return gl_launch(memory_divide_kernel, dim3((unsigned)(want > 16384 ? 16384 : want)), dim3(256), 0, stream, 1, a);
}

template <typename TA, int DMAX, int KIND>
static int launch_memory_chunks(const MemoryChunkArgs& a, cudaStream_t stream) {
    // heads of up to 64 columns (a state-space layer's) would leave half of a block's threads without a column
    if constexpr (KIND == 3) {
        if (a.cols <= 64) return launch_memory_chunks_nt<TA, DMAX, KIND, 64>(a, stream);
    }
    return launch_memory_chunks_nt<TA, DMAX, KIND, MC_THREADS>(a, stream);
}

template <typename TA, int KIND>
static int dispatch_memory_chunks(const MemoryChunkArgs& a, cudaStream_t stream) {
    if (a.D <= 16) return launch_memory_chunks<TA, 16, KIND>(a, stream);
    if (a.D <= 32) return launch_memory_chunks<TA, 32, KIND>(a, stream);
    if (a.D <= 64) return launch_memory_chunks<TA, 64, KIND>(a, stream);
    if (a.D <= 128) return launch_memory_chunks<TA, 128, KIND>(a, stream);
    return GL_ERR_SHAPE;
}

template <typename TA>
static int dispatch_memory_chunks_kind(const MemoryChunkArgs& a, cudaStream_t stream) {
    if (a.kind == 0) return dispatch_memory_chunks<TA, 0>(a, stream);
    if (a.kind == 1) return dispatch_memory_chunks<TA, 1>(a, stream);
    return dispatch_memory_chunks<TA, 3>(a, stream);
}

// kernels that gl_memory_chunks launches
GL_API int gl_memory_chunks_launches(const MemoryChunkArgs* args, int act_dtype) {
    const int gates = args->kind == 0 ? 2 : args->kind == 3 ? 1 : 0;
    return gates + (mt_takes(*args, act_dtype) ? 3 : args->kind == 0 ? 5 : 4);
}

GL_API int gl_memory_chunks(const MemoryChunkArgs* args, int act_dtype, cudaStream_t stream) {
    const MemoryChunkArgs& a = *args;
    if (a.B <= 0 || a.T <= 0) return GL_OK;
    if (a.H <= 0 || a.D <= 0 || a.D > 128 || a.V <= 0 || a.n_chunks <= 0 || a.chunk_len <= 0) return GL_ERR_SHAPE;
    if ((a.kind != 0 && a.kind != 1 && a.kind != 3) || a.cols != a.V + (a.kind == 0 ? 1 : 0)) return GL_ERR_SHAPE;
    if ((long long)a.B * a.n_chunks > 65535 || a.H > 65535) return GL_ERR_SHAPE;
    if (!a.chunk_state || !a.chunk_decay || (a.kind == 0 && (!a.nq || !a.gates || !(a.cap > 0.f)))) return GL_ERR_SHAPE;
    if (a.kind == 3) {
        if (!a.gates || a.KVH <= 0 || a.H % a.KVH) return GL_ERR_SHAPE;
        if ((a.lower != nullptr) == (a.gates_in != nullptr)) return GL_ERR_SHAPE;
        if (a.gates_in && (!a.a_log || !a.dt_bias)) return GL_ERR_SHAPE;
        if (a.cosv && (!a.sinv || a.rot_half <= 0 || 2 * a.rot_half > a.D)) return GL_ERR_SHAPE;
    }
    if (act_dtype == GL_F32) return dispatch_memory_chunks_kind<float>(a, stream);
    if (act_dtype == GL_BF16) return dispatch_memory_chunks_kind<__nv_bfloat16>(a, stream);
    return GL_ERR_DTYPE;
}
