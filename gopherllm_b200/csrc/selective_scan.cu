// The selective state-space scan.  A library of its own: what the compiler gives its kernels (registers, inlining) then
// does not change with the matrix memories' kernels, nor theirs with it.
#include <type_traits>

#include "common.cuh"
#include "recurrent_common.cuh"

#define SS_CHUNK 16         // tokens staged at a time

// rc_decay of an x that is never positive, without a branch (the same two formulas, both taken, one chosen): in a walk over
// tokens the branches of one token's decays would keep the next tokens' from being computed beside them.
__device__ __forceinline__ float rc_decay_falling(float x) {
    float p = 2.755731922e-6f;
    p = fmaf(p, x, 2.48015873e-5f);
    p = fmaf(p, x, 1.984126984e-4f);
    p = fmaf(p, x, 1.388888889e-3f);
    p = fmaf(p, x, 8.333333333e-3f);
    p = fmaf(p, x, 4.166666667e-2f);
    p = fmaf(p, x, 1.666666667e-1f);
    p = fmaf(p, x, 0.5f);
    p = fmaf(p, x, 1.0f);
    p = fmaf(p, x, 1.0f);
    const float e = expf(x);
    return x > -0.5f ? p : e;
}

// ---------------------------------------------------------------------------
// Selective scan.  Per channel c and state n:
//   dt = softplus(dtp[t, c]);  S[c, n] <- e^(dt A[c, n]) S[c, n] + dt x[t, c] B[t, n],  A = -e^(A_log)
//   y[t, c] = (sum_n S[c, n] C[t, n] + D[c] x[t, c]) * silu(z[t, c])
// A channel's states are spread over G adjacent lanes, NPT states a lane (fewer states a lane and more lanes
// when the grid would otherwise leave the SMs with a warp or two each: a thread walks the tokens in order).
// ---------------------------------------------------------------------------
struct SelectiveScanArgs {
    const void* x;            // [T, C] activation type (the convolution's output)
    const float* dtp;         // [T, C] 32-bit: the step size before softplus, bias included
    const void* bc;           // [T, 2N] activation type: B then C
    const void* z;            // activation type, row pitch z_ld, first column z_off
    void* out;                // [T, C] activation type
    const float* a_log;       // [C, N]
    const float* d_skip;      // [C]
    float* state;             // [slots, state_stride], S [C, N] first
    const int* seq_slot;
    const int* seq_qstart;
    const int* seq_qlen;
    int B, C, N, z_ld, z_off, state_stride;
    // a long run cut into chunks of chunk_len tokens that are walked side by side (n_chunks > 1):
    //   first every chunk from a zero state, keeping its last state and the sum of its step sizes;
    //   then a carry over the chunks, S_start[k+1] = e^(A sum_k) S_start[k] + last_k (the decays of a chunk
    //   multiply to e^(A sum of its step sizes));  then every chunk again from its true start, with outputs.
    float* chunk_state;       // [B, n_chunks, C, N]
    float* chunk_dt;          // [B, n_chunks, C]
    int chunk_len, n_chunks;
    int one_token;            // every run is one token
    int by_channel;           // chunks are walked a thread a channel (N <= SC_STATE)
};

// MODE 0: a run in one piece.  MODE 1: a chunk from a zero state, no outputs.  MODE 2: a chunk from its start.
// MODE 3: a run in one piece, of one token: nothing to fetch ahead or to walk together, and so few registers that all
// blocks of a step run at once (4 sequences, 4,096 channels: 4.4 us; with the walk's 80 registers 6.9).
template <typename TA, int SS_NPT, int MODE>
__global__ void __launch_bounds__(RC_THREADS, MODE == 3 ? (SS_NPT <= 2 ? 12 : 8) : SS_NPT <= 2 ? 6 : 4)
selective_scan_kernel(SelectiveScanArgs a, int G) {
    constexpr bool ONE = MODE == 3, WHOLE = MODE == 0 || ONE;
    extern __shared__ float smem[];
    // (launched in order, not early: placed beside the kernel before, the blocks of a scan sat several to an SM
    // for its whole length, and a prompt of 2,048 tokens took 25 ms instead of 16)
    gl_grid_wait();
    const int N = a.N, C = a.C;
    const int CPB = RC_THREADS / G;
    const int b = blockIdx.y, c0 = blockIdx.x * CPB;
    const int g = threadIdx.x % G, cl = threadIdx.x / G;
    const int c = c0 + cl;
    const bool live = c < C;
    const int qlen = a.seq_qlen[b], qstart = a.seq_qstart[b];
    const int chunk = WHOLE ? 0 : blockIdx.z;
    const int t_begin = WHOLE ? 0 : chunk * a.chunk_len;
    const int t_end = WHOLE ? qlen : min(qlen, t_begin + a.chunk_len);
    if (t_begin >= qlen) return;                      // (the whole block: this sequence has no such chunk)
    float* Bs = smem;                                 // [CHUNK][N]
    float* Cs = Bs + SS_CHUNK * N;                    // [CHUNK][N]
    float* ds = Cs + SS_CHUNK * N;                    // [CHUNK][CPB] step sizes
    float* xs = ds + SS_CHUNK * CPB;                  // [CHUNK][CPB]
    float* zs = xs + SS_CHUNK * CPB;                  // [CHUNK][CPB]
    float* S_g = a.state + (size_t)a.seq_slot[b] * a.state_stride + (size_t)(live ? c : 0) * N;
    float* S_c = WHOLE ? S_g : a.chunk_state + (((size_t)b * a.n_chunks + chunk) * C + (live ? c : 0)) * N;
    float S[SS_NPT], A[SS_NPT];
#pragma unroll
    for (int i = 0; i < SS_NPT; ++i) {
        const int n = g + G * i;
        const bool ok = live && n < N;
        S[i] = (ok && MODE != 1) ? (WHOLE ? S_g[n] : S_c[n]) : 0.f;
        A[i] = ok ? -expf(a.a_log[(size_t)c * N + n]) : -1.f;      // (not zero: an infinite step times zero would be NaN)
    }
    float dt_sum = 0.f;
    // A thread's share of a chunk's inputs travels while the chunk before is walked and waits in registers: a chunk's trip
    // to memory would otherwise stand between two walks of sixteen tokens and be as long as both.  Few states a lane mean
    // few channels a block and so few elements a thread; larger shares are staged behind the walk (eight states a lane is
    // the form for many sequences, whose blocks run under one another's trips and would be fewer with more registers).
    // And a few tokens are walked together: everything that does not depend on the state (decays, what enters, what reads)
    // before the first of them, the read-outs' sums over the lanes and their stores behind the last.  One token after the
    // other, each waited out its own loads, decays, shuffles and the store that might alias the next one's loads.
    // Four prompts of 64 to 1,000 tokens, 4,096 channels of 16 states: 656 us a launch; inputs ahead and decays without a
    // branch 449, tokens together 335.  One of 1,000: 396, 320, 233; one of 2,040 in chunks 649, 516, 471.
    constexpr int PX = SS_NPT >= 2 ? 4 : 2, PB = 4, TOGETHER = ONE ? 1 : SS_NPT >= 8 ? 2 : 4;
    const bool ahead = !ONE && SS_NPT <= 2 && SS_CHUNK * CPB <= PX * RC_THREADS && SS_CHUNK * N <= PB * RC_THREADS;
    float rd[PX], rx[PX], rz[PX], rb[PB], rc[PB];
    const int my_j = threadIdx.x % CPB, my_s = threadIdx.x / CPB;      // (CPB divides RC_THREADS: one channel a thread)
    const bool my_ok = c0 + my_j < C;
    auto fetch = [&](int s0) {
        const int ns = min(SS_CHUNK, t_end - s0);
#pragma unroll
        for (int i = 0; i < PB; ++i) {
            const int e = threadIdx.x + i * RC_THREADS;
            if (e < ns * N) {
                const int s = e / N, n = e - s * N;
                const TA* row = (const TA*)a.bc + (size_t)(qstart + s0 + s) * 2 * N;
                rb[i] = gl_load(row + n);
                rc[i] = gl_load(row + N + n);
            }
        }
#pragma unroll
        for (int i = 0; i < PX; ++i) {
            const int s = my_s + i * G;
            rd[i] = rx[i] = rz[i] = 0.f;
            if (s < ns && my_ok) {
                const size_t t = (size_t)(qstart + s0 + s);
                rd[i] = a.dtp[t * C + c0 + my_j];
                rx[i] = gl_load((const TA*)a.x + t * C + c0 + my_j);
                if (MODE != 1) rz[i] = gl_load((const TA*)a.z + t * a.z_ld + a.z_off + c0 + my_j);
            }
        }
    };
    if (ahead) fetch(t_begin);
    for (int s0 = t_begin; s0 < t_end; s0 += SS_CHUNK) {
        const int ns = min(SS_CHUNK, t_end - s0);
        __syncthreads();
        if (ahead) {
#pragma unroll
            for (int i = 0; i < PB; ++i) {
                const int e = threadIdx.x + i * RC_THREADS;
                if (e < ns * N) { Bs[e] = rb[i]; Cs[e] = rc[i]; }
            }
#pragma unroll
            for (int i = 0; i < PX; ++i) {
                const int s = my_s + i * G, e = s * CPB + my_j;
                if (s < ns) { ds[e] = my_ok ? rc_softplus(rd[i]) : 0.f; xs[e] = rx[i]; zs[e] = rz[i]; }
            }
        } else {
            for (int e = threadIdx.x; e < ns * N; e += RC_THREADS) {
                const int s = e / N, n = e - s * N;
                const TA* row = (const TA*)a.bc + (size_t)(qstart + s0 + s) * 2 * N;
                Bs[e] = gl_load(row + n);
                Cs[e] = gl_load(row + N + n);
            }
            for (int e = threadIdx.x; e < ns * CPB; e += RC_THREADS) {
                const int s = e / CPB, j = e - s * CPB;
                const size_t t = (size_t)(qstart + s0 + s);
                const bool ok = c0 + j < C;
                ds[e] = ok ? rc_softplus(a.dtp[t * C + c0 + j]) : 0.f;
                xs[e] = ok ? gl_load((const TA*)a.x + t * C + c0 + j) : 0.f;
                zs[e] = ok ? gl_load((const TA*)a.z + t * a.z_ld + a.z_off + c0 + j) : 0.f;
            }
        }
        __syncthreads();
        if (ahead && s0 + SS_CHUNK < t_end) fetch(s0 + SS_CHUNK);
        int sb = 0;
        auto walk = [&](auto tokens) {
            constexpr int U = decltype(tokens)::value;
            float keep[U][SS_NPT], add[U][SS_NPT], read[U][SS_NPT], y[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int s = sb + u;
                const float dt = ds[s * CPB + cl], dx = dt * xs[s * CPB + cl];
                if (MODE == 1) dt_sum += dt;
                y[u] = 0.f;
#pragma unroll
                for (int i = 0; i < SS_NPT; ++i) {
                    const int n = g + G * i;
                    const bool ok = n < N;              // (a state that does not exist stays zero)
                    keep[u][i] = rc_decay_falling(dt * A[i]);                 // dt >= 0, A <= 0
                    add[u][i] = ok ? dx * Bs[s * N + n] : 0.f;
                    read[u][i] = ok ? Cs[s * N + n] : 0.f;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int i = 0; i < SS_NPT; ++i) {
                    S[i] = fmaf(keep[u][i], S[i], add[u][i]);
                    y[u] = fmaf(S[i], read[u][i], y[u]);
                }
            for (int o = G >> 1; o > 0; o >>= 1)
#pragma unroll
                for (int u = 0; u < U; ++u) y[u] += __shfl_xor_sync(0xffffffffu, y[u], o);
            if (g == 0) {
#pragma unroll
                for (int u = 0; u < U; ++u) ds[(sb + u) * CPB + cl] = y[u];      // the step size has been used: its place takes the sum
            }
            sb += U;
        };
#pragma unroll 1
        while (sb + TOGETHER <= ns) walk(std::integral_constant<int, TOGETHER>{});
#pragma unroll 1
        while (sb < ns) walk(std::integral_constant<int, 1>{});
        if (MODE == 1) continue;
        __syncthreads();
        // the skip connection and the gate do not go from token to token: all of the chunk's outputs at once
        for (int e = threadIdx.x; e < ns * CPB; e += RC_THREADS) {
            const int s = e / CPB, j = e - s * CPB;
            if (c0 + j < C) {
                const float y = fmaf(a.d_skip[c0 + j], xs[e], ds[e]);
                gl_store((TA*)a.out + (size_t)(qstart + s0 + s) * C + c0 + j, y * rc_silu(zs[e]));
            }
        }
    }
    if (live && (MODE != 2 || t_end == qlen)) {       // the state row takes the run's last state
        float* dst = MODE == 1 ? S_c : S_g;
#pragma unroll
        for (int i = 0; i < SS_NPT; ++i) {
            const int n = g + G * i;
            if (n < N) dst[n] = S[i];
        }
    }
    if (MODE == 1 && live && g == 0) a.chunk_dt[((size_t)b * a.n_chunks + chunk) * C + c] = dt_sum;
}

// Between the two walks: every chunk's start state from the run's start state and the chunks' last states.
__global__ void __launch_bounds__(128)
selective_carry_kernel(SelectiveScanArgs a) {
    gl_grid_launch_dependents();
    gl_grid_wait();
    const int b = blockIdx.y;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)a.C * a.N) return;
    const int c = (int)(i / a.N);
    const int chunks = (a.seq_qlen[b] + a.chunk_len - 1) / a.chunk_len;
    float S = a.state[(size_t)a.seq_slot[b] * a.state_stride + i];
    const float A = -expf(a.a_log[i]);
    // (eight chunks' last states and step sizes are asked for at once: a chunk costs no trip to memory of its own)
    for (int k0 = 0; k0 < chunks; k0 += 8) {
        float last[8], keep[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const size_t at = (size_t)b * a.n_chunks + min(k0 + j, chunks - 1);
            last[j] = a.chunk_state[at * a.C * a.N + i];
            keep[j] = a.chunk_dt[at * a.C + c];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) keep[j] = expf(A * keep[j]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (k0 + j < chunks) {
                a.chunk_state[((size_t)b * a.n_chunks + k0 + j) * a.C * a.N + i] = S;
                S = fmaf(keep[j], S, last[j]);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// The walks over chunks for states of up to SC_STATE numbers: a thread a channel, all of its states in registers, two to an
// instruction.  Chunks give the machine its threads, so a channel need not be spread over lanes: nothing is exchanged between
// lanes, the step size and the gate are taken once a channel, and a token's sixteen states are sixteen chains side by side.
// What bounds it: the FMA pipe (fifteen of a state's twenty operations a walk), active 57 % of the time, and the ALU's (48 %).
// 4,096 channels of 16 states in bfloat16, against eight lanes a channel: runs of 64, 376, 688 and 1,000 tokens in one piece
// 407 us, in chunks of 64 256; one of 1,000 221 and 123 (chunks of 32); one of 2,040 in chunks of 128 459, now 229 (of 64).
// ---------------------------------------------------------------------------
#define SC_STATE 16
#define SC_TOKENS 64        // tokens whose B and C are staged at a time
#define SC_GROUP 4          // tokens whose step size, input and gate are on their way while as many are walked

// e^x of two numbers that are never positive: x = k ln 2 + f with the logarithm in two parts (Cody and Waite: the high part has
// 15 bits, so that k, of up to 7 bits, times it is exact, and the low part is what is left of ln 2), |f| < 0.347, and
// the series of e^f to f^7 (the next term is below 2^-27).  Near zero k is 0 and f is x itself, so a slow decay is rounded once.
// Below -87 (where k would leave the exponent) it is zero.
__device__ __forceinline__ unsigned long long ss_decay2(unsigned long long x2) {
    const auto both = [](float v) { return mc_pack(v, v); };
    const float2 x = mc_unpack(x2);
    const bool gone0 = x.x < -87.f, gone1 = x.y < -87.f;
    const unsigned long long y = mc_pack(gone0 ? -87.f : x.x, gone1 ? -87.f : x.y);
    const unsigned long long t = mc_fma2(y, both(1.44269504f), both(12582912.f));       // k in the low bits
    const unsigned long long k = mc_fma2(t, both(1.f), both(-12582912.f));
    const unsigned long long f = mc_fma2(k, both(-1.42860677e-6f), mc_fma2(k, both(-0.693145752f), y));
    unsigned long long p = mc_fma2(both(1.f / 5040.f), f, both(1.f / 720.f));
    p = mc_fma2(p, f, both(1.f / 120.f));
    p = mc_fma2(p, f, both(1.f / 24.f));
    p = mc_fma2(p, f, both(1.f / 6.f));
    p = mc_fma2(p, f, both(0.5f));
    p = mc_fma2(p, f, both(1.f));
    p = mc_fma2(p, f, both(1.f));
    const float2 e = mc_unpack(p), n = mc_unpack(t);
    const float r0 = __int_as_float(__float_as_int(e.x) + (__float_as_int(n.x) << 23));
    const float r1 = __int_as_float(__float_as_int(e.y) + (__float_as_int(n.y) << 23));
    // (a NaN is handed on: the bits put together above are no NaN's)
    return mc_pack(gone0 ? 0.f : x.x != x.x ? x.x : r0, gone1 ? 0.f : x.y != x.y ? x.y : r1);
}

// MODE 1: a chunk from a zero state, no outputs.  MODE 2: a chunk from its start.  FULL: N == SC_STATE.
template <typename TA, int MODE, bool FULL>
__global__ void __launch_bounds__(RC_THREADS, 4)
selective_chunk_kernel(SelectiveScanArgs a) {
    __shared__ __align__(16) float bcs[SC_TOKENS][2 * SC_STATE];    // B, then C
    gl_grid_wait();
    const int N = a.N, C = a.C, b = blockIdx.y, chunk = blockIdx.z;
    const int c = blockIdx.x * RC_THREADS + threadIdx.x;
    const bool live = c < C;
    const int qlen = a.seq_qlen[b], qstart = a.seq_qstart[b];
    const int t_begin = chunk * a.chunk_len, t_end = min(qlen, t_begin + a.chunk_len);
    if (t_begin >= qlen) return;                      // (the whole block: this sequence has no such chunk)
    const int cc = live ? c : 0;
    float* S_c = a.chunk_state + (((size_t)b * a.n_chunks + chunk) * C + cc) * N;
    unsigned long long S[SC_STATE / 2], A[SC_STATE / 2];
#pragma unroll
    for (int i = 0; i < SC_STATE / 2; ++i) {
        float s[2], r[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int n = 2 * i + k;
            s[k] = MODE == 2 && n < N ? S_c[n] : 0.f;
            r[k] = n < N ? -expf(a.a_log[(size_t)cc * N + n]) : -1.f;        // (not zero: an infinite step times zero would be NaN)
        }
        S[i] = mc_pack(s[0], s[1]);
        A[i] = mc_pack(r[0], r[1]);
    }
    const float skip = MODE == 2 ? a.d_skip[cc] : 0.f;
    float dt_sum = 0.f;
    float rd[SC_GROUP], rx[SC_GROUP], rz[SC_GROUP];
    auto fetch = [&](int t) {
#pragma unroll
        for (int u = 0; u < SC_GROUP; ++u) {
            const size_t row = (size_t)(qstart + min(t + u, t_end - 1));
            rd[u] = a.dtp[row * C + cc];
            rx[u] = gl_load((const TA*)a.x + row * C + cc);
            rz[u] = MODE == 2 ? gl_load((const TA*)a.z + row * a.z_ld + a.z_off + cc) : 0.f;
        }
    };
    fetch(t_begin);
    for (int s0 = t_begin; s0 < t_end; s0 += SC_TOKENS) {
        const int ns = min(SC_TOKENS, t_end - s0);
        __syncthreads();
        for (int e = threadIdx.x; e < ns * 2 * SC_STATE; e += RC_THREADS) {
            const int s = e / (2 * SC_STATE), j = e - s * (2 * SC_STATE), n = j & (SC_STATE - 1);
            const TA* row = (const TA*)a.bc + (size_t)(qstart + s0 + s) * 2 * N;
            bcs[s][j] = n < N ? gl_load(row + (j < SC_STATE ? n : N + n)) : 0.f;
        }
        __syncthreads();
        for (int g0 = 0; g0 < ns; g0 += SC_GROUP) {
            float d[SC_GROUP], x[SC_GROUP], z[SC_GROUP];
#pragma unroll
            for (int u = 0; u < SC_GROUP; ++u) { d[u] = rd[u]; x[u] = rx[u]; z[u] = rz[u]; }
            if (s0 + g0 + SC_GROUP < t_end) fetch(s0 + g0 + SC_GROUP);
#pragma unroll
            for (int u = 0; u < SC_GROUP; ++u) {
                if (g0 + u >= ns) break;
                const float dt = rc_softplus(d[u]), dx = dt * x[u];
                if (MODE == 1) dt_sum += dt;
                const unsigned long long dt2 = mc_pack(dt, dt);
                // (nothing enters a state that does not exist: an infinite input times its B of zero would be NaN)
                auto dx2 = [&](int i) { return mc_pack(FULL || 2 * i < N ? dx : 0.f, FULL || 2 * i + 1 < N ? dx : 0.f); };
                unsigned long long y2 = mc_pack(0.f, 0.f);
                const ulonglong2* row = (const ulonglong2*)bcs[g0 + u];
#pragma unroll
                for (int i = 0; i < SC_STATE / 2; i += 2) {
                    const ulonglong2 B = row[i / 2];
                    S[i] = mc_fma2(ss_decay2(mc_mul2(dt2, A[i])), S[i], mc_mul2(dx2(i), B.x));
                    S[i + 1] = mc_fma2(ss_decay2(mc_mul2(dt2, A[i + 1])), S[i + 1], mc_mul2(dx2(i + 1), B.y));
                    if (MODE == 2) {
                        const ulonglong2 Cn = row[SC_STATE / 4 + i / 2];
                        y2 = mc_fma2(S[i], Cn.x, y2);
                        y2 = mc_fma2(S[i + 1], Cn.y, y2);
                    }
                }
                if (MODE == 2 && live) {
                    const float2 y = mc_unpack(y2);
                    gl_store((TA*)a.out + (size_t)(qstart + s0 + g0 + u) * C + c, fmaf(skip, x[u], y.x + y.y) * rc_silu(z[u]));
                }
            }
        }
    }
    if (!live) return;
    if (MODE == 1 || t_end == qlen) {                 // the state row takes the run's last state
        float* dst = MODE == 1 ? S_c : a.state + (size_t)a.seq_slot[b] * a.state_stride + (size_t)c * N;
#pragma unroll
        for (int i = 0; i < SC_STATE / 2; ++i) {
            const float2 s = mc_unpack(S[i]);
            if (2 * i < N) dst[2 * i] = s.x;
            if (2 * i + 1 < N) dst[2 * i + 1] = s.y;
        }
    }
    if (MODE == 1) a.chunk_dt[((size_t)b * a.n_chunks + chunk) * C + c] = dt_sum;
}

template <typename TA>
static int launch_selective_chunks(const SelectiveScanArgs& a, cudaStream_t stream) {
    const dim3 grid((a.C + RC_THREADS - 1) / RC_THREADS, a.B, a.n_chunks);
    const bool full = a.N == SC_STATE;
    int rc = full ? gl_launch_in_order(selective_chunk_kernel<TA, 1, true>, grid, dim3(RC_THREADS), 0, stream, a)
                  : gl_launch_in_order(selective_chunk_kernel<TA, 1, false>, grid, dim3(RC_THREADS), 0, stream, a);
    if (rc != 0) return rc;
    const long long n = (long long)a.C * a.N;
    rc = gl_launch(selective_carry_kernel, dim3((unsigned)((n + 127) / 128), a.B), dim3(128), 0, stream, 1, a);
    if (rc != 0) return rc;
    return full ? gl_launch_in_order(selective_chunk_kernel<TA, 2, true>, grid, dim3(RC_THREADS), 0, stream, a)
                : gl_launch_in_order(selective_chunk_kernel<TA, 2, false>, grid, dim3(RC_THREADS), 0, stream, a);
}

template <typename TA, int NPT>
static int launch_selective_scan(const SelectiveScanArgs& a, cudaStream_t stream) {
    int G = 1;
    while (G * NPT < a.N) G <<= 1;
    if (G > 32) return GL_ERR_SHAPE;
    const int CPB = RC_THREADS / G;
    const size_t smem = (size_t)SS_CHUNK * (2 * a.N + 3 * CPB) * sizeof(float);
    if (smem > 48 * 1024) return GL_ERR_SMEM;
    if (a.n_chunks <= 1) {
        const dim3 grid((a.C + CPB - 1) / CPB, a.B);
        if (a.one_token) return gl_launch_in_order(selective_scan_kernel<TA, NPT, 3>, grid, dim3(RC_THREADS), smem, stream, a, G);
        return gl_launch_in_order(selective_scan_kernel<TA, NPT, 0>, grid, dim3(RC_THREADS), smem, stream, a, G);
    }
    const dim3 grid((a.C + CPB - 1) / CPB, a.B, a.n_chunks);
    int rc = gl_launch_in_order(selective_scan_kernel<TA, NPT, 1>, grid, dim3(RC_THREADS), smem, stream, a, G);
    if (rc != 0) return rc;
    const long long n = (long long)a.C * a.N;
    rc = gl_launch(selective_carry_kernel, dim3((unsigned)((n + 127) / 128), a.B), dim3(128), 0, stream, 1, a);
    if (rc != 0) return rc;
    return gl_launch_in_order(selective_scan_kernel<TA, NPT, 2>, grid, dim3(RC_THREADS), smem, stream, a, G);
}

static int selective_scan_blocks(const SelectiveScanArgs& a, int npt) {
    int G = 1;
    while (G * npt < a.N) G <<= 1;
    if (G > 32) return -1;
    const int CPB = RC_THREADS / G;
    return ((a.C + CPB - 1) / CPB) * a.B * (a.n_chunks > 1 ? a.n_chunks : 1);
}

template <typename TA>
static int dispatch_selective_scan(const SelectiveScanArgs& a, cudaStream_t stream) {
    if (a.n_chunks > 1 && a.by_channel) return a.N <= SC_STATE ? launch_selective_chunks<TA>(a, stream) : GL_ERR_SHAPE;
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 148;
    }
    const int want = 4 * sms;
    const int b8 = selective_scan_blocks(a, 8), b2 = selective_scan_blocks(a, 2), b1 = selective_scan_blocks(a, 1);
    if (b8 >= want || (b2 < 0 && b1 < 0)) return launch_selective_scan<TA, 8>(a, stream);
    if (b2 >= want || b1 < 0) return b2 >= 0 ? launch_selective_scan<TA, 2>(a, stream) : launch_selective_scan<TA, 8>(a, stream);
    return launch_selective_scan<TA, 1>(a, stream);
}

GL_API int gl_selective_scan(const SelectiveScanArgs* args, int act_dtype, cudaStream_t stream) {
    const SelectiveScanArgs& a = *args;
    if (a.B <= 0) return GL_OK;
    if (a.C <= 0 || a.N <= 0 || a.N > 256 || a.B > 65535) return GL_ERR_SHAPE;
    if (a.n_chunks > 1 && (!a.chunk_state || !a.chunk_dt || a.chunk_len <= 0 || a.n_chunks > 65535)) return GL_ERR_SHAPE;
    if (act_dtype == GL_F32) return dispatch_selective_scan<float>(a, stream);
    if (act_dtype == GL_BF16) return dispatch_selective_scan<__nv_bfloat16>(a, stream);
    return GL_ERR_DTYPE;
}
