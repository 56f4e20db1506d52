// Attention over the paged cache with 32-bit arithmetic, for any head size and
// any element type: the kernel of the 32-bit path and the one the fast kernels
// are checked against.
//
// One warp owns one query row (token, head); the warps of a block are
// consecutive tokens of one sequence and share the key/value tiles they stage
// in shared memory.  Scores, the running maximum, the sum and the output
// accumulate in 32-bit (the reference: model.go:3346-3366, 3801-3855; it makes
// two passes, this one rescales on the fly, which differs by rounding only).
// A query at position p sees keys lo..p, lo = 0 or p-window+1
// (model.go:2707-2710); nothing else masks.
//
// A sequence that brings one token has one query row for a block of eight warps: there, from
// AG_SHARE_FROM pages on, the warps share the row's pages or half pages (ag_one_token), and their softmaxes are merged in the
// warps' order.  What bounds such a row is the chain of trips to memory, half a page after the other.  us a launch, one warp
// walking all pages / whole pages shared, values asked for behind their keys / now, 32 bits: 4 sequences of 16 to 300 positions, 32
// heads of 64 57 / 17.5 / 9; 1 x 2,000 385 / 92 / 28; 16 heads of 100, 64 x 300 - / 186 / 124, 16 x 2,000 - / 314 / 163.
// On fewer pages the tiles' wide loads are ahead (1 x 10 positions, 8 heads of 40: 12 us with tiles, 16 without; 1 x 100 23 and
// 29; 16 x 128 29 and 31).  The form depends on the sequence's own run alone, so a row still does not depend on the batch around it.
#include <type_traits>

#include "common.cuh"

struct AttnArgs {
    const void* q;            // [T, nH*hd] activation type, already scaled
    void* out;                // [T, nH*hd] activation type
    const void* k_cache;      // [pages, nKV, GL_PAGE, hd] cache type
    const void* v_cache;
    const int* seq_qstart;    // [B] row of each sequence's first token
    const int* seq_qlen;      // [B] tokens of each sequence in this step
    const int* seq_ctx;       // [B] positions cached before this step
    const int* pages;         // [B, max_pages]
    int B, nH, nKV, hd, max_pages, window, max_qlen;
    float score_scale;
    int n_pages;              // pages of the cache entry (read by builds that check indices; 0: unknown)
};

#define AG_ROWS 8
#define AG_SHARE_FROM 4               // pages a one-token row sees from which its block's warps share them

__device__ __forceinline__ float4 ag_load4(const float* p) { return *(const float4*)p; }
__device__ __forceinline__ float4 ag_load4(const __nv_bfloat16* p) {
    const uint2 raw = *(const uint2*)p;
    const float2 x = __bfloat1622float2(*(const __nv_bfloat162*)&raw.x), y = __bfloat1622float2(*(const __nv_bfloat162*)&raw.y);
    return make_float4(x.x, x.y, y.x, y.y);
}

// q . k with k in ascending order; rows of whole 16-byte (of bfloat16 also 8-byte) pieces are read as such
__device__ __forceinline__ float ag_dot(const float* q, const float* k, int hd) {
    float s = 0.f;
    if ((hd & 3) == 0 && ((uintptr_t)k & 15) == 0) {
#pragma unroll 8
        for (int d = 0; d < hd; d += 4) {
            const float4 v = *(const float4*)(k + d);
            s = fmaf(q[d], v.x, s); s = fmaf(q[d + 1], v.y, s); s = fmaf(q[d + 2], v.z, s); s = fmaf(q[d + 3], v.w, s);
        }
    } else {
        for (int d = 0; d < hd; ++d) s = fmaf(q[d], k[d], s);
    }
    return s;
}
__device__ __forceinline__ float ag_add2(float s, const float* q, unsigned pair) {
    const float2 v = __bfloat1622float2(*(const __nv_bfloat162*)&pair);
    return fmaf(q[1], v.y, fmaf(q[0], v.x, s));
}
__device__ __forceinline__ float ag_dot(const float* q, const __nv_bfloat16* k, int hd) {
    float s = 0.f;
    if ((hd & 7) == 0 && ((uintptr_t)k & 15) == 0) {
#pragma unroll 4
        for (int d = 0; d < hd; d += 8) {
            const uint4 v = *(const uint4*)(k + d);
            s = ag_add2(s, q + d, v.x); s = ag_add2(s, q + d + 2, v.y); s = ag_add2(s, q + d + 4, v.z); s = ag_add2(s, q + d + 6, v.w);
        }
    } else if ((hd & 3) == 0 && ((uintptr_t)k & 7) == 0) {
#pragma unroll 8
        for (int d = 0; d < hd; d += 4) {
            const uint2 v = *(const uint2*)(k + d);
            s = ag_add2(s, q + d, v.x); s = ag_add2(s, q + d + 2, v.y);
        }
    } else {
#pragma unroll 8
        for (int d = 0; d < hd; ++d) s = fmaf(q[d], gl_load(k + d), s);
    }
    return s;
}

// The row of a sequence that brings one token, its keys lo..p shared out among the block's warps, straight from the cache: by half
// pages where that spares the longest warp a half page (one to four pages more than whole rounds of eight), by whole pages where it
// does not (five: ten half pages are two rounds of eight warps, as five pages are; 64 x 300 positions, 8 heads of 256 in 32 bits, 306 us
// by halves, 266 by pages).  q0: the scaled query in shared memory; part: shared memory for the warps' sums.  A half page's values
// are asked for together with its keys (where a lane's share of them, 32 numbers a dim, fits its registers), so that it costs one
// trip to memory and not one for the keys and four for the values.
template <typename TA, typename TC, int NACC, bool AHEAD>
__device__ __forceinline__ void ag_one_token(const AttnArgs& a, const float* q0, float* part, int b, int h, int p, int lo) {
    const int hd = a.hd, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = h / (a.nH / a.nKV);
    const int* pg = a.pages + (size_t)b * a.max_pages;
    float acc[NACC];
#pragma unroll
    for (int i = 0; i < NACC; ++i) acc[i] = 0.f;
    float m = -INFINITY, l = 0.f;
    int seen = 0x7fffffff, lost = -1;      // the first key of the first half page taken, and of the last one left out for a NaN
    const int span = ((p / GL_PAGE - lo / GL_PAGE) & (AG_ROWS - 1)) < AG_ROWS / 2 ? 32 : GL_PAGE;      // keys a warp takes at a time
    for (int j1 = (lo / span + warp) * span; j1 <= p; j1 += AG_ROWS * span)
#pragma unroll 1
    for (int j0 = j1; j0 < j1 + span && j0 <= p; j0 += 32) {
        if (j0 + 31 < lo) continue;
        const int page = gl_checked(pg[gl_checked(j0 / GL_PAGE, a.max_pages, GL_BAD_POSITION)], a.n_pages > 0 ? a.n_pages : 0x7fffffff, GL_BAD_PAGE);
        const size_t at = (((size_t)page * a.nKV + g) * GL_PAGE + j0 % GL_PAGE) * hd;
        const TC* kp = (const TC*)a.k_cache + at;
        const TC* vr = (const TC*)a.v_cache + at;
        const bool ok = j0 + lane >= lo && j0 + lane <= p;
        // rows outside [lo, p] were never written or given back: they are not read
        const int k0 = max(0, lo - j0), k1 = min(32, p - j0 + 1);
        float v[AHEAD ? 32 : 1][NACC];
        if constexpr (AHEAD) {
#pragma unroll
            for (int k = 0; k < 32; ++k)
#pragma unroll
                for (int i = 0; i < NACC; ++i) {
                    const int d = lane + 32 * i;
                    v[k][i] = d < hd && k >= k0 && k < k1 ? gl_load(vr + (size_t)k * hd + d) : 0.f;
                }
        }
        const float s = ok ? ag_dot(q0, kp + (size_t)lane * hd, hd) : -INFINITY;
        const float m_new = fmaxf(m, gl_warp_max(s));
        if (m_new == -INFINITY) {
            if (__any_sync(0xffffffffu, s != s)) lost = j0;
            continue;
        }
        if (m == -INFINITY) seen = j0;
        const float pj = ok ? expf(s - m_new) : 0.f;
        const float corr = expf(m - m_new);                    // m = -inf gives 0
        l = l * corr + gl_warp_sum(pj);
        m = m_new;
#pragma unroll
        for (int i = 0; i < NACC; ++i) acc[i] *= corr;
        if constexpr (AHEAD) {
#pragma unroll
            for (int k = 0; k < 32; ++k) {
                const float pk = __shfl_sync(0xffffffffu, pj, k);
#pragma unroll
                for (int i = 0; i < NACC; ++i) acc[i] = fmaf(pk, v[k][i], acc[i]);
            }
        } else {
#pragma unroll 8
            for (int k = 0; k < 32; ++k) {
                const float pk = __shfl_sync(0xffffffffu, pj, k);
#pragma unroll
                for (int i = 0; i < NACC; ++i) {
                    const int d = lane + 32 * i;
                    if (d < hd && k >= k0 && k < k1) acc[i] = fmaf(pk, gl_load(vr + (size_t)k * hd + d), acc[i]);
                }
            }
        }
    }
    // a warp's sums, its maximum and its weight.  Scores that are NaN behind scores that are not make the row NaN, as
    // where one warp walks all pages (there a half page of nothing but NaN has no maximum and is left out only as long
    // as nothing came before it).
    // part: [AG_ROWS][hd + 2]
    int* nan_at = (int*)(part + AG_ROWS * (hd + 2));       // [AG_ROWS][2]
    float* mine = part + warp * (hd + 2);
#pragma unroll
    for (int i = 0; i < NACC; ++i)
        if (lane + 32 * i < hd) mine[lane + 32 * i] = acc[i];
    if (lane == 0) { mine[hd] = m; mine[hd + 1] = l; nan_at[2 * warp] = seen; nan_at[2 * warp + 1] = lost; }
    __syncthreads();
    float top = -INFINITY;
#pragma unroll
    for (int w = 0; w < AG_ROWS; ++w) {
        top = fmaxf(top, part[w * (hd + 2) + hd]);
        seen = min(seen, nan_at[2 * w]);
        lost = max(lost, nan_at[2 * w + 1]);
    }
    float f[AG_ROWS], den = 0.f;
#pragma unroll
    for (int w = 0; w < AG_ROWS; ++w) {
        const float mw = part[w * (hd + 2) + hd];
        f[w] = mw > -INFINITY ? expf(mw - top) : 0.f;
        den = fmaf(f[w], part[w * (hd + 2) + hd + 1], den);
    }
    const float inv = lost > seen ? NAN : den > 0.f ? 1.0f / den : 0.f;
    TA* o = (TA*)a.out + ((size_t)a.seq_qstart[b] * a.nH + h) * hd;
    for (int d = threadIdx.x; d < hd; d += AG_ROWS * 32) {
        float y = 0.f;
#pragma unroll
        for (int w = 0; w < AG_ROWS; ++w) y = fmaf(f[w], part[w * (hd + 2) + d], y);
        gl_store(o + d, y * inv);
    }
}

template <typename TA, typename TC, int NACC>
__device__ __forceinline__ void ag_rows(const AttnArgs& a) {
    extern __shared__ float smem[];
    const int hd = a.hd, ks = hd + 1;
    float* Ks = smem;                       // [GL_PAGE][hd+1]
    float* Vs = Ks + GL_PAGE * ks;          // [GL_PAGE][hd]
    float* Qs = Vs + GL_PAGE * hd;          // [AG_ROWS][hd]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b = blockIdx.z, h = blockIdx.y;
    const int qlen = a.seq_qlen[b];
    const int row0 = blockIdx.x * AG_ROWS;
    if (row0 >= qlen) return;
    const int ctx = a.seq_ctx[b];
    const int total = ctx + qlen;
    const int g = h / (a.nH / a.nKV);
    const int idx = row0 + warp;
    const bool live = idx < qlen;
    const int p = ctx + idx;                               // this row's position
    const int lo = (a.window > 0 && p - a.window + 1 > 0) ? p - a.window + 1 : 0;
    const int rows_here = min(AG_ROWS, qlen - row0);
    const int p_first = ctx + row0, p_last = ctx + row0 + rows_here - 1;
    const int lo_cta = (a.window > 0 && p_first - a.window + 1 > 0) ? p_first - a.window + 1 : 0;

    float* qv = Qs + warp * hd;
    if (live) {
        const TA* qsrc = (const TA*)a.q + ((size_t)(a.seq_qstart[b] + idx) * a.nH + h) * hd;
        for (int d = lane; d < hd; d += 32) qv[d] = gl_load(qsrc + d) * a.score_scale;
    }
    float acc[NACC];
#pragma unroll
    for (int i = 0; i < NACC; ++i) acc[i] = 0.f;
    float m = -INFINITY, l = 0.f;

    const int* pg = a.pages + (size_t)b * a.max_pages;
    if (qlen == 1 && p_first / GL_PAGE - lo_cta / GL_PAGE + 1 >= AG_SHARE_FROM) {
        __syncthreads();
        ag_one_token<TA, TC, NACC, false>(a, Qs, smem, b, h, p_first, lo_cta);
        return;
    }
    for (int page_i = lo_cta / GL_PAGE; page_i <= p_last / GL_PAGE; ++page_i) {
        const int page = gl_checked(pg[gl_checked(page_i, a.max_pages, GL_BAD_POSITION)], a.n_pages > 0 ? a.n_pages : 0x7fffffff, GL_BAD_PAGE);
        const TC* kp = (const TC*)a.k_cache + ((size_t)page * a.nKV + g) * GL_PAGE * hd;
        const TC* vp = (const TC*)a.v_cache + ((size_t)page * a.nKV + g) * GL_PAGE * hd;
        const int j0 = page_i * GL_PAGE;
        __syncthreads();
        for (int e = threadIdx.x; e < GL_PAGE * hd; e += blockDim.x) {
            const int r = e / hd, d = e - r * hd;
            const bool ok = j0 + r < total;       // rows past the sequence were never written
            Ks[r * ks + d] = ok ? gl_load(kp + e) : 0.f;
            Vs[r * hd + d] = ok ? gl_load(vp + e) : 0.f;
        }
        __syncthreads();
        if (!live) continue;
#pragma unroll 1
        for (int half = 0; half < GL_PAGE / 32; ++half) {
            const int jj = half * 32 + lane, j = j0 + jj;
            const bool ok = j >= lo && j <= p;
            float s = -INFINITY;
            if (ok) {
                const float* kr = Ks + jj * ks;
                float d0 = 0.f;
                for (int d = 0; d < hd; ++d) d0 = fmaf(qv[d], kr[d], d0);
                s = d0;
            }
            const float m_new = fmaxf(m, gl_warp_max(s));
            if (m_new == -INFINITY) continue;
            const float pj = ok ? expf(s - m_new) : 0.f;
            const float corr = expf(m - m_new);            // m = -inf gives 0
            l = l * corr + gl_warp_sum(pj);
            m = m_new;
#pragma unroll
            for (int i = 0; i < NACC; ++i) acc[i] *= corr;
            const float* vr = Vs + half * 32 * hd;
            for (int k = 0; k < 32; ++k) {
                const float pk = __shfl_sync(0xffffffffu, pj, k);
#pragma unroll
                for (int i = 0; i < NACC; ++i) {
                    const int d = lane + 32 * i;
                    if (d < hd) acc[i] = fmaf(pk, vr[k * hd + d], acc[i]);
                }
            }
        }
    }
    if (!live) return;
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    TA* o = (TA*)a.out + ((size_t)(a.seq_qstart[b] + idx) * a.nH + h) * hd;
#pragma unroll
    for (int i = 0; i < NACC; ++i) {
        const int d = lane + 32 * i;
        if (d < hd) gl_store(o + d, acc[i] * inv);
    }
}

template <typename TA, typename TC, int NACC>
__global__ void __launch_bounds__(AG_ROWS * 32)
attn_generic_kernel(AttnArgs a) { ag_rows<TA, TC, NACC>(a); }

// Heads of more than 96 (of them those that are no whole 16-byte pieces come here): as many blocks an SM as shared memory allows (a prompt
// of 1,000 tokens, 16 heads of 100 in bfloat16, 742 us with the compiler's choice of registers, 627 so; smaller heads lose by any limit).
template <typename TA, typename TC, int NACC>
__global__ void __launch_bounds__(AG_ROWS * 32, NACC <= 4 ? 4 : NACC <= 6 ? 3 : 2)
attn_generic_wide_kernel(AttnArgs a) { ag_rows<TA, TC, NACC>(a); }

// Many rows of a sequence: a warp takes R consecutive ones, which share every key and value it reads from the tiles, and R
// independent chains of multiply-adds in the place of one.  A row's sums run in the order of ag_rows (keys in ascending order of
// their dims, half pages one after the other, values in ascending order of their keys), so it is the same number from either.
// What bounds it: shared-memory loads (four rows a warp, heads of 64: their pipe is active 42 % of the time, the FMA pipe 29 %, two blocks
// an SM).  hd: a multiple of 4.
template <typename TA, typename TC, int NACC, int R>
__global__ void __launch_bounds__(AG_ROWS * 32, R == 1 && NACC == 4 ? 3 : 2)
attn_generic_rows_kernel(AttnArgs a) {
    extern __shared__ __align__(16) float smem[];
    const int hd = a.hd, ks = hd + 4;       // (eight rows' 16-byte pieces fall on different banks)
    float* Ks = smem;                       // [GL_PAGE][hd+4]
    float* Vs = Ks + GL_PAGE * ks;          // [GL_PAGE][hd]
    float* Qs = Vs + GL_PAGE * hd;          // [AG_ROWS * R][hd]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // (in a prompt the next kernel's blocks, launched early, would only take these blocks' places)
    if (R == 1) gl_grid_launch_dependents();
    gl_grid_wait();
    const int b = blockIdx.z, h = blockIdx.y;
    const int qlen = a.seq_qlen[b];
    const int row0 = blockIdx.x * (AG_ROWS * R);
    if (row0 >= qlen) return;
    const int ctx = a.seq_ctx[b], total = ctx + qlen, g = h / (a.nH / a.nKV);
    const int rows_here = min(AG_ROWS * R, qlen - row0);
    const int p_first = ctx + row0, p_last = ctx + row0 + rows_here - 1;
    const int lo_cta = (a.window > 0 && p_first - a.window + 1 > 0) ? p_first - a.window + 1 : 0;
    for (int e = threadIdx.x; e < rows_here * hd; e += AG_ROWS * 32) {
        const int r = e / hd, d = e - r * hd;
        Qs[e] = gl_load((const TA*)a.q + ((size_t)(a.seq_qstart[b] + row0 + r) * a.nH + h) * hd + d) * a.score_scale;
    }
    if (qlen == 1 && p_first / GL_PAGE - lo_cta / GL_PAGE + 1 >= AG_SHARE_FROM) {
        __syncthreads();
        ag_one_token<TA, TC, NACC, NACC <= 2>(a, Qs, smem, b, h, p_first, lo_cta);
        return;
    }
    const int mine = warp * R, live = min(R, rows_here - mine);             // this warp's rows (live may be <= 0)
    const int p0 = p_first + mine, p_top = p0 + live - 1;
    const float* qv = Qs + min(mine, rows_here - 1) * hd;
    float acc[R][NACC], m[R], l[R];
    int lo[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.f;
        lo[r] = (a.window > 0 && p0 + r - a.window + 1 > 0) ? p0 + r - a.window + 1 : 0;
#pragma unroll
        for (int i = 0; i < NACC; ++i) acc[r][i] = 0.f;
    }
    const int* pg = a.pages + (size_t)b * a.max_pages;
    for (int page_i = lo_cta / GL_PAGE; page_i <= p_last / GL_PAGE; ++page_i) {
        const int page = gl_checked(pg[gl_checked(page_i, a.max_pages, GL_BAD_POSITION)], a.n_pages > 0 ? a.n_pages : 0x7fffffff, GL_BAD_PAGE);
        const TC* kp = (const TC*)a.k_cache + ((size_t)page * a.nKV + g) * GL_PAGE * hd;
        const TC* vp = (const TC*)a.v_cache + ((size_t)page * a.nKV + g) * GL_PAGE * hd;
        const int j0 = page_i * GL_PAGE, h4 = hd / 4;
        __syncthreads();
#pragma unroll 4
        for (int e = threadIdx.x; e < GL_PAGE * h4; e += AG_ROWS * 32) {
            const int r = e / h4, d = (e - r * h4) * 4;
            const bool ok = j0 + r < total;       // rows past the sequence were never written
            *(float4*)(Ks + r * ks + d) = ok ? ag_load4(kp + 4 * (size_t)e) : make_float4(0.f, 0.f, 0.f, 0.f);
            *(float4*)(Vs + r * hd + d) = ok ? ag_load4(vp + 4 * (size_t)e) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
        if (live <= 0) continue;
#pragma unroll 1
        for (int half = 0; half < GL_PAGE / 32; ++half) {
            const int jh = j0 + half * 32, j = jh + lane;
            if (jh > p_top) break;                // (no row of this warp sees a key from here on)
            float s[R];
#pragma unroll
            for (int r = 0; r < R; ++r) s[r] = 0.f;
            const float* kr = Ks + (half * 32 + lane) * ks;
#pragma unroll 4
            for (int d = 0; d < hd; d += 4) {
                const float4 k = *(const float4*)(kr + d);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float4 q = *(const float4*)(qv + (r < live ? r : 0) * hd + d);
                    s[r] = fmaf(q.x, k.x, s[r]); s[r] = fmaf(q.y, k.y, s[r]); s[r] = fmaf(q.z, k.z, s[r]); s[r] = fmaf(q.w, k.w, s[r]);
                }
            }
            float pj[R];
            bool all = true;
            unsigned on = 0;                      // rows that have seen a key
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const bool ok = r < live && j >= lo[r] && j <= p0 + r;
                const float m_new = fmaxf(m[r], gl_warp_max(ok ? s[r] : -INFINITY));
                pj[r] = 0.f;
                if (m_new == -INFINITY) { all = false; continue; }
                on |= 1u << r;
                pj[r] = ok ? expf(s[r] - m_new) : 0.f;
                const float corr = expf(m[r] - m_new);            // m = -inf gives 0
                l[r] = l[r] * corr + gl_warp_sum(pj[r]);
                m[r] = m_new;
#pragma unroll
                for (int i = 0; i < NACC; ++i) acc[r][i] *= corr;
            }
            const float* vr = Vs + half * 32 * hd + lane;
            auto values = [&](auto every) {
#pragma unroll 8
                for (int k = 0; k < 32; ++k) {
                    float v[NACC];
#pragma unroll
                    for (int i = 0; i < NACC; ++i) v[i] = lane + 32 * i < hd ? vr[k * hd + 32 * i] : 0.f;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float pk = __shfl_sync(0xffffffffu, pj[r], k);
                        // (a row that has seen no key stays zero whatever the values are)
                        if (!decltype(every)::value && !(on >> r & 1)) continue;
#pragma unroll
                        for (int i = 0; i < NACC; ++i) acc[r][i] = fmaf(pk, v[i], acc[r][i]);
                    }
                }
            };
            if (all) values(std::true_type{});
            else values(std::false_type{});
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
        if (r >= live) break;
        const float inv = l[r] > 0.f ? 1.0f / l[r] : 0.f;
        TA* o = (TA*)a.out + ((size_t)(a.seq_qstart[b] + row0 + mine + r) * a.nH + h) * hd;
#pragma unroll
        for (int i = 0; i < NACC; ++i) {
            const int d = lane + 32 * i;
            if (d < hd) gl_store(o + d, acc[r][i] * inv);
        }
    }
}

static int ag_sm_count() {
    static int sms = 0;                    // (the same whichever thread finds it first)
    if (!sms) {
        int dev = 0, n = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        sms = n > 0 ? n : 148;
    }
    return sms;
}

template <typename TA, typename TC, int NACC, int R>
static int launch_generic_rows(const AttnArgs& a, cudaStream_t stream) {
    const size_t smem = ((size_t)GL_PAGE * (a.hd + 4) + (size_t)GL_PAGE * a.hd + (size_t)AG_ROWS * R * a.hd) * sizeof(float);
    void (*kern)(AttnArgs) = attn_generic_rows_kernel<TA, TC, NACC, R>;
    if (smem > 48 * 1024 && cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return GL_ERR_SMEM;
    }
    const dim3 grid((a.max_qlen + AG_ROWS * R - 1) / (AG_ROWS * R), a.nH, a.B), block(AG_ROWS * 32);
    // One token a sequence is not launched early: its blocks, few and long, would pile up on whichever SMs have room beside the kernel
    // before (32 bits, early and in order: 8 x 701 positions, 16 heads of 100 61 and 28 us, 8 of 256 107 and 60; 1 x 20, 32 of 64 3.6 and 4.0).
    const int rc = a.max_qlen == 1 ? gl_launch_in_order(kern, grid, block, smem, stream, a) : gl_launch(kern, grid, block, smem, stream, 1, a);
    return rc == 0 ? GL_OK : GL_ERR_LAUNCH;
}

// Rows a warp of attn_generic_rows_kernel, 0: ag_rows.  It takes heads of whole 16-byte pieces: as many rows, up to four, as leave the
// SMs a block each (two thirds of them with two).
// One, two and four rows a warp, 32 bits, us: 4 runs of 16 to 300 tokens, 32 heads of 64 118 / 85 / 77; 2,000 tokens 2273 / 1540 /
// 1233; 8 heads, 300 tokens 28 / 26 / 34, 100 tokens 9.8 / 10.0 / 13.9; 4 heads of 256, 500 tokens 120 / 97 / 134, 60 tokens 12 /
// 16 / 22.  (A row a warp, its numbers read one at a time: 144, 2523 and 326 for the first, second and fifth.)
// One token of each of many sequences in bfloat16, heads of up to 96: ag_rows, whose blocks are more to an SM (64 x 300 positions, rows and
// ag_rows, us: 32 heads of 64 114 and 85, of 80 183 and 121; 8 x 700 18 and 21).
static int ag_rows_a_warp(const AttnArgs& a, int cache_bytes) {
    if (a.hd % 4 || (((uintptr_t)a.k_cache | (uintptr_t)a.v_cache) & (4 * cache_bytes - 1))) return 0;
    const int sms = ag_sm_count();
    if (a.max_qlen == 1 && cache_bytes == 2 && a.hd <= 96 && (long long)a.nH * a.B > 2 * sms) return 0;
    const auto blocks = [&](int rows) { return (long long)((a.max_qlen + rows - 1) / rows) * a.nH * a.B; };
    if (a.max_qlen > AG_ROWS && blocks(4 * AG_ROWS) >= sms) return 4;
    if (a.max_qlen > AG_ROWS && 3 * blocks(2 * AG_ROWS) >= 2 * sms) return 2;
    return 1;
}

template <typename TA, typename TC, int NACC>
static int launch_generic(const AttnArgs& a, cudaStream_t stream) {
    switch (ag_rows_a_warp(a, sizeof(TC))) {
        case 4: return launch_generic_rows<TA, TC, NACC, 4>(a, stream);
        case 2: return launch_generic_rows<TA, TC, NACC, 2>(a, stream);
        case 1: return launch_generic_rows<TA, TC, NACC, 1>(a, stream);
    }
    const size_t smem = ((size_t)GL_PAGE * (a.hd + 1) + (size_t)GL_PAGE * a.hd + (size_t)AG_ROWS * a.hd) * sizeof(float);
    void (*kern)(AttnArgs);
    if constexpr (NACC > 3) kern = attn_generic_wide_kernel<TA, TC, NACC>;
    else kern = attn_generic_kernel<TA, TC, NACC>;
    if (smem > 48 * 1024) {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
            cudaGetLastError();
            return GL_ERR_SMEM;
        }
    }
    dim3 grid((a.max_qlen + AG_ROWS - 1) / AG_ROWS, a.nH, a.B);
    kern<<<grid, AG_ROWS * 32, smem, stream>>>(a);
    return gl_check_launch();
}

template <typename TA, typename TC>
static int dispatch_generic(const AttnArgs& a, cudaStream_t stream) {
    switch ((a.hd + 31) / 32) {
        case 1: return launch_generic<TA, TC, 1>(a, stream);
        case 2: return launch_generic<TA, TC, 2>(a, stream);
        case 3: return launch_generic<TA, TC, 3>(a, stream);
        case 4: return launch_generic<TA, TC, 4>(a, stream);
        case 5: return launch_generic<TA, TC, 5>(a, stream);
        case 6: return launch_generic<TA, TC, 6>(a, stream);
        case 7: return launch_generic<TA, TC, 7>(a, stream);
        case 8: return launch_generic<TA, TC, 8>(a, stream);
        default: return GL_ERR_SHAPE;
    }
}

// which form a call takes: rows a warp of the kernel for heads of whole 16-byte pieces, or 0
GL_API int gl_attention_generic_rows(const AttnArgs* args, int cache_dtype) { return ag_rows_a_warp(*args, cache_dtype == GL_BF16 ? 2 : 4); }

GL_API int gl_attention_generic(const AttnArgs* args, int act_dtype, int cache_dtype, cudaStream_t stream) {
    const AttnArgs& a = *args;
    if (a.B <= 0 || a.max_qlen <= 0) return GL_OK;
    if (a.hd <= 0 || a.hd > 256 || a.nH <= 0 || a.nKV <= 0 || a.nH % a.nKV) return GL_ERR_SHAPE;
    if (a.B > 65535 || a.nH > 65535) return GL_ERR_SHAPE;
    if (act_dtype == GL_F32 && cache_dtype == GL_F32) return dispatch_generic<float, float>(a, stream);
    if (act_dtype == GL_BF16 && cache_dtype == GL_BF16) return dispatch_generic<__nv_bfloat16, __nv_bfloat16>(a, stream);
    return GL_ERR_DTYPE;
}
