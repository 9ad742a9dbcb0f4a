// Grouped-query attention of every token of a step over its sequence's paged cache, prompts and single decoded tokens,
// for the 32-bit path and for head sizes the tensor-core kernels do not take (any head_dim that is a multiple of 2 up to
// 256).
//
// Arithmetic, float32 and the same in both kernels below: keys are taken in chunks of 32 whose boundaries lie at absolute
// key positions (multiples of 32).  A chunk by itself gives scores (one chain over the head's dimensions), their maximum,
// the sum of the weights and the weighted sum of the values (one chain over the chunk's keys); the chunks are then joined
// in order, each rescaled to the larger maximum.  The result for a token depends only on its query and on the keys it
// sees, not on how the tokens were cut into steps or batched, nor on the kernel.
// Reference: core/model.cpp:411-435 (decode) and :605-626 (prefill): query head h reads
// KV head h / (H/KVH); s_t = (q.k_t)/sqrt(hd) for keys t <= pos; softmax; o = sum s_t v_t.
// `window` > 0 restricts the keys to pos-window < t <= pos, `window` < 0 to those of the query's own chunk of -window
// positions (0 = all keys; common.cuh: oe_first_key).
// `sink` != 0 adds one to the softmax's denominator: a key of score 0 that has no value
// (the running maximum starts at 0 and the running sum at 1).
//
// attn_prompt_kernel, many tokens of few sequences: a CTA has 64 rows (a row is a token and a query head) of one KV head, 8
// a warp, and brings each chunk's keys and values into shared memory once for all of them.
// attn_token_kernel, few tokens a sequence: a CTA has one token and KV head, its eight warps take eight chunks at a time
// straight from memory and one warp per head joins them in order (with one warp per token and head walking over all chunks
// the chain of loads was the time: 260 us for 3 sequences of 200 keys, 32 heads of 64).
#include "common.cuh"
#include <type_traits>

namespace {

constexpr int MAX_HD = 256;
constexpr int RB = 8;                    // rows a warp works on at a time
constexpr int WARPS = 8;
constexpr int ROWS = RB * WARPS;         // rows of a prompt CTA

// The running softmax of one row; acc[i] belongs to dimension lane + 32 i.
template <int NI>
struct Running {
    float m, l, acc[NI];
    __device__ __forceinline__ void start(int sink) {
        m = sink ? 0.f : -INFINITY;
        l = sink ? 1.f : 0.f;
#pragma unroll
        for (int i = 0; i < NI; i++) acc[i] = 0.f;
    }
    // one chunk more: its maximum, its sum and its weighted values.  Without a key for this row the maximum is -inf and the
    // sum zero; with keys whose scores are all NaN the maximum, which passes NaN over, is -inf as well, but not the sum
    __device__ __forceinline__ void join(float mc, float lc, const float (&ac)[NI]) {
        if (mc == -INFINITY && lc == 0.f) return;
        const float m_new = fmaxf(m, mc);
        const float a = expf(m - m_new), b = expf(mc - m_new);
        l = fmaf(l, a, __fmul_rn(lc, b));
#pragma unroll
        for (int i = 0; i < NI; i++) acc[i] = fmaf(acc[i], a, __fmul_rn(ac[i], b));
        m = m_new;
    }
};

template <typename T> struct Four;
template <> struct Four<float> {
    static __device__ __forceinline__ float4 load(const float* p) { return *(const float4*)p; }
};
template <> struct Four<bf16> {
    static __device__ __forceinline__ float4 load(const bf16* p) {
        const uint2 v = *(const uint2*)p;
        const float2 a = __bfloat1622float2(*(const __nv_bfloat162*)&v.x), b = __bfloat1622float2(*(const __nv_bfloat162*)&v.y);
        return make_float4(a.x, a.y, b.x, b.y);
    }
};
__device__ __forceinline__ float dot4(float4 a, float4 b, float s) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, s))));
}

// ------------------------------------------------------------------------------------------------------------------
template <typename T, int NI>
__global__ void __launch_bounds__(WARPS * 32)
attn_prompt_kernel(T* out, const T* q, int q_stride, const T* cache, const int* __restrict__ tables, int max_pages,
                   const int* __restrict__ tok_seq, const int* __restrict__ tok_pos, int n_tokens, int H, int KVH, int hd,
                   int window, float scale, int sink) {
    extern __shared__ __align__(16) float smem[];
    const int hp = (hd + 3) / 4 * 4, row_words = hp + 4;      // rows of keys: no bank conflicts for 16-byte loads
    float* ks = smem;                                         // [32][row_words]
    float* vs = ks + 32 * row_words;                          // [32][hp]
    float* qs = vs + 32 * hp;                                 // [ROWS][hp]
    float* ps = qs + ROWS * hp;                               // [WARPS][32][RB]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kvh = blockIdx.x % KVH, G = H / KVH;
    const long long row0 = (long long)(blockIdx.x / KVH) * ROWS, n_rows = (long long)n_tokens * G;
    pdl_launch_dependents();
    pdl_wait();
    const int t0 = (int)(row0 / G), t1 = (int)((min(row0 + ROWS, n_rows) - 1) / G);
    for (int e = threadIdx.x; e < ROWS * hp; e += WARPS * 32) {
        const long long row = row0 + e / hp;
        const int d = e % hp;
        float v = 0.f;
        if (row < n_rows && d < hd) v = to_f32(q[(size_t)(row / G) * q_stride + (size_t)(kvh * G + row % G) * hd + d]);
        qs[e] = v;
    }
    int tok[RB], lo[RB], pos[RB];
    Running<NI> run[RB];
#pragma unroll
    for (int r = 0; r < RB; r++) {
        const long long row = row0 + warp * RB + r;
        tok[r] = row < n_rows ? (int)(row / G) : -1;
        pos[r] = tok[r] >= 0 ? tok_pos[tok[r]] : -1;
        lo[r] = oe_first_key(pos[r], window);
        run[r].start(sink);
    }
    const float* qw = qs + warp * RB * hp;
    float* pw = ps + warp * 32 * RB;

    for (int a = t0; a <= t1;) {                              // the runs of one sequence's tokens
        const int b = tok_seq[a];
        int e = a, first = 0x7fffffff, last = -1;
        for (; e <= t1 && tok_seq[e] == b; e++) {
            const int p = tok_pos[e];
            first = min(first, oe_first_key(p, window));
            last = max(last, p);
        }
        if (b < 0) { a = e; continue; }
        const int* trow = tables + (size_t)b * max_pages;
        for (int c0 = first / 32 * 32; c0 <= last; c0 += 32) {
            __syncthreads();
            // a chunk lies in one page; keys behind the run's last one are not read
            const long long ko = page_row_offset(trow, c0, 0, kvh, KVH, hd), vo = page_row_offset(trow, c0, 1, kvh, KVH, hd);
            const int have = ko < 0 ? 0 : min(32, last - c0 + 1);
#pragma unroll
            for (int j = warp; j < 32; j += WARPS)
#pragma unroll
                for (int i = 0; i < NI; i++) {
                    const int d = lane + 32 * i;
                    if (d >= hp) continue;
                    const bool on = j < have && d < hd;
                    ks[j * row_words + d] = on ? to_f32(cache[ko + (size_t)j * hd + d]) : 0.f;
                    vs[j * hp + d] = on ? to_f32(cache[vo + (size_t)j * hd + d]) : 0.f;
                }
            __syncthreads();
            bool any = false, full = have == 32;
            int jlo[RB], jhi[RB];                             // the row's keys in this chunk (none: jhi < jlo)
#pragma unroll
            for (int r = 0; r < RB; r++) {
                const bool mine = tok[r] >= a && tok[r] < e;
                jlo[r] = max(lo[r] - c0, 0);
                jhi[r] = mine ? min(pos[r] - c0, 31) : -1;
                if (jhi[r] < jlo[r]) jhi[r] = -1;
                any |= jhi[r] >= 0;
                full &= jlo[r] == 0 && jhi[r] == 31;
            }
            if (!any) continue;
            float s[RB];
#pragma unroll
            for (int r = 0; r < RB; r++) s[r] = 0.f;
            const float* kr = ks + lane * row_words;
            for (int d = 0; d < hp; d += 4) {
                const float4 k4 = *(const float4*)(kr + d);
#pragma unroll
                for (int r = 0; r < RB; r++) s[r] = dot4(*(const float4*)(qw + r * hp + d), k4, s[r]);
            }
            float mc[RB], lc[RB];
#pragma unroll
            for (int r = 0; r < RB; r++) {
                const float v = lane < have && lane >= jlo[r] && lane <= jhi[r] ? s[r] * scale : -INFINITY;
                mc[r] = warp_max(v);
                s[r] = v == -INFINITY ? 0.f : expf(v - mc[r]);
                lc[r] = warp_sum(s[r]);
            }
            __syncwarp();
#pragma unroll
            for (int r = 0; r < RB; r += 4) *(float4*)(pw + lane * RB + r) = make_float4(s[r], s[r + 1], s[r + 2], s[r + 3]);
            __syncwarp();
            float ac[RB][NI];
#pragma unroll
            for (int r = 0; r < RB; r++)
#pragma unroll
                for (int i = 0; i < NI; i++) ac[r][i] = 0.f;
            for (int j = 0; j < 32; j++) {
                float p[RB];
#pragma unroll
                for (int r = 0; r < RB; r += 4) *(float4*)(p + r) = *(const float4*)(pw + j * RB + r);
#pragma unroll
                for (int i = 0; i < NI; i++) {
                    const int d = lane + 32 * i;
                    const float v = d < hp ? vs[j * hp + d] : 0.f;
                    if (full) {
#pragma unroll
                        for (int r = 0; r < RB; r++) ac[r][i] = fmaf(p[r], v, ac[r][i]);
                    } else {                                  // a key that a row does not see must not touch its sum
#pragma unroll
                        for (int r = 0; r < RB; r++) { const float u = fmaf(p[r], v, ac[r][i]); ac[r][i] = j >= jlo[r] && j <= jhi[r] ? u : ac[r][i]; }
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < RB; r++) run[r].join(mc[r], lc[r], ac[r]);
        }
        a = e;
    }
#pragma unroll
    for (int r = 0; r < RB; r++) {
        if (tok[r] < 0) continue;
        T* o = out + (size_t)tok[r] * H * hd + (size_t)(kvh * G + (row0 + warp * RB + r) % G) * hd;
        const float inv = tok_seq[tok[r]] < 0 ? 0.f : 1.f / run[r].l;     // a padding row: zeros
#pragma unroll
        for (int i = 0; i < NI; i++) {
            const int d = lane + 32 * i;
            if (d < hd) o[d] = from_f32<T>(run[r].acc[i] * inv);
        }
    }
}

// ------------------------------------------------------------------------------------------------------------------
template <typename T, int NI, bool QUADS>
__global__ void __launch_bounds__(WARPS * 32)
attn_token_kernel(T* out, const T* q, int q_stride, const T* cache, const int* __restrict__ tables, int max_pages,
                  const int* __restrict__ tok_seq, const int* __restrict__ tok_pos, int H, int KVH, int hd, int window,
                  float scale, int sink) {
    __shared__ __align__(16) float qs[RB * MAX_HD];
    __shared__ __align__(16) float ps[WARPS][32 * RB];
    __shared__ float pm[WARPS][RB], pl[WARPS][RB];
    extern __shared__ __align__(16) float part[];             // [WARPS][RB][32 NI]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kvh = blockIdx.x % KVH, t = blockIdx.x / KVH, G = H / KVH;
    pdl_launch_dependents();
    pdl_wait();
    const int b = tok_seq[t];
    T* ot = out + (size_t)t * H * hd + (size_t)kvh * G * hd;
    if (b < 0) {                                              // padding row
        for (int d = threadIdx.x; d < G * hd; d += WARPS * 32) ot[d] = from_f32<T>(0.f);
        return;
    }
    const int pos = tok_pos[t], lo = oe_first_key(pos, window);
    const int* trow = tables + (size_t)b * max_pages;
    const T* qt = q + (size_t)t * q_stride + (size_t)kvh * G * hd;
    for (int g0 = 0; g0 < G; g0 += RB) {
        __syncthreads();
        for (int x = threadIdx.x; x < RB * hd; x += WARPS * 32) qs[x / hd * MAX_HD + x % hd] = g0 + x / hd < G ? to_f32(qt[(size_t)g0 * hd + x]) : 0.f;
        __syncthreads();
        Running<NI> run;                                      // of head g0 + warp
        run.start(sink);
        for (int r0 = lo / 32 * 32; r0 <= pos; r0 += 32 * WARPS) {
            const int c0 = r0 + 32 * warp;
            // a chunk for R heads of the group: 4 where it has no more (8 for all groups: 16.4 us for 3
            // tokens of 32 heads over 8, 11.0 so)
            auto chunk = [&](auto rows) {
            constexpr int R = decltype(rows)::value;
            float s[R];
#pragma unroll
            for (int r = 0; r < R; r++) s[r] = 0.f;
            if (c0 <= pos) {
                const long long ko = page_row_offset(trow, c0, 0, kvh, KVH, hd), vo = page_row_offset(trow, c0, 1, kvh, KVH, hd);
                const int jlo = max(lo - c0, 0), jhi = min(pos - c0, 31);
                const bool seen = lane >= jlo && lane <= jhi && ko >= 0;
                const T* kr = cache + (seen ? ko + (size_t)lane * hd : 0);
                if (QUADS) {
#pragma unroll 4
                    for (int d = 0; d < hd; d += 4) {
                        const float4 k4 = seen ? Four<T>::load(kr + d) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                        for (int r = 0; r < R; r++) s[r] = dot4(*(const float4*)(qs + r * MAX_HD + d), k4, s[r]);
                    }
                } else {
                    for (int d = 0; d < hd; d++) {
                        const float k = seen ? to_f32(kr[d]) : 0.f;
#pragma unroll
                        for (int r = 0; r < R; r++) s[r] = fmaf(qs[r * MAX_HD + d], k, s[r]);
                    }
                }
                float mc[R], lc[R];
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const float v = seen ? s[r] * scale : -INFINITY;
                    mc[r] = warp_max(v);
                    s[r] = v == -INFINITY ? 0.f : expf(v - mc[r]);
                    lc[r] = warp_sum(s[r]);
                }
                float* pw = ps[warp];
#pragma unroll
                for (int r = 0; r < R; r += 4) *(float4*)(pw + lane * RB + r) = make_float4(s[r], s[r + 1], s[r + 2], s[r + 3]);
                __syncwarp();
                float ac[R][NI];
#pragma unroll
                for (int r = 0; r < R; r++)
#pragma unroll
                    for (int i = 0; i < NI; i++) ac[r][i] = 0.f;
                if (ko >= 0) {
#pragma unroll 4
                    for (int j = jlo; j <= jhi; j++) {
                        float p[R];
#pragma unroll
                        for (int r = 0; r < R; r += 4) *(float4*)(p + r) = *(const float4*)(pw + j * RB + r);
#pragma unroll
                        for (int i = 0; i < NI; i++) {
                            const int d = lane + 32 * i;
                            const float v = d < hd ? to_f32(cache[vo + (size_t)j * hd + d]) : 0.f;
#pragma unroll
                            for (int r = 0; r < R; r++) ac[r][i] = fmaf(p[r], v, ac[r][i]);
                        }
                    }
                }
                __syncwarp();
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if (lane == 0) { pm[warp][r] = mc[r]; pl[warp][r] = lc[r]; }
#pragma unroll
                    for (int i = 0; i < NI; i++) part[(warp * RB + r) * NI * 32 + lane + 32 * i] = ac[r][i];
                }
            }
            };
            if (G - g0 <= 4) chunk(std::integral_constant<int, 4>{});
            else chunk(std::integral_constant<int, RB>{});
            __syncthreads();
            for (int w = 0; w < WARPS && r0 + 32 * w <= pos; w++) {
                float ac[NI];
#pragma unroll
                for (int i = 0; i < NI; i++) ac[i] = part[(w * RB + warp) * NI * 32 + lane + 32 * i];
                run.join(pm[w][warp], pl[w][warp], ac);
            }
            __syncthreads();
        }
        if (g0 + warp < G) {
            const float inv = 1.f / run.l;
#pragma unroll
            for (int i = 0; i < NI; i++) {
                const int d = lane + 32 * i;
                if (d < hd) ot[(size_t)(g0 + warp) * hd + d] = from_f32<T>(run.acc[i] * inv);
            }
        }
    }
}

template <typename T, int NI>
int launch_sized(T* out, const T* q, int q_stride, const T* cache, const int* tables, int max_pages, const int* tok_seq,
                 const int* tok_pos, int n_tokens, int n_seqs, int H, int KVH, int hd, int window, float scale, int sink, int kind,
                 cudaStream_t st) {
    const long long n_rows = (long long)n_tokens * (H / KVH), tiles = (n_rows + ROWS - 1) / ROWS;
    // A prompt CTA loads a chunk once for 64 rows of one sequence, chunk after chunk; with few tokens a sequence most of its
    // rows would idle, and with few CTAs most SMs: a CTA a token walks eight chunks at a time.
    const bool by_token = kind == 1 || (kind == 0 && (n_tokens <= 4LL * n_seqs || tiles * KVH < 74));
    // a grid of one dimension, the KV heads of a token or tile side by side: the others end at 65,535
    const long long ctas = (by_token ? (long long)n_tokens : tiles) * KVH;
    if (ctas > 2147483647LL) return OE_ERR_UNSUPPORTED;
    const dim3 grid((unsigned)ctas);
    if (by_token) {
        const bool quads = hd % 4 == 0 && ((uintptr_t)cache & 15) == 0;
        const size_t bytes = (size_t)WARPS * RB * NI * 32 * 4;
        cudaError_t e = cudaFuncSetAttribute(quads ? attn_token_kernel<T, NI, true> : attn_token_kernel<T, NI, false>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
        if (e != cudaSuccess) return (int)e;
        if (quads) return oe_launch(attn_token_kernel<T, NI, true>, grid, dim3(WARPS * 32), bytes, st, out, q, q_stride, cache, tables,
                                  max_pages, tok_seq, tok_pos, H, KVH, hd, window, scale, sink);
        return oe_launch(attn_token_kernel<T, NI, false>, grid, dim3(WARPS * 32), bytes, st, out, q, q_stride, cache, tables,
                         max_pages, tok_seq, tok_pos, H, KVH, hd, window, scale, sink);
    }
    const int hp = (hd + 3) / 4 * 4;
    const size_t bytes = (size_t)(32 * (hp + 4) + 32 * hp + ROWS * hp + WARPS * 32 * RB) * 4;
    cudaError_t e = cudaFuncSetAttribute(attn_prompt_kernel<T, NI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    return oe_launch(attn_prompt_kernel<T, NI>, grid, dim3(WARPS * 32), bytes, st, out, q, q_stride, cache, tables, max_pages,
                     tok_seq, tok_pos, n_tokens, H, KVH, hd, window, scale, sink);
}

template <typename T>
int launch(T* out, const T* q, int q_stride, const T* cache, const int* tables, int max_pages, const int* tok_seq,
           const int* tok_pos, int n_tokens, int n_seqs, int H, int KVH, int hd, int window, float scale, int sink, int kind, cudaStream_t st) {
    if (n_tokens <= 0) return 0;
    if (hd <= 0 || hd > MAX_HD || (hd % 2) || H % KVH) return OE_ERR_UNSUPPORTED;
#define OE_ATTN_GO(NI) launch_sized<T, NI>(out, q, q_stride, cache, tables, max_pages, tok_seq, tok_pos, n_tokens, n_seqs, H, KVH, hd, window, scale, sink, kind, st)
    if (hd <= 64) return OE_ATTN_GO(2);
    if (hd <= 128) return OE_ATTN_GO(4);
    return OE_ATTN_GO(8);
#undef OE_ATTN_GO
}

}  // namespace

// kind: 0 by the numbers of tokens and sequences, 1 a CTA per token, 2 a CTA per 64 rows (the same bits)
extern "C" {
int oe_attn_paged_f32(float* out, const float* q, int q_stride, const float* cache, const int* tables,
                      int max_pages, const int* tok_seq, const int* tok_pos, int n_tokens, int n_seqs, int H, int KVH,
                      int hd, int window, float scale, int sink, int kind, cudaStream_t st) {
    return launch<float>(out, q, q_stride, cache, tables, max_pages, tok_seq, tok_pos, n_tokens, n_seqs, H, KVH, hd,
                         window, scale, sink, kind, st);
}
int oe_attn_paged_bf16(bf16* out, const bf16* q, int q_stride, const bf16* cache, const int* tables,
                       int max_pages, const int* tok_seq, const int* tok_pos, int n_tokens, int n_seqs, int H, int KVH,
                       int hd, int window, float scale, int sink, int kind, cudaStream_t st) {
    return launch<bf16>(out, q, q_stride, cache, tables, max_pages, tok_seq, tok_pos, n_tokens, n_seqs, H, KVH, hd,
                        window, scale, sink, kind, st);
}
}
