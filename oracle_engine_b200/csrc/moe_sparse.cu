// Mixtures of experts of which a token uses a few (bfloat16): what computes the chosen experts alone.
//
// `dense` [T, W] float32 is the routing (csrc/moe.cu): an expert's weight where the token chose it, zero elsewhere, and in
// a last column (W = E + 1) the shared expert's.  The expert's unit, from float32 sums g and u of its gate and up rows, is
//   0: silu(g) u w     1: g' sigmoid(1.702 g') (u' + 1) w with g' = min(g, L), u' = clamp(u, -L, L)     2: silu(w g) (w u).
//
// Up to 16 tokens (a decode step): moe_up_stream_kernel and moe_down_stream_kernel, the weight-streaming product
// (gemm_skinny.cu) over the rows, and the columns, of those experts that some token of the step chose.  Both are bound by
// the weights they read; at one token and two of eight experts that is a quarter of the matrices.  A thread block of the
// first has eight gate rows and the eight up rows that belong to them, so that the unit is its epilogue.  The sums run in
// an order that does not depend on which experts are skipped (a skipped one would add zeros), so that a token's result
// does not depend on its neighbours.
//
// More tokens: moe_count_kernel and moe_place_kernel sort the (token, expert) pairs by expert, every expert's rows padded
// to the row tile of the grouped product (gemm_tcgen05_pair.cu), and copy the tokens' rows there; moe_combine_kernel adds a
// token's results in order of the experts.
#include "common.cuh"

namespace {

constexpr int ROWS = 16, CHUNK = 64;
constexpr int MAX_GROUPS = 64;                // experts
constexpr int MAX_CHUNKS = 2048;              // chunks of 64 columns that the down product's list holds

__device__ __forceinline__ uint4 ld_weight(const bf16* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::128B.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The group (expert, or shared expert) of column c.
__device__ __forceinline__ int group_of(int c, int E, int ff) { const int g = c / ff; return g < E ? g : E; }

// h [M, D] (rows of lda), w [2 F, D]: F gate rows, then F up rows.  a [M, F] = the unit; columns of experts that no token
// chose are not written.  F = E ff + shared columns, ff and F multiples of 8.
// AHEAD: a lane has a round's weights in registers before it uses the first, so that 5 CTAs fill an SM, and the shared expert's
// columns, which every token uses, come first and are asked for while the kernel before this one still routes.  Otherwise 10 CTAs an
// SM (8 for 16 tokens), for more columns than that holds at once (ops.moe_up_ahead has both sides' times; as many registers for all
// sizes cost 8 experts of 1,024 and a shared one of 2,048 for 4 tokens 3 us of 14).  16 tokens, 8 experts of 512: 12.7 us with 56
// registers, 10.1 with 64 (of 1,024 and 2,048, which 56 hold in one round: 17.9 and 20.2).
template <int NT, int WARPS, int UNROLL, bool AHEAD>
__global__ void __launch_bounds__(WARPS * 32, AHEAD ? 5 : NT == 1 ? 10 : 8)
moe_up_stream_kernel(bf16* a, const bf16* h, const bf16* __restrict__ w, const float* dense, int M, int D, int F, int E, int ff, int W,
                     long long lda, int unit, float limit) {
    __shared__ float red[WARPS][ROWS][8 * NT + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int col0 = (AHEAD ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * 8, grp = group_of(col0, E, ff);
    const bf16* w0 = w + (size_t)(col0 + g) * D;
    const bf16* w1 = w0 + (size_t)F * D;
    const int n_chunks = (D + CHUNK - 1) / CHUNK, per = (n_chunks + WARPS - 1) / WARPS;
    const int c_begin = warp * per, c_end = min(n_chunks, c_begin + per);
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    auto weights = [&](uint4 (&wa)[UNROLL][2], uint4 (&wb)[UNROLL][2], int c) {
#pragma unroll
        for (int u = 0; u < UNROLL; u++)
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
                const int k8 = (c + u) * CHUNK + t * 16 + hh * 8;
                const bool kv = c + u < c_end && k8 < D;
                wa[u][hh] = kv ? ld_weight(w0 + k8) : zero;
                wb[u][hh] = kv ? ld_weight(w1 + k8) : zero;
            }
    };
    const bool shared = AHEAD && grp >= E;
    uint4 wa0[UNROLL][2], wb0[UNROLL][2];
    if (shared) weights(wa0, wb0, c_begin);
    pdl_wait();                                   // the routing comes from the kernel before
    float mine = 0.f;
    if (lane < M && grp < W) mine = dense[(size_t)lane * W + grp];
    if (!__any_sync(0xffffffffu, mine != 0.f)) { pdl_launch_dependents(); return; }      // every warp alike
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    auto products = [&](const uint4 (&wa)[UNROLL][2], const uint4 (&wb)[UNROLL][2], int c) {
#pragma unroll
        for (int u = 0; u < UNROLL; u++)
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
                const int k8 = (c + u) * CHUNK + t * 16 + hh * 8;
                const bool kv = c + u < c_end && k8 < D;
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    const int tok = n * 8 + g;
                    uint4 x = zero;
                    if (kv && tok < M) x = *(const uint4*)(h + (size_t)tok * lda + k8);
                    mma_bf16(acc[n], wa[u][hh].x, wb[u][hh].x, wa[u][hh].y, wb[u][hh].y, x.x, x.y);
                    mma_bf16(acc[n], wa[u][hh].z, wb[u][hh].z, wa[u][hh].w, wb[u][hh].w, x.z, x.w);
                }
            }
    };
    for (int c = c_begin; c < c_end; c += UNROLL) {
        if constexpr (AHEAD) {
            if (!shared || c > c_begin) weights(wa0, wb0, c);
            __syncwarp();                         // all loads are asked for before the first is used
            products(wa0, wb0, c);
        } else {
            uint4 wa[UNROLL][2], wb[UNROLL][2];
            weights(wa, wb, c);
            __syncwarp();
            products(wa, wb, c);
        }
    }
    pdl_launch_dependents();
#pragma unroll
    for (int n = 0; n < NT; n++) {
        red[warp][g][n * 8 + t * 2] = acc[n][0];
        red[warp][g][n * 8 + t * 2 + 1] = acc[n][1];
        red[warp][g + 8][n * 8 + t * 2] = acc[n][2];
        red[warp][g + 8][n * 8 + t * 2 + 1] = acc[n][3];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 64 * NT; i += WARPS * 32) {
        const int r = i % 8, tok = i / 8;
        if (tok >= M) continue;
        float gs = 0.f, us = 0.f;
#pragma unroll
        for (int q = 0; q < WARPS; q++) { gs += red[q][r][tok]; us += red[q][r + 8][tok]; }
        const float wt = grp < W ? dense[(size_t)tok * W + grp] : 0.f;
        a[(size_t)tok * F + col0 + r] = wt != 0.f ? __float2bfloat16_rn(oe_moe_unit(unit, gs, us, wt, limit)) : __float2bfloat16_rn(0.f);
    }
}

// out [M, N] float32 (+)= a [M, F] . w [N, F]^T over the columns of the experts that some token chose.  The warps take
// chunks of 64 columns in turn (an expert's run is shared out evenly), whatever is skipped.
template <int NT, int WARPS, int UNROLL>
__global__ void __launch_bounds__(WARPS * 32)
moe_down_stream_kernel(float* out, const bf16* a, const bf16* __restrict__ w, const float* dense, int M, int N, int F, int E, int ff, int W,
                       long long ldc, int accumulate) {
    __shared__ float red[WARPS][ROWS][8 * NT + 1];
    __shared__ unsigned char used[MAX_GROUPS + 1];
    __shared__ short list[WARPS][MAX_CHUNKS / WARPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int row0 = blockIdx.x * ROWS;
    const bool rv0 = row0 + g < N, rv1 = row0 + g + 8 < N;
    const bf16* w0 = w + (size_t)(rv0 ? row0 + g : 0) * F;
    const bf16* w1 = w + (size_t)(rv1 ? row0 + g + 8 : 0) * F;
    const int n_chunks = (F + CHUNK - 1) / CHUNK;
    const bool whole = ff % CHUNK == 0;               // a chunk belongs to one group
    // the shared expert's columns count whatever is chosen: into the L2 while the kernel before this one drains
    if (W > E)
        for (int c = E * ff / CHUNK + warp * 2 + (lane >> 4); c < n_chunks; c += 2 * WARPS) {
            const int row = row0 + (lane & 15);
            if (row < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(w + (size_t)row * F + c * CHUNK));
        }
    pdl_wait();
    if (threadIdx.x <= E) used[threadIdx.x] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < M * W; i += WARPS * 32)        // a weight a thread: token after token the loads were a chain
        if (dense[i] != 0.f && i % W <= E) used[i % W] = 1;
    __syncthreads();
    // the warp's chunks with a column that counts, in order
    int count = 0;
    for (int i = lane; __any_sync(0xffffffffu, warp + WARPS * i < n_chunks); i += 32) {
        const int c = warp + WARPS * i;
        bool on = false;
        if (c < n_chunks) {
            const int last = group_of(min(c * CHUNK + CHUNK, F) - 1, E, ff);
            for (int q = group_of(c * CHUNK, E, ff); q <= last; q++) on |= used[q] != 0;
        }
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (on) list[warp][count + __popc(m & ((1u << lane) - 1u))] = (short)c;
        count += __popc(m);
    }
    __syncwarp();
    float acc[NT][4];
#pragma unroll
    for (int n = 0; n < NT; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (int i = 0; i < count; i += UNROLL) {
        uint4 wa[UNROLL][2], wb[UNROLL][2];
        int k8[UNROLL][2];                            // F: no column that counts
#pragma unroll
        for (int u = 0; u < UNROLL; u++) {
            const int c = i + u < count ? list[warp][i + u] : n_chunks;
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
                int k = min(c * CHUNK + t * 16 + hh * 8, F);
                if (!whole && k < F && !used[group_of(k, E, ff)]) k = F;         // eight columns of one group
                k8[u][hh] = k;
                wa[u][hh] = k < F && rv0 ? ld_weight(w0 + k) : zero;
                wb[u][hh] = k < F && rv1 ? ld_weight(w1 + k) : zero;
            }
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < UNROLL; u++)
#pragma unroll
            for (int hh = 0; hh < 2; hh++)
#pragma unroll
                for (int n = 0; n < NT; n++) {
                    const int tok = n * 8 + g;
                    uint4 x = zero;
                    if (k8[u][hh] < F && tok < M) x = *(const uint4*)(a + (size_t)tok * F + k8[u][hh]);
                    mma_bf16(acc[n], wa[u][hh].x, wb[u][hh].x, wa[u][hh].y, wb[u][hh].y, x.x, x.y);
                    mma_bf16(acc[n], wa[u][hh].z, wb[u][hh].z, wa[u][hh].w, wb[u][hh].w, x.z, x.w);
                }
    }
    pdl_launch_dependents();
#pragma unroll
    for (int n = 0; n < NT; n++) {
        red[warp][g][n * 8 + t * 2] = acc[n][0];
        red[warp][g][n * 8 + t * 2 + 1] = acc[n][1];
        red[warp][g + 8][n * 8 + t * 2] = acc[n][2];
        red[warp][g + 8][n * 8 + t * 2 + 1] = acc[n][3];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < ROWS * 8 * NT; i += WARPS * 32) {
        const int r = i % ROWS, tok = i / ROWS;
        if (tok >= M || row0 + r >= N) continue;
        float s = 0.f;
#pragma unroll
        for (int q = 0; q < WARPS; q++) s += red[q][r][tok];
        float* o = out + (size_t)tok * ldc + row0 + r;
        *o = accumulate ? *o + s : s;
    }
}

// ------------------------------------------------------------------------------------------------------------------
constexpr int PT = 8;                             // tokens of a block of the two sorting kernels

// counts[block][e]: how many of the block's tokens chose expert e.
__global__ void __launch_bounds__(256)
moe_count_kernel(const float* dense, int T, int E, int W, int* counts) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, t = lane < PT ? blockIdx.x * PT + lane : T;
    for (int e = threadIdx.x >> 5; e < E; e += 8) {
        const unsigned m = __ballot_sync(0xffffffffu, t < T && dense[(size_t)t * W + e] != 0.f);
        if (lane == 0) counts[(size_t)blockIdx.x * E + e] = __popc(m);
    }
}

// Expert e's rows begin at a multiple of `tile`; within them the tokens stand in order.  place[t][j]: the row of token t's
// j-th expert (in order of the experts; -1: none); row_w: the rows' weights; xs: the tokens' rows of h, copied (16 bytes at
// a time); tile_expert: the expert of every tile of rows, n_tiles[0] how many there are.
__global__ void __launch_bounds__(256)
moe_place_kernel(const float* dense, int T, int E, int W, int top, int tile, const int* counts, int n_blocks, const bf16* h, long long ldh,
                 int D, bf16* xs, int* place, float* row_w, int* tile_expert, int* n_tiles, int max_tiles) {
    __shared__ int before[MAX_GROUPS], all[MAX_GROUPS], start[MAX_GROUPS + 1];
    __shared__ int s_place[PT][8];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, b = blockIdx.x;
    for (int e = warp; e < E; e += 8) {
        int n = 0, m = 0;
        for (int i = lane; i < n_blocks; i += 32) {
            const int c = counts[(size_t)i * E + e];
            m += c;
            if (i < b) n += c;
        }
        n = __reduce_add_sync(0xffffffffu, n);
        m = __reduce_add_sync(0xffffffffu, m);
        if (lane == 0) { before[e] = n; all[e] = m; }
    }
    for (int i = threadIdx.x; i < PT * 8; i += 256) s_place[i / 8][i % 8] = -1;
    __syncthreads();
    if (threadIdx.x == 0) {
        int at = 0;
        for (int e = 0; e < E; e++) { start[e] = at; at += (all[e] + tile - 1) / tile * tile; }
        start[E] = at;
    }
    __syncthreads();
    if (b == 0) {
        const int n = min(start[E] / tile, max_tiles);
        if (threadIdx.x == 0) n_tiles[0] = n;
        for (int i = threadIdx.x; i < n; i += 256) {
            int e = 0;
            while (e + 1 < E && start[e + 1] <= i * tile) e++;
            tile_expert[i] = e;
        }
    }
    if (warp == 0) {                              // one warp, a token a lane, expert after expert
        const int t = lane < PT ? b * PT + lane : T;
        int j = 0;
        for (int e = 0; e < E; e++) {
            const float w = t < T ? dense[(size_t)t * W + e] : 0.f;
            const unsigned m = __ballot_sync(0xffffffffu, w != 0.f);
            if (w != 0.f && j < top) {
                const int row = start[e] + before[e] + __popc(m & ((1u << lane) - 1u));
                s_place[lane][j] = row;
                row_w[row] = w;
                j++;
            }
        }
        if (t < T) for (int i = 0; i < top; i++) place[(size_t)t * top + i] = s_place[lane][i];
    }
    __syncthreads();
    const int quads = D / 8;                      // 16-byte pieces of a row
    for (int i = warp; i < PT * top; i += 8) {
        const int row = s_place[i / top][i % top];
        if (row < 0) continue;
        const uint4* src = (const uint4*)(h + (size_t)(b * PT + i / top) * ldh);
        uint4* dst = (uint4*)(xs + (size_t)row * D);
        for (int q = lane; q < quads; q += 32) dst[q] = src[q];
    }
}

// out[t] (+)= the sum of y[place[t][j]] over j, four columns a thread.
__global__ void __launch_bounds__(256)
moe_combine_kernel(float* out, long long ldc, const float* y, const int* place, int top, int T, int D, int accumulate) {
    pdl_launch_dependents();
    pdl_wait();
    const int per = D / 4;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < (long long)T * per; i += (long long)gridDim.x * 256) {
        const int t = (int)(i / per), c = (int)(i % per) * 4;
        float4* o = (float4*)(out + (size_t)t * ldc + c);
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int j = 0; j < top; j++) {
            const int row = place[(size_t)t * top + j];
            if (row < 0) break;
            const float4 v = *(const float4*)(y + (size_t)row * D + c);
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        if (accumulate) { const float4 v = *o; s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w; }
        *o = s;
    }
}

bool unit_ok(int unit, float limit) { return unit >= 0 && unit <= 2 && (unit != 1 || limit > 0.f); }

}  // namespace

extern "C" {

// ahead: which of the two kernels (moe_up_stream_kernel says what for); the same bits.
int oe_moe_up_stream(bf16* a, const bf16* h, const bf16* w, const float* dense, int M, int D, int F, int E, int ff, int W, long long lda,
                     int unit, float limit, int ahead, cudaStream_t st) {
    if (M <= 0) return 0;
    if (M > 16 || D % 8 || lda % 8 || ff < 8 || ff % 8 || F % 8 || F < E * ff || E < 1 || E > MAX_GROUPS || W < E || !unit_ok(unit, limit)) return OE_ERR_UNSUPPORTED;
    if (((uintptr_t)h | (uintptr_t)w) & 15) return OE_ERR_UNSUPPORTED;
    if (M > 8) return oe_launch(moe_up_stream_kernel<2, 4, 4, false>, dim3(F / 8), dim3(128), 0, st, a, h, w, dense, M, D, F, E, ff, W, lda, unit, limit);
    return oe_launch(ahead ? moe_up_stream_kernel<1, 4, 4, true> : moe_up_stream_kernel<1, 4, 4, false>, dim3(F / 8), dim3(128), 0, st, a, h, w, dense, M, D, F, E, ff, W, lda, unit, limit);
}

int oe_moe_down_stream(float* out, const bf16* a, const bf16* w, const float* dense, int M, int N, int F, int E, int ff, int W, long long ldc,
                       int accumulate, cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    if (M > 16 || ff < 8 || ff % 8 || F % 8 || F < E * ff || E < 1 || E > MAX_GROUPS || W < E || F > CHUNK * MAX_CHUNKS) return OE_ERR_UNSUPPORTED;
    if (((uintptr_t)a | (uintptr_t)w) & 15) return OE_ERR_UNSUPPORTED;
    const int blocks = (N + ROWS - 1) / ROWS;
    if (M > 8) return oe_launch(moe_down_stream_kernel<2, 8, 3>, dim3(blocks), dim3(256), 0, st, out, a, w, dense, M, N, F, E, ff, W, ldc, accumulate);
    return oe_launch(moe_down_stream_kernel<1, 8, 4>, dim3(blocks), dim3(256), 0, st, out, a, w, dense, M, N, F, E, ff, W, ldc, accumulate);
}

// counts: at least ceil(T / 8) E integers; xs [max_tiles tile, D]; place [T, top]; row_w [max_tiles tile].  Two launches.
int oe_moe_place(const float* dense, int T, int E, int W, int top, int tile, int* counts, const bf16* h, long long ldh, int D, bf16* xs,
                 int* place, float* row_w, int* tile_expert, int* n_tiles, int max_tiles, cudaStream_t st) {
    if (T <= 0) return 0;
    if (E < 1 || E > MAX_GROUPS || W < E || top < 1 || top > 8 || tile < 1 || D % 8 || ldh % 8) return OE_ERR_UNSUPPORTED;
    if ((long long)max_tiles < (long long)T * top / tile + E || (((uintptr_t)h | (uintptr_t)xs) & 15)) return OE_ERR_UNSUPPORTED;
    const int blocks = (T + PT - 1) / PT;
    int rc = oe_launch(moe_count_kernel, dim3(blocks), dim3(256), 0, st, dense, T, E, W, counts);
    if (rc) return rc;
    return oe_launch(moe_place_kernel, dim3(blocks), dim3(256), 0, st, dense, T, E, W, top, tile, (const int*)counts, blocks, h, ldh, D, xs, place,
                     row_w, tile_expert, n_tiles, max_tiles);
}

int oe_moe_combine(float* out, long long ldc, const float* y, const int* place, int top, int T, int D, int accumulate, cudaStream_t st) {
    if (T <= 0) return 0;
    if (D % 4 || ldc % 4 || (((uintptr_t)out | (uintptr_t)y) & 15)) return OE_ERR_UNSUPPORTED;
    long long blocks = ((long long)T * (D / 4) + 255) / 256;
    if (blocks > 148 * 16) blocks = 148 * 16;
    return oe_launch(moe_combine_kernel, dim3((unsigned)blocks), dim3(256), 0, st, out, ldc, y, place, top, T, D, accumulate);
}

}  // extern "C"
