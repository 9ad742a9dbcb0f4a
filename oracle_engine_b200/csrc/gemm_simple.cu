// C[M,N] (+)= A[M,K] . W[N,K]^T on the CUDA cores, float32 accumulation.
//
// This is the matrix product of the true 32-bit path (no tensor cores, no reduced-
// precision mode) and the product for shapes the tensor-core kernels refuse.  Every
// output element is summed in ONE order, whatever kernel computes it: up to K = 512 one chain
// of fused multiply-adds over k; beyond, k is cut into segments of 64, segment s belongs to
// class s mod 8, a class is one chain over its segments in order of k, and the eight classes are
// added in order.  An element's value therefore does not depend on M, on the tile it falls in, or
// on what else is in the batch: the 32-bit logits are identical under every way of cutting
// the work.  Eight chains instead of one are what lets a handful of rows stream a weight
// matrix at the speed of the memory: eight threads share an output element.
// Role of the reference's `ops::matmul` / `gemm_q` (core/ops.cpp:207-289,
// core/gguf_parser.cpp:919-997): out[m,n] = A[m,k] . B[n,k]^T.
//
// Three kernels: `gemm_stream_kernel` for a few rows (bound by the weights' bytes), `gemm_tile_kernel` for more (bound
// by the multiply-adds), both float32 with 16-byte aligned rows, and `gemm_nt_kernel` for everything else.
#include "common.cuh"

namespace {

constexpr int CLASSES = 8, ONE_CHAIN = 512;

// A segment's length (a multiple of 64), the classes that have a segment, and how many rounds of segments there are.
__host__ __device__ __forceinline__ int segment(int K) { return K > ONE_CHAIN ? 64 : (K + 63) / 64 * 64; }
__host__ __device__ __forceinline__ int class_count(int K) { return K > ONE_CHAIN ? CLASSES : 1; }
__host__ __device__ __forceinline__ int class_rounds(int K) { return (K + segment(K) * CLASSES - 1) / (segment(K) * CLASSES); }

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool on) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = on ? 16 : 0;                      // 0: sixteen zero bytes, the source is not read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ------------------------------------------------------------------------------------------------------------------
// A few rows.  A warp owns 8 R weight rows and four classes (lane = row mod 8 and class), two warps share a set of rows, a
// CTA of four warps has 16 R rows, and CTAs walk over the tiles of rows.  Every warp has a ring of its own: a stage is KS
// values of k of its rows and classes (4 KS consecutive bytes a row and class) and the same k of MT rows of A; the ring
// runs on from tile to tile, so that loads stay in flight while a tile's classes are added up.  A lane reads its weights
// and A's values from the stage (rows four words apart from a multiple of 32: no eight lanes meet in a bank).  The next
// stage is asked for behind the products: before them it cost 5 to 15 %.
// ------------------------------------------------------------------------------------------------------------------
template <int R, int MT>
struct StreamShape {
    static constexpr int KS = R == 1 && MT <= 4 ? 32 : 16;                                 // k per stage and class
    static constexpr int CLS = KS;                                           // words between two classes of a row
    static constexpr int WROW = 4 * CLS + 4;                                     // words of a weight row in a stage
    static constexpr int STAGE = 8 * R * WROW + MT * 4 * CLS;                    // floats
    static constexpr int PER_SM = R == 4 ? 1 : 2;                                // CTAs an SM
    static constexpr int BUDGET = ((PER_SM == 1 ? 208 : 104) * 1024 - 16 * R * CLASSES * MT * 4) / (4 * STAGE * 4);
    static constexpr int STAGES = BUDGET > 10 ? 10 : BUDGET;
    static constexpr size_t BYTES = (size_t)(4 * STAGES * STAGE + 16 * R * CLASSES * MT) * 4;
};

template <int R, int MT, int MODE>
__global__ void __launch_bounds__(128)
gemm_stream_kernel(float* C, const float* A, const float* __restrict__ W, int M, int N, int K, long long lda, long long ldc,
                   int tiles_m, int tiles) {
    using S = StreamShape<R, MT>;
    constexpr int KS = S::KS, WROW = S::WROW, CLS = S::CLS;
    const int seg = segment(K), steps = seg / KS;
    extern __shared__ __align__(16) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int half = warp & 1, group = warp >> 1;    // classes 4 half .. 4 half + 3; rows 8 R group .. of the tile
    const int rl = lane & 7, sub = lane >> 3;
    float* ring = smem + warp * S::STAGES * S::STAGE;
    float* part = smem + 4 * S::STAGES * S::STAGE;   // [class][row of the tile][MT]
    const int per_tile = class_rounds(K) * steps;
    const int mine = tiles > (int)blockIdx.x ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int total = mine * per_tile;

    // what a lane loads in each stage: 16 bytes (k 4 lq .. 4 lq + 3) of class ls of weight rows lr, lr + LROWS, ...
    constexpr int LQ = KS / 4, LROWS = 8 / LQ;       // 16-byte pieces a row and class; rows a load instruction covers
    const int lq = lane % LQ, ls = lane / LQ % 4, lr = lane / LQ / 4;
    struct Place {                                   // where the next stage comes from and goes
        int tile, it, stage;
    };
    auto next = [&](Place& p) {
        if (++p.it == per_tile) { p.it = 0; p.tile += gridDim.x; }
        if (++p.stage == S::STAGES) p.stage = 0;
    };
    auto k_of = [&](const Place& p) { return (p.it / steps * CLASSES + 4 * half + ls) * seg + p.it % steps * KS + 4 * lq; };
    auto load_w = [&](const Place& p) {
        const int n0 = p.tile / tiles_m * (16 * R) + group * 8 * R, k = k_of(p);
        float* st = ring + p.stage * S::STAGE + ls * CLS + 4 * lq;
        const float* src = W + (size_t)n0 * K + k;
#pragma unroll
        for (int r0 = 0; r0 < 8 * R; r0 += LROWS) {
            const int r = r0 + lr;
            const bool on = k < K && n0 + r < N;
            cp_async16(st + r * WROW, on ? src + (size_t)r * K : W, on);
        }
    };
    auto load_a = [&](const Place& p) {
        const int m0 = p.tile % tiles_m * MT, k = k_of(p);
        float* st = ring + p.stage * S::STAGE + 8 * R * WROW + ls * CLS + 4 * lq;
#pragma unroll
        for (int r0 = 0; r0 < MT; r0 += LROWS) {
            const int m = r0 + lr;
            if (m < MT) {
                const bool on = k < K && m0 + m < M;
                cp_async16(st + m * 4 * CLS, on ? A + (size_t)(m0 + m) * lda + k : W, on);
            }
        }
    };
    // the first weights are asked for while the kernel before this one drains
    Place pw = {(int)blockIdx.x, 0, 0}, pa = pw;
#pragma unroll
    for (int i = 0; i < S::STAGES - 1; i++) if (i < total) { load_w(pw); next(pw); }
    pdl_wait();
#pragma unroll
    for (int i = 0; i < S::STAGES - 1; i++) {
        if (i < total) { load_a(pa); next(pa); }
        cp_commit();
    }
    float acc[R][MT];
#pragma unroll
    for (int j = 0; j < R; j++)
#pragma unroll
        for (int m = 0; m < MT; m++) acc[j][m] = 0.f;

    int it = 0, tile = blockIdx.x, stage = 0;
    for (int i = 0; i < total; i++) {
        cp_wait<S::STAGES - 2>();
        __syncwarp();                                 // the stage is there, and the one before it is free
        const float* st = ring + stage * S::STAGE;
        if (++stage == S::STAGES) stage = 0;
        const float* wr = st + rl * WROW + sub * CLS;
        const float* ar = st + 8 * R * WROW + sub * CLS;
#pragma unroll
        for (int kk = 0; kk < KS; kk += 4) {
            float4 w[R];
#pragma unroll
            for (int j = 0; j < R; j++) w[j] = *(const float4*)(wr + j * 8 * WROW + kk);
#pragma unroll
            for (int m = 0; m < MT; m++) {
                const float4 a = *(const float4*)(ar + m * 4 * CLS + kk);
#pragma unroll
                for (int j = 0; j < R; j++) {
                    acc[j][m] = fmaf(a.x, w[j].x, acc[j][m]);
                    acc[j][m] = fmaf(a.y, w[j].y, acc[j][m]);
                    acc[j][m] = fmaf(a.z, w[j].z, acc[j][m]);
                    acc[j][m] = fmaf(a.w, w[j].w, acc[j][m]);
                }
            }
        }
        __syncwarp();
        if (i + S::STAGES - 1 < total) { load_w(pa); load_a(pa); next(pa); }
        cp_commit();
        if (++it < per_tile) continue;
        it = 0;
        const int n0 = tile / tiles_m * (16 * R), m0 = tile % tiles_m * MT;
        tile += gridDim.x;
        float* p = part + ((4 * half + sub) * 16 * R + group * 8 * R + rl) * MT;
#pragma unroll
        for (int j = 0; j < R; j++)
#pragma unroll
            for (int m = 0; m < MT; m++) { p[j * 8 * MT + m] = acc[j][m]; acc[j][m] = 0.f; }
        __syncthreads();
        const int classes = class_count(K);
        for (int e = threadIdx.x; e < 16 * R * MT; e += 128) {
            const int r = e % (16 * R), m = e / (16 * R);
            float v = part[r * MT + m];
            for (int c = 1; c < classes; c++) v += part[(c * 16 * R + r) * MT + m];
            if (n0 + r < N && m0 + m < M) {
                float* o = C + (size_t)(m0 + m) * ldc + n0 + r;
                *o = MODE == 1 ? *o + v : v;
            }
        }
        __syncthreads();
    }
    pdl_launch_dependents();
}

// ------------------------------------------------------------------------------------------------------------------
// Many rows.  256 threads of 8 x 8 outputs: a tile of 128 x 128 (KG = 1), or of 64 x 64 whose classes are shared out over
// KG = 4 groups of 64 threads (small products, for which tiles of 128 would leave SMs idle).  Stages of 16 values of k come
// by cp.async as they lie in memory; a thread reads four k at a time of its rows (rows 20 words apart: no bank conflicts
// between the eight lanes that differ), 16 16-byte loads for 256 multiply-adds.
// ------------------------------------------------------------------------------------------------------------------
constexpr int TK = 16, TROW = TK + 4;

template <int BM, int BN, int KG>
struct TileShape {
    static constexpr int STAGE = (BM + BN) * TROW, STAGES = 3;
    static constexpr size_t RING = (size_t)KG * STAGES * STAGE * 4;
    static constexpr size_t BYTES = RING + (KG > 1 ? (size_t)KG * BM * BN * 4 : 0);   // the first of a group's two classes
};

template <int BM, int BN, int KG, int MODE>
__global__ void __launch_bounds__(256)
gemm_tile_kernel(float* C, const float* A, const float* __restrict__ W, int M, int N, int K, long long lda, long long ldc) {
    using S = TileShape<BM, BN, KG>;
    constexpr int GT = 256 / KG;                     // threads of a group
    static_assert((BM / 8) * (BN / 8) == GT, "8 x 8 outputs a thread");
    extern __shared__ __align__(16) float smem[];
    const int g = threadIdx.x / GT, t = threadIdx.x % GT, warp = t >> 5, lane = t & 31;
    const int wn = warp % (BN / 64), wm = warp / (BN / 64);
    const int ty = lane >> 3, tx = lane & 7;         // outputs (32 wm + ty + 4 i, 64 wn + tx + 8 j)
    const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
    float* ring = smem + g * S::STAGES * S::STAGE;
    const int classes = class_count(K), rounds = class_rounds(K);
    constexpr int CPG = CLASSES / KG;                // classes of a group
    const int seg = segment(K), steps = seg / TK, per_class = rounds * steps;
    const int total = (KG == 1 ? classes : CPG) * per_class;

    const int lq = t & 3, lr = t >> 2;
    auto load = [&](int i) {
        const int c = g * CPG + i / per_class, it = i % per_class;
        const int k = (it / steps * CLASSES + c) * seg + it % steps * TK + 4 * lq;
        float* st = ring + (i % S::STAGES) * S::STAGE + 4 * lq;
#pragma unroll
        for (int r = lr; r < BM; r += GT / 4) {
            const bool on = k < K && m0 + r < M;
            cp_async16(st + r * TROW, on ? A + (size_t)(m0 + r) * lda + k : W, on);
        }
#pragma unroll
        for (int r = lr; r < BN; r += GT / 4) {
            const bool on = k < K && n0 + r < N;
            cp_async16(st + (BM + r) * TROW, on ? W + (size_t)(n0 + r) * K + k : W, on);
        }
    };
    pdl_launch_dependents();
    pdl_wait();
#pragma unroll
    for (int i = 0; i < S::STAGES - 1; i++) { if (i < total) load(i); cp_commit(); }
    float acc[8][8], tot[KG == 1 ? 8 : 1][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) { acc[i][j] = 0.f; if (KG == 1) tot[KG == 1 ? i : 0][j] = 0.f; }
    float* kept = smem + KG * S::STAGES * S::STAGE + g * BM * BN;
    const int row = 32 * wm + ty, col = 64 * wn + tx;

    int it = 0, c = 0;
    for (int i = 0; i < total; i++) {
        cp_wait<S::STAGES - 2>();
        __syncthreads();
        if (i + S::STAGES - 1 < total) load(i + S::STAGES - 1);
        cp_commit();
        const float* as = ring + (i % S::STAGES) * S::STAGE + row * TROW;
        const float* ws = ring + (i % S::STAGES) * S::STAGE + (BM + col) * TROW;
#pragma unroll
        for (int kk = 0; kk < TK; kk += 4) {
            float4 a[8], b[8];
#pragma unroll
            for (int j = 0; j < 8; j++) { a[j] = *(const float4*)(as + 4 * j * TROW + kk); b[j] = *(const float4*)(ws + 8 * j * TROW + kk); }
#pragma unroll
            for (int ii = 0; ii < 8; ii++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[ii][j] = fmaf(a[ii].x, b[j].x, acc[ii][j]);
#pragma unroll
            for (int ii = 0; ii < 8; ii++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[ii][j] = fmaf(a[ii].y, b[j].y, acc[ii][j]);
#pragma unroll
            for (int ii = 0; ii < 8; ii++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[ii][j] = fmaf(a[ii].z, b[j].z, acc[ii][j]);
#pragma unroll
            for (int ii = 0; ii < 8; ii++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[ii][j] = fmaf(a[ii].w, b[j].w, acc[ii][j]);
        }
        if (++it < per_class) continue;
        it = 0;                                       // a class is complete
        if (KG == 1) {
#pragma unroll
            for (int ii = 0; ii < 8; ii++)
#pragma unroll
                for (int j = 0; j < 8; j++) { tot[KG == 1 ? ii : 0][j] = c == 0 ? acc[ii][j] : tot[KG == 1 ? ii : 0][j] + acc[ii][j]; acc[ii][j] = 0.f; }
        } else if (c == 0) {
#pragma unroll
            for (int ii = 0; ii < 8; ii++)
#pragma unroll
                for (int j = 0; j < 8; j++) { kept[(row + 4 * ii) * BN + col + 8 * j] = acc[ii][j]; acc[ii][j] = 0.f; }
        }
        c++;
    }
    if constexpr (KG > 1) {
        // the second classes go where the stages were; then every thread adds up a share of the outputs
        cp_wait<0>();
        __syncthreads();
        float* second = smem + g * BM * BN;
        static_assert(KG == 1 || (size_t)KG * BM * BN * 4 <= S::RING, "the ring holds the second classes");
#pragma unroll
        for (int ii = 0; ii < 8; ii++)
#pragma unroll
            for (int j = 0; j < 8; j++) second[(row + 4 * ii) * BN + col + 8 * j] = acc[ii][j];
        __syncthreads();
        const float* first = smem + KG * S::STAGES * S::STAGE;
        for (int e = threadIdx.x; e < BM * BN; e += 256) {
            const int m = m0 + e / BN, n = n0 + e % BN;
            if (m >= M || n >= N) continue;
            float v = first[e];
            for (int q = 1; q < classes; q++) v += ((q & 1) ? smem : first)[(q >> 1) * BM * BN + e];
            float* o = C + (size_t)m * ldc + n;
            *o = MODE == 1 ? *o + v : v;
        }
    } else
#pragma unroll
    for (int ii = 0; ii < 8; ii++) {
        const int m = m0 + row + 4 * ii;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int n = n0 + col + 8 * j;
            if (n >= N) continue;
            float* o = C + (size_t)m * ldc + n;
            const float v = tot[KG == 1 ? ii : 0][j];
            *o = MODE == 1 ? *o + v : v;
        }
    }
}

// ------------------------------------------------------------------------------------------------------------------
// Any types, sizes and alignments.
// ------------------------------------------------------------------------------------------------------------------
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

// MODE 0: C = acc (type TC);  MODE 1: C += acc (TC must be float: the residual stream)
template <typename TA, typename TC, int MODE>
__global__ void __launch_bounds__(256)
gemm_nt_kernel(TC* C, const TA* A, const TA* __restrict__ W,
               int M, int N, int K, long long lda, long long ldc) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int lr = tid / 4, lk = (tid % 4) * 4;      // loader: row lr, k lk..lk+3

    pdl_launch_dependents();
    pdl_wait();
    float acc[TM][TN], tot[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) acc[i][j] = tot[i][j] = 0.f;

    const int seg = segment(K);
    for (int c = 0; c < class_count(K); c++) {
    for (int s = c * seg; s < K; s += seg * CLASSES)
    for (int k0 = s; k0 < s + seg && k0 < K; k0 += BK) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int k = k0 + lk + j;
            const int am = m0 + lr, wn = n0 + lr;
            As[lk + j][lr] = (am < M && k < K) ? to_f32(A[(size_t)am * lda + k]) : 0.f;
            Ws[lk + j][lr] = (wn < N && k < K) ? to_f32(W[(size_t)wn * K + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; i++) a[i] = As[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; j++) b[j] = Ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j++) { tot[i][j] = c == 0 ? acc[i][j] : tot[i][j] + acc[i][j]; acc[i][j] = 0.f; }
    }
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const int n = n0 + tx * TN + j;
            if (n >= N) continue;
            TC* p = C + (size_t)m * ldc + n;
            if (MODE == 1) *p = from_f32<TC>(to_f32(*p) + tot[i][j]);
            else *p = from_f32<TC>(tot[i][j]);
        }
    }
}

template <typename TA, typename TC, int MODE>
int launch(TC* C, const TA* A, const TA* W, int M, int N, int K, long long lda, long long ldc,
           cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return OE_ERR_UNSUPPORTED;
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return OE_ERR_UNSUPPORTED;
    const int launch_rc = oe_launch(gemm_nt_kernel<TA, TC, MODE>, dim3(grid), dim3(256), 0, st, C, A, W, M, N, K, lda, ldc);
    return launch_rc;
}

template <int R, int MT, int MODE>
int launch_stream(float* C, const float* A, const float* W, int M, int N, int K, long long lda, long long ldc, int sms, cudaStream_t st) {
    constexpr size_t bytes = StreamShape<R, MT>::BYTES;
    static_assert(StreamShape<R, MT>::STAGES >= 3, "stages");
    cudaError_t e = cudaFuncSetAttribute(gemm_stream_kernel<R, MT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    const int tiles_m = (M + MT - 1) / MT, tiles = tiles_m * ((N + 16 * R - 1) / (16 * R));
    const int most = StreamShape<R, MT>::PER_SM * sms, grid = tiles < most ? tiles : most;
    return oe_launch(gemm_stream_kernel<R, MT, MODE>, dim3(grid), dim3(128), bytes, st, C, A, W, M, N, K, lda, ldc, tiles_m, tiles);
}
template <int MT, int MODE>
int launch_stream_rows(float* C, const float* A, const float* W, int M, int N, int K, long long lda, long long ldc, int sms, cudaStream_t st) {
    // Weight rows a lane: A's values are read from shared memory once for R rows, so more of them help as soon as there are
    // tiles for every SM.
    if (MT > 2 && N >= 64 * sms) return launch_stream<4, MT, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
    if (N >= 32 * sms) return launch_stream<2, MT, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
    return launch_stream<1, MT, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
}
template <int BM_, int BN_, int KG, int MODE>
int launch_tile(float* C, const float* A, const float* W, int M, int N, int K, long long lda, long long ldc, cudaStream_t st) {
    constexpr size_t bytes = TileShape<BM_, BN_, KG>::BYTES;
    cudaError_t e = cudaFuncSetAttribute(gemm_tile_kernel<BM_, BN_, KG, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    dim3 grid((N + BN_ - 1) / BN_, (M + BM_ - 1) / BM_);
    if (grid.y > 65535) return OE_ERR_UNSUPPORTED;
    return oe_launch(gemm_tile_kernel<BM_, BN_, KG, MODE>, grid, dim3(256), bytes, st, C, A, W, M, N, K, lda, ldc);
}

constexpr int STREAM_MAX_M = 32;

// kind: 0 by size, else 1 streaming, 2 tiles of 64, 3 tiles of 128, 4 the general kernel (tests).
template <int MODE>
int launch_f32(float* C, const float* A, const float* W, int M, int N, int K, long long lda, long long ldc, int kind, cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return OE_ERR_UNSUPPORTED;
    const bool aligned = K % 4 == 0 && lda % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
    if (!aligned || kind == 4) return kind == 0 || kind == 4 ? launch<float, float, MODE>(C, A, W, M, N, K, lda, ldc, st) : OE_ERR_UNSUPPORTED;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (kind == 0) {
        const long long t128 = (long long)((M + 127) / 128) * ((N + 127) / 128);
        const long long t64 = (long long)((M + 63) / 64) * ((N + 63) / 64);
        // Eight chains are what tiles of 64 share out over a CTA's groups: up to K = 512 there is one, and tiles of 128 it is.
        // Up to 64 rows a narrow weight has too few tiles of 64 for the SMs (64 x 2,048 x 2,048: 58 us streamed, 78 by tiles; 64 x
        // 16,384 x 2,048: 249 and 153); below 1.5 tiles of 128 an SM, tiles of 64 leave less of the last round empty
        kind = M <= STREAM_MAX_M || (M <= 64 && 2 * t64 < sms) ? 1 : K <= ONE_CHAIN || 2 * t128 >= 3 * sms ? 3 : 2;
    }
    if (kind == 3) return launch_tile<128, 128, 1, MODE>(C, A, W, M, N, K, lda, ldc, st);
    if (kind == 2) return launch_tile<64, 64, 4, MODE>(C, A, W, M, N, K, lda, ldc, st);
    if (M == 1) return launch_stream_rows<1, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
    if (M == 2) return launch_stream_rows<2, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
    if (M <= 4) return launch_stream_rows<4, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
    return launch_stream_rows<8, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
}

}  // namespace

extern "C" {
// out_kind: 0 = same type as the inputs, 1 = float32 store, 2 = float32 accumulate (C += A.W^T)
int oe_gemm_simple_f32(void* C, const float* A, const float* W, int M, int N, int K, long long lda,
                       long long ldc, int out_kind, cudaStream_t st) {
    if (out_kind == 2) return launch_f32<1>((float*)C, A, W, M, N, K, lda, ldc, 0, st);
    return launch_f32<0>((float*)C, A, W, M, N, K, lda, ldc, 0, st);
}
// The same through one kernel of the three, whatever the size: they give the same bits.
int oe_gemm_simple_kind_f32(float* C, const float* A, const float* W, int M, int N, int K, long long lda, long long ldc,
                            int accumulate, int kind, cudaStream_t st) {
    if (accumulate) return launch_f32<1>(C, A, W, M, N, K, lda, ldc, kind, st);
    return launch_f32<0>(C, A, W, M, N, K, lda, ldc, kind, st);
}
int oe_gemm_simple_bf16(void* C, const bf16* A, const bf16* W, int M, int N, int K, long long lda,
                        long long ldc, int out_kind, cudaStream_t st) {
    if (out_kind == 2) return launch<bf16, float, 1>((float*)C, A, W, M, N, K, lda, ldc, st);
    if (out_kind == 1) return launch<bf16, float, 0>((float*)C, A, W, M, N, K, lda, ldc, st);
    return launch<bf16, bf16, 0>((bf16*)C, A, W, M, N, K, lda, ldc, st);
}
}
