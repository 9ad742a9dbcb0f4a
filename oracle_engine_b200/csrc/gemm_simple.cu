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
// Four kernels: `gemm_rows_kernel` for a few rows (bound by the weights' bytes), `gemm_tile_kernel` for some dozens and
// `gemm_wide_kernel` for more (bound by the multiply-adds), all float32 with 16-byte aligned rows, and `gemm_nt_kernel` for
// everything else.
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
// A few rows: bound by the weights' bytes.  A CTA takes tiles of 16 weight rows in turn, a stage at a time: 512 k of every row,
// that is 2 KB in one piece from memory, where the eight classes lie side by side.  Two warps multiply, a lane rows rl and
// rl + 8 of one class (A's values, four fifths of what was read from shared memory when a lane had one row, are read once for
// two); two warps load the weights and one the rows of A, so that the ring runs on from tile to tile.  Rows four words apart
// from a multiple of 32: no eight lanes meet in a bank.  In the decode step of the 1B shape (3 rows), against a kernel whose
// warps loaded 128 bytes of every other segment for themselves: 8,192 -> 2,048 43.5 -> 19.4 us (67 MB), 2,048 -> 2,048
// 9.5 -> 5.2, 2,048 -> 3,072 12.4 -> 10, 2,048 -> 16,384 34.7 -> 32.8 (134 MB).  Up to 512 k eight lanes of one warp have all there is
// to add up, and it is still faster than the kernel before, whose sixteen did (K = 64 / 128 / 192 / 512 to 2,048 rows: 1 row 2.5 / 3.8 /
// 5.0 / 10.8 -> 2.0 / 2.1 / 2.5 / 4.2, 3 rows 2.9 / 4.8 / 6.7 / 16.1 -> 2.5 / 3.3 / 4.1 / 8.1, 16 rows 5.0 / 8.5 / 12.1 / 29.3 -> 3.6 / 4.8 /
// 7.3 / 14).  Where the ring leaves room for one or two CTAs an SM anyway the registers are theirs: left to itself the compiler
// took 64 and loaded no value ahead of its use (2 rows of 64 x 2,048 6.7 -> 5.0 us, of 2,048 x 8,192 22 -> 16.3; 8 rows 39 -> 28).
// ------------------------------------------------------------------------------------------------------------------
constexpr int RT = 16, RK = 512, RPITCH = RK + 4;    // weight rows of a tile, k of a stage, words between a stage's rows

template <int MT, int S>
struct RowsShape {
    static constexpr int STAGE = (RT + MT) * RPITCH;
    static constexpr size_t BYTES = ((size_t)S * STAGE + CLASSES * RT * MT) * 4;
};
__device__ __forceinline__ void rows_sync(int id) { asm volatile("barrier.cta.sync %0, 160;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void rows_arrive(int id) { asm volatile("barrier.cta.arrive %0, 160;" ::"r"(id) : "memory"); }

template <int MT, int S, int MODE>
__global__ void __launch_bounds__(160, MT == 8 && S == 2 ? 0 : 1)
gemm_rows_kernel(float* C, const float* A, const float* __restrict__ W, int M, int N, int K, long long lda, long long ldc,
                 int tiles_m, int tiles) {
    constexpr int STAGE = RowsShape<MT, S>::STAGE;
    constexpr int READY = 1, TAKEN = 1 + S, PAIR = 1 + 2 * S;      // barriers: of stage s READY + s, TAKEN + s; of the multiplying warps
    extern __shared__ __align__(16) float smem[];
    float* part = smem + S * STAGE;                  // [class][row][MT]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int per_tile = (K + RK - 1) / RK;
    const int mine = tiles > (int)blockIdx.x ? (tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int total = mine * per_tile;

    if (warp >= 2) {
        const bool weights = warp < 4;               // two warps load the weights, which no kernel writes, one the rows of A
        if (!weights) pdl_wait();
        for (int i = 0; i < total + S - 1; i++) {
            if (i < total) {
                if (i >= S) rows_sync(TAKEN + i % S);
                const int tile = blockIdx.x + i / per_tile * (int)gridDim.x, k0 = i % per_tile * RK;
                const int pieces = min(RK, K - k0) / 4;             // of 16 bytes in a row
                float* st = smem + i % S * STAGE;
                if (weights) {
                    const int n0 = tile / tiles_m * RT, rows = min(RT, N - n0);
                    const float* from = W + (size_t)n0 * K + k0;
                    for (int p = (threadIdx.x & 31); p < pieces; p += 32) {
#pragma unroll
                        for (int r = warp - 2; r < RT; r += 2) if (r < rows) cp_async16(st + r * RPITCH + 4 * p, from + (size_t)r * K + 4 * p, true);
                    }
                } else {
                    const int m0 = tile % tiles_m * MT, rows = min(MT, M - m0);
                    const float* from = A + (size_t)m0 * lda + k0;
                    for (int p = lane; p < pieces; p += 32) {
#pragma unroll
                        for (int m = 0; m < MT; m++) if (m < rows) cp_async16(st + (RT + m) * RPITCH + 4 * p, from + (size_t)m * lda + 4 * p, true);
                    }
                }
            }
            cp_commit();
            if (i >= S - 1) {
                cp_wait<S - 1>();
                rows_arrive(READY + (i - (S - 1)) % S);
            }
        }
        if (weights) pdl_wait();
        return;
    }
    pdl_wait();
    // a lane: rows rl and rl + 8, class c
    const int rl = lane & 7, c = 4 * warp + (lane >> 3), seg = segment(K), classes = class_count(K);
    float acc[2][MT];
#pragma unroll
    for (int m = 0; m < MT; m++) acc[0][m] = acc[1][m] = 0.f;
    int it = 0, tile = blockIdx.x;
    for (int i = 0; i < total; i++) {
        const int left = K - (it * CLASSES + c) * seg, n = left < 0 ? 0 : left < seg ? left : seg;    // values of this lane's class
        rows_sync(READY + i % S);
        const float* w0 = smem + i % S * STAGE + rl * RPITCH + c * seg;
        const float* a0 = smem + i % S * STAGE + RT * RPITCH + c * seg;
        auto four = [&](int k) {
            const float4 u = *(const float4*)(w0 + k), v = *(const float4*)(w0 + 8 * RPITCH + k);
#pragma unroll
            for (int m = 0; m < MT; m++) {
                const float4 a = *(const float4*)(a0 + m * RPITCH + k);
                acc[0][m] = fmaf(a.x, u.x, acc[0][m]); acc[1][m] = fmaf(a.x, v.x, acc[1][m]);
                acc[0][m] = fmaf(a.y, u.y, acc[0][m]); acc[1][m] = fmaf(a.y, v.y, acc[1][m]);
                acc[0][m] = fmaf(a.z, u.z, acc[0][m]); acc[1][m] = fmaf(a.z, v.z, acc[1][m]);
                acc[0][m] = fmaf(a.w, u.w, acc[0][m]); acc[1][m] = fmaf(a.w, v.w, acc[1][m]);
            }
        };
        if (__all_sync(0xffffffffu, n == 64)) {
#pragma unroll
            for (int k = 0; k < 64; k += 4) four(k);
        } else {
            for (int k = 0; k < n; k += 4) four(k);
            __syncwarp();
        }
        if (i + S < total) rows_arrive(TAKEN + i % S);
        if (++it < per_tile) continue;
        it = 0;
        const int n0 = tile / tiles_m * RT, m0 = tile % tiles_m * MT;
        tile += gridDim.x;
#pragma unroll
        for (int m = 0; m < MT; m++) {
            part[(c * RT + rl) * MT + m] = acc[0][m];
            part[(c * RT + rl + 8) * MT + m] = acc[1][m];
            acc[0][m] = acc[1][m] = 0.f;
        }
        asm volatile("barrier.cta.sync %0, 64;" ::"r"(PAIR) : "memory");
        for (int e = threadIdx.x; e < RT * MT; e += 64) {
            const int r = e % RT, m = e / RT;
            float v = part[r * MT + m];
            for (int q = 1; q < classes; q++) v += part[(q * RT + r) * MT + m];
            if (n0 + r < N && m0 + m < M) {
                float* o = C + (size_t)(m0 + m) * ldc + n0 + r;
                *o = MODE == 1 ? *o + v : v;
            }
        }
        asm volatile("barrier.cta.sync %0, 64;" ::"r"(PAIR) : "memory");
    }
    pdl_launch_dependents();
}

// ------------------------------------------------------------------------------------------------------------------
// Some dozens of rows of a wide weight.  256 threads of 8 x 8 outputs: a tile of 64 x 64 whose classes are shared out over
// KG = 4 groups of 64 threads.  Stages of 16 values of k come by cp.async as they lie in memory; a thread reads four k at a
// time of its rows (rows 20 words apart: no bank conflicts between the eight lanes that differ), 16 16-byte loads for 256
// multiply-adds.
// ------------------------------------------------------------------------------------------------------------------
constexpr int TK = 16, TROW = TK + 4;

template <int BM, int BN, int KG>
struct TileShape {
    static constexpr int STAGE = (BM + BN) * TROW, STAGES = 3;
    static constexpr size_t RING = (size_t)KG * STAGES * STAGE * 4;
    static constexpr size_t BYTES = RING + (size_t)KG * BM * BN * 4;                  // the first of a group's two classes
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
    const int total = CPG * per_class;

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
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0.f;
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
        if (c == 0) {
#pragma unroll
            for (int ii = 0; ii < 8; ii++)
#pragma unroll
                for (int j = 0; j < 8; j++) { kept[(row + 4 * ii) * BN + col + 8 * j] = acc[ii][j]; acc[ii][j] = 0.f; }
        }
        c++;
    }
    // the second classes go where the stages were; then every thread adds up a share of the outputs
    cp_wait<0>();
    __syncthreads();
    float* second = smem + g * BM * BN;
    static_assert((size_t)KG * BM * BN * 4 <= S::RING, "the ring holds the second classes");
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
}

// ------------------------------------------------------------------------------------------------------------------
// Many rows, tiles of 128 x 128.  Four warps multiply, 16 x 8 outputs a thread; four others load (setmaxnreg gives the first
// the others' registers); two CTAs an SM.  A thread of 8 x 8 outputs reads 16 values from shared memory for 64 products, at
// which the two take the same time; 16 x 8 read 24 for 128.  Stages of 16 k lie transposed, k by k, so that a thread's values
// of one k are 16-byte pieces; the loading warps turn 4 x 4 values in registers.  Loaded by the multiplying warps themselves the
// same kernel was a quarter slower, with cp.async of 4 bytes as with 16-byte loads.  The products are done two rows at a time
// (fma.rn.f32x2: each half is rounded as by itself), which leaves issue slots to the loads from shared memory.
// KG = 1: a single chain (K up to 512).  KG = 4, 8: the classes of a tile are shared out over the CTAs of a cluster, class
// p KG + rank in phase p; behind each phase every CTA adds up its share of the rows, class by class, from the shared memory
// of all.  468 rows, tiles of 8 x 8 outputs before -> now: 2,048 -> 16,384 997 -> 734 us (43 TFLOP/s; the multiply-adds of
// tiles that are full to the last row would take 470), 2,048 -> 3,072 228 -> 162, 2,048 -> 2,048 156 -> 118, 8,192 -> 2,048
// 578 -> 406.
// ------------------------------------------------------------------------------------------------------------------
constexpr int WT = 128, WLD = WT;

struct WideShape {
    static constexpr int STAGE = 2 * TK * WLD;
    static constexpr size_t BYTES = ((size_t)2 * STAGE + 2 * WT * TK + WT * WT) * 4;      // 112 KB: two CTAs an SM, no more
    static constexpr size_t ALONE = 120 * 1024;                                           // one
};

__device__ __forceinline__ unsigned long long two(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float2 halves(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(unsigned long long& c, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 load_shared_of(const float* local, unsigned rank) {
    const unsigned here = (unsigned)__cvta_generic_to_shared(local);
    unsigned there;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(here), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(there) : "memory");
    return v;
}
__device__ __forceinline__ float4 add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

// Four neighbouring outputs of a row.
template <int MODE>
__device__ __forceinline__ void store4(float* C, float4 v, int m, int n, int M, int N, long long ldc, bool vec) {
    if (m >= M) return;
    float* o = C + (size_t)m * ldc + n;
    if (vec && n + 4 <= N) {
        if (MODE == 1) v = add4(*(const float4*)o, v);
        *(float4*)o = v;
        return;
    }
    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; i++) if (n + i < N) o[i] = MODE == 1 ? o[i] + e[i] : e[i];
}

__device__ __forceinline__ void named_sync(int id) { asm volatile("barrier.cta.sync %0, 256;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void named_arrive(int id) { asm volatile("barrier.cta.arrive %0, 256;" ::"r"(id) : "memory"); }
constexpr int FULL = 1, FREE = 3;                    // the barriers of stage s: FULL + s, FREE + s

template <int KG, int MODE>
__global__ void __launch_bounds__(256, 2)
gemm_wide_kernel(float* C, const float* A, const float* __restrict__ W, int M, int N, int K, long long lda, long long ldc, int tiles_m) {
    extern __shared__ __align__(16) float smem[];
    float4* landing = (float4*)(smem + 2 * WideShape::STAGE);        // what the loading threads have asked for, [piece][thread]
    float* sums = smem + 2 * WideShape::STAGE + 2 * WT * TK;         // a class's sums, [row][column]
    const int tid = threadIdx.x & 127, warp = tid >> 5, lane = tid & 31;
    const int rank = KG == 1 ? 0 : (int)(blockIdx.x % KG), tile = blockIdx.x / KG;
    const int m0 = tile % tiles_m * WT, n0 = tile / tiles_m * WT;
    const int seg = segment(K), steps = seg / TK, per_class = class_rounds(K) * steps;
    const int phases = KG == 1 ? 1 : CLASSES / KG, total = phases * per_class;
    pdl_launch_dependents();
    pdl_wait();
    if (KG > 1) cluster_barrier();                   // every CTA of the cluster is there before its memory is read

    if (threadIdx.x >= 128) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
        // k 4 lk .. 4 lk + 3 of rows 4 lr .. 4 lr + 3
        const int lr = lane & 7 | warp << 3, lk = lane >> 3;
        const float* a_at = A + (size_t)(m0 + 4 * lr) * lda;
        const float* w_at = W + (size_t)(n0 + 4 * lr) * K;
        const int a_rows = M - m0 - 4 * lr, w_rows = N - n0 - 4 * lr;
        auto ask = [&](int i) {
            const int c = i / per_class * KG + rank, it = i % per_class;
            const int k = (it / steps * CLASSES + c) * seg + it % steps * TK + 4 * lk;
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const bool on = k < K && r < a_rows;
                cp_async16((float*)(landing + r * 128 + tid), on ? a_at + r * lda + k : A, on);
            }
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const bool on = k < K && r < w_rows;
                cp_async16((float*)(landing + (4 + r) * 128 + tid), on ? w_at + (size_t)r * K + k : W, on);
            }
        };
        auto turn = [&](const float4* from, float* st) {
            const float4 p0 = from[0], p1 = from[128], p2 = from[256], p3 = from[384];
            float* to = st + 4 * lk * WLD + 4 * lr;
            *(float4*)to = make_float4(p0.x, p1.x, p2.x, p3.x);
            *(float4*)(to + WLD) = make_float4(p0.y, p1.y, p2.y, p3.y);
            *(float4*)(to + 2 * WLD) = make_float4(p0.z, p1.z, p2.z, p3.z);
            *(float4*)(to + 3 * WLD) = make_float4(p0.w, p1.w, p2.w, p3.w);
        };
        ask(0);
        for (int i = 0; i < total; i++) {
            // two stages may lie ahead of the multiplying warps, which meet the other CTAs behind the first class
            if (KG > 1 && i == per_class + 2) cluster_barrier();
            cp_commit();
            cp_wait<0>();
            if (i >= 2) named_sync(FREE + (i & 1));
            float* st = smem + (i & 1) * WideShape::STAGE;
            turn(landing + tid, st);
            turn(landing + 512 + tid, st + TK * WLD);
            named_arrive(FULL + (i & 1));
            if (i + 1 < total) ask(i + 1);            // (a thread reads only what it has asked for)
        }
        if (KG > 1) {                                 // the barriers of the multiplying warps that are left
            for (int b = phases > 1 ? 1 : 0; b < 2 * phases; b++) cluster_barrier();
        }
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
    // outputs (row + 16 i + r, col + 32 j + c), i, r, c < 4, j < 2
    const int row = (warp >> 1) * 64 + (lane >> 3) * 4, col = (warp & 1) * 64 + (lane & 7) * 4;
    unsigned long long acc[8][8];                    // rows 2 p, 2 p + 1 of the thread's sixteen; columns
#pragma unroll
    for (int p = 0; p < 8; p++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[p][j] = 0ull;
    constexpr int SHARE = KG == 1 ? 1 : WT * WT / KG / 128 / 4;      // 16-byte pieces of the tile that a thread adds up
    float4 share[SHARE];

    const bool vec = (ldc & 3) == 0 && ((size_t)C & 15) == 0;

    int it = 0, phase = 0;
    for (int i = 0; i < total; i++) {
        named_sync(FULL + (i & 1));
        const float* as = smem + (i & 1) * WideShape::STAGE + row;
        const float* ws = smem + (i & 1) * WideShape::STAGE + TK * WLD + col;
#pragma unroll
        for (int kk = 0; kk < TK; kk++) {
            unsigned long long a[8], b[8];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const ulonglong2 v = *(const ulonglong2*)(as + kk * WLD + 16 * q);
                a[2 * q] = v.x; a[2 * q + 1] = v.y;
            }
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const float4 v = *(const float4*)(ws + kk * WLD + 32 * q);
                b[4 * q] = two(v.x, v.x); b[4 * q + 1] = two(v.y, v.y); b[4 * q + 2] = two(v.z, v.z); b[4 * q + 3] = two(v.w, v.w);
            }
#pragma unroll
            for (int p = 0; p < 8; p++)
#pragma unroll
                for (int j = 0; j < 8; j++) fma2(acc[p][j], a[p], b[j]);
        }
        if (i + 2 < total) named_arrive(FREE + (i & 1));
        if (++it < per_class) continue;
        it = 0;                                       // a class is complete
        const bool first = phase++ == 0;
        if (KG > 1 && !first) cluster_barrier();      // the class before has been read
#pragma unroll
        for (int p = 0; p < 8; p++) {
#pragma unroll
            for (int j = 0; j < 2; j++) {
                float2 h[4];
#pragma unroll
                for (int c = 0; c < 4; c++) { h[c] = halves(acc[p][4 * j + c]); acc[p][4 * j + c] = 0ull; }
                const float4 even = make_float4(h[0].x, h[1].x, h[2].x, h[3].x), odd = make_float4(h[0].y, h[1].y, h[2].y, h[3].y);
                const int r = row + 16 * (p >> 1) + 2 * (p & 1), c = col + 32 * j;
                if (KG == 1) {
                    store4<MODE>(C, even, m0 + r, n0 + c, M, N, ldc, vec);
                    store4<MODE>(C, odd, m0 + r + 1, n0 + c, M, N, ldc, vec);
                } else {
                    float4* to = (float4*)(sums + r * WT + c);
                    to[0] = even; to[WT / 4] = odd;
                }
            }
        }
        if (KG > 1) {
            cluster_barrier();
#pragma unroll
            for (int e = 0; e < SHARE; e++) {
                const int place = rank * (WT * WT / KG) + (e * 128 + tid) * 4;
                float4 v = load_shared_of(sums + place, 0);
                if (!first) v = add4(share[e], v);
#pragma unroll
                for (int g = 1; g < KG; g++) v = add4(v, load_shared_of(sums + place, g));
                share[e] = v;
            }
        }
    }
    if (KG > 1) {
#pragma unroll
        for (int e = 0; e < SHARE; e++) {
            const int place = rank * (WT * WT / KG) + (e * 128 + tid) * 4;
            store4<MODE>(C, share[e], m0 + place / WT, n0 + place % WT, M, N, ldc, vec);
        }
        cluster_barrier();                            // no CTA leaves while its memory is read
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

template <int MT, int S, int MODE>
int launch_rows(float* C, const float* A, const float* W, int M, int N, int K, long long lda, long long ldc, int most, cudaStream_t st) {
    constexpr size_t bytes = RowsShape<MT, S>::BYTES;
    cudaError_t e = cudaFuncSetAttribute(gemm_rows_kernel<MT, S, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    const int tiles_m = (M + MT - 1) / MT, tiles = tiles_m * ((N + RT - 1) / RT);
    return oe_launch(gemm_rows_kernel<MT, S, MODE>, dim3(tiles < most ? tiles : most), dim3(160), bytes, st, C, A, W, M, N, K, lda, ldc, tiles_m, tiles);
}
template <int MT, int MODE>
int launch_rows_for(float* C, const float* A, const float* W, int M, int N, int K, long long lda, long long ldc, int sms, cudaStream_t st) {
    // While the tiles leave an SM each, one CTA with a deep ring; beyond, two an SM (8 x 2,048 x 8,192: 43 us with the deep ring,
    // 45 with two stages, 16 rows 82 and 53; 3 x 128,256 x 2,048: 265 and 202).
    constexpr int DEEP = MT == 8 ? 4 : 5;
    const long long tiles = (long long)((M + MT - 1) / MT) * ((N + RT - 1) / RT);
    if (tiles > 0x7fffffffll) return OE_ERR_UNSUPPORTED;
    if (tiles <= sms) return launch_rows<MT, DEEP, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
    return launch_rows<MT, 2, MODE>(C, A, W, M, N, K, lda, ldc, 2 * sms, st);
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

template <int KG, int MODE>
int launch_wide(float* C, const float* A, const float* W, int M, int N, int K, long long lda, long long ldc, int sms, cudaStream_t st) {
    if ((KG == 1) != (K <= ONE_CHAIN)) return OE_ERR_UNSUPPORTED;
    const int tiles_m = (M + WT - 1) / WT;
    const long long ctas = (long long)tiles_m * ((N + WT - 1) / WT) * KG;
    // An SM for each CTA where there are enough: a kernel that starts while the one before it still holds the SMs otherwise gets two
    // places each on those that are free first, and two CTAs take turns there while other SMs idle (in a row of such products, 1,111 x
    // 2,048 x 512, 144 CTAs: 97 us, so 58; 130 x 8,192 x 512, 128: 97 and 58).  Clusters of four and eight would not all fit so.
    const size_t bytes = KG == 1 && ctas <= sms ? WideShape::ALONE : WideShape::BYTES;
    cudaError_t e = cudaFuncSetAttribute(gemm_wide_kernel<KG, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WideShape::ALONE);
    if (e != cudaSuccess) return (int)e;
    if (tiles_m > 65535 || ctas > 0x7fffffffll) return OE_ERR_UNSUPPORTED;
    if (KG == 1) return oe_launch(gemm_wide_kernel<KG, MODE>, dim3((unsigned)ctas), dim3(256), bytes, st, C, A, W, M, N, K, lda, ldc, tiles_m);
    return oe_launch_cluster(gemm_wide_kernel<KG, MODE>, KG, dim3((unsigned)ctas), dim3(256), bytes, st, C, A, W, M, N, K, lda, ldc, tiles_m);
}

constexpr int ROWS_MAX_M = 32;

// The kernel for a product (1 few rows, 2 tiles of 64, 3 tiles of 128, 5, 6 tiles of 128 whose classes four, eight CTAs share).
int f32_kind(int M, int N, int K, int sms) {
    const long long t128 = (long long)((M + 127) / 128) * ((N + 127) / 128), t64 = (long long)((M + 63) / 64) * ((N + 63) / 64);
    // Up to 64 rows a tile of 128 is half empty.  A weight of few rows is streamed (64 x 2,048 x 8,192: 174 us, 191 by tiles of
    // 128, 297 by tiles of 64; 40 x 3,072 x 3,072: 70, 79, 113; 48 x 2,048 x 2,048: 41, 56, 80); beyond that, while there are two
    // CTAs an SM for eight shares of every tile, tiles of 128 (64 x 3,072 x 3,072: 137 us streamed by the kernel before, 80, 119); a
    // weight of more rows has tiles of 64 enough for all SMs (64 x 16,384 x 2,048: 156 us, 197 by tiles of 128; 32 rows 154
    // streamed, 150).
    if (M <= ROWS_MAX_M || (M <= 64 && M * t128 <= 1024)) return 1;
    // A single chain cannot be shared out, and a tile of 128 takes as long for a few columns as for all: small products stream, up to
    // two tiles of 8 x 16 for each of two CTAs an SM (1,111 x 64 x 64: 6.1 us, 9.9 by tiles of 128; 468 x 64 x 512 16 and 55; 130 x 512 x
    // 64 6.0 and 9.4; beyond, 1,111 x 128 x 64 10.3 and 9.6, 130 x 2,048 x 64 18 and 9.7)
    if (K <= ONE_CHAIN) return M > 64 && (long long)((M + 7) / 8) * ((N + 15) / 16) <= 4 * sms ? 1 : 3;
    if (M <= 64) return 8 * t128 <= 2 * sms ? 6 : 2;
    // From 65 rows on tiles of 64 are faster only where they are one round of CTAs and eight shares of every tile of 128 are more
    // (clusters of eight leave a few SMs of each group of them out: up to 8/9 of two CTAs an SM), or two rounds and four shares are
    // more (192 x 3,072 x 3,072: 113 us, 148 by tiles of 128; 1,111 x 512 x 1,024 40 and 45; 160 x 6,144 x 2,048 149 and 155; else 256 x
    // 2,048 x 2,048 76 and 57, 300 x 3,072 x 2,048 149 and 127).
    if ((t64 <= sms && 9 * t128 > 2 * sms) || (t64 <= 2 * sms && 4 * t128 > 2 * sms)) return 2;
    // eight shares of a tile while four would not fill the SMs (192 x 4,096 x 4,096, 64 tiles: 211 us, 240 with four; 300 rows, 96
    // tiles: 301 and 301; 468 x 16,384 x 2,048: 769 and 734: a share's adding up costs what it costs)
    return 4 * t128 <= 2 * sms ? 6 : 5;
}

// kind: 0 by size, 4 the general kernel, else as f32_kind says (tests).
template <int MODE>
int launch_f32(float* C, const float* A, const float* W, int M, int N, int K, long long lda, long long ldc, int kind, cudaStream_t st) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return OE_ERR_UNSUPPORTED;
    const bool aligned = K % 4 == 0 && lda % 4 == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0;
    if (!aligned || kind == 4) return kind == 0 || kind == 4 ? launch<float, float, MODE>(C, A, W, M, N, K, lda, ldc, st) : OE_ERR_UNSUPPORTED;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (kind == 0) kind = f32_kind(M, N, K, sms);
    if (kind == 3) {
        if (K <= ONE_CHAIN) return launch_wide<1, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
        kind = 4ll * ((M + 127) / 128) * ((N + 127) / 128) <= 2 * sms ? 6 : 5;
    }
    if (kind == 5) return launch_wide<4, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
    if (kind == 6) return launch_wide<8, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
    if (kind == 2) return launch_tile<64, 64, 4, MODE>(C, A, W, M, N, K, lda, ldc, st);
    if (M == 1) return launch_rows_for<1, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
    if (M == 2) return launch_rows_for<2, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
    if (M <= 4) return launch_rows_for<4, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
    return launch_rows_for<8, MODE>(C, A, W, M, N, K, lda, ldc, sms, st);
}

}  // namespace

extern "C" {
// out_kind: 0 = same type as the inputs, 1 = float32 store, 2 = float32 accumulate (C += A.W^T)
int oe_gemm_simple_f32(void* C, const float* A, const float* W, int M, int N, int K, long long lda,
                       long long ldc, int out_kind, cudaStream_t st) {
    if (out_kind == 2) return launch_f32<1>((float*)C, A, W, M, N, K, lda, ldc, 0, st);
    return launch_f32<0>((float*)C, A, W, M, N, K, lda, ldc, 0, st);
}
// Which kernel takes a product of aligned operands on a device of `sms` SMs.
int oe_gemm_simple_f32_kind(int M, int N, int K, int sms) { return f32_kind(M, N, K, sms); }
// The same through one kernel, whatever the size: they give the same bits.
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
