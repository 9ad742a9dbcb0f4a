// The decaying time mixing over prompts, in chunks of 32 tokens (bfloat16 path; csrc/recurrent.cu walks token by token):
//   o = (S + diag(u) k v^T)^T r;  S <- diag(w) S + k v^T,  w = exp(-exp(z + w0))     S [d, d] per head and sequence, float32
// With S0 the state before a chunk and P_st = w_(s+1) * ... * w_(t-1) per channel (empty: one), the chunk's outputs are
//   o_t = (r_t P_0t)^T S0 + sum_(s<t) (r_t P_st . k_s) v_s + (r_t u . k_t) v_t,   S = P_0(n+1) S0 + sum_s (P_s(n+1) k_s) v_s^T,
// all decays as products, never as quotients: a channel may forget everything within a chunk.
//
// Token by token the chain of dependent steps is the time: 1,111 tokens, 32 heads of 64 x 64, 379 us there, 150 us here (3 us a
// chunk, still a chain); 8 heads of 128 x 128 553 and 157 us.  Errors against 64 bits as the walk's (5.2e-7 both).  Here
// decay_chunk_prepare_kernel makes a chunk's decayed vectors and its 32 x 32 scores for all chunks and heads side by side, and
// decay_chunk_scan_kernel carries 16 columns of a head's state, in registers, from chunk to chunk.
#include "scan_chunks.cuh"

namespace {

// What the scan reads of a chunk and head: [Kd: CH d | Qd: CH d | V: CH d | M: CH CH | the chunk's decays: d].
__host__ __device__ __forceinline__ size_t block_floats(int d) { return (size_t)CH * (3 * d + CH) + d; }

template <int D>
__global__ void __launch_bounds__(256)
decay_chunk_prepare_kernel(float* blocks, const float* r, const float* k, const float* v, const float* z, long long stride,
                           const float* __restrict__ u, const float* __restrict__ w0, const int* __restrict__ seq_slot,
                           const int* __restrict__ cu_q, int n_seqs, int H) {
    constexpr int LD = D + 4, PER = D / 32;
    extern __shared__ __align__(16) float smem[];
    float *Rs = smem, *Ks = Rs + CH * LD, *Ws = Ks + CH * LD;          // [CH][LD] each
    const int h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    int chunk = blockIdx.x, b = 0;
    for (; b < n_seqs; b++) {
        const int n = chunks_of(cu_q, seq_slot, b);
        if (chunk < n) break;
        chunk -= n;
    }
    pdl_wait();
    pdl_launch_dependents();
    if (b == n_seqs) return;
    const int row0 = cu_q[b] + chunk * CH, n = min(CH, cu_q[b + 1] - row0);
    float* out = blocks + ((size_t)blockIdx.x * H + h) * block_floats(D);
    float *oK = out, *oQ = oK + CH * D, *oV = oQ + CH * D, *oM = oV + CH * D, *oW = oM + CH * CH;
    for (int e = tid; e < CH * D; e += 256) {
        const int t = e / D, i = e % D;
        const size_t at = (size_t)(row0 + t) * stride + (size_t)h * D + i;
        const bool on = t < n;
        Rs[t * LD + i] = on ? r[at] : 0.f;
        Ks[t * LD + i] = on ? k[at] : 0.f;
        Ws[t * LD + i] = on ? expf(-expf(z[at] + w0[(size_t)h * D + i])) : 1.f;
        oV[e] = on ? v[at] : 0.f;
    }
    __syncthreads();
    if (tid < D) {                                     // a channel a thread: the decays from the chunk's start on, and to its end
        float p = 1.f;
        for (int t = 0; t < CH; t++) { oQ[t * D + tid] = Rs[t * LD + tid] * p; p *= Ws[t * LD + tid]; }
        oW[tid] = p;
        p = 1.f;
        for (int t = CH - 1; t >= 0; t--) { oK[t * D + tid] = Ks[t * LD + tid] * p; p *= Ws[t * LD + tid]; }
    }
    for (int s = warp; s < CH; s += 8) {               // a key a warp: its scores with the queries behind it
        float kp[PER], uu = 0.f;
#pragma unroll
        for (int q = 0; q < PER; q++) {
            const int i = lane + 32 * q;
            kp[q] = Ks[s * LD + i];
            uu = fmaf(Rs[s * LD + i], u[(size_t)h * D + i] * kp[q], uu);
        }
        uu = warp_sum(uu);
        for (int t = lane; t < s; t += 32) oM[t * CH + s] = 0.f;
        if (lane == 0) oM[s * CH + s] = uu;
#pragma unroll 4
        for (int t = s + 1; t < CH; t++) {
            float a = 0.f;
#pragma unroll
            for (int q = 0; q < PER; q++) {
                a = fmaf(Rs[t * LD + lane + 32 * q], kp[q], a);
                kp[q] *= Ws[t * LD + lane + 32 * q];
            }
            a = warp_sum(a);
            if (lane == 0) oM[t * CH + s] = a;
        }
    }
}

// grid (H * d / 16, sequences).  Thread (rg, j): rows rg ROWS .. of column j.  What a chunk's block holds comes by
// asynchronous copies while the chunk before it is worked on.
template <int ROWS>
__global__ void __launch_bounds__(COLS * GROUPS)
decay_chunk_scan_kernel(float* o, float* state, const float* blocks, const int* __restrict__ seq_slot, const int* __restrict__ cu_q, int H) {
    constexpr int D = ROWS * GROUPS, WARPS = COLS * GROUPS / 32;
    constexpr int STAGE = CH * 2 * D + CH * COLS + CH * CH + D;
    extern __shared__ __align__(16) float smem[];
    float* part = smem + 2 * STAGE;                    // [WARPS][CH][COLS]
    const int tiles = D / COLS, h = blockIdx.x / tiles, col0 = blockIdx.x % tiles * COLS, b = blockIdx.y;
    const int tid = threadIdx.x, j = tid % COLS, rg = tid / COLS, warp = tid >> 5, lane = tid & 31;
    int first = 0;
    for (int q = 0; q < b; q++) first += chunks_of(cu_q, seq_slot, q);
    const int chunks = chunks_of(cu_q, seq_slot, b), slot = seq_slot[b];
    pdl_wait();
    pdl_launch_dependents();
    if (chunks == 0) return;
    const int row0 = cu_q[b], n_all = cu_q[b + 1] - row0;
    float* S = state + ((size_t)slot * H + h) * D * D + col0 + j;
    float s[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; r++) s[r] = S[(size_t)(rg * ROWS + r) * D];
    auto load = [&](int chunk, float* st) {
        const float* src = blocks + ((size_t)(first + chunk) * H + h) * block_floats(D);
        for (int e = tid; e < CH * 2 * D / 4; e += COLS * GROUPS) cp_async16(st + 4 * e, src + 4 * e);
        float* d = st + CH * 2 * D;
        const float* v = src + CH * 2 * D + col0;
        for (int e = tid; e < CH * COLS / 4; e += COLS * GROUPS) cp_async16(d + 4 * e, v + (size_t)(e / (COLS / 4)) * D + e % (COLS / 4) * 4);
        d += CH * COLS;
        const float* m = src + CH * 3 * D;
        for (int e = tid; e < (CH * CH + D) / 4; e += COLS * GROUPS) cp_async16(d + 4 * e, m + 4 * e);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load(0, smem);
    for (int chunk = 0; chunk < chunks; chunk++) {
        const float* st = smem + (chunk & 1) * STAGE;
        if (chunk + 1 < chunks) { load(chunk + 1, smem + ((chunk + 1) & 1) * STAGE); asm volatile("cp.async.wait_group 1;" ::: "memory"); }
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const float *Kd = st, *Qd = Kd + CH * D, *V = Qd + CH * D, *M = V + CH * COLS, *Wd = M + CH * CH;
        // Qd S0: this thread's rows, then the warp's two row groups, then the warps (eight rows' loads before the first store into
        // `part`: the compiler moves none across one)
        constexpr int AT_ONCE = 8;
#pragma unroll 1
        for (int t0 = 0; t0 < CH; t0 += AT_ONCE) {
            float q[AT_ONCE];
#pragma unroll
            for (int t = 0; t < AT_ONCE; t++) {
                q[t] = 0.f;
#pragma unroll
                for (int r = 0; r < ROWS; r += 4) {
                    const float4 c = *(const float4*)(Qd + (t0 + t) * D + rg * ROWS + r);
                    q[t] = fmaf(c.w, s[r + 3], fmaf(c.z, s[r + 2], fmaf(c.y, s[r + 1], fmaf(c.x, s[r], q[t]))));
                }
            }
#pragma unroll
            for (int t = 0; t < AT_ONCE; t++) q[t] += __shfl_xor_sync(0xffffffffu, q[t], 16);
#pragma unroll
            for (int t = 0; t < AT_ONCE; t++) if (lane < 16) part[(warp * CH + t0 + t) * COLS + lane] = q[t];
        }
        // the state at the chunk's end does not wait for the outputs
#pragma unroll
        for (int r = 0; r < ROWS; r++) s[r] *= Wd[rg * ROWS + r];
#pragma unroll 8
        for (int t = 0; t < CH; t++) {
            const float v = V[t * COLS + j];
#pragma unroll
            for (int r = 0; r < ROWS; r += 4) {
                const float4 k = *(const float4*)(Kd + t * D + rg * ROWS + r);
                s[r] = fmaf(k.x, v, s[r]); s[r + 1] = fmaf(k.y, v, s[r + 1]); s[r + 2] = fmaf(k.z, v, s[r + 2]); s[r + 3] = fmaf(k.w, v, s[r + 3]);
            }
        }
        __syncthreads();
#pragma unroll
        for (int e = 0; e < CH / GROUPS; e++) {        // (t, j) = (rg + 16 e, j)
            const int t = rg + GROUPS * e;
            float a = 0.f;
#pragma unroll
            for (int p = 0; p < WARPS; p++) a += part[(p * CH + t) * COLS + j];
#pragma unroll 8
            for (int q = 0; q < CH; q++) {             // a later token's value must not touch this one, were it infinite
                const float m = fmaf(M[t * CH + q], V[q * COLS + j], a);
                a = q <= t ? m : a;
            }
            if (chunk * CH + t < n_all) o[(size_t)(row0 + chunk * CH + t) * H * D + (size_t)h * D + col0 + j] = a;
        }
        __syncthreads();                               // the stage and part are free
    }
#pragma unroll
    for (int r = 0; r < ROWS; r++) S[(size_t)(rg * ROWS + r) * D] = s[r];
}

template <int D>
int launch(float* o, float* state, float* blocks, const float* r, const float* k, const float* v, const float* z, long long stride, const float* u,
           const float* w0, const int* seq_slot, const int* cu_q, int n_tokens, int n_seqs, int H, cudaStream_t st) {
    constexpr int ROWS = D / GROUPS;
    const size_t b1 = (size_t)3 * CH * (D + 4) * 4;
    const size_t b2 = (size_t)(2 * (CH * 2 * D + CH * COLS + CH * CH + D) + COLS * GROUPS / 32 * CH * COLS) * 4;
    cudaError_t e = cudaFuncSetAttribute(decay_chunk_prepare_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(decay_chunk_scan_kernel<ROWS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)b2);
    if (e != cudaSuccess) return (int)e;
    int rc = oe_launch(decay_chunk_prepare_kernel<D>, dim3(n_tokens / CH + n_seqs, H), dim3(256), b1, st, blocks, r, k, v, z, stride, u, w0, seq_slot,
                       cu_q, n_seqs, H);
    if (rc) return rc;
    return oe_launch(decay_chunk_scan_kernel<ROWS>, dim3(H * (D / COLS), n_seqs), dim3(COLS * GROUPS), b2, st, o, state, blocks, seq_slot, cu_q, H);
}

}  // namespace

extern "C" {

int oe_decay_chunks_supported(int d) { return d == 64 || d == 128; }

// blocks: scratch of at least (n_tokens / 32 + n_seqs) H (32 (3 d + 32) + d) floats, 16-byte aligned.  r, k, v, z: rows of
// `stride` floats, [T, H d].  d 64 or 128.
int oe_decay_chunks(float* o, float* state, float* blocks, const float* r, const float* k, const float* v, const float* z, long long stride,
                    const float* u, const float* w0, const int* seq_slot, const int* cu_q, int n_tokens, int n_seqs, int H, int d, cudaStream_t st) {
    if (n_seqs <= 0 || n_tokens <= 0) return 0;
    if (!oe_decay_chunks_supported(d) || H < 1 || H > 65535 || n_seqs > 65535 || ((uintptr_t)blocks & 15)) return OE_ERR_UNSUPPORTED;
    if (d == 64) return launch<64>(o, state, blocks, r, k, v, z, stride, u, w0, seq_slot, cu_q, n_tokens, n_seqs, H, st);
    return launch<128>(o, state, blocks, r, k, v, z, stride, u, w0, seq_slot, cu_q, n_tokens, n_seqs, H, st);
}

}  // extern "C"
