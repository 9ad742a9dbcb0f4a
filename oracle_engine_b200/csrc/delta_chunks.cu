// The gated delta rule over prompts, in chunks of 32 tokens (bfloat16 path; csrc/recurrent.cu walks token by token):
//   S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q          S [dk, dv] per head and sequence, all float32
// With S0 the state before a chunk, R_ij = g_(j+1) ... g_i and G_i = g_1 ... g_i within it, the chunk's u solve
//   u_i + beta_i sum_(j<i) R_ij (k_i . k_j) u_j = beta_i (v_i - G_i S0^T k_i),   that is   U = Uv - W S0,
// where Uv and W are the solutions of the unit lower triangular system for the right sides beta V and beta G K: they do not
// depend on the state.  Then o_i = G_i S0^T q_i + sum_(j<=i) R_ij (q_i . k_j) u_j and S = G_n S0 + sum_j R_nj k_j u_j^T.
// (The form is that of Yang, Wang, Zhang, Shen, Kim, "Parallelizing Linear Transformers with the Delta Rule over Sequence
// Length", with a decay.)
//
// Token by token the chain of dependent steps was the time (1,111 tokens, 16 heads of 128 x 128: 414 us, 0.37 us a token,
// 64 CTAs of which a scheduler had one or two warps).  Here delta_chunk_solve_kernel does what does not depend on the state
// for all chunks and heads side by side, and delta_chunk_scan_kernel carries 16 columns of a head's state, in registers,
// from chunk to chunk: the chain has 32 times fewer links.  Products of decays are formed as such, without dividing.
#include "scan_chunks.cuh"

namespace {

// What the scan reads of a chunk and head, one block of floats: [W: CH dk | Kd: CH dk | Qg: CH dk | Uv: CH dv | M: CH CH | G: 4].
__host__ __device__ __forceinline__ size_t block_floats(int dk, int dv) { return (size_t)CH * (3 * dk + dv + CH) + 4; }

// Two blocks an SM where there are more blocks than SMs: with the 246 registers that the compiler would take, 560 blocks are four
// rounds: 62 us for 1,111 tokens, 48 so, although 240 bytes a thread are then stored to memory and loaded again.  Up to a
// block an SM that is only lost time (16 heads of 128 x 128, both kernels: 33 tokens 30.5 us, 24.0 with all registers, 200 51.4 and 44.5;
// 240 blocks 88 and 93).
template <int PER_SM>
__global__ void __launch_bounds__(256, PER_SM)
delta_chunk_solve_kernel(float* blocks, const float* qkv, const float* gb, const int* __restrict__ seq_slot, const int* __restrict__ cu_q,
                         int n_seqs, int G, int H, int dk, int dv) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float gs[CH], bs[CH], Gs[CH], R[CH][CH + 1];
    __shared__ __align__(16) float L[CH][CH + 4];
    const int h = blockIdx.y, g = h / (H / G), tid = threadIdx.x;
    int chunk = blockIdx.x, b = 0;
    for (; b < n_seqs; b++) {
        const int n = chunks_of(cu_q, seq_slot, b);
        if (chunk < n) break;
        chunk -= n;
    }
    pdl_wait();
    pdl_launch_dependents();
    if (b == n_seqs) return;
    const int row0 = cu_q[b] + chunk * CH, n = min(CH, cu_q[b + 1] - row0), C = 2 * G * dk + H * dv;
    const int ld = dk + 4;
    float* K = smem;                                   // [CH][ld]
    float* Q = K + CH * ld;
    float* out = blocks + ((size_t)blockIdx.x * H + h) * block_floats(dk, dv);
    float *oW = out, *oKd = oW + CH * dk, *oQg = oKd + CH * dk, *oUv = oQg + CH * dk, *oM = oUv + CH * dv;
    for (int e = tid; e < CH * dk / 4; e += 256) {
        const int i = e / (dk / 4), c = e % (dk / 4) * 4;
        const float* row = qkv + (size_t)(row0 + i) * C + g * dk + c;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        *(float4*)(Q + i * ld + c) = i < n ? *(const float4*)row : zero;
        *(float4*)(K + i * ld + c) = i < n ? *(const float4*)(row + G * dk) : zero;
    }
    if (tid < CH) {
        gs[tid] = tid < n ? gb[(size_t)(row0 + tid) * 2 * H + h] : 1.f;
        bs[tid] = tid < n ? gb[(size_t)(row0 + tid) * 2 * H + H + h] : 0.f;
    }
    __syncthreads();
    if (tid < CH) {                                    // column tid of R, down the rows
        float r = 1.f;
        for (int i = 0; i < CH; i++) {
            r = i <= tid ? 1.f : r * gs[i];
            R[i][tid] = i < tid ? 0.f : r;
        }
    } else if (tid == CH) {
        float r = 1.f;
        for (int i = 0; i < CH; i++) { r *= gs[i]; Gs[i] = r; }
    }
    __syncthreads();
    // k_i . k_j and q_i . k_j: a thread has rows i, i + 16 and columns j, j + 16
    {
        const int i = tid / 16, j = tid % 16;
        float kk[2][2] = {}, qk[2][2] = {};
        for (int c = 0; c < dk; c += 4) {
            float4 ki[2], qi[2], kj[2];
#pragma unroll
            for (int a = 0; a < 2; a++) {
                ki[a] = *(const float4*)(K + (i + 16 * a) * ld + c);
                qi[a] = *(const float4*)(Q + (i + 16 * a) * ld + c);
                kj[a] = *(const float4*)(K + (j + 16 * a) * ld + c);
            }
#pragma unroll
            for (int a = 0; a < 2; a++)
#pragma unroll
                for (int d = 0; d < 2; d++) {
                    kk[a][d] = fmaf(ki[a].w, kj[d].w, fmaf(ki[a].z, kj[d].z, fmaf(ki[a].y, kj[d].y, fmaf(ki[a].x, kj[d].x, kk[a][d]))));
                    qk[a][d] = fmaf(qi[a].w, kj[d].w, fmaf(qi[a].z, kj[d].z, fmaf(qi[a].y, kj[d].y, fmaf(qi[a].x, kj[d].x, qk[a][d]))));
                }
        }
#pragma unroll
        for (int a = 0; a < 2; a++)
#pragma unroll
            for (int d = 0; d < 2; d++) {
                const int ii = i + 16 * a, jj = j + 16 * d;
                L[ii][jj] = jj < ii ? bs[ii] * R[ii][jj] * kk[a][d] : 0.f;
                oM[ii * CH + jj] = jj <= ii ? R[ii][jj] * qk[a][d] : 0.f;
            }
    }
    __syncthreads();
    // a column a thread: columns of Uv (right side beta V), then of W (right side beta G K)
    for (int c = tid; c < dv + dk; c += 256) {
        float x[CH];
#pragma unroll
        for (int i = 0; i < CH; i++) {
            if (c < dv) x[i] = i < n ? bs[i] * qkv[(size_t)(row0 + i) * C + 2 * G * dk + (size_t)h * dv + c] : 0.f;
            else x[i] = bs[i] * Gs[i] * K[i * ld + c - dv];
        }
#pragma unroll
        for (int i = 1; i < CH; i++) {
            float a0 = 0.f, a1 = 0.f;
#pragma unroll
            for (int j = 0; j < i; j += 4) {           // a later token's value must not touch this one, were it infinite
                const float4 l = *(const float4*)&L[i][j];
                a0 = fmaf(l.x, x[j], a0);
                if (j + 1 < i) a1 = fmaf(l.y, x[j + 1], a1);
                if (j + 2 < i) a0 = fmaf(l.z, x[j + 2], a0);
                if (j + 3 < i) a1 = fmaf(l.w, x[j + 3], a1);
            }
            x[i] -= a0 + a1;
        }
        float* o = c < dv ? oUv + c : oW + c - dv;
        const int step = c < dv ? dv : dk;
#pragma unroll
        for (int i = 0; i < CH; i++) o[(size_t)i * step] = x[i];
    }
    for (int e = tid; e < CH * dk; e += 256) {
        const int i = e / dk, c = e % dk;
        oKd[e] = i < n ? R[n - 1][i] * K[i * ld + c] : 0.f;
        oQg[e] = Gs[i] * Q[i * ld + c];
    }
    if (tid == 0) oM[CH * CH] = Gs[n - 1];
}

// grid (H * dv / 16, sequences), DK threads.  A thread has four rows of four columns of the state: a row of W, Qg or Kd is read
// from shared memory once for four columns, and eight rows are asked for before the first sum is stored (with eight rows of one
// column a thread, and every row's loads behind the store before it, a chunk took 5.4 us; now 4.1).  What a chunk's block holds
// comes by asynchronous copies while the chunk before it is worked on.
template <int DK>
__global__ void __launch_bounds__(DK)
delta_chunk_scan_kernel(float* o, float* state, const float* blocks, const int* __restrict__ seq_slot, const int* __restrict__ cu_q, int H, int dv) {
    constexpr int WARPS = DK / 32;
    constexpr int MROW = CH + 4;                       // rows of M in a stage: eight lanes of eight rows meet in no bank
    constexpr int STAGE = CH * 3 * DK + CH * COLS + CH * MROW + 4;
    extern __shared__ __align__(16) float smem[];
    float* part = smem + 2 * STAGE;                    // [WARPS][CH][2][COLS]
    float* U = part + WARPS * 2 * CH * COLS;           // [CH][COLS]
    const int tiles = dv / COLS, h = blockIdx.x / tiles, col0 = blockIdx.x % tiles * COLS, b = blockIdx.y;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int cg = lane & 3, rg = warp * 8 + (lane >> 2);        // columns 4 cg .., rows 4 rg ..
    int first = 0;
    for (int q = 0; q < b; q++) first += chunks_of(cu_q, seq_slot, q);
    const int chunks = chunks_of(cu_q, seq_slot, b), slot = seq_slot[b];
    pdl_wait();
    pdl_launch_dependents();
    if (chunks == 0) return;
    const int row0 = cu_q[b], n_all = cu_q[b + 1] - row0;
    float* S = state + ((size_t)slot * H + h) * DK * dv + (size_t)4 * rg * dv + col0 + 4 * cg;
    float s[4][4];                                     // [row][column]
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) s[r][c] = S[(size_t)r * dv + c];
    auto load = [&](int chunk, float* st) {
        const float* src = blocks + ((size_t)(first + chunk) * H + h) * block_floats(DK, dv);
#pragma unroll 8
        for (int e = tid; e < CH * 3 * DK / 4; e += DK) cp_async16(st + 4 * e, src + 4 * e);
        float* d = st + CH * 3 * DK;
        const float* uv = src + CH * 3 * DK + col0;
        for (int e = tid; e < CH * COLS / 4; e += DK) cp_async16(d + 4 * e, uv + (size_t)(e / (COLS / 4)) * dv + e % (COLS / 4) * 4);
        d += CH * COLS;
        const float* m = src + CH * (3 * DK + dv);
        for (int e = tid; e < CH * CH / 4 + 1; e += DK) cp_async16(d + e / (CH / 4) * MROW + e % (CH / 4) * 4, m + 4 * e);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load(0, smem);
    for (int chunk = 0; chunk < chunks; chunk++) {
        const float* st = smem + (chunk & 1) * STAGE;
        if (chunk + 1 < chunks) { load(chunk + 1, smem + ((chunk + 1) & 1) * STAGE); asm volatile("cp.async.wait_group 1;" ::: "memory"); }
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        const float *W = st, *Kd = W + CH * DK, *Qg = Kd + CH * DK, *Uv = Qg + CH * DK, *M = Uv + CH * COLS;
        // W S0 and Qg S0: this thread's rows, then the warp's eight row groups (each exchange halves what a lane carries on: at the
        // end it has one value, of W for the lower half of the warp, of Qg for the upper), then the warps
        // (eight rows' loads before the first store into `part`: the compiler moves none across one)
        const bool up = lane & 16, high = lane & 8, odd = lane & 4;
        float* own = part + (warp * CH * 2 + (up ? 1 : 0)) * COLS + 4 * cg + (high ? 2 : 0) + (odd ? 1 : 0);
        constexpr int AT_ONCE = 8;
#pragma unroll 1
        for (int i0 = 0; i0 < CH; i0 += AT_ONCE) {
            float4 a[AT_ONCE], q[AT_ONCE];
            float y[AT_ONCE][4], sum[AT_ONCE];
#pragma unroll
            for (int i = 0; i < AT_ONCE; i++) {
                a[i] = *(const float4*)(W + (i0 + i) * DK + 4 * rg);
                q[i] = *(const float4*)(Qg + (i0 + i) * DK + 4 * rg);
            }
#pragma unroll
            for (int i = 0; i < AT_ONCE; i++) {
                float x[8];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    x[c] = fmaf(a[i].w, s[3][c], fmaf(a[i].z, s[2][c], fmaf(a[i].y, s[1][c], a[i].x * s[0][c])));
                    x[4 + c] = fmaf(q[i].w, s[3][c], fmaf(q[i].z, s[2][c], fmaf(q[i].y, s[1][c], q[i].x * s[0][c])));
                }
#pragma unroll
                for (int c = 0; c < 4; c++) y[i][c] = (up ? x[4 + c] : x[c]) + __shfl_xor_sync(0xffffffffu, up ? x[c] : x[4 + c], 16);
            }
#pragma unroll
            for (int i = 0; i < AT_ONCE; i++) {
                float z[2];
#pragma unroll
                for (int c = 0; c < 2; c++) z[c] = (high ? y[i][2 + c] : y[i][c]) + __shfl_xor_sync(0xffffffffu, high ? y[i][c] : y[i][2 + c], 8);
                sum[i] = (odd ? z[1] : z[0]) + __shfl_xor_sync(0xffffffffu, odd ? z[0] : z[1], 4);
            }
#pragma unroll
            for (int i = 0; i < AT_ONCE; i++) own[(i0 + i) * 2 * COLS] = sum[i];
        }
        __syncthreads();
        float4 qs[CH * 4 / DK];
#pragma unroll
        for (int e = 0; e < CH * 4 / DK; e++) {        // four columns of row i
            const int at = e * DK + tid, i = at / 4, c = at % 4 * 4;
            float4 w = make_float4(0.f, 0.f, 0.f, 0.f), q = w;
#pragma unroll
            for (int p = 0; p < WARPS; p++) {
                const float4 a = *(const float4*)(part + (p * CH + i) * 2 * COLS + c), d = *(const float4*)(part + ((p * CH + i) * 2 + 1) * COLS + c);
                w.x += a.x; w.y += a.y; w.z += a.z; w.w += a.w;
                q.x += d.x; q.y += d.y; q.z += d.z; q.w += d.w;
            }
            const float4 v = *(const float4*)(Uv + i * COLS + c);
            *(float4*)(U + i * COLS + c) = make_float4(v.x - w.x, v.y - w.y, v.z - w.z, v.w - w.w);
            qs[e] = q;
        }
        __syncthreads();
        const float decay = M[CH * MROW];
#pragma unroll
        for (int r = 0; r < 4; r++)
#pragma unroll
            for (int c = 0; c < 4; c++) s[r][c] *= decay;
#pragma unroll 8
        for (int i = 0; i < CH; i++) {
            const float4 u = *(const float4*)(U + i * COLS + 4 * cg), k = *(const float4*)(Kd + i * DK + 4 * rg);
            const float kr[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
            for (int r = 0; r < 4; r++) {
                s[r][0] = fmaf(kr[r], u.x, s[r][0]); s[r][1] = fmaf(kr[r], u.y, s[r][1]);
                s[r][2] = fmaf(kr[r], u.z, s[r][2]); s[r][3] = fmaf(kr[r], u.w, s[r][3]);
            }
        }
#pragma unroll
        for (int e = 0; e < CH * 4 / DK; e++) {
            const int at = e * DK + tid, i = at / 4, c = at % 4 * 4, most = (e * DK + (tid | 31)) / 4;       // the warp's last row
            float4 a = qs[e];
#pragma unroll 8
            for (int l = 0; l <= most; l++) {          // a later token's value must not touch this one, were it infinite
                const float m = M[i * MROW + l];
                const float4 u = *(const float4*)(U + l * COLS + c);
                const float4 n = make_float4(fmaf(m, u.x, a.x), fmaf(m, u.y, a.y), fmaf(m, u.z, a.z), fmaf(m, u.w, a.w));
                a = l <= i ? n : a;
            }
            const int t = chunk * CH + i;
            if (t < n_all) {
                float* to = o + (size_t)(row0 + t) * H * dv + (size_t)h * dv + col0 + c;
                to[0] = a.x; to[1] = a.y; to[2] = a.z; to[3] = a.w;
            }
        }
        __syncthreads();                               // the stage, part and U are free
    }
#pragma unroll
    for (int r = 0; r < 4; r++)
#pragma unroll
        for (int c = 0; c < 4; c++) S[(size_t)r * dv + c] = s[r][c];
}

constexpr size_t SM_SHARED = 227 * 1024;              // what the blocks resident on an SM share, each with 1 KB of the system's on top

template <int DK>
int launch_scan(float* o, float* state, const float* blocks, const int* seq_slot, const int* cu_q, int n_seqs, int H, int dv, int sms, cudaStream_t st) {
    size_t bytes = (size_t)(2 * (CH * 3 * DK + CH * COLS + CH * (CH + 4) + 4) + DK / 32 * 2 * CH * COLS + CH * COLS) * 4;
    // No more blocks an SM than one round of them needs: this kernel starts while the one before it drains, and otherwise gets three
    // places each on the SMs that are free first while others stay empty (heads of 64: 32 of 64 x 64, 1,111 tokens, both kernels 297 -> 241
    // us, 4,000 1,091 -> 883; 16 of 64 x 128 249 -> 189).
    const size_t ctas = (size_t)H * (dv / COLS) * n_seqs, share = SM_SHARED / ((ctas + sms - 1) / sms);
    if (share > bytes + 1024) bytes = (share - 1024) / 16 * 16;
    cudaError_t e = cudaFuncSetAttribute(delta_chunk_scan_kernel<DK>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    return oe_launch(delta_chunk_scan_kernel<DK>, dim3(H * (dv / COLS), n_seqs), dim3(DK), bytes, st, o, state, blocks, seq_slot, cu_q, H, dv);
}

}  // namespace

extern "C" {

int oe_delta_chunks_supported(int G, int H, int dk, int dv) {
    return G >= 1 && H >= 1 && H % G == 0 && (dk == 64 || dk == 128) && dv >= COLS && dv % COLS == 0 && dv <= 4096;
}

// blocks: scratch of at least (n_tokens / 32 + n_seqs) H (32 (3 dk + dv + 32) + 4) floats, 16-byte aligned.
int oe_delta_chunks(float* o, float* state, float* blocks, const float* qkv, const float* gb, const int* seq_slot, const int* cu_q, int n_tokens,
                    int n_seqs, int G, int H, int dk, int dv, cudaStream_t st) {
    if (n_seqs <= 0 || n_tokens <= 0) return 0;
    if (!oe_delta_chunks_supported(G, H, dk, dv) || n_seqs > 65535 || H > 65535 || (((uintptr_t)qkv | (uintptr_t)blocks) & 15)) return OE_ERR_UNSUPPORTED;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const dim3 grid(n_tokens / CH + n_seqs, H);
    const auto solve = (long long)(n_tokens / CH) * H <= sms ? delta_chunk_solve_kernel<1> : delta_chunk_solve_kernel<2>;
    const size_t bytes = (size_t)2 * CH * (dk + 4) * 4;
    cudaError_t e = cudaFuncSetAttribute(solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return (int)e;
    int rc = oe_launch(solve, grid, dim3(256), bytes, st, blocks, qkv, gb, seq_slot, cu_q, n_seqs, G, H, dk, dv);
    if (rc) return rc;
    if (dk == 64) return launch_scan<64>(o, state, blocks, seq_slot, cu_q, n_seqs, H, dv, sms, st);
    return launch_scan<128>(o, state, blocks, seq_slot, cu_q, n_seqs, H, dv, sms, st);
}

}  // extern "C"
