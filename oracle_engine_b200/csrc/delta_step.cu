// One token of every sequence of a decode step through a gated delta rule (csrc/recurrent.cu has the mixer for steps of any
// tokens), from the input projection's row to the gated read-out, in one launch:
//   causal convolution per channel + silu (q, k, v), q and k unit vectors, g = exp(-exp(A) softplus(a + dt)), beta = sigmoid(b)
//   S <- g S;  u = beta (v - S^T k);  S <- S + k u^T;  o = S^T q;  y = o / sqrt(mean(o^2) + eps) * w * silu(gate)
// and the convolution's kept rows moved on by one.
//
// A step of one sequence is bound by its launches and the round trips to memory in each (16 heads of 128 x 128: 4 launches
// of 2 to 4 us for 1 MB of state): here a CTA has one head of one sequence, has its state and the kept rows brought into the
// L2 before it waits for the projection, and keeps the state in registers, four columns and up to 16 rows a thread.  The heads that share
// a key head are a cluster: the last one to have read the kept rows of q and k lets the first one overwrite them.
#include "common.cuh"

namespace {

constexpr int THREADS = 256, MAX_ROWS = 16, MAX_KEPT = 7, MAX_CHANNELS = 3;     // rows a thread, kept rows, channels a thread

__device__ __forceinline__ void prefetch_l2(const float* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ float silu_f(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return z > 20.f ? z : log1pf(expf(z)); }

__global__ void __launch_bounds__(THREADS)
delta_step_kernel(bf16* y, float* state, float* conv_state, const float* proj, int P, const float* __restrict__ conv_w, int taps,
                  const float* __restrict__ A_log, const float* __restrict__ dt_bias, const float* __restrict__ norm_w,
                  const int* __restrict__ seq_slot, const int* __restrict__ cu_q, int G, int H, int dk, int dv, float q_scale, float eps) {
    extern __shared__ __align__(16) float smem[];
    __shared__ float red[32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int h = blockIdx.x, b = blockIdx.y, g = h / (H / G), rank = h % (H / G);
    const int slot = seq_slot[b], t = cu_q[b];
    if (slot < 0 || cu_q[b + 1] <= t) { pdl_launch_dependents(); pdl_wait(); return; }      // the whole cluster
    const int quads = dv / 4, groups = THREADS / quads;
    const int cq = tid % quads, rg = tid / quads;     // columns 4 cq ..; rows rg, rg + groups, ...
    const bool works = rg < groups;
    float* vec = smem;                                // [q: dk | k: dk | v: dv]
    float* part = vec + 2 * dk + dv;                  // [groups][dv]
    float* S = state + ((size_t)slot * H + h) * dk * dv;
    const int C = 2 * G * dk + H * dv, channels = 2 * dk + dv;
    auto channel = [&](int c) { return c < dk ? g * dk + c : c < 2 * dk ? G * dk + g * dk + (c - dk) : 2 * G * dk + h * dv + (c - 2 * dk); };
    float* kept = conv_state + (size_t)slot * (taps - 1) * C;
    // An earlier kernel of the stream may still write both (a slot's reset, this kernel a token earlier): they are read behind
    // the wait, and before it only asked into the L2, 128 bytes at a time.  (Reading them before it saved 0.4 us a layer: six of
    // eight layers of width 2,048, one sequence, 393 and 396 us a decode step.)
    for (int i = tid; i < dk * dv / 32; i += THREADS) prefetch_l2(S + 32 * i);
    if (tid % 32 == 0)
        for (int c = tid; c < channels; c += THREADS)
            for (int j = 0; j < taps - 1; j++) prefetch_l2(kept + (size_t)j * C + channel(c));
    // what no kernel writes: read before the wait, since it has left the L2 since the step before
    float tap[MAX_CHANNELS][MAX_KEPT + 1];
#pragma unroll
    for (int e = 0; e < MAX_CHANNELS; e++) {
        const int c = tid + e * THREADS;
#pragma unroll
        for (int j = 0; j <= MAX_KEPT; j++) tap[e][j] = c < channels && j < taps ? conv_w[(size_t)channel(c) * taps + j] : 0.f;
    }
    const float a_log = A_log[h], dt = dt_bias[h], out_w = tid < dv ? norm_w[tid] : 0.f;
    pdl_wait();
    pdl_launch_dependents();
    float4 s[MAX_ROWS];
#pragma unroll
    for (int i = 0; i < MAX_ROWS; i++) {
        const int r = rg + groups * i;
        s[i] = works && r < dk ? *(const float4*)(S + (size_t)r * dv + 4 * cq) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float old[MAX_CHANNELS][MAX_KEPT];
#pragma unroll
    for (int e = 0; e < MAX_CHANNELS; e++) {
        const int c = tid + e * THREADS;
#pragma unroll
        for (int j = 0; j < MAX_KEPT; j++) old[e][j] = c < channels && j < taps - 1 ? kept[(size_t)j * C + channel(c)] : 0.f;
    }
    const float* row = proj + (size_t)t * P;
    const float beta = 1.f / (1.f + expf(-row[C + H * dv + h]));
    const float decay = expf(-expf(a_log) * softplus_f(row[C + H * dv + H + h] + dt));
    const float gate = tid < dv ? row[C + (size_t)h * dv + tid] : 0.f;
    float now[MAX_CHANNELS];
#pragma unroll
    for (int e = 0; e < MAX_CHANNELS; e++) {
        const int c = tid + e * THREADS;
        if (c >= channels) continue;
        const int ch = channel(c);
        now[e] = row[ch];
        float acc = 0.f;
#pragma unroll
        for (int j = 0; j < MAX_KEPT; j++) if (j < taps - 1) acc = fmaf(tap[e][j], old[e][j], acc);
        float last = 0.f;
#pragma unroll
        for (int j = 0; j <= MAX_KEPT; j++) last = j == taps - 1 ? tap[e][j] : last;
        vec[c] = silu_f(fmaf(last, now[e], acc));
    }
    // every CTA of the cluster has read the kept rows of q and k
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    __syncthreads();
    if (warp < 2) {                                   // the lengths of q and k
        float ss = 0.f;
        for (int d = lane; d < dk; d += 32) ss = fmaf(vec[warp * dk + d], vec[warp * dk + d], ss);
        ss = warp_sum(ss);
        if (lane == 0) red[warp] = 1.f / sqrtf(ss + 1e-6f) * (warp == 0 ? q_scale : 1.f);
    }
    __syncthreads();
    const float qs = red[0], ks = red[1];
    float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < MAX_ROWS; i++) {
        const int r = rg + groups * i;
        const float k = r < dk ? vec[dk + r] * ks : 0.f;
        d.x = fmaf(k, s[i].x, d.x); d.y = fmaf(k, s[i].y, d.y); d.z = fmaf(k, s[i].z, d.z); d.w = fmaf(k, s[i].w, d.w);
    }
    if (works) *(float4*)(part + rg * dv + 4 * cq) = d;
    __syncthreads();
    float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = 0; q < groups; q++) {
        const float4 p = *(const float4*)(part + q * dv + 4 * cq);
        u.x += p.x; u.y += p.y; u.z += p.z; u.w += p.w;
    }
    const float4 v = *(const float4*)(vec + 2 * dk + 4 * cq);
    u.x = beta * (v.x - decay * u.x); u.y = beta * (v.y - decay * u.y); u.z = beta * (v.z - decay * u.z); u.w = beta * (v.w - decay * u.w);
    __syncthreads();
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < MAX_ROWS; i++) {
        const int r = rg + groups * i;
        if (!works || r >= dk) continue;
        const float k = vec[dk + r] * ks, q = vec[r] * qs;
        s[i].x = fmaf(k, u.x, decay * s[i].x); s[i].y = fmaf(k, u.y, decay * s[i].y);
        s[i].z = fmaf(k, u.z, decay * s[i].z); s[i].w = fmaf(k, u.w, decay * s[i].w);
        o.x = fmaf(q, s[i].x, o.x); o.y = fmaf(q, s[i].y, o.y); o.z = fmaf(q, s[i].z, o.z); o.w = fmaf(q, s[i].w, o.w);
        *(float4*)(S + (size_t)r * dv + 4 * cq) = s[i];
    }
    if (works) *(float4*)(part + rg * dv + 4 * cq) = o;
    __syncthreads();
    float out = 0.f;
    if (tid < dv) for (int q = 0; q < groups; q++) out += part[q * dv + tid];
    const float ss = block_sum(out * out, red);
    const float scale = 1.f / sqrtf(ss / (float)dv + eps);
    if (tid < dv) y[((size_t)t * H + h) * dv + tid] = __float2bfloat16_rn(out * scale * out_w * silu_f(gate));
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
#pragma unroll
    for (int e = 0; e < MAX_CHANNELS; e++) {
        const int c = tid + e * THREADS;
        if (c >= channels || (c < 2 * dk && rank != 0)) continue;
#pragma unroll
        for (int j = 0; j < MAX_KEPT; j++)
            if (j < taps - 1) kept[(size_t)j * C + channel(c)] = j + 1 < taps - 1 ? old[e][j + 1 < MAX_KEPT ? j + 1 : j] : now[e];
    }
}

}  // namespace

extern "C" {

// 1 if the kernel takes these sizes.
int oe_delta_step_supported(int G, int H, int dk, int dv, int taps) {
    if (G < 1 || H < 1 || H % G || H / G > 8 || dv < 4 || dv % 4 || dv > 256 || dk < 1 || taps < 1 || taps - 1 > MAX_KEPT) return 0;
    return dk <= MAX_ROWS * (THREADS / (dv / 4)) && 2 * dk + dv <= MAX_CHANNELS * THREADS && (2 * dk) % 4 == 0;
}

// Every sequence b with a slot has one token, row cu_q[b] of proj [T, P] = [q | k | v | gate | beta | a] and of y [T, H dv].
int oe_delta_step(bf16* y, float* state, float* conv_state, const float* proj, int P, const float* conv_w, int taps, const float* A_log,
                  const float* dt_bias, const float* norm_w, const int* seq_slot, const int* cu_q, int n_seqs, int G, int H, int dk, int dv,
                  float q_scale, float eps, cudaStream_t st) {
    if (n_seqs <= 0) return 0;
    if (!oe_delta_step_supported(G, H, dk, dv, taps) || n_seqs > 65535 || ((uintptr_t)state & 15)) return OE_ERR_UNSUPPORTED;
    const size_t smem = (size_t)(2 * dk + dv + THREADS / (dv / 4) * dv) * sizeof(float);
    return oe_launch_cluster(delta_step_kernel, (unsigned)(H / G), dim3(H, n_seqs), dim3(THREADS), smem, st, y, state, conv_state, proj, P, conv_w,
                             taps, A_log, dt_bias, norm_w, seq_slot, cu_q, G, H, dk, dv, q_scale, eps);
}

}  // extern "C"
