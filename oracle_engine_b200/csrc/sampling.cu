// Token selection on the device: first-maximum argmax, and the reference's sampling
// chain  repeat penalty -> temperature -> softmax -> top-k -> top-p -> draw
// (core/sampler.cpp:15-27, 35-39, 48-86, 91-97), one block or one cluster of blocks per row of float32 logits.
//
// Differences from the reference, on purpose:
//  * the draw is one uniform per (sequence, draw number) from a counter-based generator
//    kept in the per-sequence state (the reference seeds std::mt19937 from the clock,
//    core/engine.cpp:109-111), and the kept tokens are walked in index order, which gives
//    the same distribution as walking them by probability;
//  * top-k and top-p are applied as probability thresholds found by bisection over the
//    bit patterns, so tokens whose probability equals the cut exactly are all kept.
// The logits row is overwritten (the reference's sampler also works in place).
#include "common.cuh"

namespace {

constexpr int SAMPLE_THREADS = 1024;

__device__ __forceinline__ float uniform_from_counter(unsigned long long seed, unsigned long long counter) {
    unsigned long long z = seed + (counter + 1ull) * 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z = z ^ (z >> 31);
    return (float)(z >> 40) * (1.0f / 16777216.0f);
}

// First maximum of a row (strict >, lowest index wins ties; core/ops.cpp:490-497).
__device__ int block_argmax(const float* x, int V, float* s_val, int* s_idx) {
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
        const float v = x[i];
        if (v > best || bi == 0x7fffffff) { best = v; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __syncthreads();
    if (lane == 0) { s_val[warp] = best; s_idx[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        best = lane < nw ? s_val[lane] : -INFINITY;
        bi = lane < nw ? s_idx[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (lane == 0) s_idx[0] = bi;
    }
    __syncthreads();
    const int r = s_idx[0];
    __syncthreads();
    return r;
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
argmax_rows_kernel(const float* logits, int* out, int V) {
    __shared__ float s_val[32];
    __shared__ int s_idx[32];
    pdl_launch_dependents();
    pdl_wait();
    const int r = block_argmax(logits + (size_t)blockIdx.x * V, V, s_val, s_idx);
    if (threadIdx.x == 0) out[blockIdx.x] = r;
}

// Two-stage first-maximum for wide rows: each block takes one slice of a row, then one warp
// per row combines the slices (lowest index wins ties, as in block_argmax).
constexpr int ARGMAX_SLICES = 32;

__global__ void __launch_bounds__(256)
argmax_partial_kernel(const float* logits, float* part_val, int* part_idx, int V) {
    __shared__ float s_val[32];
    __shared__ int s_idx[32];
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.y, slice = blockIdx.x;
    const int per = (V + ARGMAX_SLICES - 1) / ARGMAX_SLICES;
    const int lo = slice * per, hi = min(V, lo + per);
    const float* x = logits + (size_t)row * V;
    float best = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        const float v = x[i];
        if (v > best || bi == 0x7fffffff) { best = v; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) { s_val[warp] = best; s_idx[warp] = bi; }
    __syncthreads();
    if (warp == 0) {
        best = lane < (int)(blockDim.x >> 5) ? s_val[lane] : -INFINITY;
        bi = lane < (int)(blockDim.x >> 5) ? s_idx[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
        }
        if (lane == 0) { part_val[row * ARGMAX_SLICES + slice] = best; part_idx[row * ARGMAX_SLICES + slice] = bi; }
    }
}

__global__ void argmax_final_kernel(const float* part_val, const int* part_idx, int* out) {
    pdl_launch_dependents();
    pdl_wait();
    const int row = blockIdx.x, lane = threadIdx.x;
    float best = part_val[row * ARGMAX_SLICES + lane];
    int bi = part_idx[row * ARGMAX_SLICES + lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) { best = ov; bi = oi; }
    }
    if (lane == 0) out[row] = bi;
}

struct SampleState {
    const long long* rng_seed;   // [slots]
    int* rng_counter;            // [slots] draws made so far
    int* hist;                   // [slots, hist_cap] ring of recorded tokens
    int* hist_count;             // [slots] tokens recorded so far
    int hist_cap;
};

constexpr int PENALTY_CAP = 256;                    // the longest history whose tokens fit the kernels' shared arrays

// The repeat penalty over the last `repeat_last` recorded tokens, for those in [lo, hi), by the whole block: the first of
// equal tokens is penalised once for each of them.  (One thread going through the history took 1.2 us a token.)
__device__ void penalise(float* x, int lo, int hi, int slot, float repeat_pen, int repeat_last, const SampleState& st, int* s_ids) {
    const int count = st.hist_count[slot];
    int n = count < repeat_last ? count : repeat_last;
    if (n > st.hist_cap) n = st.hist_cap;
    const int* ring = st.hist + (size_t)slot * st.hist_cap;
    for (int j = threadIdx.x; j < n; j += blockDim.x) s_ids[j] = ring[(count - n + j) % st.hist_cap];
    __syncthreads();
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        const int id = s_ids[j];
        if (id < lo || id >= hi) continue;
        bool first = true;
        int times = 1;
        for (int i = 0; i < j; i++) first &= s_ids[i] != id;
        if (!first) continue;
        for (int i = j + 1; i < n; i++) times += s_ids[i] == id;
        float v = x[id];
        for (int i = 0; i < times; i++) v = v > 0.f ? v / repeat_pen : v * repeat_pen;
        x[id] = v;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_rows_kernel(float* __restrict__ logits, int* __restrict__ out, const int* __restrict__ row_slot,
                   int V, float temperature, int top_k, float top_p, float repeat_pen, int repeat_last,
                   SampleState st, int record) {
    __shared__ float red[32];
    __shared__ float s_val[32];
    __shared__ int s_idx[32];
    __shared__ float s_scan[SAMPLE_THREADS];
    __shared__ int s_pick, s_ids[PENALTY_CAP];
    pdl_launch_dependents();
    pdl_wait();
    const int slot = row_slot[blockIdx.x];
    if (slot < 0) { if (threadIdx.x == 0) out[blockIdx.x] = -1; return; }
    float* x = logits + (size_t)blockIdx.x * V;
    const int tid = threadIdx.x;

    // 1. repeat penalty over the last `repeat_last` recorded tokens, in order
    if (repeat_pen > 1.f && st.hist != nullptr && st.hist_cap <= PENALTY_CAP) {
        penalise(x, 0, V, slot, repeat_pen, repeat_last, st, s_ids);
    } else if (repeat_pen > 1.f && st.hist != nullptr) {
        if (tid == 0) {
            const int count = st.hist_count[slot];
            int n = count < repeat_last ? count : repeat_last;
            if (n > st.hist_cap) n = st.hist_cap;
            const int* ring = st.hist + (size_t)slot * st.hist_cap;
            for (int j = count - n; j < count; j++) {
                const int id = ring[j % st.hist_cap];
                if (id < 0 || id >= V) continue;
                const float v = x[id];
                x[id] = v > 0.f ? v / repeat_pen : v * repeat_pen;
            }
        }
        __syncthreads();
    }

    int token;
    if (temperature <= 0.f) {
        token = block_argmax(x, V, s_val, s_idx);
    } else {
        // 2. temperature, 3. softmax (probabilities stored in place)
        const float inv_t = (temperature == 1.f) ? 1.f : 1.f / temperature;
        float mx = -INFINITY;
        for (int i = tid; i < V; i += blockDim.x) { const float v = x[i] * inv_t; x[i] = v; mx = fmaxf(mx, v); }
        mx = block_max(mx, red);
        float sum = 0.f;
        for (int i = tid; i < V; i += blockDim.x) { const float e = expf(x[i] - mx); x[i] = e; sum += e; }
        sum = block_sum(sum, red);
        const float inv = 1.f / sum;
        for (int i = tid; i < V; i += blockDim.x) x[i] *= inv;
        __syncthreads();

        // 4. top-k: largest threshold with at least k probabilities at or above it
        unsigned thr = 0u;
        if (top_k > 0 && top_k < V) {
            for (int bit = 30; bit >= 0; bit--) {
                const unsigned cand = thr | (1u << bit);
                float cnt = 0.f;
                for (int i = tid; i < V; i += blockDim.x) cnt += (__float_as_uint(x[i]) >= cand) ? 1.f : 0.f;
                cnt = block_sum(cnt, red);
                if (cnt >= (float)top_k) thr = cand;
            }
        }
        // 5. top-p within those: largest threshold whose kept mass reaches top_p
        if (top_p < 1.f) {
            unsigned thp = 0u;
            for (int bit = 30; bit >= 0; bit--) {
                const unsigned cand = thp | (1u << bit);
                const unsigned eff = cand > thr ? cand : thr;
                float mass = 0.f;
                for (int i = tid; i < V; i += blockDim.x) mass += (__float_as_uint(x[i]) >= eff) ? x[i] : 0.f;
                mass = block_sum(mass, red);
                if (mass >= top_p) thp = cand;
            }
            if (thp > thr) thr = thp;
        }
        // 6. draw: first kept index (ascending) whose running mass exceeds u * kept mass
        const int chunk = (V + blockDim.x - 1) / blockDim.x;
        const int i0 = tid * chunk, i1 = (i0 + chunk < V) ? i0 + chunk : V;
        float local = 0.f;
        for (int i = i0; i < i1; i++) local += (__float_as_uint(x[i]) >= thr) ? x[i] : 0.f;
        s_scan[tid] = local;
        if (tid == 0) s_pick = -1;
        __syncthreads();
        if (tid == 0) {
            float run = 0.f;
            for (int t = 0; t < (int)blockDim.x; t++) { const float v = s_scan[t]; s_scan[t] = run; run += v; }
            red[0] = run;
        }
        __syncthreads();
        const float total = red[0];
        const float u = uniform_from_counter((unsigned long long)st.rng_seed[slot],
                                             (unsigned long long)st.rng_counter[slot]);
        const float r = u * total;
        const float excl = s_scan[tid];
        const float next = (tid + 1 < (int)blockDim.x) ? s_scan[tid + 1] : total;
        if (local > 0.f && excl <= r && r < next) {
            float run = excl;
            int pick = -1, last = -1;
            for (int i = i0; i < i1; i++) {
                if (__float_as_uint(x[i]) >= thr) {
                    last = i;
                    run += x[i];
                    if (run > r) { pick = i; break; }
                }
            }
            s_pick = pick >= 0 ? pick : last;
        }
        __syncthreads();
        if (s_pick < 0) {
            // r fell at or beyond the total through rounding: the last kept index
            int last = -1;
            for (int i = i0; i < i1; i++) if (__float_as_uint(x[i]) >= thr && x[i] > 0.f) last = i;
            if (last >= 0) atomicMax(&s_pick, last);
            __syncthreads();
        }
        token = s_pick;
    }
    if (tid == 0) {
        out[blockIdx.x] = token;
        if (record) {
            if (temperature > 0.f) st.rng_counter[slot] += 1;
            if (st.hist != nullptr) {
                const int c = st.hist_count[slot];
                st.hist[(size_t)slot * st.hist_cap + (c % st.hist_cap)] = token;
                st.hist_count[slot] = c + 1;
            }
        }
    }
}

// ------------------------------------------------------------------------------------------------------------------
// The same chain for wide rows (a temperature above zero): a cluster of eight CTAs per row, the row's values in registers
// (up to 32 a thread) from the first pass to the draw.  What bounds it is the number of exchanges between the CTAs (a cluster
// barrier and what stands on both sides of it, 1.2 us each), not the row's bytes.
//   * The usual case (BOUND), a top-k of fewer tokens than the cluster has warps (128): the k-th largest of the warps' maxima
//     is a lower bound of the k-th largest value, and few values are at or above it (about 50 for k = 40 where the order of the
//     tokens is unrelated to their values).  Those go to the first CTA with the exchange of the softmax's sums, which ends the
//     row alone by comparing them all with one another: two exchanges in all.  8 rows of 128,256: 34 -> 15 us a launch (12 without the repeat penalty).
//   * Otherwise, or where more values are at or above the bound than there is room for, passes over the registers: one
//     settles two bits of a threshold (three candidates), and a search ends as soon as the tokens it keeps are known: top-k
//     when a candidate keeps exactly k, top-p when one token is left between the bounds.
// With one block per row the row came from the L2 again for each of the 62 passes of the two searches: 1.35 ms for 128,256
// tokens whatever the number of rows.
// ------------------------------------------------------------------------------------------------------------------
constexpr int CL = 8, CT = 512, CW = CT / 32;        // CTAs of a cluster, threads and warps of a CTA
constexpr int SEG = 16, FEW = 512;                   // values at or above the bound: room for a warp's and for all of them
constexpr int KEPT = 1 << 30;                        // marks a kept token's index

struct __align__(16) Sums { float a[4]; unsigned n[4]; };

__device__ __forceinline__ unsigned cluster_rank() { unsigned r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_barrier() { cluster_arrive(); cluster_wait(); }
__device__ __forceinline__ void store_remote(void* local, unsigned rank, float4 v) {
    const unsigned here = (unsigned)__cvta_generic_to_shared(local);
    unsigned there;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(here), "r"(rank));
    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(there), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// Every thread of the cluster gets the sums (or, MAX, the largest first value) over all threads, added in one order.
template <bool MAX>
__device__ __forceinline__ Sums cluster_sums(Sums v, Sums (*box)[CL * CW], int& turn) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (MAX) v.a[0] = fmaxf(v.a[0], __shfl_xor_sync(0xffffffffu, v.a[0], o));
        else {
#pragma unroll
            for (int c = 0; c < 3; c++) v.a[c] += __shfl_xor_sync(0xffffffffu, v.a[c], o);
        }
    }
    if (!MAX) {
#pragma unroll
        for (int c = 0; c < 3; c++) v.n[c] = __reduce_add_sync(0xffffffffu, v.n[c]);
    }
    Sums* b = box[turn];
    turn ^= 1;                                        // the other box may still be read by a slower CTA
    if (lane < CL) {
        Sums* at = b + cluster_rank() * CW + warp;
        store_remote(&at->a[0], lane, make_float4(v.a[0], v.a[1], v.a[2], 0.f));
        store_remote(&at->n[0], lane, make_float4(__uint_as_float(v.n[0]), __uint_as_float(v.n[1]), __uint_as_float(v.n[2]), 0.f));
    }
    cluster_barrier();
    Sums t = b[lane];
#pragma unroll
    for (int i = 1; i < CL * CW / 32; i++) {
        const Sums u = b[lane + 32 * i];
        if (MAX) t.a[0] = fmaxf(t.a[0], u.a[0]);
        else {
#pragma unroll
            for (int c = 0; c < 3; c++) { t.a[c] += u.a[c]; t.n[c] += u.n[c]; }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        if (MAX) t.a[0] = fmaxf(t.a[0], __shfl_xor_sync(0xffffffffu, t.a[0], o));
        else {
#pragma unroll
            for (int c = 0; c < 3; c++) t.a[c] += __shfl_xor_sync(0xffffffffu, t.a[c], o);
        }
    }
    if (!MAX) {
#pragma unroll
        for (int c = 0; c < 3; c++) t.n[c] = __reduce_add_sync(0xffffffffu, t.n[c]);
    }
    return t;
}

// A sum of probabilities, RUN of them at a time: pairs of pairs, then with what rounding left of the sum so far.  No further from the
// sum in 64 bits than the passes' trees (50 values 1e-8 on average, 7e-8 at most; 320 4e-9 and 7e-8), where one value after another in 32
// bits was up to six times further off.
constexpr int RUN = 8;
struct Sum {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void add(const float (&q)[RUN]) {
        const float y = ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7])) - c, t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ double value() const { return (double)s - (double)c; }
};

// drawn, recorded: what the slot's counters hold.
__device__ __forceinline__ void record_token(int token, int row, int slot, int drawn, int recorded, int* out, const SampleState& st, int record) {
    out[row] = token;
    if (record) {
        st.rng_counter[slot] = drawn + 1;
        if (st.hist != nullptr) {
            st.hist[(size_t)slot * st.hist_cap + (recorded % st.hist_cap)] = token;
            st.hist_count[slot] = recorded + 1;
        }
    }
}

template <int EPT, bool BOUND>
__global__ void __launch_bounds__(CT)
sample_cluster_kernel(float* logits, int* out, const int* row_slot, int V, float temperature, int top_k, float top_p, float repeat_pen,
                      int repeat_last, SampleState st, int record) {
    __shared__ Sums box[2][CL * CW];
    __shared__ float2 s_seg[BOUND ? CL * CW : 1][SEG];       // of the first CTA: per warp of the cluster its (value, index) at or above the bound
    __shared__ __align__(16) float2 s_few[BOUND ? FEW : 1];  // the same side by side
    __shared__ int2 s_place[BOUND ? CL * CW : 1];     // of a warp's values in s_few: the first, how many
    __shared__ unsigned s_hit[CT];
    __shared__ int s_ids[PENALTY_CAP];
    __shared__ float s_part[EPT * CW], s_excl[EPT * CW], s_total[CL];
    __shared__ int s_entry, s_again, s_last[CL], s_warp_last[CW];
    __shared__ float s_bound;
    __shared__ unsigned s_cut;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = (int)cluster_rank(), row = blockIdx.y;
    pdl_launch_dependents();
    pdl_wait();
    const int slot = row_slot[row];
    float* x = logits + (size_t)row * V;
    const int slice = EPT * CT, base = rank * slice;  // this CTA's values are base + 512 j + tid
    int turn = 0;
    float v[EPT];
#pragma unroll
    for (int j = 0; j < EPT; j++) {
        const int i = base + j * CT + tid;
        v[j] = i < V ? x[i] : -INFINITY;
    }
    if (slot < 0) { if (rank == 0 && tid == 0) out[row] = -1; return; }      // the whole cluster
    cluster_arrive();                                 // (waited for before another CTA's memory is written)
    const unsigned long long seed = (unsigned long long)st.rng_seed[slot];
    const int drawn = st.rng_counter[slot], recorded = st.hist != nullptr ? st.hist_count[slot] : 0;
    // Repeat penalty, while the values are on their way: the recorded tokens in this CTA's slice are marked, and the thread that
    // has a marked one penalises it, as often as it was recorded.
    if (repeat_pen > 1.f && st.hist != nullptr) {
        int n = recorded < repeat_last ? recorded : repeat_last;
        if (n > st.hist_cap) n = st.hist_cap;
        // place p of the ring holds one of the last n if it lies less than n places, going round, before the next one's
        int id = -1;
        if (tid < st.hist_cap) {
            id = st.hist[(size_t)slot * st.hist_cap + tid];
            int back = recorded % st.hist_cap - tid;
            if (back <= 0) back += st.hist_cap;
            if (back > n) id = -1;
        }
        if (id < base || id >= min(base + slice, V)) id = -1;
        s_hit[tid] = 0u;
        if (tid < PENALTY_CAP) s_ids[tid] = id;
        if (tid == 0) s_again = 0;
        __syncthreads();
        if (id >= 0) {
            const unsigned bit = 1u << ((id - base) / CT);
            if (atomicOr(&s_hit[(id - base) % CT], bit) & bit) s_again = 1;
        }
        __syncthreads();
        for (unsigned mine = s_hit[tid]; mine != 0u; mine &= mine - 1u) {
            const int at = __ffs(mine) - 1, token = base + at * CT + tid;
            int times = s_again ? 0 : 1;
            if (s_again) for (int i = 0; i < PENALTY_CAP; i++) times += s_ids[i] == token ? 1 : 0;
            float p = 0.f;
#pragma unroll
            for (int j = 0; j < EPT; j++) p = j == at ? v[j] : p;
            for (int i = 0; i < times; i++) p = p > 0.f ? p / repeat_pen : p * repeat_pen;
            x[token] = p;
#pragma unroll
            for (int j = 0; j < EPT; j++) v[j] = j == at ? p : v[j];
        }
    }

    // temperature, softmax
    const float inv_t = temperature == 1.f ? 1.f : 1.f / temperature;
    Sums sums = {};
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < EPT; j++) { v[j] *= inv_t; mx = fmaxf(mx, v[j]); }
    __syncwarp();
    cluster_wait();
    sums.a[0] = mx;
    mx = cluster_sums<true>(sums, box, turn).a[0];
    // the bound: the top_k-th largest of the warps' maxima.  At least top_k values are at or above it.
    float least = INFINITY;                           // exponentials from here on are marked: a little below the bound's, so
    if (BOUND) {                                      // that whatever rounds to the bound's probability is among them
        const Sums* maxima = box[turn ^ 1];
        if (tid < CL * CW) {
            const float own = maxima[tid].a[0];
            int above = 0, from_it_on = 0;
#pragma unroll 16
            for (int i = 0; i < CL * CW; i++) { const float m = maxima[i].a[0]; above += m > own ? 1 : 0; from_it_on += m >= own ? 1 : 0; }
            if (above < top_k && top_k <= from_it_on) s_bound = own;
        }
        __syncthreads();
        least = fmaxf(expf(s_bound - mx) * 0.9999f, 1e-45f);
    }
    sums = {};
    unsigned marked = 0u;
#pragma unroll
    for (int j = 0; j < EPT; j++) {
        v[j] = base + j * CT + tid < V ? expf(v[j] - mx) : 0.f;
        if (BOUND) marked |= v[j] >= least ? 1u << j : 0u;
        sums.a[0] += v[j];
    }
    if (BOUND) {
        const int mine = __popc(marked), all = __reduce_add_sync(0xffffffffu, mine);
        if (all > 0 && all <= SEG) {
            int at = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, at, o); if (lane >= o) at += u; }
            at -= mine;
            const unsigned here = (unsigned)__cvta_generic_to_shared(&s_seg[rank * CW + warp][0]);
            unsigned there;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"(here), "r"(0));
#pragma unroll
            for (int j = 0; j < EPT; j++) {
                if (marked >> j & 1u) {
                    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(there + 8u * at), "f"(v[j]),
                                 "f"(__int_as_float(base + j * CT + tid)) : "memory");
                    at++;
                }
            }
        }
        if (lane == 0) { sums.n[0] = all; sums.n[1] = all > SEG ? 1u : 0u; }
    }
    const Sums softmax = cluster_sums<false>(sums, box, turn);
    const float inv = 1.f / softmax.a[0];

    // (a sum that is no number takes the passes, which choose no token)
    if (BOUND && softmax.n[1] == 0u && softmax.n[0] <= FEW && softmax.a[0] >= 1.f) {
        if (rank != 0) return;                        // nothing is written to another CTA any more
        const int n = (int)softmax.n[0], whole = (n + RUN - 1) / RUN * RUN;
        // side by side, in the warps' order
        if (warp == 0) {
            const Sums* of = box[turn ^ 1];
            int count[CL * CW / 32], before = 0;
#pragma unroll
            for (int i = 0; i < CL * CW / 32; i++) { count[i] = (int)of[lane * (CL * CW / 32) + i].n[0]; before += count[i]; }
            int scan = before;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, scan, o); if (lane >= o) scan += u; }
            before = scan - before;
#pragma unroll
            for (int i = 0; i < CL * CW / 32; i++) { s_place[lane * (CL * CW / 32) + i] = make_int2(before, count[i]); before += count[i]; }
        }
        if (tid == 0) { s_cut = 0u; s_entry = 0x7fffffff; }
        __syncthreads();
        {
            static_assert(CT == 4 * CL * CW, "four threads a warp's values");
            const int2 place = s_place[tid >> 2];
            for (int i = tid & 3; i < place.y; i += 4) { const float2 c = s_seg[tid >> 2][i]; s_few[place.x + i] = make_float2(c.x * inv, c.y); }
            if (tid < RUN && n + tid < whole) s_few[n + tid] = make_float2(-1.f, 0.f);      // kept by nothing
        }
        __syncthreads();
        // kept by top-k: fewer than top_k are above it; the cut of top-p: the largest value with which the mass reaches top_p
        for (int i = tid; i < n; i += CT) {
            const float p = s_few[i].x;
            int above = 0;
            Sum mass;
            for (int j = 0; j < whole; j += RUN) {
                float q[RUN];
#pragma unroll
                for (int e = 0; e < RUN; e++) { const float o = s_few[j + e].x; above += o > p ? 1 : 0; q[e] = o >= p ? o : 0.f; }
                mass.add(q);
            }
            if (above < top_k) {
                if (top_p < 1.f && (float)mass.value() >= top_p) atomicMax(&s_cut, __float_as_uint(p));
                s_few[i].y = __int_as_float(__float_as_int(s_few[i].y) | KEPT);
            }
        }
        __syncthreads();
        const unsigned cut = s_cut;
        const float u = uniform_from_counter(seed, (unsigned long long)drawn);
        // the draw: the first kept token, by index, whose running mass exceeds u x the kept mass
        int last_kept = -1;
        for (int i = tid; i < n; i += CT) {
            const float2 c = s_few[i];
            const int id = __float_as_int(c.y);
            if (!(id & KEPT) || __float_as_uint(c.x) < cut) continue;
            Sum run, total;
            for (int j = 0; j < whole; j += RUN) {
                float q[RUN], r[RUN];
#pragma unroll
                for (int e = 0; e < RUN; e++) {
                    const float2 o = s_few[j + e];
                    const int other = __float_as_int(o.y);
                    q[e] = (other & KEPT) && __float_as_uint(o.x) >= cut ? o.x : 0.f;
                    r[e] = other <= id ? q[e] : 0.f;
                }
                total.add(q);
                run.add(r);
            }
            if (run.value() > (double)u * total.value()) atomicMin(&s_entry, id & ~KEPT);
            last_kept = max(last_kept, id & ~KEPT);
        }
        __syncthreads();
        if (s_entry == 0x7fffffff) {                  // rounding left u x the mass at or beyond the last one: the last kept token
            if (tid == 0) s_last[0] = -1;
            __syncthreads();
            if (last_kept >= 0) atomicMax(&s_last[0], last_kept);
            __syncthreads();
            if (tid == 0) s_entry = s_last[0];
        }
        if (tid == 0) record_token(s_entry, row, slot, drawn, recorded, out, st, record);
        return;
    }
#pragma unroll
    for (int j = 0; j < EPT; j++) v[j] *= inv;

    // top-k: the largest threshold with at least k probabilities at or above it; positions behind V hold 0 and are below
    // any candidate.  No probability reaches 2, so that bit 30 is never set.
    unsigned thr = 0u;
    if (top_k > 0 && top_k < V) {
        for (int bit = 28; bit >= 0; bit -= 2) {
            sums = {};
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const unsigned cand = thr | ((unsigned)(c + 1) << bit);
#pragma unroll
                for (int j = 0; j < EPT; j++) sums.n[c] += __float_as_uint(v[j]) >= cand ? 1u : 0u;
            }
            const Sums t = cluster_sums<false>(sums, box, turn);
            unsigned add = 0;
            bool exact = false;
#pragma unroll
            for (int c = 0; c < 3; c++) if (t.n[c] >= (unsigned)top_k) { add = c + 1; exact = t.n[c] == (unsigned)top_k; }
            thr |= add << bit;
            if (exact) break;
        }
    }
    // top-p within those: the largest threshold whose kept mass reaches top_p
    if (top_p < 1.f) {
        unsigned thp = 0u, above = 0u, kept = 0xffffffffu;    // tokens kept at the upper bound and at thp
        for (int bit = 28; bit >= 0; bit -= 2) {
            sums = {};
#pragma unroll
            for (int c = 0; c < 3; c++) {
                const unsigned cand = thp | ((unsigned)(c + 1) << bit), eff = cand > thr ? cand : thr;
#pragma unroll
                for (int j = 0; j < EPT; j++) {
                    const bool in = __float_as_uint(v[j]) >= eff;
                    sums.a[c] += in ? v[j] : 0.f;
                    sums.n[c] += in ? 1u : 0u;
                }
            }
            const Sums t = cluster_sums<false>(sums, box, turn);
            if (t.a[0] < top_p && (thp | (1u << bit)) <= thr) break;      // all that top-k left does not reach top_p
            unsigned add = 0;
            bool open = true;                         // the first candidate that is not reached is the upper bound
#pragma unroll
            for (int c = 0; c < 3; c++) {
                if (t.a[c] >= top_p) { add = c + 1; kept = t.n[c]; }
                else if (open) { above = t.n[c]; open = false; }
            }
            thp |= add << bit;
            if (kept != 0xffffffffu && kept - above <= 1u) break;     // nothing but the last kept token lies between the bounds
        }
        if (thp > thr) thr = thp;
    }

    // the draw: kept tokens in order of their index; first the sums of runs of 32 of them
    int last = -1;
#pragma unroll
    for (int j = 0; j < EPT; j++) {
        const bool in = __float_as_uint(v[j]) >= thr && base + j * CT + tid < V;
        v[j] = in ? v[j] : 0.f;
        if (in && v[j] > 0.f) last = base + j * CT + tid;
        const float s = warp_sum(v[j]);
        if (lane == 0) s_part[j * CW + warp] = s;
    }
    last = __reduce_max_sync(0xffffffffu, last);
    if (lane == 0) s_warp_last[warp] = last;
    __syncthreads();
    constexpr int PER = EPT * CW / 32;                // runs a lane of warp 0 adds up
    float mine = 0.f;
    if (warp == 0) {
#pragma unroll
        for (int i = 0; i < PER; i++) mine += s_part[lane * PER + i];
        float scan = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const float u = __shfl_up_sync(0xffffffffu, scan, o); if (lane >= o) scan += u; }
        const float before = __shfl_up_sync(0xffffffffu, scan, 1);
        float run = lane == 0 ? 0.f : before;
#pragma unroll
        for (int i = 0; i < PER; i++) { s_excl[lane * PER + i] = run; run += s_part[lane * PER + i]; }
        last = __reduce_max_sync(0xffffffffu, lane < CW ? s_warp_last[lane] : -1);
        const float total = __shfl_sync(0xffffffffu, scan, 31);
        if (lane < CL) store_remote(&box[turn][rank], lane, make_float4(total, __int_as_float(last), 0.f, 0.f));
        if (lane == 0) s_entry = -1;
    }
    cluster_barrier();
    if (tid < CL) { s_total[tid] = box[turn][tid].a[0]; s_last[tid] = __float_as_int(box[turn][tid].a[1]); }
    turn ^= 1;
    __syncthreads();
    float from = 0.f, total = 0.f;
#pragma unroll
    for (int c = 0; c < CL; c++) { if (c == rank) from = total; total += s_total[c]; }
    float to = from + s_total[rank];
    const float u = uniform_from_counter(seed, (unsigned long long)drawn);
    const float r = u * total;
    int pick = -1;
    if (from <= r && r < to) {                        // one CTA at most
        for (int e = tid; e < EPT * CW; e += CT) {
            // the last run that begins at or below r among those that hold something
            if (s_part[e] > 0.f && from + s_excl[e] <= r) atomicMax(&s_entry, e);
        }
        __syncthreads();
        const int e = s_entry;
        if (e >= 0 && e % CW == warp) {
            float mass = 0.f;
#pragma unroll
            for (int j = 0; j < EPT; j++) if (j == e / CW) mass = v[j];
            float run = from + s_excl[e];
            int at = -1, some = -1;
            for (int l = 0; l < 32; l++) {
                const float m = __shfl_sync(0xffffffffu, mass, l);
                if (m <= 0.f) continue;
                run += m;
                some = l;
                if (at < 0 && run > r) at = l;
            }
            pick = base + e / CW * CT + warp * 32 + (at >= 0 ? at : some);
            if (lane == 0) store_remote(&box[turn][0], 0, make_float4(__int_as_float(pick), 0.f, 0.f, 0.f));
        }
    } else if (tid == 0 && rank == 0 && !(r < total)) {
        // r fell at or beyond the total through rounding (or nothing is kept): the last kept token
        int l = -1;
        for (int c = 0; c < CL; c++) l = max(l, s_last[c]);
        box[turn][0].a[0] = __int_as_float(l);
    }
    cluster_barrier();
    if (rank == 0 && tid == 0) record_token(__float_as_int(box[turn][0].a[0]), row, slot, drawn, recorded, out, st, record);
}

// Whether a row's top-k goes by the bound.  Of W warps that hold values, as many as k have their maximum at or above it where it
// has W / (W - k + 1) + .. + W / W values at or above it on average, wherever they lie in the row.  Comparing n values with one
// another takes n^2 / 32 steps, so that beyond some 320 the passes are as fast (8 rows of 128,256: top-k 40 14 us, 104 19, 110 22, by
// passes 32 to 35; 128, of which 700 values are at or above the bound, 91; 64 of 65,536, 300 values, 30 and 31, 64 rows 67 and 135).  The
// attempt costs a row that it does not settle 2.6 us (one whose values are all the same, 25 -> 28 us), and the kernel without it is
// 1 us faster than one that has both.
bool by_bound(int top_k, int V, int slice) {
    if (top_k <= 0 || top_k >= V) return false;
    const int rest = V % slice, warps = V / slice * CW + (rest < CT ? (rest + 31) / 32 : CW);
    if (top_k > warps) return false;
    if (16 * top_k <= 13 * warps) return true;        // 1.7 W at most
    float values = 0.f;
    for (int i = warps - top_k + 1; i <= warps; i++) values += (float)warps / (float)i;
    return values <= 320.f;
}

template <int EPT>
int launch_cluster(float* logits, int* out, const int* row_slot, int rows, int V, float temperature, int top_k, float top_p,
                   float repeat_pen, int repeat_last, const SampleState& state, int record, cudaStream_t st) {
    const auto kernel = by_bound(top_k, V, EPT * CT) ? sample_cluster_kernel<EPT, true> : sample_cluster_kernel<EPT, false>;
    return oe_launch_cluster(kernel, CL, dim3(CL, rows), dim3(CT), 0, st, logits, out, row_slot, V, temperature, top_k, top_p, repeat_pen,
                             repeat_last, state, record);
}

// Row `row` of every tensor of a table of (address, bytes of a row), four bytes at a time.  grid (pieces, tensors)
__global__ void __launch_bounds__(256)
zero_rows_kernel(const long long* table, int row) {
    pdl_launch_dependents();
    pdl_wait();
    const long long bytes = table[2 * blockIdx.y + 1];
    unsigned* p = (unsigned*)(table[2 * blockIdx.y] + (long long)row * bytes);
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < bytes / 4; i += (long long)gridDim.x * 256) p[i] = 0u;
}

// A sequence's first sampler state.  The recorded tokens come as a kernel argument: no copy to the device.
struct Ring { int id[PENALTY_CAP]; };
__global__ void __launch_bounds__(PENALTY_CAP)
sampler_start_kernel(long long* rng_seed, int* rng_counter, int* hist, int* hist_count, int slot, long long seed, int count, int cap,
                     int with_ring, const __grid_constant__ Ring ring) {
    pdl_launch_dependents();
    pdl_wait();
    if (threadIdx.x == 0) { rng_seed[slot] = seed; rng_counter[slot] = 0; hist_count[slot] = count; }
    if (with_ring && (int)threadIdx.x < cap) hist[(size_t)slot * cap + threadIdx.x] = ring.id[threadIdx.x];
}

}  // namespace

extern "C" {

int oe_zero_rows(const long long* table, int n, long long largest, int row, cudaStream_t st) {
    if (n <= 0) return 0;
    if (n > 65535 || row < 0 || largest < 0) return OE_ERR_UNSUPPORTED;
    long long pieces = (largest / 4 + 1023) / 1024;
    if (pieces < 1) pieces = 1;
    if (pieces > 64) pieces = 64;
    return oe_launch(zero_rows_kernel, dim3((unsigned)pieces, n), dim3(256), 0, st, table, row);
}

// tail: null, or the last `n_tail` (up to `cap`) of the `count` recorded tokens in host memory, read before the call returns; they
// go where a ring of `cap` places has them, the other places are zero.  null: the history stays as it is.
int oe_sampler_start(long long* rng_seed, int* rng_counter, int* hist, int* hist_count, int cap, int slot, long long seed, int count,
                     const int* tail, int n_tail, cudaStream_t st) {
    if (cap < 1 || cap > PENALTY_CAP || slot < 0 || n_tail < 0 || n_tail > cap || (tail && n_tail > count)) return OE_ERR_UNSUPPORTED;
    Ring r = {};
    if (tail) for (int i = 0, at = (count - n_tail) % cap; i < n_tail; i++, at = at + 1 == cap ? 0 : at + 1) r.id[at] = tail[i];
    return oe_launch(sampler_start_kernel, dim3(1), dim3(PENALTY_CAP), 0, st, rng_seed, rng_counter, hist, hist_count, slot, seed, count, cap,
                     tail != nullptr ? 1 : 0, r);
}

// Wide rows in two stages; scratch: rows * 32 floats and rows * 32 ints.
int oe_argmax_rows_wide(const float* logits, int* out, float* part_val, int* part_idx, int rows, int V, cudaStream_t st) {
    if (rows <= 0) return 0;
    if (V <= 0 || rows > 65535) return OE_ERR_UNSUPPORTED;
    int rc = oe_launch(argmax_partial_kernel, dim3(ARGMAX_SLICES, rows), dim3(256), 0, st, logits, part_val, part_idx, V);
    if (rc) return rc;
    return oe_launch(argmax_final_kernel, dim3(rows), dim3(32), 0, st, (const float*)part_val, (const int*)part_idx, out);
}

int oe_argmax_rows(const float* logits, int* out, int rows, int V, cudaStream_t st) {
    if (rows <= 0) return 0;
    if (V <= 0) return OE_ERR_UNSUPPORTED;
    const int launch_rc = oe_launch(argmax_rows_kernel, dim3(rows), dim3(SAMPLE_THREADS), 0, st, logits, out, V);
    return launch_rc;
}

// Whether a draw of wide rows looks for a small top-k's values by a bound.
int oe_sample_by_bound(int top_k, int V) { return by_bound(top_k, V, (V <= CL * CT * 8 ? 8 : 32) * CT) ? 1 : 0; }

int oe_sample_rows(float* logits, int* out, const int* row_slot, int rows, int V, float temperature,
                   int top_k, float top_p, float repeat_pen, int repeat_last, const long long* rng_seed,
                   int* rng_counter, int* hist, int* hist_count, int hist_cap, int record,
                   cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (V <= 0 || (hist != nullptr && hist_cap <= 0)) return OE_ERR_UNSUPPORTED;
    SampleState st{rng_seed, rng_counter, hist, hist_count, hist_cap};
    // A row per cluster from 8,192 tokens on (below that the row fits a block's first-level cache) up to what the registers of a
    // cluster hold, 131,072; the history's bound is that of the ring in shared memory.
    if (temperature > 0.f && V >= 8192 && V <= CL * CT * 32 && rows <= 65535 && (hist == nullptr || hist_cap <= PENALTY_CAP)) {
        if (V <= CL * CT * 8)
            return launch_cluster<8>(logits, out, row_slot, rows, V, temperature, top_k, top_p, repeat_pen, repeat_last, st, record, stream);
        return launch_cluster<32>(logits, out, row_slot, rows, V, temperature, top_k, top_p, repeat_pen, repeat_last, st, record, stream);
    }
    const int launch_rc = oe_launch(sample_rows_kernel, dim3(rows), dim3(SAMPLE_THREADS), 0, stream, logits, out, row_slot, V, temperature, top_k, top_p,
                                                            repeat_pen, repeat_last, st, record);
    return launch_rc;
}

}  // extern "C"
