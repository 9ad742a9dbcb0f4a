// What the scans in chunks (delta_chunks.cu, decay_chunks.cu) share: how a step's sequences are cut, and the split of a head's
// state over CTAs and threads.
#pragma once
#include "common.cuh"

namespace {

constexpr int CH = 32;                 // tokens of a chunk
constexpr int COLS = 16;               // columns of the state that a CTA of the scan carries
constexpr int GROUPS = 16;             // threads that share a column, each a sixteenth of its rows

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem) : "memory");
}

// The chunks of sequence b stand behind those of the sequences before it.
__device__ __forceinline__ int chunks_of(const int* __restrict__ cu_q, const int* __restrict__ seq_slot, int b) {
    return seq_slot[b] < 0 ? 0 : (cu_q[b + 1] - cu_q[b] + CH - 1) / CH;
}

}  // namespace
