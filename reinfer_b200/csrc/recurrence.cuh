// What the two files of the linear recurrences share: the arguments, the pointwise functions, 16-byte asynchronous copies.
#pragma once
#include "common.cuh"

struct RecurArgs {
    const void* q; long long ldq;          // [T, Hk * dk]   (activation dtype)
    const void* k; long long ldk;          // [T, Hk * dk]
    const void* v; long long ldv;          // [T, H * dv]
    const float* z; long long ldz;         // [T, H * dk] gate pre-activation without its bias ([T, H] with z_per_head)
    const float* z_bias;                   // [H * dk] or null ([H] with z_per_head)
    int z_per_head;                        // one gate per head and token instead of one per key channel
    const void* a_pre; long long lda;      // form 1: removal rate before the sigmoid [T, H * dk] (activation dtype)
    const float* a_bias;                   // form 1: [H * dk] or null
    const void* b_pre; long long ldb;      // form 2: write strength before the sigmoid [T, H]
    const float* rate;                     // gate 2: [H]
    const float* bonus;                    // form 3: [H * dk]
    float gate_param;                      // gate 0: 1 / tau;  gate 1: c
    float q_scale;                         // q is multiplied by this (after it was made a unit vector, if it is)
    int unit_qk;                           // q and k are made unit vectors: x / sqrt(sum x^2 + 1e-6)
    int gate;
    float* state;                          // [slots, H, dk, dv]
    float* out;                            // [T, H, dv]
    const int* cu_q; const int* entry_slot;
    int H, Hk, dk, dv, tile;
    float* prep;                           // [T, H, record] vectors prepared ahead (null: the walking kernel prepares them)
    int n_tokens;
    int rec_floats;                        // floats of a record made ahead: the vectors, then v of the head padded to RR_COLS columns
};

__device__ __forceinline__ void rr_cp_async16(void* dst, const void* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void rr_cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void rr_cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ float softplus_f(float x) { return fmaxf(x, 0.0f) + log1pf(expf(-fabsf(x))); }
__device__ __forceinline__ float sigmoid_f(float x) { return 1.0f / (1.0f + expf(-x)); }

// The gate of one key channel from its pre-activation (bias included), as ln g: the four kinds that recurrence.cu lists.
__device__ __forceinline__ float recur_log_gate(const RecurArgs& A, float z, float rate) {
    if (A.gate == 0) return -softplus_f(-z) * A.gate_param;
    if (A.gate == 1) return -A.gate_param * sigmoid_f(z);
    if (A.gate == 2) return -rate * softplus_f(z);
    return -expf(z);
}

// recurrence_chunk.cu: long portions of 16-bit tokens, four tokens at a time.
int recurrence_chunks(const RecurArgs& A, int form, int n_entries, cudaStream_t st);
long long recurrence_chunks_scratch(int form, int dk, int dv, int H, int n_tokens, int n_entries);
