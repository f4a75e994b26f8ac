// The fixed-size states of newly admitted requests, set to zero: every state tensor's row of every new slot in one launch.
// (A fill per tensor and slot is 10 launches a request for a model of six recurrent layers; eight requests that arrive together
// cost the host 0.7 ms, and their first step as much.)
#include "common.cuh"

#define SLOTS_BATCH 64                        // slots of one launch (they travel as an argument)

struct RbZeroRow { unsigned char* rows; long long bytes; };           // a state tensor's first row, the bytes from one row to the next
struct RbSlots { int slot[SLOTS_BATCH]; };

// grid: (pieces of a row, tensors, slots)
__global__ void __launch_bounds__(256)
zero_slots_kernel(const RbZeroRow* __restrict__ table, const RbSlots slots) {
    pdl_trigger();
    const RbZeroRow row = table[blockIdx.y];                          // made when the storage was: nothing here waits
    pdl_wait();
    unsigned char* p = row.rows + (size_t)slots.slot[blockIdx.z] * row.bytes;
    const size_t first = (size_t)blockIdx.x * 256 + threadIdx.x, step = (size_t)gridDim.x * 256;
    if (((uintptr_t)p & 15) == 0) {
        const size_t whole = (size_t)row.bytes / 16;
        for (size_t i = first; i < whole; i += step) reinterpret_cast<uint4*>(p)[i] = make_uint4(0, 0, 0, 0);
        if (first < (size_t)row.bytes % 16) p[whole * 16 + first] = 0;
    } else {
        for (size_t i = first; i < (size_t)row.bytes; i += step) p[i] = 0;
    }
}

// table [n_tensors] on the device, largest_row the bytes of the longest row; slots on the host.
extern "C" int rb_zero_slots(const void* table, int n_tensors, long long largest_row, const int* slots, int n_slots, void* stream) {
    if (n_tensors <= 0 || n_slots <= 0 || largest_row <= 0) return 0;
    if (n_tensors > 65535) RB_REFUSE("zero_slots: %d tensors", n_tensors);
    const long long pieces = (largest_row + 256 * 64 - 1) / (256 * 64);       // four stores of 16 bytes a thread of the longest row
    for (int at = 0; at < n_slots; at += SLOTS_BATCH) {
        RbSlots some;
        const int n = n_slots - at < SLOTS_BATCH ? n_slots - at : SLOTS_BATCH;
        for (int i = 0; i < n; ++i) some.slot[i] = slots[at + i];
        const int e = rb_launch(zero_slots_kernel, dim3((unsigned)(pieces < 4096 ? pieces : 4096), n_tensors, n), dim3(256), 0, (cudaStream_t)stream,
                                (const RbZeroRow*)table, some);
        if (e) return e;
    }
    return 0;
}
