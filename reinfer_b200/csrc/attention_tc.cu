// Paged causal flash attention for prompt portions on the fifth-generation tensor cores.
//
// The formulas are the reference's attention (crates/cuda/kernels/dense_kernels.cu:173-231: scores, causal
// mask, softmax in float, weighted sum of the values), tiled as flash attention.  A CTA owns 256 query rows: two
// row tiles A and B of 128 rows each (a row = a token x one of the Gc grouped query heads of one kv head; tile B
// holds the tokens after tile A's), and walks the request's keys in tiles of 64.  Both row tiles use every key
// tile that comes in, so a key tile is fetched once for 256 rows.  For every key tile j and row tile t
//     S_t = Q_t K^T        tcgen05.mma, 128 x 64 x 128, operands in shared memory, S in tensor memory (two buffers a row tile)
//     P_t = exp2(S_t - m)  128 threads, one row each (tcgen05.ld gives a thread its whole row: the row maximum and
//                          sum need no shuffles), P rounded to bfloat16 and written back to tensor memory, over the scores
//     O_t += P_t V         tcgen05.mma, 128 x 128 x 64, P from tensor memory, accumulated there over all key tiles: P and O are
//                          scaled to a maximum that follows the true one only when it rose by more than 2^8 (then the
//                          row's thread rescales its lane of O in tensor memory, which is rare), so the rows read O once
// Warp 0 feeds key and value tiles by TMA into a ring of four each: ONE request brings the keys (or the values) of a page for this kv
// head, laid out as [8-key group][64-dim half][8 keys][64 dims] whatever the page size is (the 5-D map of runtime.cu).  Warp 1
// allocates tensor memory and issues the products of tile A, warp 3 those of tile B; warps 4-7 are the rows of tile A,
// warps 8-11 the rows of tile B.  Q [rows][d] and K [keys][d] are K-major operands; V [keys][d] is
// used as it lands, as an MN-major operand (instruction descriptor bit 16; in the shared-memory descriptor the
// leading offset steps to the second 64 dims, the stride offset to the next 8 keys) - nothing is transposed.
//
// What runs ahead of what.  The scores of tile j + 2 go into the columns that P of tile j lay in: their product is issued right behind
// the weighted sum that reads P, by the same warp, and runs behind it; the rows meanwhile work on tile j + 1 in the other buffer.  So no
// hand-over lies on the rows' path from one key tile to the next.  P does not pass through shared memory: with P there, its
// writes, the products' two reads of every operand and the copies wanted 3,070 cycles of shared memory per 128 keys, at 128 bytes a
// cycle, where the tensor cores want 2,048.
//
// What bounds it (-DRB_TIMELINE, cycles per 64 keys; 2,048 tokens behind 14,336 others, 32 query over 8 kv heads): a row warp works
// 1,480, of them 1,230 in the exponentials (the special-function unit needs 1,024 for the two row warps of a scheduler), and waits 220
// for scores; the tensor pipe is busy 1,280 (a 128 x 64 product of scores reads 6 KB of shared memory, 48 cycles for 32 of arithmetic).
// 473 us (1,090 TFLOP/s); with P in shared memory, scores of 128 keys and a third issuing warp for the weighted sums 526.  256 CTAs of
// equal length are 1.73 rounds over 148 SMs, which costs another seventh.  Measured beside it: products of 128 x 128 scores with P over
// them, whose rows wait for product, hand-over and product again (664 us); one score buffer and two of P beside it (554); barriers of
// keys and values looked at only when they are needed (500: a wait costs an issuer 135 cycles however long ago the bytes came).
// Scaling, sums and maxima are packed or three-input instructions, and the code of the options is in instantiations of its
// own, for the rows' loop has to fit the instruction cache: with all options in it, a fifth of the rows' stalls were
// instruction fetches.  Built, measured, left out before P moved: two threads per row (the row's maximum agreed through shared memory:
// 11 % slower); a part of the exponentials as a cubic on the FMA pipe (8 to 16 % slower); P rounded by integer instructions.
// Registers follow the roles (setmaxnreg): 64 for the control warps, 216 for the rows - what the control warps give up
// (128 threads x 104) must cover what the rows take (256 threads x 48), for the registers come from the CTA's own
// allocation (384 x 168) and a request for more than it holds waits for ever.
//
// Options on top: a distance penalty, a learned bias by distance, chunks, a soft cap on the scores (before penalty and
// bias), a sink in the denominator and a sigmoid gate on the output - each skipped when not asked for.
// Head size 128, page size a power of two >= 8.  Every wait is bounded (2 s); a CTA that gives up raises the
// error word, lets its copies land, frees its tensor memory and leaves; CTAs that start after that leave at once.
#define RB_UNIT 3
#include "sm100.cuh"
#include <stdlib.h>

#define FC_BN 64                              // keys per key tile
#define FC_ROWS 128                           // query rows per row tile
#define FC_TILES 2                            // row tiles per CTA
#define FC_D 128
#define FC_THREADS 384                        // a control group (TMA, products of tile A, -, products of tile B) and two groups of four row warps
#define FC_RING 4                             // key tiles, and value tiles, in shared memory
#define FC_SLOTS (2 * FC_RING)                // keys in slots 0 .., values behind them
#define FC_KSLOT(tile) ((tile) % FC_RING)
#define FC_VSLOT(tile) (FC_RING + (tile) % FC_RING)
#define FC_PHASE(tile) ((uint32_t)(((tile) / FC_RING) & 1))
#define FC_KV_BYTES (FC_BN * 256)             // a slot: 64 keys (or values) x 256 bytes, as 8 groups of [2 halves][8 keys][128 bytes]
#define FC_GROUP 2048                         // bytes from one 8-key group to the next
#define FC_HALF 1024                          // bytes from a group's first 64 dims to its second
#define FC_QHALF (FC_ROWS * 128)              // 128 rows x 128 bytes: one 64-column half of a Q tile
#define FC_RESCALE 8.0f                       // O is brought to a new maximum only when it rose by more than this (log2)
#define FC_TMEM_COLS 512                      // S_A: columns 0..63 and 64..127, P_A in the first half of either; S_B 128..255; O_A 256..383; O_B 384..511
#define FC_S(t, tile) ((uint32_t)((t) * 2 * FC_BN + ((tile) & 1) * FC_BN))
#define FC_O(t) ((uint32_t)(FC_TILES * 2 * FC_BN + (t) * FC_D))

struct FcArgs {
    const bf16* q;
    const int* block_table;
    const int* cu_q;
    const int* kv_len;
    bf16* out;
    int QH, KH, page_size, page_shift, max_pages, window;
    int Gc, chunks, first_entry, n_entries;
    float scale_log2;
    // Options for attention that is local to chunks of positions: a row sees only the keys from the start of its own
    // chunk of `chunk` positions (a multiple of the 64-key tile; 0: off), its scores lose r1[h] ln(1 + r2[h] (i - j))
    // (null: no penalty), and the output is multiplied by out_scale.
    int chunk;
    const float* r1;
    const float* r2;
    float out_scale;
    // A learned bias by distance: score += bias[h][min(i - j, bias_last)] (a float table [QH, bias_last + 1] in units of
    // the scaled score; null: none).  Its last column stands for every greater distance.
    const float* bias;
    int bias_last;
    // A soft cap: score <- cap tanh(score / cap) on the scaled score; here in units of the raw score (cap / scale), with
    // 2 log2(e) / that for the exponential the tanh is made of (0: none).
    float cap_raw, cap_arg;
    // A sink: one more term exp(sink[h]) in a row's denominator, with no key and no value (null: none).
    const float* sink;
    // An output gate: out *= sigmoid(gate[t * gate_stride + h * 128 + i]) (null: none).
    // gate_heads: one number a head, gate[t * gate_stride + h].
    const float* gate;
    long long gate_stride;
    int gate_heads;
};

struct FcShared {
    unsigned long long full[FC_SLOTS];
    unsigned long long done[FC_RING];                              // [i % FC_RING]: either issuer's scores of tile i and weighted sum of tile i - 2
    unsigned long long s_full[FC_TILES][2], p_full[FC_TILES][2];
    unsigned long long o_full[FC_TILES][2];                        // the weighted sums up to the last tile but one; up to the last (one use each)
    int uses[FC_SLOTS];                                            // copies issued into each slot
    uint32_t tmem_base;
    int abort_flag;
};

// byte offset of 16-byte chunk c (8 elements) of row `row` in a K-major tile of 128-byte rows with the 128-byte
// swizzle; chunks 8.. lie in the next 64-column half, half_bytes further
__device__ __forceinline__ uint32_t fc_off(int row, int c, int half_bytes) {
    return (uint32_t)((c >> 3) * half_bytes + row * 128 + (((c & 7) ^ (row & 7)) << 4));
}
// the same for a key/value tile as the 5-D map lays it out: [8-key group][half][8 keys][128 bytes]
__device__ __forceinline__ uint32_t fc_kv_off(int key, int c) {
    return (uint32_t)((key >> 3) * FC_GROUP + (c >> 3) * FC_HALF + (key & 7) * 128 + (((c & 7) ^ (key & 7)) << 4));
}
// D += A B with A in tensor memory (a lane a row, two 16-bit elements along K a column); see fc_mma_ss.
__device__ __forceinline__ void fc_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(lead) : "memory");
}
// Sixteen 32-bit columns of this warp's 32 lanes back into tensor memory (the counterpart of tc_ld16).
__device__ __forceinline__ void fc_st16(uint32_t taddr, const uint32_t* r) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]) : "memory");
}
__device__ __forceinline__ void fc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// An issuing warp runs its loop with all lanes (addresses and descriptors are the same in all of them, so they live in
// uniform registers) and one lane issues: the instruction carries the predicate itself, no branch surrounds it.  A loop
// run by one lane alone cost well over a hundred clocks per MMA in moving its operands into uniform registers, and
// the tensor pipe waited for the issuing thread.
__device__ __forceinline__ void fc_mma_ss(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(lead) : "memory");
}
__device__ __forceinline__ void fc_commit_lead(uint32_t bar, uint32_t lead) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
        ::"r"(bar), "r"(lead) : "memory");
}

// 2^x by the special-function unit alone: one instruction (exp2f adds range handling around it, and so does
// ex2.approx without .ftz: a compare and two multiplications per call for results below 2^-126, which are flushed to
// zero here - P is rounded to bfloat16 anyway).  Accurate to two units in the last place.  The arguments that count are at most
// FC_RESCALE, or -inf; a pass against an old maximum may see any larger one and overflow: such a maximum moves, and the pass
// is done again.
__device__ __forceinline__ float fc_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Two floats in a 64-bit register pair, for the packed instructions (one issue slot for two results, each rounded as the
// scalar instruction rounds it).
__device__ __forceinline__ unsigned long long fc_pair(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ void fc_unpair(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long fc_fma2(unsigned long long x, unsigned long long y, unsigned long long z) {
    unsigned long long v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(x), "l"(y), "l"(z));
    return v;
}
__device__ __forceinline__ unsigned long long fc_add2(unsigned long long x, unsigned long long y) {
    unsigned long long v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(x), "l"(y));
    return v;
}
__device__ __forceinline__ float fc_max3(float x, float y, float z) {
    float v;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(v) : "f"(x), "f"(y), "f"(z));
    return v;
}
__device__ __forceinline__ uint32_t fc_pack(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// try_wait with a suspend-time hint: the thread sleeps in the barrier unit until the phase completes or the time is
// up, and issues nothing meanwhile.  (A bare poll loop spins: a waiting warp was seen to execute a fifth of all the
// kernel's instructions, taking issue slots from the row warps on its scheduler.)
__device__ __forceinline__ bool fc_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity), "r"(20000u) : "memory");
    return ok != 0;
}
// The bounded wait of sm100.cuh on top of it.
__device__ __forceinline__ bool fc_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int where) {
    if (fc_try(bar, parity)) return true;
    unsigned long long t0 = 0;
    for (uint32_t it = 0; it < RB_SPIN_LIMIT; ++it) {
        if (fc_try(bar, parity)) return true;
        if ((it & 7u) == 7u) {
            if (*abort_flag) return false;
            const unsigned long long now = rb_globaltimer();
            if (t0 == 0) t0 = now;
            else if (now - t0 > RB_WAIT_NS) break;
        }
    }
    *abort_flag = where;
    rb_raise(where);
    return false;
}

// With -DRB_TIMELINE lane 0 of every warp adds up, over the key tiles of its CTA, the cycles it spent in each of its
// waits and in its own work, into the buffer of rb_fa_tc_trace(): [warp][8] sums over all CTAs (atomics) and, in word 7
// of a warp's row, the number of (CTA, key tile) pairs counted.  A development aid: where a key tile's time goes.
#ifdef RB_TIMELINE
__device__ unsigned long long* g_fc_trace = nullptr;
extern "C" int rb_fa_tc_trace(unsigned long long* buf) { return (int)cudaMemcpyToSymbol(g_fc_trace, &buf, sizeof(buf)); }
#define FC_T0() const long long fc_t0 = clock64()
#define FC_ADD(slot) do { fc_acc[slot] += clock64() - fc_t0; } while (0)
#define FC_FLUSH(n) do { if (g_fc_trace && lane == 0) { for (int q = 0; q < 7; ++q) atomicAdd(g_fc_trace + warp * 8 + q, (unsigned long long)fc_acc[q]); \
                         atomicAdd(g_fc_trace + warp * 8 + 7, (unsigned long long)(n)); } } while (0)
#else
#define FC_T0() do { } while (0)
#define FC_ADD(slot) do { } while (0)
#define FC_FLUSH(n) do { } while (0)
#endif

// OPTIONS: which options on the scores there may be (FC_CAP | FC_PENALTY | FC_BIAS).  They are instantiations because their
// unrolled code would stand in the rows' loop: with all of it there the loop did not fit the instruction cache and the rows
// spent a fifth of a key tile fetching code that they jumped over.
#define FC_CAP 1
#define FC_PENALTY 2
#define FC_BIAS 4
template <int OPTIONS>
__global__ void __launch_bounds__(FC_THREADS, 1)
fa_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_kv, const FcArgs a) {
    RB_TL(11);
    if (*(volatile int*)&g_rb_kernel_error) return;                // an earlier wait gave up: fail fast, the host sees the word
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* stages = smem;                                  // [FC_SLOTS]
    unsigned char* sQ = stages + FC_SLOTS * FC_KV_BYTES;           // [row tile][two halves of [128 rows][64 dims]]
    FcShared* sh = (FcShared*)(sQ + FC_TILES * 2 * FC_QHALF);
    const uint32_t stages_u = smem_u32(stages), sQ_u = smem_u32(sQ);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int* abort_flag = &sh->abort_flag;

    if (threadIdx.x == 0) {
        for (int s = 0; s < FC_SLOTS; ++s) {
            mbar_init(smem_u32(&sh->full[s]), 1);
            sh->uses[s] = 0;
        }
        for (int s = 0; s < FC_RING; ++s) mbar_init(smem_u32(&sh->done[s]), 2);
        for (int t = 0; t < FC_TILES; ++t) {
            for (int b = 0; b < 2; ++b) {
                mbar_init(smem_u32(&sh->s_full[t][b]), 1);
                mbar_init(smem_u32(&sh->p_full[t][b]), 4);         // one arrival per row warp: P is written
            }
            for (int b = 0; b < 2; ++b) mbar_init(smem_u32(&sh->o_full[t][b]), 1);
        }
        sh->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh->tmem_base)), "r"(FC_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // Nothing that a copy or a thread of this CTA did not write reaches the results: value rows at or beyond the
    // request's length are zeroed before use, scores of such keys and of rows without a token are replaced by
    // -inf whatever they are, P is written whole before it is read.
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    pdl_trigger();
    pdl_wait();

    // which rows: heavy CTAs (late in a request: more keys) first
    const int tpt = FC_ROWS / a.Gc;                                // tokens per row tile
    const int tpc = FC_TILES * tpt;                                // tokens per CTA
    int tile = (int)gridDim.y - 1 - (int)blockIdx.y, e = a.first_entry, q_len = 0;   // CTAs start in order of x, then y
    for (; e < a.first_entry + a.n_entries; ++e) {
        q_len = a.cu_q[e + 1] - a.cu_q[e];
        const int nt = (q_len + tpc - 1) / tpc;
        if (tile < nt) break;
        tile -= nt;
    }
    const bool none = e >= a.first_entry + a.n_entries;            // uniform: a CTA beyond the last entry
    int n_tiles = 0, q0 = 0, n_tok = 0, kv_end = 0, start_pos = 0, tok_base = 0, t_begin = 0, head0 = 0, kh = 0;
    const int* bt = a.block_table;
    if (!none) {
        q0 = tile * tpc;
        n_tok = min(tpc, q_len - q0);                              // tokens of this CTA: the first tpt in tile A, the rest in B
        kh = blockIdx.x / a.chunks;
        head0 = kh * (a.QH / a.KH) + (blockIdx.x % a.chunks) * a.Gc;
        kv_end = a.kv_len[e];
        start_pos = kv_end - q_len;
        tok_base = a.cu_q[e] + q0;
        bt = a.block_table + (size_t)e * a.max_pages;
        const int pos_min = start_pos + q0, pos_max = start_pos + q0 + n_tok - 1;
        int lo_min = a.window > 0 ? max(0, pos_min - a.window + 1) : 0;
        if (a.chunk > 0) lo_min = max(lo_min, pos_min / a.chunk * a.chunk);
        t_begin = lo_min / FC_BN;
        n_tiles = pos_max / FC_BN + 1 - t_begin;
        // Q rows (row r of the CTA = token r / Gc, grouped head r % Gc; rows 128.. are tile B) into the swizzled K-major layout
        for (int i = threadIdx.x; i < n_tok * a.Gc * (FC_D / 8); i += FC_THREADS) {
            const int row = i / (FC_D / 8), c = i % (FC_D / 8);
            const uint4 v = *reinterpret_cast<const uint4*>(a.q + ((size_t)(tok_base + row / a.Gc) * a.QH + head0 + row % a.Gc) * FC_D + c * 8);
            *reinterpret_cast<uint4*>(sQ + (row >> 7) * 2 * FC_QHALF + fc_off(row & 127, c, FC_QHALF)) = v;
        }
        if (a.window > 0) {
            // With a window the first key tile of a row block may hold pages that went back to the pool: their copies
            // are skipped and their keys masked, but the values at those places are multiplied all the same (by P = 0,
            // and 0 x NaN is NaN).  So the slots start as zeros; what a later use leaves there is this request's own
            // finite data.
            for (int i = threadIdx.x; i < FC_SLOTS * (FC_KV_BYTES / 16); i += FC_THREADS)
                *reinterpret_cast<uint4*>(stages + i * 16) = make_uint4(0, 0, 0, 0);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();

    [[maybe_unused]] long long fc_acc[7] = {0, 0, 0, 0, 0, 0, 0};
    if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");           // the control group gives registers up ...
    if (warp == 0) {
        // ---- producer: keys 0, keys 1, values 0, keys 2, values 1, ... each into its ring.
        // Block-table entries 32 at a time, in windows that begin at multiples of 32, which a tile's pages (eight at most) never
        // cross: the window of the keys, the one before it (values lie up to 24 pages behind the keys that went out before them), and
        // the one after it, asked for a window ahead of its use.
        const int box_keys = min(a.page_size, FC_BN);              // keys that one request brings
        const int subs = FC_BN / box_keys;
        const uint32_t lead = lane == 0 ? 1u : 0u;
        auto entries = [&](int w) { return w * 32 + lane < a.max_pages ? bt[w * 32 + lane] : -1; };
        int window = ((t_begin * FC_BN) >> a.page_shift) >> 5;
        int before = -1, here = entries(window), after = entries(window + 1);
        bool ok = true;
        for (int step = 0; step < 2 * n_tiles + 2 && ok; ++step) {
            const int values = step >= 2 && !(step & 1), tile = values ? step / 2 - 1 : (step + 1) / 2;
            if (tile < n_tiles) {
                const int k0 = (t_begin + tile) * FC_BN;
                const int own = (k0 >> a.page_shift) >> 5;         // (a tile is at most eight pages behind the last: one window further)
                if (own > window) { before = here; here = after; after = entries(++window + 1); }
                const int s = values ? FC_VSLOT(tile) : FC_KSLOT(tile), use = tile / FC_RING;
                const uint32_t full = smem_u32(&sh->full[s]);
                const uint32_t dst0 = stages_u + s * FC_KV_BYTES;
                // A lane for each page of this tile, which makes the page's request itself, all in one instruction.  (Lane 0 making them
                // one after the other took some 200 cycles a request: 16 of them per 64 keys and values in pages of 8 keys are more than
                // the products and rows need.  32 query over 8 kv heads, 2,048 tokens behind 14,336 others: pages of 8 keys 548 us, of
                // 16 and 64 473; one after the other 951, 652 and 531 with P in shared memory, 618, 526 and 525 in one instruction.)
                const int my_key = k0 + lane * box_keys;
                const int my_page = __shfl_sync(0xffffffffu, own == window ? here : before, (my_key >> a.page_shift) & 31);
                const uint32_t there = __ballot_sync(0xffffffffu, lane < subs && my_key < kv_end && my_page >= 0);
                const int my_index = (my_page * 2 + values) * a.KH + kh, grp = (k0 & (a.page_size - 1)) >> 3;
                // What was here before has been used: keys by the scores of the tile FC_RING before, values by that tile's weighted sum,
                // which goes with the scores two tiles on.
                const int user = values ? tile - FC_RING + 2 : tile - FC_RING;
                { FC_T0(); if (use && !fc_wait(smem_u32(&sh->done[user % FC_RING]), FC_PHASE(user), abort_flag, 11)) { ok = false; break; } FC_ADD(0); }
                FC_T0();
                mbar_expect_tx_lead(full, (uint32_t)(__popc(there) * box_keys * 256), lead);
                __syncwarp();                                      // the barrier expects the bytes before the first of them can arrive
                tma_load_5d_lead(dst0 + (uint32_t)((lane & 7) * (box_keys >> 3) * FC_GROUP), &map_kv, 0, 0, 0, grp, my_index, full, (there >> lane) & 1u);
                if (lead) sh->uses[s] = use + 1;
                FC_ADD(1);
            }
        }
        FC_FLUSH(n_tiles);
    } else if (warp == 1 || warp == 3) {
        // ---- issuers, one warp per row tile: every lane runs the loop, lane 0's instructions take effect
        // O_t += P_t(i) V(i) once the rows have written P, then S_t(i + 2) = Q_t K(i + 2)^T into the columns that P(i) lay in: one warp
        // issues both, and the products of one issuer run in the order they were issued in, so nothing waits between them.  d =
        // 128 is two 64-column halves of four 16-wide steps each; the keys' 8-row groups lie 2,048 bytes apart, their second half
        // 1,024 bytes on.  V [keys][d] as it lies in its slot is an MN-major operand: a key's 64 dims (128 bytes) contiguous, keys
        // 128 bytes apart, groups of 8 keys 2,048 bytes apart (SBO), the second 64 dims 1,024 bytes on (LBO); an MMA takes 16 keys =
        // two groups of V and eight columns of P.  (One warp for both row tiles had twice the products and commits to issue, about 65
        // cycles each: more than the products take to run.)
        const uint32_t lead = lane == 0 ? 1u : 0u;
        const int t = warp == 1 ? 0 : 1;
        constexpr uint32_t idesc_s = make_idesc(FC_BN), idesc_mn = make_idesc(FC_D) | (1u << 16);      // B of the weighted sum is MN-major
        const uint64_t dq0 = make_smem_desc(sQ_u + (t * 2) * FC_QHALF), dq1 = make_smem_desc(sQ_u + (t * 2 + 1) * FC_QHALF);
        // Whether keys and values have landed is asked while the products before theirs are issued: a wait costs over a hundred
        // cycles however long ago the bytes came, and the tensor pipe runs dry meanwhile.
        bool keys_there = false, values_there = false;
        auto scores = [&](int i) -> bool {
            const int s = FC_KSLOT(i);
            { FC_T0(); if (!keys_there && !fc_wait(smem_u32(&sh->full[s]), FC_PHASE(i), abort_flag, 12)) return false; FC_ADD(0); }
            FC_T0();
            const uint32_t sK = stages_u + s * FC_KV_BYTES;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint64_t dq = h ? dq1 : dq0;
                const uint64_t dk = make_smem_desc_lbo_sbo(sK + h * FC_HALF, 16, FC_GROUP);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    fc_mma_ss(tmem + FC_S(t, i), dq + (uint64_t)(k * 2), dk + (uint64_t)(k * 2), idesc_s, (h | k) != 0, lead);
            }
            fc_commit_lead(smem_u32(&sh->s_full[t][i & 1]), lead);
            FC_ADD(2);
            return true;
        };
        auto done = [&](int i) { fc_commit_lead(smem_u32(&sh->done[i % FC_RING]), lead); };
        bool ok = n_tiles < 1 || scores(0);
        if (ok) done(0);
        ok = ok && (n_tiles < 2 || scores(1));
        if (ok) done(1);
        for (int i = 0; i < n_tiles && ok; ++i) {
            const int s = FC_VSLOT(i);
            const uint32_t par = (uint32_t)((i >> 1) & 1);
            { FC_T0(); if (!values_there && !fc_wait(smem_u32(&sh->full[s]), FC_PHASE(i), abort_flag, 21)) break; FC_ADD(1); }
            { FC_T0(); if (!fc_wait(smem_u32(&sh->p_full[t][i & 1]), par, abort_flag, 13)) break; FC_ADD(3); }
            // the request's last values: rows of tile A have set what lies behind them to zero before they said that P is there
            if (t == 1 && (t_begin + i + 1) * FC_BN > kv_end && !fc_wait(smem_u32(&sh->p_full[0][i & 1]), par, abort_flag, 20)) break;
            FC_T0();
            tc_fence_after();
            const uint64_t dv = make_smem_desc_lbo_sbo(stages_u + s * FC_KV_BYTES, FC_HALF, FC_GROUP);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                fc_mma_ts(tmem + FC_O(t), tmem + FC_S(t, i) + (uint32_t)(k * 8), dv + (uint64_t)(k * ((2 * FC_GROUP) >> 4)), idesc_mn, (i > 0) || k != 0, lead);
                if (k == 0) {
                    keys_there = i + 2 < n_tiles && mbar_test(smem_u32(&sh->full[FC_KSLOT(i + 2)]), FC_PHASE(i + 2));
                    values_there = i + 1 < n_tiles && mbar_test(smem_u32(&sh->full[FC_VSLOT(i + 1)]), FC_PHASE(i + 1));
                }
            }
            if (i + 2 >= n_tiles) fc_commit_lead(smem_u32(&sh->o_full[t][i + 1 == n_tiles]), lead);
            FC_ADD(2);
            if (i + 2 < n_tiles && !scores(i + 2)) break;
            done(i + 2);
        }
        FC_FLUSH(n_tiles);
    }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");      // ... and the rows take them
        // ---- softmax rows: thread = row = tensor-memory lane; group t owns row tile t through all key tiles ----------
        const int t = (warp - 4) >> 2;
        const int quad = warp & 3;                                 // the lanes this warp may read: 32 * (warp % 4) ..
        const int row = quad * 32 + lane;                          // row of the tile
        const int ti = t * tpt + row / a.Gc;                       // token of the CTA
        const bool live = !none && ti < n_tok;
        const int pos = live ? start_pos + q0 + ti : -1;
        int lo = a.window > 0 ? max(0, pos - a.window + 1) : 0;
        if (a.chunk > 0) lo = max(lo, max(pos, 0) / a.chunk * a.chunk);
        // the distance penalty of this row's head, in units of the raw score (the scale is applied to the difference)
        const bool pen = (OPTIONS & FC_PENALTY) && a.r1 != nullptr;
        const float pen_a = pen ? a.r1[head0 + row % a.Gc] / a.scale_log2 : 0.0f, pen_b = pen ? a.r2[head0 + row % a.Gc] : 0.0f;
        // the bias by distance of this row's head, in units of the raw score like the penalty; a tile whose keys all lie
        // at least bias_last behind the row gets one constant
        const float* brow = (OPTIONS & FC_BIAS) && a.bias ? a.bias + (size_t)(head0 + row % a.Gc) * (a.bias_last + 1) : nullptr;
        const float bias_unit = 1.4426950408889634f / a.scale_log2;
        const float bias_far = brow ? brow[a.bias_last] * bias_unit : 0.0f;
        // m: the maximum that P and O are scaled to (it follows the true maximum only in steps larger than
        // FC_RESCALE, so that O can stay in tensor memory and be accumulated by the MMA itself); l: the sum in that scale
        float m = -INFINITY, l = 0.0f;
        const uint32_t lane_base = tmem + ((uint32_t)(quad * 32) << 16);
        const uint32_t o_col = FC_O(t);
        bool ok = true;
        for (int it = 0; it < n_tiles && ok; ++it) {
            // S: this row's 64 scores in one go (one wait for tensor memory)
            const int b = it & 1, k0 = (t_begin + it) * FC_BN;
            uint32_t sr[FC_BN];
            { FC_T0(); if (!fc_wait(smem_u32(&sh->s_full[t][b]), (uint32_t)((it >> 1) & 1), abort_flag, 15)) { ok = false; break; } FC_ADD(0); }
#ifdef RB_TIMELINE
            const long long fc_tile0 = clock64();
#endif
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < FC_BN / 16; ++c) tc_ld16(lane_base + FC_S(t, it) + (uint32_t)(c * 16), sr + c * 16);
            tc_ld_wait();
#ifdef RB_TIMELINE
            fc_acc[1] += clock64() - fc_tile0;
#endif
            const bool edge = k0 + FC_BN - 1 > pos || k0 < lo;     // these keys cross this row's causal edge or window
            if ((OPTIONS & FC_CAP) && a.cap_raw > 0.0f) {
                // tanh z = 1 - 2 / (e^(2z) + 1): one exponential and one reciprocal of the special-function unit, exact
                // at both ends (e = inf gives 1, e = 0 gives -1); the error is an absolute 2^-23 or so of the cap
#pragma unroll
                for (int j = 0; j < FC_BN; ++j) {
                    const float e2 = fc_ex2(__uint_as_float(sr[j]) * a.cap_arg);
                    sr[j] = __float_as_uint(fmaf(-a.cap_raw, __fdividef(2.0f, e2 + 1.0f), a.cap_raw));
                }
            }
            if (pen) {                                             // (places beyond the row's position are replaced below)
                const float dist0 = (float)(pos - k0);
#pragma unroll
                for (int j = 0; j < FC_BN; ++j)
                    sr[j] = __float_as_uint(fmaf(-pen_a, __log2f(fmaf(pen_b, dist0 - (float)j, 1.0f)), __uint_as_float(sr[j])));
            }
            if (brow) {
                const int d0 = pos - k0;                           // distance of the tile's first key (a dead row: below zero)
                if (d0 - (FC_BN - 1) >= a.bias_last) {
#pragma unroll
                    for (int j = 0; j < FC_BN; ++j) sr[j] = __float_as_uint(__uint_as_float(sr[j]) + bias_far);
                } else {
#pragma unroll
                    for (int j = 0; j < FC_BN; ++j) {
                        const int dist = min(max(d0 - j, 0), a.bias_last);
                        sr[j] = __float_as_uint(fmaf(brow[dist], bias_unit, __uint_as_float(sr[j])));
                    }
                }
            }
            if (edge) {
#pragma unroll
                for (int j = 0; j < FC_BN; ++j) {
                    const int key = k0 + j;
                    if (key < lo || key > pos) sr[j] = 0xff800000u;            // -inf
                }
            }
            if (t == 0 && k0 + FC_BN > kv_end) {
                // the request's last keys: slots of its last page beyond its length hold foreign data - the values
                // there are zeroed before the tensor core multiplies them (by P = 0, but 0 x NaN is NaN).  The rows of
                // tile A do it, and the issuer of tile B's product waits for them.  (Scores of this tile stand behind the product of the
                // tile two before, so this slot's barrier cannot be two phases behind.)
                const int s = FC_VSLOT(it);
                if (!fc_wait(smem_u32(&sh->full[s]), FC_PHASE(it), abort_flag, 14)) { ok = false; break; }
                unsigned char* sV = stages + s * FC_KV_BYTES;
                for (int i = row; i < FC_BN * 16; i += FC_ROWS) {
                    const int r = i / 16, c = i % 16;
                    if (k0 + r >= kv_end) *reinterpret_cast<uint4*>(sV + fc_kv_off(r, c)) = make_uint4(0, 0, 0, 0);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the zeros, before the tensor core reads the values
            }
            // P = 2^(S * scale - base), rounded to bfloat16, two a register; its row sum; and, beside the exponentials (nothing
            // here waits for it), the maximum of the raw scores in `top`
            uint32_t pr[FC_BN / 2];
            float top = -INFINITY;
            auto emit = [&](float base) -> float {
                unsigned long long sum2[2] = {0ull, 0ull};             // four running sums, packed in pairs
                float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
                const unsigned long long scale2 = fc_pair(a.scale_log2, a.scale_log2), base2 = fc_pair(-base, -base);
#pragma unroll
                for (int c = 0; c < FC_BN / 8; ++c) {
                    float p[8];
#pragma unroll
                    for (int j = 0; j < 8; j += 2) {
                        const float s0 = __uint_as_float(sr[c * 8 + j]), s1 = __uint_as_float(sr[c * 8 + j + 1]);
                        mx4[j >> 1] = fc_max3(mx4[j >> 1], s0, s1);
                        fc_unpair(fc_fma2(fc_pair(s0, s1), scale2, base2), p[j], p[j + 1]);
                        p[j] = fc_ex2(p[j]);
                        p[j + 1] = fc_ex2(p[j + 1]);
                        sum2[(j >> 1) & 1] = fc_add2(sum2[(j >> 1) & 1], fc_pair(p[j], p[j + 1]));
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) pr[c * 4 + j] = fc_pack(p[2 * j], p[2 * j + 1]);
                }
                top = fmaxf(fc_max3(mx4[0], mx4[1], mx4[2]), mx4[3]);
                float s0, s1, s2, s3;
                fc_unpair(sum2[0], s0, s1);
                fc_unpair(sum2[1], s2, s3);
                return (s0 + s1) + (s2 + s3);
            };
            // The scale m follows the true maximum only when that rose by more than FC_RESCALE (P then stays below
            // 2^FC_RESCALE, which bfloat16 and the float accumulators hold as well as values below 1).  So in nearly every
            // tile the old scale stays, and the exponentials need not wait for this tile's maximum: both are computed side
            // by side, and only a warp in which some row's scale has to move (always in a row's first tile) does its
            // exponentials again.
#ifdef RB_TIMELINE
            const long long fc_c5 = clock64();
#endif
            // (one copy of the exponentials' code, run once or twice: see OPTIONS)
            float sum = 0.0f;
#pragma unroll 1
            for (int again = 0; ; ++again) {
                sum = emit(m == -INFINITY ? 0.0f : m);
                const float mx = top * a.scale_log2;               // the scale is positive
                const bool moves = (m == -INFINITY) ? (mx != -INFINITY) : (mx > m + FC_RESCALE);
                if (again || !__any_sync(0xffffffffu, moves)) break;
                float alpha = 1.0f;
                if (m == -INFINITY) m = mx;
                else if (moves) { alpha = fc_ex2(m - mx); m = mx; }
                l *= alpha;
                if (it == 0 || !__any_sync(0xffffffffu, alpha != 1.0f)) continue;
                // rare: O = O * alpha in tensor memory, every lane of the warp with its own factor (1 for most); the
                // product of the 64 keys before (the last one that can have been issued) must have landed in O first
                // (the next tile's scores, issued behind it, say so; behind the last tile there are none)
                if (it + 1 < n_tiles ? !fc_wait(smem_u32(&sh->s_full[t][b ^ 1]), (uint32_t)(((it + 1) >> 1) & 1), abort_flag, 18)
                                     : !fc_wait(smem_u32(&sh->o_full[t][0]), 0u, abort_flag, 16)) { ok = false; break; }
                tc_fence_after();
#pragma unroll 1
                for (int c = 0; c < FC_D / 32; ++c) {
                    uint32_t ov[32];
                    tc_ld16(lane_base + o_col + (uint32_t)(c * 32), ov);
                    tc_ld16(lane_base + o_col + (uint32_t)(c * 32 + 16), ov + 16);
                    tc_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) ov[j] = __float_as_uint(__uint_as_float(ov[j]) * alpha);
                    fc_st16(lane_base + o_col + (uint32_t)(c * 32), ov);
                    fc_st16(lane_base + o_col + (uint32_t)(c * 32 + 16), ov + 16);
                }
                fc_st_wait();
            }
            if (!ok) break;
#ifdef RB_TIMELINE
            fc_acc[5] += clock64() - fc_c5;
#endif
            l += sum;
#ifdef RB_TIMELINE
            const long long fc_c6 = clock64();
#endif
            fc_st16(lane_base + FC_S(t, it), pr);                  // over the scores, which are in registers
            fc_st16(lane_base + FC_S(t, it) + 16u, pr + 16);
            fc_st_wait();
            tc_fence_before();                                     // P (and O, if touched) is written: the product may go on
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&sh->p_full[t][b]));
#ifdef RB_TIMELINE
            fc_acc[6] += clock64() - fc_c6;
#endif
#ifdef RB_TIMELINE
            fc_acc[4] += clock64() - fc_tile0;
#endif
        }
        FC_FLUSH(n_tiles);
        // the row of O, once the last product is done
        if (ok && n_tiles > 0) ok = fc_wait(smem_u32(&sh->o_full[t][1]), 0u, abort_flag, 17);
        if (ok && n_tiles > 0 && !*abort_flag) {
            // (the loads from tensor memory are the whole warp's: every lane takes part, only live rows store)
            tc_fence_after();
            if (a.sink && m != -INFINITY) l += fc_ex2(fmaf(a.sink[head0 + row % a.Gc], 1.4426950408889634f, -m));   // in the scale of l
            float inv = l > 0.0f ? a.out_scale / l : 0.0f;
            if (a.gate && a.gate_heads && live) inv /= 1.0f + expf(-a.gate[(size_t)(tok_base + ti) * a.gate_stride + head0 + row % a.Gc]);
            bf16* dst = a.out + ((size_t)(tok_base + (live ? ti : 0)) * a.QH + head0 + row % a.Gc) * FC_D;
            const float* grow = (a.gate && !a.gate_heads && live) ? a.gate + (size_t)(tok_base + ti) * a.gate_stride + (size_t)(head0 + row % a.Gc) * FC_D : nullptr;
#pragma unroll
            for (int c = 0; c < FC_D / 32; ++c) {
                uint32_t ov[32];
                tc_ld16(lane_base + o_col + (uint32_t)(c * 32), ov);
                tc_ld16(lane_base + o_col + (uint32_t)(c * 32 + 16), ov + 16);
                tc_ld_wait();
                if (!live) continue;
                if (grow) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) ov[j] = __float_as_uint(__uint_as_float(ov[j]) / (1.0f + expf(-grow[c * 32 + j])));
                }
#pragma unroll
                for (int q4 = 0; q4 < 4; ++q4) {
                    uint4 pk;
                    pk.x = fc_pack(__uint_as_float(ov[q4 * 8 + 0]) * inv, __uint_as_float(ov[q4 * 8 + 1]) * inv);
                    pk.y = fc_pack(__uint_as_float(ov[q4 * 8 + 2]) * inv, __uint_as_float(ov[q4 * 8 + 3]) * inv);
                    pk.z = fc_pack(__uint_as_float(ov[q4 * 8 + 4]) * inv, __uint_as_float(ov[q4 * 8 + 5]) * inv);
                    pk.w = fc_pack(__uint_as_float(ov[q4 * 8 + 6]) * inv, __uint_as_float(ov[q4 * 8 + 7]) * inv);
                    reinterpret_cast<uint4*>(dst)[c * 4 + q4] = pk;
                }
            }
            tc_fence_before();
        } else if (ok && live && n_tiles == 0) {
            // a row without a single key (cannot happen for a causal row, which sees itself): zeros
            bf16* dst = a.out + ((size_t)(tok_base + ti) * a.QH + head0 + row % a.Gc) * FC_D;
            for (int c = 0; c < FC_D / 8; ++c) reinterpret_cast<uint4*>(dst)[c] = make_uint4(0, 0, 0, 0);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0) {
        // copies that were issued but never consumed still write this CTA's shared memory: wait for them
        for (int s = 0; s < FC_SLOTS; ++s)
            if (sh->uses[s]) mbar_drain(smem_u32(&sh->full[s]), (uint32_t)((sh->uses[s] - 1) & 1));
    }
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(FC_TMEM_COLS) : "memory");
    }
}

template <int OPTIONS>
static int fc_launch(dim3 grid, size_t smem, cudaStream_t s, const CUtensorMap& map, const FcArgs& a) {
    static RbPerDevice limit;
    if (int e = rb_allow_shared(limit, fa_prefill_tc_kernel<OPTIONS>, smem)) return e;
    return rb_launch(fa_prefill_tc_kernel<OPTIONS>, grid, dim3(FC_THREADS), smem, s, map, a);
}

// q [T, QH, 128] bfloat16; cache: one layer's [num_pages, 2, KH, page_size, 128]; entries first_entry .. bring
// cu_q[e+1] - cu_q[e] tokens each and hold kv_len[e] tokens after this step.  n_tiles: the sum over these
// entries of ceil(tokens / (256 / Gc)), Gc = the largest of 16, 8, 4, 2, 1 that divides QH / KH.
extern "C" int rb_fa_prefill_tc(const void* q, const void* cache, long long num_pages, const int* block_table, const int* cu_q,
                                const int* kv_len, void* out, int first_entry, int n_entries, int n_tiles, int QH, int KH, int d,
                                int page_size, int max_pages, int window, float scale, int chunk, const float* r1, const float* r2,
                                float out_scale, const float* bias, int bias_rows, float softcap, const float* sink,
                                const float* gate, long long gate_stride, int gate_heads, void* stream) {
    if (n_entries <= 0 || n_tiles <= 0) return 0;
    if (QH <= 0 || KH <= 0 || QH % KH) RB_REFUSE("attention: %d query heads over %d kv heads", QH, KH);
    if (softcap < 0.0f || (softcap > 0.0f && !(scale > 0.0f))) RB_REFUSE("attention (tcgen05): a soft cap of %g at scale %g", (double)softcap, (double)scale);
    if (bias && bias_rows <= 0) RB_REFUSE("attention: a distance bias of %d rows", bias_rows);
    if (d != FC_D) RB_REFUSE("attention (tcgen05): head_dim %d, only 128 is built", d);
    // a chunk that starts inside a key tile would leave the tile's first keys to pages that may have gone back to the pool
    if (chunk < 0 || chunk % FC_BN || (r1 == nullptr) != (r2 == nullptr)) RB_REFUSE("attention (tcgen05): chunk %d (a multiple of %d), or half a distance penalty", chunk, FC_BN);
    int shift = -1;
    for (int s = 3; s < 16; ++s) if ((1 << s) == page_size) shift = s;
    if (shift < 0) RB_REFUSE("attention (tcgen05): page size %d is not a power of two >= 8", page_size);
    if (((uintptr_t)cache & 15) || ((uintptr_t)q & 15) || ((uintptr_t)out & 15)) RB_REFUSE("attention (tcgen05): operands must be 16-byte aligned");
    FcArgs a{};
    a.q = (const bf16*)q; a.block_table = block_table; a.cu_q = cu_q; a.kv_len = kv_len; a.out = (bf16*)out;
    a.QH = QH; a.KH = KH; a.page_size = page_size; a.page_shift = shift; a.max_pages = max_pages; a.window = window;
    const int G = QH / KH;
    a.Gc = 1;
    for (int c = 16; c >= 1; c >>= 1) if (G % c == 0) { a.Gc = c; break; }
    a.chunks = G / a.Gc; a.first_entry = first_entry; a.n_entries = n_entries;
    a.scale_log2 = scale * 1.4426950408889634f;
    a.chunk = chunk; a.r1 = r1; a.r2 = r2; a.out_scale = out_scale;
    a.bias = bias; a.bias_last = bias_rows - 1;
    if (softcap > 0.0f) { a.cap_raw = softcap / scale; a.cap_arg = 2.0f * 1.4426950408889634f * scale / softcap; }
    a.sink = sink; a.gate = gate; a.gate_stride = gate_stride; a.gate_heads = gate_heads;
    CUtensorMap map;
    if (rb_tensor_map_kv_pages(cache, num_pages, KH, page_size, &map)) return -1;
    constexpr size_t smem = (size_t)FC_SLOTS * FC_KV_BYTES + FC_TILES * 2 * FC_QHALF + sizeof(FcShared) + 1024;
    static_assert(smem <= 232448, "more than the shared memory of an SM");
    if (n_tiles > 65535) RB_REFUSE("attention (tcgen05): %d row tiles in one launch", n_tiles);
    const int options = (softcap > 0.0f ? FC_CAP : 0) | (r1 ? FC_PENALTY : 0) | (bias ? FC_BIAS : 0);
    const dim3 grid(KH * a.chunks, n_tiles);
    switch (options) {
        case 0: return fc_launch<0>(grid, smem, (cudaStream_t)stream, map, a);
        case FC_CAP: return fc_launch<FC_CAP>(grid, smem, (cudaStream_t)stream, map, a);
        case FC_PENALTY: return fc_launch<FC_PENALTY>(grid, smem, (cudaStream_t)stream, map, a);
        case FC_BIAS: return fc_launch<FC_BIAS>(grid, smem, (cudaStream_t)stream, map, a);
        default: return fc_launch<FC_CAP | FC_PENALTY | FC_BIAS>(grid, smem, (cudaStream_t)stream, map, a);
    }
}

// The group of query heads that share a CTA's rows, as rb_fa_prefill_tc chooses it, and the rows of a CTA (for the
// caller's count of CTAs: a CTA takes rows / group tokens).
extern "C" int rb_fa_prefill_tc_group(int QH, int KH) {
    if (QH <= 0 || KH <= 0 || QH % KH) return 0;
    const int G = QH / KH;
    for (int c = 16; c >= 1; c >>= 1) if (G % c == 0) return c;
    return 1;
}
extern "C" int rb_fa_prefill_tc_rows() { return FC_TILES * FC_ROWS; }

// The error word of this file's kernels (0 = none); synchronises the device.  With reset != 0 it is cleared.
RB_STATUS_EXPORTS(rb_attn_tc_error, rb_attn_tc_bind_status)

RB_TL_SETTER(rb_attn_tc_step_timeline)
