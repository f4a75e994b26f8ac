// The plain attention over the paged cache: any number of new tokens per request,
// causal, grouped heads, optional window.  Keys are walked in blocks of 32 that are aligned
// to absolute positions, with one online-softmax update per block: by several warps of a
// CTA per (token, query heads of a kv head), their results added in a fixed order, where
// rows are multiples of four numbers (the second kernel below), else in ascending order by
// one warp per (token, query head).  The sequence of operations for a token depends only
// on its position and its mask, never on how the request was cut into steps, on the
// batch, or on the page size - so the same bits come out under every cut.  It is the
// attention of the 32-bit path and the yardstick of the faster bfloat16 kernels.
// Beyond the plain form it takes: a value head size of its own (dv != d), a chunk mask (a token sees the
// keys of its own chunk of `chunk` positions, counted from position 0), a logarithmic distance penalty per
// query head (score -= r1[h] * ln(1 + r2[h] * (i - j))), a learned bias by distance (score += bias[h][min(i - j,
// rows - 1)], a float table [QH, rows] whose last column stands for every greater distance), and a factor on the output.
// Further options: scores squashed to cap * tanh(score / cap) (softcap > 0); a sink per query head, a number that joins
// the softmax's denominator as exp(sink[h]) and brings no value; values that are the first dv columns of the key rows
// (v_in_k: a page then holds keys only, [KH][page_size][d]); and a gate on the output, out *= sigmoid(gate[t][h * dv + i])
// (float rows with a stride of their own).
// (reference semantics: crates/cuda/kernels/decode_gqa_kernels.cu:99-136 page lookup
//  page[t/block_len]; decode_flash_kernels.cu:212-349 max/exp/sum/PV in f32.)
#include "common.cuh"

#define RA_WARPS 4
#define RA_MAX_D 512

// q        [T, QH, d];  out [T, QH, dv]
// cache    one layer: [page][ K: [KH][page_size][d] | V: [KH][page_size][dv] ]   (dv == d: [page][2][KH][page_size][d])
// block_table [rows, max_pages] (page id of the i-th page of a request's row)
// tok_row  [T] row of block_table for token t;  positions [T] absolute position of token t
// A token at position p attends keys max(0, p-window+1) .. p  (window <= 0: all of them); with chunk > 0 also
// only keys from floor(p / chunk) * chunk on.
template <typename TA, typename TC>
__global__ void __launch_bounds__(RA_WARPS * 32)
paged_attention_ref_kernel(const TA* __restrict__ q, const TC* __restrict__ cache,
                           const int* __restrict__ block_table, const int* __restrict__ tok_row,
                           const int* __restrict__ positions, TA* __restrict__ out,
                           int QH, int KH, int d, int dv, int page_size, int max_pages, int window, float scale,
                           int chunk, const float* __restrict__ r1, const float* __restrict__ r2, float out_scale,
                           const float* __restrict__ bias, int bias_rows, float softcap, const float* __restrict__ sink,
                           int v_in_k, const float* __restrict__ gate, long long gate_stride) {
    pdl_trigger(); pdl_wait();
    extern __shared__ float qs_all[];                         // RA_WARPS * d floats
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x;
    const int hq = blockIdx.y * RA_WARPS + warp;
    if (hq >= QH) return;                                     // no block-wide barrier below
    float* qs = qs_all + warp * d;
    const TA* qp = q + ((size_t)t * QH + hq) * d;
    for (int i = lane; i < d; i += 32) qs[i] = to_f32(qp[i]);
    __syncwarp();
    const int kh = hq / (QH / KH);
    const int pos = positions[t];
    int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    if (chunk > 0) lo = max(lo, pos / chunk * chunk);
    const float pen1 = r1 ? r1[hq] : 0.0f, pen2 = r1 ? r2[hq] : 0.0f;
    const int* bt = block_table + (size_t)tok_row[t] * max_pages;
    const size_t head_stride = (size_t)page_size * d;         // one (page, k, head) tile
    const size_t vhead_stride = v_in_k ? head_stride : (size_t)page_size * dv;   // one (page, v, head) tile
    const size_t page_stride = v_in_k ? (size_t)KH * head_stride : (size_t)KH * (head_stride + vhead_stride);
    const size_t v_offset = v_in_k ? 0 : (size_t)KH * head_stride;                // values behind the keys, or inside them
    const int v_row = v_in_k ? d : dv;
    const float inv_cap = softcap > 0.0f ? 1.0f / softcap : 0.0f;

    constexpr int NACC = RA_MAX_D / 32;
    float acc[NACC];
#pragma unroll
    for (int i = 0; i < NACC; ++i) acc[i] = 0.0f;
    float m = -INFINITY, l = 0.0f;

    for (int b0 = (lo / 32) * 32; b0 <= pos; b0 += 32) {
        const int key = b0 + lane;
        bool valid = key >= lo && key <= pos;
        float s = -INFINITY;
        const TC* vrow = nullptr;
        const int page = (valid && key / page_size < max_pages) ? bt[key / page_size] : -1;
        valid = valid && page >= 0;                            // a page that is not held: an inert padding row
        if (valid) {
            const int off = key % page_size;
            const TC* krow = cache + (size_t)page * page_stride + (size_t)kh * head_stride + (size_t)off * d;
            vrow = cache + (size_t)page * page_stride + v_offset + (size_t)kh * vhead_stride + (size_t)off * v_row;
            float dot = 0.0f;
            for (int i = 0; i < d; ++i) dot = fmaf(qs[i], to_f32(krow[i]), dot);
            s = dot * scale;
            if (softcap > 0.0f) s = softcap * tanhf(s * inv_cap);
            if (r1) s -= pen1 * log1pf(pen2 * (float)(pos - key));
            if (bias) s += bias[(size_t)hq * bias_rows + min(pos - key, bias_rows - 1)];
        }
        const float bm = warp_max(s);
        if (bm == -INFINITY) continue;                         // no key in this block (warp-uniform)
        const float m_new = fmaxf(m, bm);
        const float corr = expf(m - m_new);                    // first block: exp(-inf) = 0
        const float p = valid ? expf(s - m_new) : 0.0f;
        l = l * corr + warp_sum(p);
#pragma unroll
        for (int i = 0; i < NACC; ++i) acc[i] *= corr;
        for (int j = 0; j < 32; ++j) {
            const float pj = __shfl_sync(0xffffffffu, p, j);
            const unsigned long long vj = __shfl_sync(0xffffffffu, (unsigned long long)vrow, j);
            if (vj == 0ull) continue;                          // warp-uniform
            const TC* vr = (const TC*)vj;
#pragma unroll
            for (int i = 0; i < NACC; ++i) {
                const int dim = lane + 32 * i;
                if (dim < dv) acc[i] = fmaf(pj, to_f32(vr[dim]), acc[i]);
            }
        }
        m = m_new;
    }
    if (sink) {                                                // one more term in the denominator, no value
        const float sk = sink[hq];
        const float m_new = fmaxf(m, sk);
        const float corr = expf(m - m_new);
        l = l * corr + expf(sk - m_new);
#pragma unroll
        for (int i = 0; i < NACC; ++i) acc[i] *= corr;
    }
    const float inv = l > 0.0f ? 1.0f / l : 0.0f;
    TA* op = out + ((size_t)t * QH + hq) * dv;
    const float* gp = gate ? gate + (size_t)t * gate_stride + (size_t)hq * dv : nullptr;
#pragma unroll
    for (int i = 0; i < NACC; ++i) {
        const int dim = lane + 32 * i;
        if (dim < dv) {
            float val = out_scale == 1.0f ? acc[i] * inv : acc[i] * inv * out_scale;
            if (gp) val *= 1.0f / (1.0f + expf(-gp[dim]));
            op[dim] = from_f32<TA>(val);
        }
    }
}

// The same attention with the keys of a (token, query heads of one kv head) shared out among the WARPS warps of a CTA (8; fewer for
// short masks), for head sizes that are multiples of four: warp w walks the 32-key blocks whose index is w modulo WARPS, in
// ascending order, with its own running maximum; the partial results are added in warp order.  Blocks are aligned to absolute positions, so what is
// added in which order still depends on nothing but the token's position and mask.  A lane scores one key for G query heads
// at once (rows read 16 bytes at a time, the queries broadcast from shared memory), and sums four columns of the values.
// Bound by latency: a block's 32 scores are one chain of d loads and FMAs per lane.  727 tokens in four prompts of 40 to 300, 32
// query over 8 kv heads of 128, 32 bits: the prompts and seven decode steps of four requests take 68 us a
// launch on average, with the kernel above 493.
template <typename T> __device__ __forceinline__ float4 load4(const T* p);
template <> __device__ __forceinline__ float4 load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 load4<bf16>(const bf16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
}

// G query heads of one kv head per CTA, value heads of at most 128 * NV numbers (G * NV <= 4).
template <typename TA, typename TC, int G, int NV, int WARPS>
__global__ void __launch_bounds__(WARPS * 32)
paged_attention_split_kernel(const TA* __restrict__ q, const TC* __restrict__ cache,
                             const int* __restrict__ block_table, const int* __restrict__ tok_row,
                             const int* __restrict__ positions, TA* __restrict__ out,
                             int QH, int KH, int d, int dv, int page_size, int max_pages, int window, float scale,
                             int chunk, const float* __restrict__ r1, const float* __restrict__ r2, float out_scale,
                             const float* __restrict__ bias, int bias_rows, float softcap, const float* __restrict__ sink,
                             int v_in_k, const float* __restrict__ gate, long long gate_stride) {
    pdl_trigger(); pdl_wait();
    extern __shared__ __align__(16) float rp_smem[];
    __shared__ __align__(16) float ps[WARPS][32][G];
    __shared__ const TC* rows[WARPS][32];
    __shared__ float ms[WARPS][G], ls[WARPS][G];
    float* qs = rp_smem;                                       // [G][d]
    float* parts = rp_smem + G * d;                            // [WARPS][G][dv]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x, hq0 = blockIdx.y * G;
    const TA* qp = q + ((size_t)t * QH + hq0) * d;
    for (int i = threadIdx.x; i < G * d; i += WARPS * 32) qs[i] = to_f32(qp[i]);
    __syncthreads();
    const int kh = hq0 / (QH / KH);
    const int pos = positions[t];
    int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    if (chunk > 0) lo = max(lo, pos / chunk * chunk);
    const int* bt = block_table + (size_t)tok_row[t] * max_pages;
    const size_t head_stride = (size_t)page_size * d;
    const size_t vhead_stride = v_in_k ? head_stride : (size_t)page_size * dv;
    const size_t page_stride = v_in_k ? (size_t)KH * head_stride : (size_t)KH * (head_stride + vhead_stride);
    const size_t v_offset = v_in_k ? 0 : (size_t)KH * head_stride;
    const int v_row = v_in_k ? d : dv;
    const float inv_cap = softcap > 0.0f ? 1.0f / softcap : 0.0f;

    float4 acc[G][NV];
    float m[G], l[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        m[g] = -INFINITY; l[g] = 0.0f;
#pragma unroll
        for (int n = 0; n < NV; ++n) acc[g][n] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int b = lo / 32 + ((warp - lo / 32) & (WARPS - 1)); b * 32 <= pos; b += WARPS) {
        const int key = b * 32 + lane;
        bool valid = key >= lo && key <= pos;
        const int page = (valid && key / page_size < max_pages) ? bt[key / page_size] : -1;
        valid = valid && page >= 0;
        float sc[G];
        const TC* vrow = nullptr;
        if (valid) {
            const int off = key % page_size;
            const TC* krow = cache + (size_t)page * page_stride + (size_t)kh * head_stride + (size_t)off * d;
            vrow = cache + (size_t)page * page_stride + v_offset + (size_t)kh * vhead_stride + (size_t)off * v_row;
            float dot[G];
#pragma unroll
            for (int g = 0; g < G; ++g) dot[g] = 0.0f;
#pragma unroll 8
            for (int i = 0; i < d; i += 4) {
                const float4 k4 = load4(krow + i);
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const float4 q4 = *reinterpret_cast<const float4*>(qs + g * d + i);
                    dot[g] = fmaf(q4.w, k4.w, fmaf(q4.z, k4.z, fmaf(q4.y, k4.y, fmaf(q4.x, k4.x, dot[g]))));
                }
            }
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float s = dot[g] * scale;
                if (softcap > 0.0f) s = softcap * tanhf(s * inv_cap);
                if (r1) s -= r1[hq0 + g] * log1pf(r2[hq0 + g] * (float)(pos - key));
                if (bias) s += bias[(size_t)(hq0 + g) * bias_rows + min(pos - key, bias_rows - 1)];
                sc[g] = s;
            }
        }
        __syncwarp();                                          // the block before has been read
        rows[warp][lane] = vrow;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float s = valid ? sc[g] : -INFINITY;
            const float m_new = fmaxf(m[g], warp_max(s));
            const float corr = m_new == -INFINITY ? 1.0f : expf(m[g] - m_new);
            const float p = s == -INFINITY ? 0.0f : expf(s - m_new);
            ps[warp][lane][g] = p;
            l[g] = l[g] * corr + warp_sum(p);
#pragma unroll
            for (int n = 0; n < NV; ++n) { acc[g][n].x *= corr; acc[g][n].y *= corr; acc[g][n].z *= corr; acc[g][n].w *= corr; }
            m[g] = m_new;
        }
        __syncwarp();
#pragma unroll 4
        for (int j = 0; j < 32; ++j) {
            const TC* vr = rows[warp][j];
            if (!vr) continue;                                 // warp-uniform
            float p[G];
#pragma unroll
            for (int g = 0; g < G; ++g) p[g] = ps[warp][j][g];
#pragma unroll
            for (int n = 0; n < NV; ++n) {
                const int dim = lane * 4 + n * 128;
                if (dim >= dv) continue;
                const float4 v4 = load4(vr + dim);
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    acc[g][n].x = fmaf(p[g], v4.x, acc[g][n].x);
                    acc[g][n].y = fmaf(p[g], v4.y, acc[g][n].y);
                    acc[g][n].z = fmaf(p[g], v4.z, acc[g][n].z);
                    acc[g][n].w = fmaf(p[g], v4.w, acc[g][n].w);
                }
            }
        }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (lane == 0) { ms[warp][g] = m[g]; ls[warp][g] = l[g]; }
#pragma unroll
        for (int n = 0; n < NV; ++n) {
            const int dim = lane * 4 + n * 128;
            if (dim < dv) *reinterpret_cast<float4*>(parts + (size_t)(warp * G + g) * dv + dim) = acc[g][n];
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < G * dv; i += WARPS * 32) {
        const int g = i / dv, dim = i - g * dv, hq = hq0 + g;
        float top = sink ? sink[hq] : -INFINITY;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) top = fmaxf(top, ms[w][g]);
        float sum = 0.0f, val = 0.0f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float f = ms[w][g] == -INFINITY ? 0.0f : expf(ms[w][g] - top);
            sum += f * ls[w][g];
            val += f * parts[(size_t)(w * G + g) * dv + dim];
        }
        if (sink) sum += expf(sink[hq] - top);
        val *= sum > 0.0f ? 1.0f / sum : 0.0f;
        if (out_scale != 1.0f) val *= out_scale;
        if (gate) val *= 1.0f / (1.0f + expf(-gate[(size_t)t * gate_stride + (size_t)hq * dv + dim]));
        out[((size_t)t * QH + hq) * dv + dim] = from_f32<TA>(val);
    }
}

// dv: the value heads' size (0: as d).  chunk 0: no chunk mask.  r1, r2 [QH] float: the distance penalty (null: none).
// bias [QH, bias_rows] float: the bias by distance (null: none).  softcap 0: none.  sink [QH] float (null: none).
// v_in_k != 0: the values are the first dv columns of the keys.  gate: float rows of stride gate_stride (null: none).
extern "C" int rb_paged_attention_ref(const void* q, const void* cache, int dtype,
                                      const int* block_table, const int* tok_row, const int* positions,
                                      void* out, int n_tokens, int QH, int KH, int d, int page_size,
                                      int max_pages, int window, float scale, int dv, int chunk, const float* r1,
                                      const float* r2, float out_scale, const float* bias, int bias_rows, float softcap,
                                      const float* sink, int v_in_k, const float* gate, long long gate_stride, void* stream) {
    if (n_tokens <= 0) return 0;
    if (dv <= 0) dv = d;
    if (QH <= 0 || KH <= 0 || QH % KH != 0) RB_REFUSE("attention: %d query heads over %d kv heads", QH, KH);
    if (d <= 0 || d > RA_MAX_D || dv > RA_MAX_D) RB_REFUSE("attention: head sizes %d, %d (supported: 1..%d)", d, dv, RA_MAX_D);
    if (page_size <= 0 || max_pages <= 0) RB_REFUSE("attention: page_size %d max_pages %d", page_size, max_pages);
    if (chunk < 0 || (r1 == nullptr) != (r2 == nullptr)) RB_REFUSE("attention: chunk %d, or half a distance penalty", chunk);
    if (bias && bias_rows <= 0) RB_REFUSE("attention: a distance bias of %d rows", bias_rows);
    if (v_in_k && dv > d) RB_REFUSE("attention: values inside the keys cannot be wider (%d) than the keys (%d)", dv, d);
    if (softcap < 0.0f) RB_REFUSE("attention: a soft cap of %g", (double)softcap);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype != RB_F32 && dtype != RB_BF16) RB_REFUSE("attention: dtype %d", dtype);
    // rows of four numbers at a time: a rule on sizes and alignment only, so that a token takes the same kernel under every cut
    const int group = QH / KH, most = 512 / ((dv + 127) / 128 * 128);
    const int G = group % 4 == 0 && most >= 4 ? 4 : group % 2 == 0 && most >= 2 ? 2 : 1;
    if (d % 4 == 0 && dv % 4 == 0 && ((uintptr_t)cache & (dtype == RB_F32 ? 15 : 7)) == 0 && QH / G <= 65535) {
        // How many warps share a token's keys: as there can be 32-key blocks in a chunk or a window.  Eight of which most find nothing
        // still start, and are merged (2,047 tokens, 5 heads of 80, chunks of 64 keys, 16 bits: 165 us with eight warps, 65 with two,
        // one warp a head as in the kernel at the top 92).
        int blocks = 8;
        if (chunk > 0) blocks = min(blocks, chunk % 32 ? chunk / 32 + 2 : chunk / 32);
        if (window > 0 && window < 256) blocks = min(blocks, (window + 30) / 32 + 1);
        const int warps = blocks <= 3 ? 2 : blocks <= 6 ? 4 : 8;
        const size_t smem = (size_t)(G * d + warps * G * dv) * sizeof(float);
        const dim3 grid(n_tokens, QH / G);
#define RP_LAUNCH(TT, GG) (warps == 2 ? RP_LAUNCH_W(TT, GG, 2) : warps == 4 ? RP_LAUNCH_W(TT, GG, 4) : RP_LAUNCH_W(TT, GG, 8))
#define RP_LAUNCH_W(TT, GG, WW) rb_launch(paged_attention_split_kernel<TT, TT, GG, 4 / GG, WW>, grid, dim3(WW * 32), smem, s, \
            (const TT*)q, (const TT*)cache, block_table, tok_row, positions, (TT*)out, QH, KH, d, dv, page_size, max_pages, window, scale, \
            chunk, r1, r2, out_scale, bias, bias_rows, softcap, sink, v_in_k, gate, gate_stride)
        if (dtype == RB_F32) return G == 4 ? RP_LAUNCH(float, 4) : G == 2 ? RP_LAUNCH(float, 2) : RP_LAUNCH(float, 1);
        return G == 4 ? RP_LAUNCH(bf16, 4) : G == 2 ? RP_LAUNCH(bf16, 2) : RP_LAUNCH(bf16, 1);
#undef RP_LAUNCH
#undef RP_LAUNCH_W
    }
    dim3 grid(n_tokens, rb_ceil_div(QH, RA_WARPS));
    const size_t smem = (size_t)RA_WARPS * d * sizeof(float);
    if (dtype == RB_F32)
        return rb_launch(paged_attention_ref_kernel<float, float>, grid, dim3(RA_WARPS * 32), smem, s,
            (const float*)q, (const float*)cache, block_table, tok_row, positions, (float*)out,
            QH, KH, d, dv, page_size, max_pages, window, scale, chunk, r1, r2, out_scale, bias, bias_rows,
            softcap, sink, v_in_k, gate, gate_stride);
    return rb_launch(paged_attention_ref_kernel<bf16, bf16>, grid, dim3(RA_WARPS * 32), smem, s,
            (const bf16*)q, (const bf16*)cache, block_table, tok_row, positions, (bf16*)out,
            QH, KH, d, dv, page_size, max_pages, window, scale, chunk, r1, r2, out_scale, bias, bias_rows,
            softcap, sink, v_in_k, gate, gate_stride);
}
