// Pointwise kernels that the statistics-free layers need: the Dynamic Tanh norm (with the
// residual sum in front, like the RMS norm of elementwise.cu), the soft cap on logits, a unary
// function on a strided block, and the per-head output stage of the recurrent mixers (unit root
// mean square over a head, weight, gate).  All arithmetic is 32-bit.
#include "common.cuh"

// ------------------------------------------------------------------ Dynamic Tanh
// x[r,:] += sum_s delta[s][r,:] (ascending s; x is float and is written back), then
// out[r,:] = tanh(alpha * x) * w + b.  No mean, no variance: nothing crosses a row.
// With row_idx the input row of output row r is row_idx[r] and x stays as it is.
template <typename TW, typename TO>
__global__ void dyt_kernel(float* __restrict__ x, const float* __restrict__ delta, int n_delta, long long delta_stride,
                           const TW* __restrict__ w, const TW* __restrict__ b, const TW* __restrict__ alpha,
                           TO* __restrict__ out, const int* __restrict__ row_idx, int h) {
    pdl_trigger();
    const float a = to_f32(alpha[0]);                   // weights never change: read before the wait
    pdl_wait();
    const int r = blockIdx.x;
    const size_t in_row = row_idx ? (size_t)row_idx[r] : (size_t)r;
    float* xr = x + in_row * h;
    const bool keep = delta && !row_idx;
    TO* o = out + (size_t)r * h;
    for (int i = threadIdx.x; i < h; i += blockDim.x) {
        float v = xr[i];
        if (delta) {
            for (int s = 0; s < n_delta; ++s) v += delta[(size_t)s * delta_stride + in_row * h + i];
            if (keep) xr[i] = v;
        }
        o[i] = from_f32<TO>(fmaf(tanhf(a * v), to_f32(w[i]), to_f32(b[i])));
    }
}

// The same for bfloat16 rows of whole 16-byte pieces: float4 loads, all on their way before the first is used, weights ahead of the wait.
// 2,048 rows of 2,048
// between two products: 6.2 us, 11.0 by elements.
#define DV_THREADS 128
template <int VPER>
__global__ void __launch_bounds__(DV_THREADS)
dyt_vec_kernel(float* __restrict__ x, const float* __restrict__ delta, int n_delta, long long delta_stride, const bf16* __restrict__ w,
               const bf16* __restrict__ b, const bf16* __restrict__ alpha, bf16* __restrict__ out, const int* __restrict__ row_idx, int h) {
    pdl_trigger();
    const float a = to_f32(alpha[0]);
    uint2 wv[VPER], bv[VPER];
#pragma unroll
    for (int k = 0; k < VPER; ++k) {
        const int i = (threadIdx.x + k * DV_THREADS) * 4;
        wv[k] = bv[k] = make_uint2(0, 0);
        if (i < h) { wv[k] = *reinterpret_cast<const uint2*>(w + i); bv[k] = *reinterpret_cast<const uint2*>(b + i); }
    }
    pdl_wait();
    const int r = blockIdx.x;
    float* xr = x + (row_idx ? (size_t)row_idx[r] : (size_t)r) * h;
    float4 v[VPER];
#pragma unroll
    for (int k = 0; k < VPER; ++k) {
        const int i = (threadIdx.x + k * DV_THREADS) * 4;
        v[k] = i < h ? *reinterpret_cast<const float4*>(xr + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (delta) {
        const float* dr = delta + (row_idx ? (size_t)row_idx[r] : (size_t)r) * h;
        for (int p = 0; p < n_delta; ++p)                              // ascending
#pragma unroll
            for (int k = 0; k < VPER; ++k) {
                const int i = (threadIdx.x + k * DV_THREADS) * 4;
                if (i < h) {
                    const float4 d = *reinterpret_cast<const float4*>(dr + (size_t)p * delta_stride + i);
                    v[k].x += d.x; v[k].y += d.y; v[k].z += d.z; v[k].w += d.w;
                }
            }
        if (!row_idx)
#pragma unroll
            for (int k = 0; k < VPER; ++k) {
                const int i = (threadIdx.x + k * DV_THREADS) * 4;
                if (i < h) *reinterpret_cast<float4*>(xr + i) = v[k];
            }
    }
#pragma unroll
    for (int k = 0; k < VPER; ++k) {
        const int i = (threadIdx.x + k * DV_THREADS) * 4;
        if (i >= h) continue;
        const float2 w0 = __bfloat1622float2(*(const __nv_bfloat162*)&wv[k].x), w1 = __bfloat1622float2(*(const __nv_bfloat162*)&wv[k].y);
        const float2 b0 = __bfloat1622float2(*(const __nv_bfloat162*)&bv[k].x), b1 = __bfloat1622float2(*(const __nv_bfloat162*)&bv[k].y);
        const __nv_bfloat162 lo = __floats2bfloat162_rn(fmaf(tanhf(a * v[k].x), w0.x, b0.x), fmaf(tanhf(a * v[k].y), w0.y, b0.y));
        const __nv_bfloat162 hi = __floats2bfloat162_rn(fmaf(tanhf(a * v[k].z), w1.x, b1.x), fmaf(tanhf(a * v[k].w), w1.y, b1.y));
        *reinterpret_cast<uint2*>(out + (size_t)r * h + i) = make_uint2(*(const uint32_t*)&lo, *(const uint32_t*)&hi);
    }
}

extern "C" int rb_dyt(float* x, const float* delta, int n_delta, long long delta_stride, const void* w, const void* b,
                      const void* alpha, int w_dtype, void* out, int out_dtype, const int* row_idx, int rows, int h,
                      void* stream) {
    if (rows <= 0) return 0;
    if (h <= 0) RB_REFUSE("dyt: width %d", h);
    cudaStream_t s = (cudaStream_t)stream;
    if (w_dtype == RB_BF16 && out_dtype == RB_BF16 && h % 4 == 0 && h <= DV_THREADS * 4 * 8 && delta_stride % 4 == 0 &&
        (((uintptr_t)x | (uintptr_t)delta) & 15) == 0 && (((uintptr_t)w | (uintptr_t)b | (uintptr_t)out) & 7) == 0) {
        const int pieces = rb_ceil_div(h, DV_THREADS * 4);
#define RB_DV(V) if (pieces <= V) return rb_launch(dyt_vec_kernel<V>, dim3(rows), dim3(DV_THREADS), 0, s, x, delta, n_delta, delta_stride, \
                                                   (const bf16*)w, (const bf16*)b, (const bf16*)alpha, (bf16*)out, row_idx, h)
        RB_DV(1); RB_DV(2); RB_DV(4); RB_DV(5); RB_DV(8);
#undef RB_DV
    }
    const int threads = h >= 2048 ? 512 : (h >= 512 ? 256 : 128);
#define RB_DYT(TW, TO) return rb_launch(dyt_kernel<TW, TO>, dim3(rows), dim3(threads), 0, s, x, delta, n_delta, delta_stride, \
                                        (const TW*)w, (const TW*)b, (const TW*)alpha, (TO*)out, row_idx, h)
    if (w_dtype == RB_F32 && out_dtype == RB_F32) RB_DYT(float, float);
    if (w_dtype == RB_BF16 && out_dtype == RB_BF16) RB_DYT(bf16, bf16);
    if (w_dtype == RB_F32 && out_dtype == RB_BF16) RB_DYT(float, bf16);
    if (w_dtype == RB_BF16 && out_dtype == RB_F32) RB_DYT(bf16, float);
#undef RB_DYT
    RB_REFUSE("dyt: dtypes %d, %d", w_dtype, out_dtype);
}

// ------------------------------------------------------------------ soft cap
// x <- cap * tanh(x / cap), in place on float rows.
__global__ void softcap_kernel(float* __restrict__ x, size_t n, float cap) {
    pdl_trigger(); pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] = cap * tanhf(x[i] / cap);
}
extern "C" int rb_softcap(float* x, long long n, float cap, void* stream) {
    if (n <= 0) return 0;
    if (!(cap > 0.0f)) RB_REFUSE("softcap: cap %f", cap);
    return rb_launch(softcap_kernel, dim3(rb_ceil_div(n, 256)), dim3(256), 0, (cudaStream_t)stream, x, (size_t)n, cap);
}

// ------------------------------------------------------------------ unary function on a strided block
// x[r, c] <- f(x[r, c]) for r < rows, c < cols, row stride ld.  kind 0: tanh.
template <typename TA>
__global__ void unary_kernel(TA* __restrict__ x, long long ld, int rows, int cols, int kind) {
    pdl_trigger(); pdl_wait();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)rows * cols) return;
    TA* p = x + (i / cols) * ld + (i % cols);
    const float v = to_f32(*p);
    *p = from_f32<TA>(kind == 0 ? tanhf(v) : v);
}
extern "C" int rb_unary(void* x, int dtype, long long ld, int rows, int cols, int kind, void* stream) {
    if (rows <= 0 || cols <= 0) return 0;
    if (kind != 0) RB_REFUSE("unary: kind %d", kind);
    const int blocks = rb_ceil_div((long long)rows * cols, 256);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == RB_F32) return rb_launch(unary_kernel<float>, dim3(blocks), dim3(256), 0, s, (float*)x, ld, rows, cols, kind);
    if (dtype == RB_BF16) return rb_launch(unary_kernel<bf16>, dim3(blocks), dim3(256), 0, s, (bf16*)x, ld, rows, cols, kind);
    RB_REFUSE("unary: dtype %d", dtype);
}

// ------------------------------------------------------------------ per-head output stage
// o [T, H, dv] float (what a recurrence read out).  For every (token, head):
//   y = o / sqrt(mean(o^2) + eps) * w * act(gate) * out_scale
// w: [dv] shared by the heads (w_heads = 0) or [H * dv] (w_heads = 1).  gate [T, H * dv] with row stride ldg;
// act 0: sigmoid, 1: silu.  One warp per (token, head); a lane sums its strided elements in ascending order.
template <typename TA>
__global__ void head_norm_gate_kernel(const float* __restrict__ o, const float* __restrict__ w, int w_heads,
                                      const TA* __restrict__ gate, long long ldg, int act, TA* __restrict__ out, long long ldo,
                                      int n_tokens, int H, int dv, float eps, float out_scale) {
    pdl_trigger(); pdl_wait();
    const long long wg = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (wg >= (long long)n_tokens * H) return;
    const int t = (int)(wg / H), hh = (int)(wg % H);
    const float* src = o + ((size_t)t * H + hh) * dv;
    float ss = 0.0f;
    for (int i = lane; i < dv; i += 32) { const float v = src[i]; ss = fmaf(v, v, ss); }
    ss = warp_sum(ss);
    const float rstd = 1.0f / sqrtf(ss / (float)dv + eps);
    const TA* g = gate + (size_t)t * ldg + (size_t)hh * dv;
    TA* dst = out + (size_t)t * ldo + (size_t)hh * dv;
    const float* wv = w + (w_heads ? (size_t)hh * dv : 0);
    for (int i = lane; i < dv; i += 32) {
        const float z = to_f32(g[i]);
        const float sg = 1.0f / (1.0f + expf(-z));
        const float gv = act == 1 ? z * sg : sg;
        dst[i] = from_f32<TA>(src[i] * rstd * wv[i] * gv * out_scale);
    }
}
// The same for bfloat16 heads of 64, 128 or 256: LANES lanes a head with PER pieces of four neighbours each, every load on its way before
// the head's sum is formed, the weight ahead of the wait.  2,048 tokens, 32 heads of 64 / 16 of 128:
// 10.3 / 10.1 us, 27.5 / 17.5 element by element.
template <int LANES, int PER>
__global__ void __launch_bounds__(128)
head_norm_gate_vec_kernel(const float* __restrict__ o, const float* __restrict__ w, int w_heads, const bf16* __restrict__ gate, long long ldg, int act,
                          bf16* __restrict__ out, long long ldo, int n_tokens, int H, float eps, float out_scale) {
    constexpr int DV = LANES * PER * 4;
    pdl_trigger();
    const long long hd = ((long long)blockIdx.x * 128 + threadIdx.x) / LANES;
    const int l = threadIdx.x % LANES;
    const bool live = hd < (long long)n_tokens * H;
    const int t = live ? (int)(hd / H) : 0, hh = live ? (int)(hd % H) : 0;
    float4 wv[PER], v[PER];
    uint2 g[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) wv[k] = *reinterpret_cast<const float4*>(w + (w_heads ? (size_t)hh * DV : 0) + (k * LANES + l) * 4);
    pdl_wait();
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const int i = (k * LANES + l) * 4;
        v[k] = *reinterpret_cast<const float4*>(o + ((size_t)t * H + hh) * DV + i);
        g[k] = *reinterpret_cast<const uint2*>(gate + (size_t)t * ldg + (size_t)hh * DV + i);
    }
    float ss = 0.0f;
#pragma unroll
    for (int k = 0; k < PER; ++k) ss += (v[k].x * v[k].x + v[k].y * v[k].y) + (v[k].z * v[k].z + v[k].w * v[k].w);
#pragma unroll
    for (int s = LANES / 2; s > 0; s >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, s);
    const float rstd = 1.0f / sqrtf(ss / (float)DV + eps);
    if (!live) return;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
        const float2 g0 = __bfloat1622float2(*(const __nv_bfloat162*)&g[k].x), g1 = __bfloat1622float2(*(const __nv_bfloat162*)&g[k].y);
        const float z[4] = {g0.x, g0.y, g1.x, g1.y}, a[4] = {v[k].x, v[k].y, v[k].z, v[k].w}, b[4] = {wv[k].x, wv[k].y, wv[k].z, wv[k].w};
        float r[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float sg = 1.0f / (1.0f + expf(-z[j]));
            r[j] = a[j] * rstd * b[j] * (act == 1 ? z[j] * sg : sg) * out_scale;
        }
        const __nv_bfloat162 lo = __floats2bfloat162_rn(r[0], r[1]), hi = __floats2bfloat162_rn(r[2], r[3]);
        *reinterpret_cast<uint2*>(out + (size_t)t * ldo + (size_t)hh * DV + (k * LANES + l) * 4) = make_uint2(*(const uint32_t*)&lo, *(const uint32_t*)&hi);
    }
}

extern "C" int rb_head_norm_gate(const float* o, const float* w, int w_heads, const void* gate, long long ldg, int act,
                                 void* out, long long ldo, int dtype, int n_tokens, int H, int dv, float eps, float out_scale,
                                 void* stream) {
    if (n_tokens <= 0) return 0;
    if (H <= 0 || dv <= 0) RB_REFUSE("head_norm_gate: %d heads of %d", H, dv);
    if (act != 0 && act != 1) RB_REFUSE("head_norm_gate: gate function %d", act);
    const int blocks = rb_ceil_div((long long)n_tokens * H, 4);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == RB_BF16 && (dv == 64 || dv == 128 || dv == 256) && ldg % 4 == 0 && ldo % 4 == 0 && (((uintptr_t)o | (uintptr_t)w) & 15) == 0 &&
        (((uintptr_t)gate | (uintptr_t)out) & 7) == 0) {
#define RB_HV(L, P) return rb_launch(head_norm_gate_vec_kernel<L, P>, dim3(rb_ceil_div((long long)n_tokens * H * L, 128)), dim3(128), 0, s, o, w, w_heads, \
                                     (const bf16*)gate, ldg, act, (bf16*)out, ldo, n_tokens, H, eps, out_scale)
        if (dv == 64) RB_HV(16, 1);
        if (dv == 128) RB_HV(32, 1);
        RB_HV(32, 2);
#undef RB_HV
    }
    if (dtype == RB_F32) return rb_launch(head_norm_gate_kernel<float>, dim3(blocks), dim3(128), 0, s, o, w, w_heads, (const float*)gate, ldg, act, (float*)out, ldo, n_tokens, H, dv, eps, out_scale);
    if (dtype == RB_BF16) return rb_launch(head_norm_gate_kernel<bf16>, dim3(blocks), dim3(128), 0, s, o, w, w_heads, (const bf16*)gate, ldg, act, (bf16*)out, ldo, n_tokens, H, dv, eps, out_scale);
    RB_REFUSE("head_norm_gate: dtype %d", dtype);
}
