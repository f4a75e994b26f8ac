// The plain matrix product of the model:  C[M,N] (=|+=) A[M,K] * W[N,K]^T, both
// operands K-major as checkpoints store them, FMA on the CUDA cores in true 32-bit.
//
// It is the product of the 32-bit path of the whole model and the fallback of the
// bfloat16 path for operand types that the tensor-core kernels do not take (a weight
// kept in 32 bits beside 16-bit activations).  What order an output element's terms are
// added in depends on K and on the operands' types and alignment, never on M or on where
// the element lies in a tile: a token's result does not depend on what else is in the batch.
// (The reference uses cublasGemmEx for M>1 and a split-K gemv pair for small M,
//  crates/cuda/src/gemm.rs:226-372, crates/cuda/kernels/gemm_m1.cu:63-235.)
#include "common.cuh"

#define RG_BM 64
#define RG_BN 64
#define RG_BK 16

// Any operands: each output element is one chain of FMAs over k = 0..K-1 in ascending order.
// MODE 0: C = acc (type TO).  MODE 1: C(float) += acc.
template <typename TA, typename TW, typename TO, int MODE>
__global__ void __launch_bounds__(256)
gemm_ref_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TO* __restrict__ C,
                int M, int N, int K, long long lda, long long ldw, long long ldc) {
    __shared__ float As[RG_BK][RG_BM + 4];
    __shared__ float Ws[RG_BK][RG_BN + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;       // 16 x 16 threads, 4x4 outputs each
    const int m0 = blockIdx.y * RG_BM, n0 = blockIdx.x * RG_BN;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += RG_BK) {
        // 64 rows x 16 k = 1024 elements per operand, 4 per thread; k fastest for coalescing
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int idx = threadIdx.x + e * 256;
            const int r = idx >> 4, kk = idx & 15;
            const int gk = k0 + kk;
            const int gm = m0 + r, gn = n0 + r;
            As[kk][r] = (gm < M && gk < K) ? to_f32(A[(size_t)gm * lda + gk]) : 0.0f;
            Ws[kk][r] = (gn < N && gk < K) ? to_f32(W[(size_t)gn * ldw + gk]) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < RG_BK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn >= N) continue;
            TO* c = C + (size_t)gm * ldc + gn;
            if (MODE == 0) *c = from_f32<TO>(acc[i][j]);
            else *c = from_f32<TO>(to_f32(*c) + acc[i][j]);
        }
    }
}

template <typename TA, typename TW>
static int gemm_ref_dispatch(const void* A, const void* W, void* C, int c_dtype, int accumulate,
                             int M, int N, int K, long long lda, long long ldw, long long ldc, cudaStream_t s) {
    dim3 grid(rb_ceil_div(N, RG_BN), rb_ceil_div(M, RG_BM));
    if (accumulate) {
        if (c_dtype != RB_F32) RB_REFUSE("gemm: accumulation needs a float destination");
        gemm_ref_kernel<TA, TW, float, 1><<<grid, 256, 0, s>>>((const TA*)A, (const TW*)W, (float*)C, M, N, K, lda, ldw, ldc);
    } else if (c_dtype == RB_F32) {
        gemm_ref_kernel<TA, TW, float, 0><<<grid, 256, 0, s>>>((const TA*)A, (const TW*)W, (float*)C, M, N, K, lda, ldw, ldc);
    } else if (c_dtype == RB_BF16) {
        gemm_ref_kernel<TA, TW, bf16, 0><<<grid, 256, 0, s>>>((const TA*)A, (const TW*)W, (bf16*)C, M, N, K, lda, ldw, ldc);
    } else RB_REFUSE("gemm: destination dtype %d", c_dtype);
    return RB_LAUNCH_RESULT();
}

// ---- 32-bit operands that 16-byte copies can address -----------------------------------------------------------
// K is cut into F32_SEGMENTS segments (each a multiple of F32_UNIT long, the last ones shorter or empty).  Within a segment
// an output element is one chain of FMAs over ascending k from zero; the segments' sums are added in ascending order.  The
// kernels below all do exactly that, so a token has the same bits whichever of them computes it.
// The first two keep rows along K in shared memory ([row][steps of BK + 4] floats: with BK 16 or 32 eight rows' 16 bytes fall into
// eight different groups of four banks), brought by cp.async; nothing is transposed: a thread reads four consecutive k of a
// row at once.
#define F32_UNIT 32
#define F32_SEGMENTS 4

__host__ __device__ static inline int f32_segment(int K) {          // length of a segment
    const int units = (K + F32_UNIT - 1) / F32_UNIT;
    return (units + F32_SEGMENTS - 1) / F32_SEGMENTS * F32_UNIT;
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool real) {
    const int n = real ? 16 : 0;                                    // 0: the 16 bytes are filled with zeros, nothing is read
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void fma4(float& acc, const float4& a, const float4& b) {
    acc = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}

// Many tokens: a tile of BM tokens x BN features per CTA, TM x TN outputs a thread.  The segments follow one another; their
// running sum waits in shared memory.
// Bound by the FMA pipes' issue: 12 loads of 16 bytes from shared memory feed 128 FMAs with 8 x 4 outputs a thread.  727 tokens over
// 19,456 x 2,560 weights take 1.86 ms (39 TFLOP/s), over 2,560 x 9,728 1.10 ms; the kernel of 64 x 64 tiles at the top of this
// file takes 3.31 and 2.19 ms.  Measured beside it: 128 x 128 tiles of 8 x 8 outputs (2.29 ms: their registers leave 8 warps
// an SM) and packed FMAs (fma.rn.f32x2: 2.0 ms, they issue at half the rate).
#define F32_BK 16
template <int BM, int BN, int TM, int TN, int STAGES>
struct F32Tile {
    static constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY, ROW = F32_BK + 4;
    static constexpr int STAGE_FLOATS = (BM + BN) * ROW;
    static constexpr size_t SMEM = ((size_t)STAGES * STAGE_FLOATS + (size_t)BM * BN) * sizeof(float);
};

template <int BM, int BN, int TM, int TN, int STAGES, int MODE>
__global__ void __launch_bounds__(F32Tile<BM, BN, TM, TN, STAGES>::THREADS)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                     long long lda, long long ldw, long long ldc) {
    using Tile = F32Tile<BM, BN, TM, TN, STAGES>;
    constexpr int NT = Tile::THREADS, ROW = Tile::ROW;
    static_assert(Tile::TX % 8 == 0 && Tile::TY % 4 == 0, "a warp is 8 feature lanes x 4 token lanes");
    static_assert(NT % 4 == 0 && BM % (NT / 4) == 0 && BN % (NT / 4) == 0, "every thread copies as many pieces");
    extern __shared__ __align__(16) float f32_smem[];
    float* run = f32_smem + STAGES * Tile::STAGE_FLOATS + threadIdx.x;      // [TM * TN][THREADS]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tx = (warp % (Tile::TX / 8)) * 8 + (lane & 7), ty = (warp / (Tile::TX / 8)) * 4 + (lane >> 3);
    const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
    const int steps = (K + F32_BK - 1) / F32_BK, seg = f32_segment(K) / F32_BK;
    // a thread copies 16 bytes of every (NT / 4)-th row; what lies outside an operand becomes zero
    const int r0 = threadIdx.x >> 2, c0 = (threadIdx.x & 3) * 4;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(f32_smem) + (uint32_t)(r0 * ROW + c0) * 4u;
    const float* wp = W + (size_t)(n0 + r0) * ldw + c0;
    const float* ap = A + (size_t)(m0 + r0) * lda + c0;
    auto load = [&](int step) {
        const uint32_t dst = base + (uint32_t)((step % STAGES) * Tile::STAGE_FLOATS) * 4u;
        const int k = step * F32_BK;
#pragma unroll
        for (int i = 0; i < BN / (NT / 4); ++i) {
            const bool real = n0 + r0 + i * (NT / 4) < N && k + c0 < K;
            cp_async16(dst + (uint32_t)(i * (NT / 4) * ROW) * 4u, real ? wp + (size_t)(i * (NT / 4)) * ldw + k : W, real);
        }
#pragma unroll
        for (int i = 0; i < BM / (NT / 4); ++i) {
            const bool real = m0 + r0 + i * (NT / 4) < M && k + c0 < K;
            cp_async16(dst + (uint32_t)((BN + i * (NT / 4)) * ROW) * 4u, real ? ap + (size_t)(i * (NT / 4)) * lda + k : A, real);
        }
    };
    pdl_trigger();
    pdl_wait();
#pragma unroll 1
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) load(s);
        cp_async_commit();
    }
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;

#pragma unroll 1
    for (int step = 0; step < steps; ++step) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();                                            // this step has landed, and all are done with the one before
        if (step + STAGES - 1 < steps) load(step + STAGES - 1);
        cp_async_commit();
        if (step && step % seg == 0) {                              // a segment begins
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    float* r = run + (i * TN + j) * NT;
                    *r = step == seg ? acc[i][j] : *r + acc[i][j];
                    acc[i][j] = 0.0f;
                }
        }
        const float* ws = f32_smem + (step % STAGES) * Tile::STAGE_FLOATS + tx * ROW;
        const float* as = f32_smem + (step % STAGES) * Tile::STAGE_FLOATS + (BN + ty) * ROW;
#pragma unroll
        for (int k = 0; k < F32_BK; k += 4) {
            float4 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * Tile::TY * ROW + k);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const float4 b = *reinterpret_cast<const float4*>(ws + j * Tile::TX * ROW + k);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].x, b.x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].y, b.y, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].z, b.z, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].w, b.w, acc[i][j]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty + i * Tile::TY;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx + j * Tile::TX;
            if (gn >= N) continue;
            float sum = acc[i][j];
            if (steps > seg) sum = run[(i * TN + j) * NT] + sum;
            float* c = C + (size_t)gm * ldc + gn;
            *c = MODE == 0 ? sum : *c + sum;
        }
    }
}

// Few tokens (2 * TM per CTA): 16 features per CTA, warp w sums segment w.  A warp has a pipeline of its own - it copies its rows'
// next 32 k itself and waits for nobody - and is 16 feature lanes x 2 halves of the tokens; a weight that has arrived is read
// twice from shared memory.  The sums of the segments meet in shared memory.
// Bound by the stream of weights up to four tokens, then by its own loads and FMAs.  Launches back to back, 4 tokens over 151,936 x
// 2,560: 255 us (6.1 TB/s; the kernel at the top of this file 2.22 ms), 8 tokens 310 to 370; 4 tokens over 19,456 x 2,560: 39 us
// (424); over 2,560 x 9,728: 34 us (972), where 160 CTAs are too few to keep memory busy.
#define F32_ROW (F32_UNIT + 4)
template <int TM>
struct F32Few {
    static constexpr int ROWS = 16 + 2 * TM;                                // of a stage: 16 weight rows, then the tokens
    static constexpr int STAGES = TM <= 2 ? 5 : 4;                          // 52 to 58 KB a CTA
    static constexpr int STAGE_FLOATS = ROWS * F32_ROW;
    static constexpr size_t SMEM = (size_t)F32_SEGMENTS * STAGES * STAGE_FLOATS * sizeof(float);
};

template <int TM, int MODE>
__global__ void __launch_bounds__(F32_SEGMENTS * 32)
gemm_f32_few_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                    long long lda, long long ldw, long long ldc) {
    using Few = F32Few<TM>;
    constexpr int STAGES = Few::STAGES;
    extern __shared__ __align__(16) float f32_smem[];
    __shared__ float sums[F32_SEGMENTS][2 * TM][16];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n0 = blockIdx.y * 16;
    A += (size_t)blockIdx.x * (2 * TM) * lda;                       // this CTA's tokens: CTAs of the same weights are neighbours
    C += (size_t)blockIdx.x * (2 * TM) * ldc;
    M = min(M - (int)blockIdx.x * 2 * TM, 2 * TM);
    const int all = (K + F32_UNIT - 1) / F32_UNIT, seg = f32_segment(K) / F32_UNIT;
    const int first = min(warp * seg, all), steps = min(seg, all - first);
    const float* own = f32_smem + (size_t)warp * STAGES * Few::STAGE_FLOATS;
    // a lane copies 16 bytes of every fourth row: rows lane / 8 + 4 i, columns 4 (lane % 8) of a step
    const int r0 = lane >> 3, c0 = (lane & 7) * 4;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(own) + (uint32_t)(r0 * F32_ROW + c0) * 4u;
    const float* wp = W + (size_t)(n0 + r0) * ldw + first * F32_UNIT + c0;
    const float* ap = A + (size_t)r0 * lda + first * F32_UNIT + c0;
    const int k_left = K - first * F32_UNIT - c0;                     // a step's 16 bytes lie inside K while step * F32_UNIT < k_left
    auto dst = [&](int s) { return base + (uint32_t)((s % STAGES) * Few::STAGE_FLOATS) * 4u; };
    auto load_w = [&](int s) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const bool real = n0 + r0 + 4 * i < N && s * F32_UNIT < k_left;
            cp_async16(dst(s) + (uint32_t)(4 * i * F32_ROW) * 4u, real ? wp + (size_t)(4 * i) * ldw + s * F32_UNIT : W, real);
        }
    };
    auto load_a = [&](int s) {
#pragma unroll
        for (int i = 0; i < (2 * TM + 3) / 4; ++i) {
            const bool real = r0 + 4 * i < M && s * F32_UNIT < k_left;
            if (r0 + 4 * i < 2 * TM) cp_async16(dst(s) + (uint32_t)((16 + 4 * i) * F32_ROW) * 4u, real ? ap + (size_t)(4 * i) * lda + s * F32_UNIT : A, real);
        }
    };
    // The first tiles of W are called into L2 while the kernels before still run, and read behind the wait: one of those may be
    // making W.
    pdl_trigger();
#pragma unroll 1
    for (int i = lane; i < 16 * (STAGES - 1); i += 32) {
        const int row = n0 + (i & 15), s = i >> 4;
        if (row < N && s < steps) asm volatile("prefetch.global.L2 [%0];" ::"l"(W + (size_t)row * ldw + (first + s) * F32_UNIT));
    }
    pdl_wait();
#pragma unroll 1
    for (int s = 0; s < STAGES - 1 && s < steps; ++s) load_w(s);
#pragma unroll 1
    for (int s = 0; s < STAGES - 1; ++s) {
        if (s < steps) load_a(s);
        cp_async_commit();
    }
    float acc[TM];
#pragma unroll
    for (int i = 0; i < TM; ++i) acc[i] = 0.0f;
    const int n = lane & 15, half = lane >> 4;
#pragma unroll 1
    for (int s = 0; s < steps; ++s) {
        cp_async_wait<STAGES - 2>();
        __syncwarp();                                               // every lane's copies have landed; all are done with the step before
        if (s + STAGES - 1 < steps) {
            load_w(s + STAGES - 1);
            load_a(s + STAGES - 1);
        }
        cp_async_commit();
        const float* ws = own + (s % STAGES) * Few::STAGE_FLOATS + n * F32_ROW;
        const float* as = own + (s % STAGES) * Few::STAGE_FLOATS + (16 + half * TM) * F32_ROW;
        // operands of 16 k at a time, all loads before the chains that wait for them
#pragma unroll
        for (int k = 0; k < F32_UNIT; k += 16) {
            float4 b[4], a[TM][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) b[q] = *reinterpret_cast<const float4*>(ws + k + q * 4);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int q = 0; q < 4; ++q) a[i][q] = *reinterpret_cast<const float4*>(as + i * F32_ROW + k + q * 4);
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int i = 0; i < TM; ++i) fma4(acc[i], a[i][q], b[q]);
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) sums[warp][half * TM + i][n] = acc[i];
    __syncthreads();
    for (int e = threadIdx.x; e < 2 * TM * 16; e += F32_SEGMENTS * 32) {
        const int m = e >> 4, f = e & 15;
        if (m >= M || n0 + f >= N) continue;
        float sum = sums[0][m][f];
#pragma unroll
        for (int w = 1; w < F32_SEGMENTS; ++w)
            if (w * seg < all) sum += sums[w][m][f];                // (empty segments add nothing: -0 stays -0)
        float* c = C + (size_t)m * ldc + n0 + f;
        *c = MODE == 0 ? sum : *c + sum;
    }
}

template <int BM, int BN, int TM, int TN, int STAGES>
static int gemm_f32_tile(const float* A, const float* W, float* C, int accumulate, int M, int N, int K, long long lda,
                         long long ldw, long long ldc, cudaStream_t s) {
    using Tile = F32Tile<BM, BN, TM, TN, STAGES>;
    auto kernel = accumulate ? gemm_f32_tile_kernel<BM, BN, TM, TN, STAGES, 1> : gemm_f32_tile_kernel<BM, BN, TM, TN, STAGES, 0>;
    static RbPerDevice limits[2];                                   // of the form that stores and the one that adds
    if (int e = rb_allow_shared(limits[accumulate ? 1 : 0], kernel, Tile::SMEM)) return e;
    return rb_launch(kernel, dim3(rb_ceil_div(M, BM), rb_ceil_div(N, BN)), dim3(Tile::THREADS), Tile::SMEM, s, A, W, C, M, N, K, lda, ldw, ldc);
}

template <int TM>
static int gemm_f32_few(const float* A, const float* W, float* C, int accumulate, int M, int N, int K, long long lda,
                        long long ldw, long long ldc, cudaStream_t s) {
    auto kernel = accumulate ? gemm_f32_few_kernel<TM, 1> : gemm_f32_few_kernel<TM, 0>;
    static RbPerDevice limits[2];                                   // of the form that stores and the one that adds
    if (int e = rb_allow_shared(limits[accumulate ? 1 : 0], kernel, F32Few<TM>::SMEM)) return e;
    return rb_launch(kernel, dim3(rb_ceil_div(M, 2 * TM), rb_ceil_div(N, 16)), dim3(F32_SEGMENTS * 32), F32Few<TM>::SMEM, s, A, W, C, M, N, K, lda, ldw, ldc);
}

// Many tokens, 128 x 128 outputs per CTA, 8 x 8 a thread.  Here the operands are transposed on the way in ([k][row], through
// registers), so that a thread's 16 operands of one k are four loads of 16 bytes and its registers hold one k ahead, not four:
// 64 sums, 32 operands and the next step's 16 numbers fit 128 registers, and two CTAs an SM.
// 727 tokens over 19,456 x 2,560 weights 1.72 ms (42 TFLOP/s; the 64 x 128 tiles above 1.87), over 2,560 x 9,728 1.00 ms (1.11).
#define F32W_ROW (128 + 4)
template <int MODE>
__global__ void __launch_bounds__(256, 2)
gemm_f32_wide_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K,
                     long long lda, long long ldw, long long ldc) {
    constexpr int BK = 16;
    extern __shared__ __align__(16) float f32_smem[];                // [2][A: BK rows of F32W_ROW, W: the same], then the running sums
    float* run = f32_smem + 2 * 2 * BK * F32W_ROW + threadIdx.x;      // [64][256]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tx = (warp & 1) * 8 + (lane & 7), ty = (warp >> 1) * 4 + (lane >> 3);
    const int m0 = blockIdx.x * 128, n0 = blockIdx.y * 128;
    const int steps = (K + BK - 1) / BK, seg = f32_segment(K) / BK;
    // a thread brings 16 bytes of rows r0 and r0 + 64 of either operand
    const int r0 = threadIdx.x >> 2, c0 = (threadIdx.x & 3) * 4;
    const float* ap = A + (size_t)(m0 + r0) * lda + c0;
    const float* wp = W + (size_t)(n0 + r0) * ldw + c0;
    float4 next[4];
    auto fetch = [&](int step) {
        const int k = step * BK;
        const bool in = k + c0 < K;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        next[0] = in && m0 + r0 < M ? *reinterpret_cast<const float4*>(ap + k) : zero;
        next[1] = in && m0 + r0 + 64 < M ? *reinterpret_cast<const float4*>(ap + 64 * lda + k) : zero;
        next[2] = in && n0 + r0 < N ? __ldg(reinterpret_cast<const float4*>(wp + k)) : zero;
        next[3] = in && n0 + r0 + 64 < N ? __ldg(reinterpret_cast<const float4*>(wp + 64 * ldw + k)) : zero;
    };
    auto put = [&](int buf) {
        float* dst = f32_smem + buf * (2 * BK * F32W_ROW) + c0 * F32W_ROW + r0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float* d = dst + (i >> 1) * (BK * F32W_ROW) + (i & 1) * 64;
            d[0] = next[i].x; d[F32W_ROW] = next[i].y; d[2 * F32W_ROW] = next[i].z; d[3 * F32W_ROW] = next[i].w;
        }
    };
    pdl_trigger();
    pdl_wait();
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
    fetch(0);
    put(0);
    __syncthreads();
#pragma unroll 1
    for (int step = 0; step < steps; ++step) {
        if (step + 1 < steps) fetch(step + 1);
        if (step && step % seg == 0) {                              // a segment begins
#pragma unroll
            for (int i = 0; i < 64; ++i) {
                float* r = run + i * 256;
                *r = step == seg ? acc[i >> 3][i & 7] : *r + acc[i >> 3][i & 7];
                acc[i >> 3][i & 7] = 0.0f;
            }
        }
        const float* as = f32_smem + (step & 1) * (2 * BK * F32W_ROW) + ty * 4;
        const float* ws = f32_smem + (step & 1) * (2 * BK * F32W_ROW) + BK * F32W_ROW + tx * 4;
        float4 a[2][2], b[2][2];
        a[0][0] = *reinterpret_cast<const float4*>(as); a[0][1] = *reinterpret_cast<const float4*>(as + 64);
        b[0][0] = *reinterpret_cast<const float4*>(ws); b[0][1] = *reinterpret_cast<const float4*>(ws + 64);
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            if (k + 1 < BK) {
                const float* an = as + (k + 1) * F32W_ROW;
                const float* wn = ws + (k + 1) * F32W_ROW;
                a[(k + 1) & 1][0] = *reinterpret_cast<const float4*>(an); a[(k + 1) & 1][1] = *reinterpret_cast<const float4*>(an + 64);
                b[(k + 1) & 1][0] = *reinterpret_cast<const float4*>(wn); b[(k + 1) & 1][1] = *reinterpret_cast<const float4*>(wn + 64);
            }
            const float4 a0 = a[k & 1][0], a1 = a[k & 1][1], b0 = b[k & 1][0], b1 = b[k & 1][1];
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w}, bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        if (step + 1 < steps) put((step + 1) & 1);                  // (the buffer that was read in the step before)
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int gm = m0 + ty * 4 + (i & 3) + (i >> 2) * 64;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int gn = n0 + tx * 4 + (j & 3) + (j >> 2) * 64;
            if (gn >= N) continue;
            float sum = acc[i][j];
            if (steps > seg) sum = run[(i * 8 + j) * 256] + sum;
            float* c = C + (size_t)gm * ldc + gn;
            *c = MODE == 0 ? sum : *c + sum;
        }
    }
}

static int gemm_f32_wide(const float* A, const float* W, float* C, int accumulate, int M, int N, int K, long long lda,
                         long long ldw, long long ldc, cudaStream_t s) {
    constexpr size_t smem = (2 * 2 * 16 * F32W_ROW + 64 * 256) * sizeof(float);
    auto kernel = accumulate ? gemm_f32_wide_kernel<1> : gemm_f32_wide_kernel<0>;
    static RbPerDevice limits[2];                                   // of the form that stores and the one that adds
    if (int e = rb_allow_shared(limits[accumulate ? 1 : 0], kernel, smem)) return e;
    // (begun early, its CTAs would go where the kernel before leaves room, two to an SM beside idle ones)
    return rb_launch_after(kernel, dim3(rb_ceil_div(M, 128), rb_ceil_div(N, 128)), dim3(256), smem, s, A, W, C, M, N, K, lda, ldw, ldc);
}

// Which kernel: up to 16 tokens the one for few (2,560 x 9,728 weights, 16 tokens: 67 us, 32 x 64 tiles 260 us; 9 .. 16 tokens are
// two CTAs a weight, neighbours in the grid, so that the second finds it in L2 however large W is: 16 tokens over 19,456 x 2,560
// weights 82 us, 89 with the second eight behind all of W; over 151,936 x 2,560 676 and 687).  Else the tile whose busiest SM is done first: a 64 x 128 tile takes an SM 80 units
// (574 us at K = 9,728), a 128 x 128 tile 134 (140 where it is alone on its SM), a 32 x 64 tile 26 (35).
static int gemm_f32_dispatch(const float* A, const float* W, float* C, int accumulate, int M, int N, int K, long long lda,
                             long long ldw, long long ldc, cudaStream_t s) {
    if (M <= 2) return gemm_f32_few<1>(A, W, C, accumulate, M, N, K, lda, ldw, ldc, s);
    if (M <= 4) return gemm_f32_few<2>(A, W, C, accumulate, M, N, K, lda, ldw, ldc, s);
    if (M <= 16) return gemm_f32_few<4>(A, W, C, accumulate, M, N, K, lda, ldw, ldc, s);
    const int sms = rb_sm_count();
    auto busiest = [&](int bm, int bn) { return (long long)rb_ceil_div((long long)rb_ceil_div(M, bm) * rb_ceil_div(N, bn), sms); };
    const long long wide = busiest(128, 128) == 1 ? 140 : 134 * busiest(128, 128);
    const long long tile = 80 * busiest(64, 128);
    const long long mid = busiest(32, 64) == 1 ? 35 : 26 * busiest(32, 64);
    if (mid < tile && mid < wide) return gemm_f32_tile<32, 64, 4, 4, 4>(A, W, C, accumulate, M, N, K, lda, ldw, ldc, s);
    if (wide < tile) return gemm_f32_wide(A, W, C, accumulate, M, N, K, lda, ldw, ldc, s);
    return gemm_f32_tile<64, 128, 8, 4, 3>(A, W, C, accumulate, M, N, K, lda, ldw, ldc, s);
}

extern "C" int rb_gemm_ref(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype,
                           int accumulate, int M, int N, int K, long long lda, long long ldw, long long ldc,
                           void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) RB_REFUSE("gemm: K=%d", K);
    if (M > 65535 * RG_BM) RB_REFUSE("gemm: M=%d exceeds the grid", M);
    cudaStream_t s = (cudaStream_t)stream;
    // cp.async brings 16 bytes at a time: rows that start on 16 bytes and end on them (a rule without M, see above)
    if (a_dtype == RB_F32 && w_dtype == RB_F32 && c_dtype == RB_F32 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 &&
        ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & 15) == 0 && N <= 65535 * 16)
        return gemm_f32_dispatch((const float*)A, (const float*)W, (float*)C, accumulate, M, N, K, lda, ldw, ldc, s);
    if (a_dtype == RB_F32 && w_dtype == RB_F32) return gemm_ref_dispatch<float, float>(A, W, C, c_dtype, accumulate, M, N, K, lda, ldw, ldc, s);
    if (a_dtype == RB_F32 && w_dtype == RB_BF16) return gemm_ref_dispatch<float, bf16>(A, W, C, c_dtype, accumulate, M, N, K, lda, ldw, ldc, s);
    if (a_dtype == RB_BF16 && w_dtype == RB_F32) return gemm_ref_dispatch<bf16, float>(A, W, C, c_dtype, accumulate, M, N, K, lda, ldw, ldc, s);
    if (a_dtype == RB_BF16 && w_dtype == RB_BF16) return gemm_ref_dispatch<bf16, bf16>(A, W, C, c_dtype, accumulate, M, N, K, lda, ldw, ldc, s);
    RB_REFUSE("gemm: operand dtypes %d, %d", a_dtype, w_dtype);
}
