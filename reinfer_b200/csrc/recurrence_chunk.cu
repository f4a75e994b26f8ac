// The linear recurrences of recurrence.cu over long portions of 16-bit tokens, four tokens at a time.
//
// Token by token a step's chain is a dot product over the key channels, shuffles that complete it, and the state's update: some 200
// to 450 cycles that every token of a request waits for, and it was these that bounded a prompt, not the work.  Here a chunk's four
// dot products start from the state before the chunk, so that their shuffles run side by side, and what the tokens of a chunk
// do to one another is left to a few numbers that do not depend on the state (the known rearrangement of linear recurrences into
// chunks: products of the gates from one token to the next inside the chunk, and a triangular system of its size).  With g_t the gates
// and D(j,t) the product of g_(j+1) .. g_t (per key channel; D(-1,t) from the chunk's first token on), S the state before the chunk:
//
//   form 0   w_j = v_j                                                  o_t = (q_t D(-1,t))^T S + sum_(j<=t) (q_t . D(j,t) k_j) w_j
//   form 3   w_j = v_j                     o_t = (q_t D(-1,t-1))^T S + sum_(j<t) (q_t . D(j,t-1) k_j) w_j + (sum q_t u k_t) v_t
//   form 2   w_t = beta_t (v_t - (k_t D(-1,t))^T S - sum_(j<t) (k_t . D(j,t) k_j) w_j)                          o_t as in form 0
//   form 1   y_t = (u_t D(-1,t-1))^T S + sum_(j<t) (u_t . D(j,t-1) k_j) v_j - (u_t . D(j,t-1) a_j) y_j,  w_j = v_j
//            o_t = (q_t D(-1,t))^T S + sum_(j<=t) (q_t . D(j,t) k_j) v_j - (q_t . D(j,t) a_j) y_j
//   S <- S + (D(-1,3) - 1) S + sum_j (D(j,3) k_j) w_j  [ - (D(j,3) a_j) y_j in form 1 ]
//
// Only products of gates are formed, never a quotient, so a gate of zero is a gate like any other; D(-1,3) - 1 is made from the
// gates' own g - 1 (recurrence.cu), so that a memory of thousands of tokens keeps its digits.  All of it is 32-bit.  A portion's last
// pair of chunks is filled up with tokens that change nothing (k = q = a = 0, g = 1).
//
// A kernel with one warp per (chunk, head) makes the vectors and the numbers, in parallel over the step's tokens; the walking CTAs
// bring them to shared memory by asynchronous copies, two pairs of chunks ahead.  A column of S is shared by 16 lanes with RP rows
// each; a lane holds CP = 2 columns, so that what it reads from shared memory - 128 bytes a cycle and SM, however many lanes read the
// same - serves both.  Four columns a lane halve that again and were slower (2,048 tokens of one request, 16 heads of 64 x 128: 155 us
// with two, 258 with four: half the warps, each twice as long); so was one column (222).
//
// A step of 2,048 tokens (895, 589 and 564), this file's two kernels against one token after the other (16 or 8 lanes a column):
// form 0, 16 heads of 64 x 128, 180 -> 121 us; form 1, 16 of 64 x 64, 260 -> 166; form 2, 16 of 128 x 128, 348 -> 286; form 3, 32 of
// 64 x 64, 204 -> 134; 520 tokens of one request 98 / 110 / 136 / 102 -> 47 / 68 / 90 / 48 us.  The error against 64 bits is 1 to 13 %
// smaller (1.1e-7 to 1.9e-7 of the outputs' norm: fewer roundings of the state).  What bounds the walk: with one request a warp's
// own latency (shuffles, reads of shared memory: one warp a scheduler), with three the reads of shared memory.
#include "recurrence.cuh"

#define RC 4                                  // tokens of a chunk
#define RC_STAGES 3
#define RC_VPAD 32                            // a record's values are padded to a multiple of this

// A chunk's record for one head: vectors of SPLIT * RP floats in the order X (forms 1, 2: what the state's columns are multiplied with
// first), Y (the read-out's), K (into the state), A (form 1), D(-1,3) - 1; then the numbers between the tokens; then the values
// [RC][padded dv].  Lane r of the SPLIT that share a column holds the rows 4 (SPLIT j + r) .. + 3, so that they read 16 bytes side by side.
template <int FORM, int SPLIT, int RP> struct ChunkRecord {
    static constexpr int VEC = SPLIT * RP;
    static constexpr bool DOTS = FORM == 1 || FORM == 2;
    static constexpr int X = 0, Y = DOTS ? RC : 0, K = Y + RC, A = K + RC, D = FORM == 1 ? A + RC : K + RC, NVEC = D + 1;
    // numbers: XK, XA for (t, j < t) at t (t - 1) / 2 + j; B by token; YK, YA for (t, j) at 4 t + j, zero for j > t
    static constexpr int XK = 0, XA = 6, B = 8, YK = FORM == 1 ? 12 : FORM == 2 ? 12 : 0, YA = 28;
    static constexpr int NNUM = FORM == 1 ? 44 : FORM == 2 ? 28 : 16;
    static constexpr int NSUM = FORM == 1 ? 32 : 16;                 // made by one sum over the lanes: X's, then Y's (t, j <= t) at t (t + 1) / 2 + j
    static constexpr int SYK = FORM == 1 ? 12 : FORM == 2 ? 6 : 0, SYA = 22;
    static constexpr int FLOATS = NVEC * VEC + NNUM;
};

// Chunks come in pairs, one stage of the walk.  Entry e's begin at pair cu_q[e] / (2 RC) + e, which leaves room for its last one.
static __host__ __device__ __forceinline__ int chunk_base(int cu, int e) { return 2 * (cu / (2 * RC) + e); }

// n sums over the 32 lanes at once (n 16 or 32): lane l ends with the sum of value l / (32 / n).
template <int N>
__device__ __forceinline__ float lane_sums(float* v, int lane) {
    int o = 16;
#pragma unroll
    for (int n = N; n > 1; n >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
            const float keep = up ? v[i + n / 2] : v[i], give = up ? v[i] : v[i + n / 2];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}

template <typename TA, int FORM, int SPLIT, int RP>
__global__ void __launch_bounds__(128)
chunk_prepare_kernel(const RecurArgs A, int n_entries, int n_chunks) {
    using R = ChunkRecord<FORM, SPLIT, RP>;
    pdl_trigger();
    const long long w = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    const int c = (int)(w / A.H), h = (int)(w % A.H);
    const bool none = c >= n_chunks;
    const float rate = (!none && A.gate == 2) ? expf(A.rate[h]) : 0.0f;
    pdl_wait();
    if (none) return;
    // the last entry whose chunks begin at or before this one
    int e = -1;
    for (int e0 = 0; e0 < n_entries; e0 += 32) {
        const bool before = e0 + lane < n_entries && chunk_base(A.cu_q[e0 + lane], e0 + lane) <= c;
        e += __popc(__ballot_sync(0xffffffffu, before));
    }
    if (e < 0) return;
    const int first = A.cu_q[e], at = (c - chunk_base(first, e)) * RC, n = A.cu_q[e + 1] - first;
    if (at / (2 * RC) * (2 * RC) >= n) return;                       // the room an entry's last pair did not need
    const int nt = max(0, min(RC, n - at)), kvh = h / (A.H / A.Hk), dk = A.dk;
    // Tokens and channels that are not there are read at the last place that is and replaced afterwards: no branch stands between the
    // loads, which are all on their way before the first is used.
    size_t tok[RC];
#pragma unroll
    for (int t = 0; t < RC; ++t) tok[t] = (size_t)(first + min(at + t, n - 1));
    float* rec = A.prep + (size_t)w * A.rec_floats;
    const TA* qr = (const TA*)A.q + (size_t)kvh * dk;
    const TA* kr = (const TA*)A.k + (size_t)kvh * dk;
    float qn[RC], kn[RC], un[RC];
#pragma unroll
    for (int t = 0; t < RC; ++t) { qn[t] = A.q_scale; kn[t] = 1.0f; un[t] = 1.0f; }
    if (A.unit_qk || FORM == 1) {
        float sums[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) sums[i] = 0.0f;
#pragma unroll 2
        for (int i = lane; i < dk; i += 32)
#pragma unroll
            for (int t = 0; t < RC; ++t) {
                const float a = to_f32(qr[tok[t] * A.ldq + i]), b = to_f32(kr[tok[t] * A.ldk + i]);
                sums[t] = fmaf(a, a, sums[t]); sums[4 + t] = fmaf(b, b, sums[4 + t]);
            }
        const float mine = lane_sums<16>(sums, lane);                // lanes 2 t, 2 t + 1: q of token t; 8 + 2 t: k
#pragma unroll
        for (int t = 0; t < RC; ++t) {
            const float rq = 1.0f / sqrtf(__shfl_sync(0xffffffffu, mine, 2 * t) + 1e-6f), rk = 1.0f / sqrtf(__shfl_sync(0xffffffffu, mine, 8 + 2 * t) + 1e-6f);
            if (A.unit_qk) { qn[t] = A.q_scale * rq; kn[t] = rk; }
            un[t] = rk;
        }
    }
    float num[R::NSUM];
#pragma unroll
    for (int i = 0; i < R::NSUM; ++i) num[i] = 0.0f;
#pragma unroll 2
    for (int i = lane; i < SPLIT * RP; i += 32) {
        const bool in = i < dk;
        const int ci = in ? i : 0;
        const size_t zi = A.z_per_head ? (size_t)h : (size_t)h * dk + ci, hi = (size_t)h * dk + ci;
        float q[RC], k[RC], g1[RC], u[RC], a[RC];                    // g1: the gate less one
#pragma unroll
        for (int t = 0; t < RC; ++t) {
            q[t] = to_f32(qr[tok[t] * A.ldq + ci]);
            k[t] = to_f32(kr[tok[t] * A.ldk + ci]);
            g1[t] = A.z[tok[t] * A.ldz + zi];
            a[t] = FORM == 1 ? to_f32(((const TA*)A.a_pre)[tok[t] * A.lda + hi]) : 0.0f;
        }
        const float zb = A.z_bias ? A.z_bias[zi] : 0.0f, ab = FORM == 1 && A.a_bias ? A.a_bias[hi] : 0.0f;
        const float bonus = FORM == 3 ? A.bonus[hi] : 0.0f;
#pragma unroll
        for (int t = 0; t < RC; ++t) {
            const bool real = in && t < nt;
            g1[t] = real ? expm1f(recur_log_gate(A, g1[t] + zb, rate)) : 0.0f;
            u[t] = real ? k[t] * un[t] : 0.0f;
            a[t] = FORM == 1 && real ? sigmoid_f(a[t] + ab) * u[t] : 0.0f;
            q[t] = real ? q[t] * qn[t] : 0.0f;
            k[t] = real ? k[t] * kn[t] : 0.0f;
        }
        float* out = rec + i;
        float d = 1.0f, dm = 0.0f;                                   // D(-1,t) and the same less one
#pragma unroll
        for (int t = 0; t < RC; ++t) {
            const float before = d;
            d = fmaf(before, g1[t], before);
            dm = dm + fmaf(dm, g1[t], g1[t]);
            out[(R::Y + t) * R::VEC] = q[t] * (FORM == 3 ? before : d);
            if (R::DOTS) out[(R::X + t) * R::VEC] = FORM == 1 ? u[t] * before : k[t] * d;
        }
        out[R::D * R::VEC] = dm;
#pragma unroll
        for (int j = 0; j < RC; ++j) {                               // what token j leaves, and how the tokens after it see it
            float kd = k[j], ad = a[j];
#pragma unroll
            for (int t = j; t < RC; ++t) {
                const int x = t * (t - 1) / 2 + j, y = t * (t + 1) / 2 + j;
                if (t > j && FORM == 1) {
                    num[R::XK + x] = fmaf(u[t], kd, num[R::XK + x]);
                    num[R::XA + x] = fmaf(u[t], ad, num[R::XA + x]);
                }
                if (FORM == 3) num[R::SYK + y] = fmaf(q[t], t == j ? k[t] * bonus : kd, num[R::SYK + y]);
                if (t > j) { kd = fmaf(kd, g1[t], kd); ad = fmaf(ad, g1[t], ad); }
                if (t > j && FORM == 2) num[R::XK + x] = fmaf(k[t], kd, num[R::XK + x]);
                if (FORM != 3) num[R::SYK + y] = fmaf(q[t], kd, num[R::SYK + y]);
                if (FORM == 1) num[R::SYA + y] = fmaf(q[t], ad, num[R::SYA + y]);
            }
            out[(R::K + j) * R::VEC] = kd;
            if (FORM == 1) out[(R::A + j) * R::VEC] = ad;
        }
    }
    const float mine = lane_sums<R::NSUM>(num, lane);
    float* numbers = rec + R::NVEC * R::VEC;
    constexpr int LANES = 32 / R::NSUM;
    if (lane % LANES == 0) {
        const int i = lane / LANES;
        if (i < R::SYK) numbers[i] = mine;                           // XK, then XA
        else {
            const bool ya = FORM == 1 && i >= R::SYA;
            const int m = i - (ya ? R::SYA : R::SYK), t = m >= 6 ? 3 : m >= 3 ? 2 : m >= 1 ? 1 : 0;
            if (m < 10) numbers[(ya ? R::YA : R::YK) + RC * t + m - t * (t + 1) / 2] = mine;
        }
    }
    if (lane < RC * RC && lane % RC > lane / RC) {
        numbers[R::YK + lane] = 0.0f;
        if (FORM == 1) numbers[R::YA + lane] = 0.0f;
    }
    if (FORM == 2 && lane < 2) numbers[6 + lane] = 0.0f;
    if (FORM == 2 && lane < RC) numbers[R::B + lane] = lane < nt ? sigmoid_f(to_f32(((const TA*)A.b_pre)[(size_t)(first + at + lane) * A.ldb + h])) : 0.0f;
    // the head's values as floats: zeros behind the portion's end and the head's last column
    const int vpad = (A.rec_floats - R::FLOATS) / RC;
    const TA* vr = (const TA*)A.v + (size_t)h * A.dv;
#pragma unroll 2
    for (int i = lane; i < vpad; i += 32) {
        float v[RC];
#pragma unroll
        for (int t = 0; t < RC; ++t) v[t] = to_f32(vr[tok[t] * A.ldv + min(i, A.dv - 1)]);
#pragma unroll
        for (int t = 0; t < RC; ++t) rec[R::FLOATS + t * vpad + i] = t < nt && i < A.dv ? v[t] : 0.0f;
    }
}

// Columns of a warp: 32 / SPLIT groups of CP; WARPS of them a CTA.
template <int FORM, int SPLIT, int RP, int CP, int WARPS> struct ChunkWalk {
    static constexpr int COLS = WARPS * (32 / SPLIT) * CP;
    static constexpr int STAGE_FLOATS = 2 * (ChunkRecord<FORM, SPLIT, RP>::FLOATS + RC * COLS);
    static constexpr size_t SMEM = (size_t)RC_STAGES * STAGE_FLOATS * sizeof(float);
    static_assert(COLS % 8 == 0 && RC_VPAD % COLS == 0, "a CTA's values are 16-byte pieces of the record's");
};

// N values a lane carries, summed over the SPLIT lanes that share a column: every step halves the values that a lane still
// carries, as long as there is more than one.  Lane r of N <= SPLIT ends with the sum r / (SPLIT / N) in v[0], of N > SPLIT with
// the N / SPLIT sums from r * (N / SPLIT) on.
template <int N, int SPLIT>
__device__ __forceinline__ void slice_sums(float* v, int r) {
    int o = SPLIT / 2;
#pragma unroll
    for (int m = N; m > 1 && o > 0; m >>= 1, o >>= 1) {
        const bool up = r & o;
#pragma unroll
        for (int i = 0; i < m / 2; ++i) {
            const float keep = up ? v[i + m / 2] : v[i], give = up ? v[i] : v[i + m / 2];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
#pragma unroll
    for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
}

// 16 bytes of shared memory; EARLY: where the program says so, and no later (left to itself the compiler reads them right before
// their use, and a warp that is alone on its scheduler waits for every one).
template <bool EARLY> __device__ __forceinline__ float4 lds4(const float* p) {
    if (!EARLY) return *reinterpret_cast<const float4*>(p);
    float4 f;
    asm volatile("ld.volatile.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(f.x), "=f"(f.y), "=f"(f.z), "=f"(f.w) : "r"((uint32_t)__cvta_generic_to_shared(p)));
    return f;
}

template <int FORM, int SPLIT, int RP, int CP, int WARPS, bool EARLY>
__global__ void __launch_bounds__(WARPS * 32)
chunk_walk_kernel(const RecurArgs A) {
    using R = ChunkRecord<FORM, SPLIT, RP>;
    using W = ChunkWalk<FORM, SPLIT, RP, CP, WARPS>;
    constexpr int THREADS = WARPS * 32, COLS = W::COLS;
    extern __shared__ __align__(16) float sm[];
    pdl_trigger();
    const int lane = threadIdx.x & 31;
    const int h = blockIdx.y, e = blockIdx.z, c0 = blockIdx.x * COLS;
    const int r = lane % SPLIT, cl = ((threadIdx.x >> 5) * (32 / SPLIT) + lane / SPLIT) * CP;    // this lane's slice of the rows, its first column
    const int dk = A.dk, dv = A.dv, c = c0 + cl;
    pdl_wait();
    const int s0 = A.cu_q[e], n = A.cu_q[e + 1] - s0;
    if (n <= 0) return;
    const int pairs = (n + 2 * RC - 1) / (2 * RC);
    const int vpad = (A.rec_floats - R::FLOATS) / RC;
    const float* records = A.prep + ((size_t)chunk_base(s0, e) * A.H + h) * A.rec_floats;
    const size_t to_next = (size_t)A.H * A.rec_floats;               // from a chunk's record to the next one's
    auto fetch = [&](int i) {
        float* dst = sm + (i % RC_STAGES) * W::STAGE_FLOATS;
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
            const float* src = records + (size_t)(2 * i + ch) * to_next;
#pragma unroll
            for (int p0 = 0; p0 < R::FLOATS / 4; p0 += THREADS) {
                const int p = p0 + threadIdx.x;
                if (p < R::FLOATS / 4) rr_cp_async16(dst + ch * R::FLOATS + 4 * p, src + 4 * p);
            }
        }
        if (threadIdx.x < 2 * RC * COLS / 4) {
            const int t = threadIdx.x / (COLS / 4), at = 4 * (threadIdx.x % (COLS / 4));
            rr_cp_async16(dst + 2 * R::FLOATS + t * COLS + at, records + (size_t)(2 * i + t / RC) * to_next + R::FLOATS + (t % RC) * vpad + c0 + at);
        }
    };
    static_assert(2 * RC * COLS / 4 <= THREADS, "a piece of the values a thread");
#pragma unroll
    for (int i = 0; i < RC_STAGES - 1; ++i) {
        if (i < pairs) fetch(i);
        rr_cp_async_commit();
    }
    float* S = A.state + ((size_t)A.entry_slot[e] * A.H + h) * dk * dv;
    float s[CP][RP];
#pragma unroll
    for (int i = 0; i < RP; ++i) {
        const int row = ((i / 4) * SPLIT + r) * 4 + i % 4;
#pragma unroll
        for (int p = 0; p < CP; ++p) s[p][i] = (row < dk && c + p < dv) ? S[(size_t)row * dv + c + p] : 0.0f;
    }

    // what this lane holds of a pair's read-out once the slices are summed: EACH columns, from p_own on, of token t_own
    constexpr int N = 2 * RC * CP, EACH = N > SPLIT ? N / SPLIT : 1, SAME = N < SPLIT ? SPLIT / N : 1;
    static_assert(EACH <= CP, "the sums of a lane are of one token");
    const int t_own = r / SAME * EACH / CP, p_own = r / SAME * EACH % CP;
#pragma unroll 1
    for (int it = 0; it < pairs; ++it) {
        rr_cp_async_wait<RC_STAGES - 2>();
        __syncthreads();                                             // the pair has landed, and all are done with the one before
        if (it + RC_STAGES - 1 < pairs) fetch(it + RC_STAGES - 1);
        rr_cp_async_commit();
        const float* st = sm + (it % RC_STAGES) * W::STAGE_FLOATS;
        float out[2 * RC * CP];                                      // this lane's part of the read-out, [token][column]
        float own[EACH];                                             // what the tokens of its chunk add to this lane's part of it
#pragma unroll
        for (int ch = 0; ch < 2; ++ch) {
            const float* rec = st + ch * R::FLOATS + 4 * r;
            const float* num = st + ch * R::FLOATS + R::NVEC * R::VEC;
            float w[CP][RC], y[CP][RC];                              // what the tokens write; form 1: what they read
            float4 vec[R::NVEC][RP / 4];
            float nm[12];
#pragma unroll
            for (int i = 0; i < RP / 4; ++i)
#pragma unroll
                for (int j = 0; j < R::NVEC; ++j) vec[j][i] = lds4<EARLY>(rec + j * R::VEC + 4 * i * SPLIT);
            if (R::DOTS) {
#pragma unroll
                for (int i = 0; i < 12; i += 4) {
                    const float4 f = lds4<EARLY>(num + i);
                    nm[i] = f.x; nm[i + 1] = f.y; nm[i + 2] = f.z; nm[i + 3] = f.w;
                }
            }
            const float4 yk = lds4<EARLY>(num + R::YK + RC * (t_own % RC));
            const float4 ya = FORM == 1 ? lds4<EARLY>(num + R::YA + RC * (t_own % RC)) : yk;
#pragma unroll
            for (int t = 0; t < RC; ++t) {
                const float* v = st + 2 * R::FLOATS + (ch * RC + t) * COLS + cl;
#pragma unroll
                for (int p = 0; p < CP; p += 2) {
                    const float2 f = *reinterpret_cast<const float2*>(v + p);
                    w[p][t] = f.x; w[p + 1][t] = f.y;
                }
            }
            if (R::DOTS) {
                float x[RC * CP];
#pragma unroll
                for (int i = 0; i < RC * CP; ++i) x[i] = 0.0f;
#pragma unroll
                for (int i = 0; i < RP; i += 4)
#pragma unroll
                    for (int t = 0; t < RC; ++t) {
                        const float4 f = vec[R::X + t][i / 4];
#pragma unroll
                        for (int p = 0; p < CP; ++p)
                            x[t * CP + p] = fmaf(f.w, s[p][i + 3], fmaf(f.z, s[p][i + 2], fmaf(f.y, s[p][i + 1], fmaf(f.x, s[p][i], x[t * CP + p]))));
                    }
                slice_sums<RC * CP, SPLIT>(x, r);
                static_assert(RC * CP <= SPLIT, "a lane ends with one sum");
                constexpr int LANES = SPLIT / (RC * CP);             // adjacent lanes with the same one
#pragma unroll
                for (int t = 0; t < RC; ++t)
#pragma unroll
                    for (int p = 0; p < CP; ++p) y[p][t] = __shfl_sync(0xffffffffu, x[0], (t * CP + p) * LANES, SPLIT);
                // the tokens of the chunk one after the other
#pragma unroll
                for (int t = 0; t < RC; ++t)
#pragma unroll
                    for (int p = 0; p < CP; ++p) {
#pragma unroll
                        for (int j = 0; j < t; ++j) {
                            y[p][t] = fmaf(nm[R::XK + t * (t - 1) / 2 + j], w[p][j], y[p][t]);
                            if (FORM == 1) y[p][t] = fmaf(-nm[R::XA + t * (t - 1) / 2 + j], y[p][j], y[p][t]);
                        }
                        if (FORM == 2) w[p][t] = nm[R::B + t] * (w[p][t] - y[p][t]);
                    }
            }
#pragma unroll
            for (int i = 0; i < EACH; ++i) {
                float wj[RC], yj[RC];
#pragma unroll
                for (int j = 0; j < RC; ++j) {
                    wj[j] = w[i][j];
                    yj[j] = FORM == 1 ? y[i][j] : 0.0f;
#pragma unroll
                    for (int p = i + EACH; p < CP; p += EACH) {
                        wj[j] = p_own + i == p ? w[p][j] : wj[j];
                        if (FORM == 1) yj[j] = p_own + i == p ? y[p][j] : yj[j];
                    }
                }
                float o = fmaf(yk.x, wj[0], fmaf(yk.y, wj[1], fmaf(yk.z, wj[2], yk.w * wj[3])));
                if (FORM == 1) o = fmaf(-ya.x, yj[0], fmaf(-ya.y, yj[1], fmaf(-ya.z, yj[2], fmaf(-ya.w, yj[3], o))));
                own[i] = ch == 0 || t_own >= RC ? o : own[i];
            }
#pragma unroll
            for (int i = 0; i < RC * CP; ++i) out[ch * RC * CP + i] = 0.0f;
            // the read-out of the state before the chunk, then the state: the chunk's decay, and what its tokens leave
#pragma unroll
            for (int i = 0; i < RP; i += 4) {
#pragma unroll
                for (int t = 0; t < RC; ++t) {
                    const float4 f = vec[R::Y + t][i / 4];
#pragma unroll
                    for (int p = 0; p < CP; ++p) {
                        float& o = out[(ch * RC + t) * CP + p];
                        o = fmaf(f.w, s[p][i + 3], fmaf(f.z, s[p][i + 2], fmaf(f.y, s[p][i + 1], fmaf(f.x, s[p][i], o))));
                    }
                }
                const float4 dm = vec[R::D][i / 4];
#pragma unroll
                for (int p = 0; p < CP; ++p) {
                    s[p][i] = fmaf(dm.x, s[p][i], s[p][i]); s[p][i + 1] = fmaf(dm.y, s[p][i + 1], s[p][i + 1]);
                    s[p][i + 2] = fmaf(dm.z, s[p][i + 2], s[p][i + 2]); s[p][i + 3] = fmaf(dm.w, s[p][i + 3], s[p][i + 3]);
                }
#pragma unroll
                for (int j = 0; j < RC; ++j) {
                    const float4 f = vec[R::K + j][i / 4];
#pragma unroll
                    for (int p = 0; p < CP; ++p) {
                        s[p][i] = fmaf(f.x, w[p][j], s[p][i]); s[p][i + 1] = fmaf(f.y, w[p][j], s[p][i + 1]);
                        s[p][i + 2] = fmaf(f.z, w[p][j], s[p][i + 2]); s[p][i + 3] = fmaf(f.w, w[p][j], s[p][i + 3]);
                    }
                    if (FORM == 1) {
                        const float4 g = vec[FORM == 1 ? R::A + j : 0][i / 4];
#pragma unroll
                        for (int p = 0; p < CP; ++p) {
                            s[p][i] = fmaf(-g.x, y[p][j], s[p][i]); s[p][i + 1] = fmaf(-g.y, y[p][j], s[p][i + 1]);
                            s[p][i + 2] = fmaf(-g.z, y[p][j], s[p][i + 2]); s[p][i + 3] = fmaf(-g.w, y[p][j], s[p][i + 3]);
                        }
                    }
                }
            }
        }
        slice_sums<N, SPLIT>(out, r);
#pragma unroll
        for (int i = 0; i < EACH; ++i)
            if (it * 2 * RC + t_own < n && c + p_own + i < dv && (SAME == 1 || (r & (SAME - 1)) == 0))
                A.out[((size_t)(s0 + it * 2 * RC + t_own) * A.H + h) * dv + c + p_own + i] = out[i] + own[i];
    }
#pragma unroll
    for (int i = 0; i < RP; ++i) {
        const int row = ((i / 4) * SPLIT + r) * 4 + i % 4;
#pragma unroll
        for (int p = 0; p < CP; ++p)
            if (row < dk && c + p < dv) S[(size_t)row * dv + c + p] = s[p][i];
    }
}

template <int FORM, int SPLIT, int RP, int CP, int WARPS, bool EARLY>
static int chunk_walk(const RecurArgs& a, int n_entries, cudaStream_t st) {
    using W = ChunkWalk<FORM, SPLIT, RP, CP, WARPS>;
    auto kernel = chunk_walk_kernel<FORM, SPLIT, RP, CP, WARPS, EARLY>;
    static RbPerDevice limit;
    if (W::SMEM > 48 * 1024)
        if (int e = rb_allow_shared(limit, kernel, W::SMEM)) return e;
    return rb_launch_after(kernel, dim3(rb_ceil_div(a.dv, W::COLS), a.H, n_entries), dim3(WARPS * 32), W::SMEM, st, a);
}

template <int FORM, int SPLIT, int RP>
static int chunk_launch(RecurArgs a, int n_entries, cudaStream_t st) {
    using R = ChunkRecord<FORM, SPLIT, RP>;
    static_assert(R::FLOATS % 4 == 0, "a record is copied 16 bytes at a time");
    a.rec_floats = R::FLOATS + RC * rb_ceil_div(a.dv, RC_VPAD) * RC_VPAD;
    const int n_chunks = chunk_base(a.n_tokens, n_entries);          // (room, not all of it used)
    if (int e = rb_launch(chunk_prepare_kernel<bf16, FORM, SPLIT, RP>, dim3(rb_ceil_div((long long)n_chunks * a.H, 4)), dim3(128), 0, st, a, n_entries, n_chunks))
        return e;
    // Up to 64 key channels two warps a CTA and the vectors read early (a request of 520 tokens, 16 heads, form 1 with 64 x 64
    // states: 71 us, 83 the other way), beyond that four, and where the compiler puts them (form 2 with 128 x 128: 92 and 110).
    return chunk_walk<FORM, SPLIT, RP, 2, RP == 4 ? 2 : 4, RP == 4>(a, n_entries, st);
}

template <int FORM>
static int chunk_dispatch(const RecurArgs& A, int n_entries, cudaStream_t st) {
    if (A.dk <= 64) return chunk_launch<FORM, 16, 4>(A, n_entries, st);
    if (A.dk <= 128) return chunk_launch<FORM, 16, 8>(A, n_entries, st);
    return chunk_launch<FORM, 16, 16>(A, n_entries, st);
}

int recurrence_chunks(const RecurArgs& A, int form, int n_entries, cudaStream_t st) {
    if (form == 0) return chunk_dispatch<0>(A, n_entries, st);
    if (form == 1) return chunk_dispatch<1>(A, n_entries, st);
    if (form == 2) return chunk_dispatch<2>(A, n_entries, st);
    return chunk_dispatch<3>(A, n_entries, st);
}

template <int SPLIT, int RP> static int chunk_floats(int form) {
    return form == 1 ? ChunkRecord<1, SPLIT, RP>::FLOATS : form == 2 ? ChunkRecord<2, SPLIT, RP>::FLOATS : ChunkRecord<0, SPLIT, RP>::FLOATS;
}
// Floats of scratch for a step's records.
long long recurrence_chunks_scratch(int form, int dk, int dv, int H, int n_tokens, int n_entries) {
    const int rec = (dk <= 64 ? chunk_floats<16, 4>(form) : dk <= 128 ? chunk_floats<16, 8>(form) : chunk_floats<16, 16>(form)) +
                    RC * rb_ceil_div(dv, RC_VPAD) * RC_VPAD;
    return (long long)chunk_base(n_tokens, n_entries) * H * rec;
}
