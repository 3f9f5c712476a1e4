// The recurrences with a decay per head and key channel, over long prompt portions, in chunks of 16 tokens:
//
//   gated delta rule   S <- diag(g) S;  u = beta (v - S^T k);  S <- S + k u^T;   o = S^T q
//   HGRN2              S <- diag(f) S + (1 - f) v^T;                             o = S^T q
//
// Token by token (recurrent.cu) a head's state moves through a chain of dependent sums: 415 ns a token for the delta rule with
// states of 128 x 128. Over a chunk the recurrence is linear in the state S before it. With E(s, t) the product of the decays
// of the tokens s + 1 .. t (per channel; E(., t) from the chunk's start), every token's u and o are
//
//   u_t = beta_t (v_t - (k_t E(., t)) . S - sum over s < t of A(t, s) u_s),     A(t, s) = (k_t E(s, t)) . k_s
//   o_t = (q_t E(., t)) . S + sum over s <= t of B(t, s) u_s,                   B(t, s) = (q_t E(s, t)) . k_s
//
// and with T = (I + diag(beta) A)^-1 diag(beta), which is triangular and knows nothing of S,
//
//   u = U0 - W S,    W = T (k E),  U0 = T v
//   o = O0 + Q S,    Q = q E - B W,  O0 = B U0
//   S behind the chunk = diag(E(., end)) S + sum over s of (k_s E(s, end)) u_s^T
//
// (HGRN2: 1 - f in k's place, u = v, no W.) Products of decays only are formed, never a quotient, so nothing overflows however
// strong the decays are. Two kernels:
//
//   chunk_vectors   W, Q, k E(., end), E(., end), U0 and O0 of every chunk and head, all of them at once
//   chunk_walk      a block carries 16 columns of one (request, head)'s S through the chunks: two small products a chunk
//
// chunk_vectors is 32-bit fused multiply-adds, as token by token; chunk_walk takes its products with S on the tensor cores, in three
// bfloat16 parts a factor, and moves S on by 32-bit multiply-adds. Against 64 bits over 1,025 tokens, in brackets with multiply-adds
// in all of the walk (8 heads of 128 x 128, decays uniform in 0.8 .. 1): read-outs 1.13e-7 (1.16e-7), the state behind them 8.6e-8
// (8.6e-8); decays in 0.999 .. 1 and repeating keys 4.7e-7 (4.7e-7) and 5.5e-7 (5.5e-7); uniform in 0 .. 1 9.1e-8 (9.2e-8) and 5.0e-8
// (5.0e-8). HGRN2 1.06e-7 (1.09e-7), 7.8e-8 (7.8e-8); 6.4e-7 (6.4e-7), 1.0e-6 (1.0e-6); 9.1e-8 (9.1e-8), 4.3e-8 (4.3e-8). (With S moved
// by products in parts as well its error was smaller where decays are near 1 and up to 15 % larger where a chunk's last tokens prevail:
// the tensor cores cut the small terms of a sum.)
// One prompt of 2,048 tokens, 16 heads of 128 x 128: token by token 938 us, in chunks with multiply-adds 214, now 178 (55 of them
// chunk_vectors, which forms the parts).
#include <algorithm>
#include <climits>

#include "mma_tiles.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int CT = 16;          // tokens a chunk
constexpr int CB = 16;          // columns of S a block of the walk holds
constexpr int MIN_STAGES = 3, MAX_STAGES = 4;

struct ChunkArgs {
    const float *q, *k, *g, *v, *beta;      // k, beta: null for HGRN2
    long long ld_q, ld_k, ld_g, ld_v;
    int per;                                // heads that share a row of q and k
    const int *cu_seqlens, *slot_ids;
    int B, min_len, heads, dim, vd;
    float* ws;                              // a chunk's and head's numbers at ((chunk - chunk0) * heads + head) * stride floats
    long long stride;
    int chunk0, chunks;                     // the step's chunks that are in the workspace
    int stages;                             // of the walk's shared memory
};

// A (chunk, head) in the workspace, as the walk's products take it (operands of mma.sync m16n8k16 in three bfloat16 parts, a lane's
// registers side by side): for every 16 channels -W (delta rule) and Q as right operands; k E(., end) [CT][DIM]; E(., end) [DIM]; then
// per block of CB columns U0 [CB][CT] (delta rule; HGRN2's are the values themselves) and O0 [CB][CT].
template <int DIM, bool DELTA> struct Layout {
    static constexpr int KINDS = DELTA ? 2 : 1, OPERAND = 3 * 32 * 4;
    static constexpr int KE = DIM / 16 * KINDS * OPERAND, DECAY = KE + CT * DIM, ROWS = DECAY + DIM;
    static constexpr int O0 = DELTA ? CT * CB : 0, COLS = O0 + CT * CB;
    static constexpr int STAGE = ROWS + COLS;
};

// A pair of 32-bit numbers as three pairs of bfloat16 numbers whose sums they are (8 bits each, all 24; of numbers below 2^-109 the parts'
// smallest step takes the last). No product of an infinite number's parts is finite, nor of those of a number that bfloat16 rounds to
// infinity. FINITE: the first part stays finite, so that whole_of finds such numbers again (infinity is (the largest, infinity, NaN)); that
// takes more instructions, which the walk's chain has no room for.
__device__ __forceinline__ uint64_t minus_parts(uint64_t x, uint32_t part) {
    const uint64_t y = (uint64_t)(part & 0xffff0000u) << 32 | (part << 16);
    uint64_t d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
    return d;
}
__device__ __forceinline__ uint32_t pack_pair_finite(uint64_t x) {
    uint32_t y;
    asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(y) : "f"(__uint_as_float((uint32_t)(x >> 32))), "f"(__uint_as_float((uint32_t)x)));
    return y;
}
__device__ __forceinline__ uint32_t pack_pair(uint64_t x) { return pack_bf16(__uint_as_float((uint32_t)x), __uint_as_float((uint32_t)(x >> 32))); }
template <bool FINITE> __device__ __forceinline__ void split3(uint32_t& hi, uint32_t& mid, uint32_t& low, float x, float y) {
    uint64_t pair = (uint64_t)__float_as_uint(y) << 32 | __float_as_uint(x);
    hi = FINITE ? pack_pair_finite(pair) : pack_pair(pair);
    pair = minus_parts(pair, hi);
    mid = pack_pair(pair);
    low = pack_pair(minus_parts(pair, mid));
}
// The number again, of the pair's first (which = 0) or second.
__device__ __forceinline__ float whole_of(uint32_t hi, uint32_t mid, uint32_t low, int which) {
    auto part = [&](uint32_t x) { return __uint_as_float(which ? x & 0xffff0000u : x << 16); };
    const float m = part(mid), sum = part(hi) + m;
    return fabsf(m) < INFINITY ? sum + part(low) : sum;
}
// Chunks of portion b, 0 where it is short; where a warp looks through the portions, a lane takes one of 32 (one after the other they
// cost a block 0.3 us each).
__device__ __forceinline__ int chunks_of(const ChunkArgs& a, int b) {
    const int n = a.cu_seqlens[b + 1] - a.cu_seqlens[b];
    return n < a.min_len ? 0 : (n + CT - 1) / CT;
}
// The portion that chunk c of the step lies in (c: which of its chunks), or -1.
__device__ __forceinline__ int portion_of(const ChunkArgs& a, int& c, int lane) {
    for (int b0 = 0; b0 < a.B; b0 += 32) {
        int sum = b0 + lane < a.B ? chunks_of(a, b0 + lane) : 0;
        const int own = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, sum, d);
            if (lane >= d) sum += up;
        }
        const unsigned behind = __ballot_sync(0xffffffffu, sum > c);
        if (behind) {
            const int l = __ffs(behind) - 1;
            c -= __shfl_sync(0xffffffffu, sum - own, l);
            return b0 + l;
        }
        c -= __shfl_sync(0xffffffffu, sum, 31);
    }
    return -1;
}

// N values a lane, summed over 2 * TOP neighbouring lanes; a lane is left with N / (2 * TOP) of the sums, those from the
// returned index on.
template <int N, int TOP> __device__ __forceinline__ int scatter_sums(float (&x)[N], int lane) {
    int first = 0;
#pragma unroll
    for (int d = TOP, half = N / 2; d >= 1; d >>= 1, half >>= 1) {
        const bool up = lane & d;
#pragma unroll
        for (int i = 0; i < N / 2; ++i) {
            if (i >= half) break;
            const float send = up ? x[i] : x[i + half], keep = up ? x[i + half] : x[i];
            x[i] = keep + __shfl_xor_sync(0xffffffffu, send, d);
        }
        first += up ? half : 0;
    }
    return first;
}

// A block a (chunk, head), a thread a channel. Bound by the instructions of the sums over channels and by what it writes (50 KB a
// block of the delta rule with 128 x 128). The walk's operands leave here in parts, once for all of a head's blocks of columns: 47 ->
// 58 us for 2,048 tokens and 16 heads, where splitting them in every block cost the walk 20.
template <int DIM, bool DELTA>
__global__ void __launch_bounds__(DIM)
chunk_vectors_kernel(const ChunkArgs a) {
    using L = Layout<DIM, DELTA>;
    __shared__ float part[DIM / 32][CT][33];
    __shared__ __align__(16) float As[CT][CT], Bs[CT][CT], Ts[CT][CT];
    __shared__ float beta[CT];
    pdl_trigger();
    pdl_wait();
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int c = a.chunk0 + blockIdx.x;
    const int b = portion_of(a, c, lane);
    if (b < 0) return;
    const int t0 = a.cu_seqlens[b] + c * CT, len = min(CT, a.cu_seqlens[b + 1] - t0);
    float* ws = a.ws + ((size_t)blockIdx.x * a.heads + h) * a.stride;
    uint32_t* operand = reinterpret_cast<uint32_t*>(ws) + (tid >> 4) * (L::KINDS * L::OPERAND);        // those of the thread's 16 channels
    const bool mine = tid < a.dim;
    const float* qp = a.q + (size_t)t0 * a.ld_q + (h / a.per) * a.dim + tid;
    const float* gp = a.g + (size_t)t0 * a.ld_g + h * a.dim + tid;
    const float* kp = DELTA ? a.k + (size_t)t0 * a.ld_k + (h / a.per) * a.dim + tid : nullptr;
    // tokens behind the portion's last: nothing decays, nothing is written
    float q[CT], k[CT], g[CT];
#pragma unroll
    for (int t = 0; t < CT; ++t) {
        const bool in = mine && t < len;
        q[t] = in ? qp[(size_t)t * a.ld_q] : 0.f;
        g[t] = in ? gp[(size_t)t * a.ld_g] : 1.f;
        k[t] = DELTA ? (in ? kp[(size_t)t * a.ld_k] : 0.f) : 1.f - g[t];
    }
    if (DELTA && tid < CT) beta[tid] = tid < len ? a.beta[(size_t)(t0 + tid) * a.heads + h] : 0.f;
    {
        float e = 1.f;
#pragma unroll
        for (int t = CT - 1; t >= 0; --t) {
            ws[L::KE + t * DIM + tid] = k[t] * e;
            e *= g[t];
        }
        ws[L::DECAY + tid] = e;
    }
    // A and B: for every s the sums over the channels of (k_t | q_t) E(s, t) k_s, t = s .. CT - 1
    if constexpr (DELTA) {
        // the sums of s and CT - 1 - s together are 2 CT: as many as lanes
#pragma unroll
        for (int s = 0; s < CT / 2; ++s) {
            float x[2 * CT];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int from = half ? CT - 1 - s : s, at = half ? 2 * CT - 1 - 2 * s : 0, n = CT - from;
                float e = k[from];
#pragma unroll
                for (int t = 0; t < CT; ++t) {
                    if (t < from) continue;
                    if (t > from) {
                        e *= g[t];
                        x[at + n + t - from - 1] = k[t] * e;
                    }
                    x[at + t - from] = q[t] * e;
                }
            }
            scatter_sums<2 * CT, 16>(x, lane);
            part[warp][s][lane] = x[0];
            asm volatile("" ::: "memory");       // one pair's sums at a time, or the registers do not suffice
        }
    } else {
#pragma unroll
        for (int s = 0; s < CT; ++s) {
            float e = k[s], x[CT];
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                if (t > s) e *= g[t];
                x[t] = t >= s ? q[t] * e : 0.f;
            }
            scatter_sums<CT, 8>(x, lane);
            x[0] += __shfl_xor_sync(0xffffffffu, x[0], 16);
            if (lane < CT) part[warp][s][lane] = x[0];
        }
    }
    __syncthreads();
    for (int i = tid; i < CT * CT; i += DIM) {
        const int s = DELTA ? i / (2 * CT) : i / CT, l = DELTA ? i % (2 * CT) : i % CT;
        float sum = part[0][s][l];
#pragma unroll
        for (int w = 1; w < DIM / 32; ++w) sum += part[w][s][l];
        if constexpr (DELTA) {
            // lanes: B(s .., s), A(s + 1 .., s), then the same of CT - 1 - s
            const int from = l < 2 * CT - 1 - 2 * s ? s : CT - 1 - s, at = from == s ? l : l - (2 * CT - 1 - 2 * s), n = CT - from;
            if (at < n) Bs[from + at][from] = sum; else As[from + 1 + at - n][from] = sum;
        } else {
            Bs[l][s] = sum;
        }
    }
    __syncthreads();
    if constexpr (DELTA) {
        if (tid < CT) {         // column tid of T, downwards
            float x[CT];
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                float sum = t == tid ? 1.f : 0.f;
#pragma unroll
                for (int s = 0; s < t; ++s) sum = fmaf(-As[t][s], x[s], sum);
                x[t] = beta[t] * sum;
                Ts[t][tid] = x[t];
            }
        }
        __syncthreads();
    }
    {
        float e = 1.f;
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            e *= g[t];
            q[t] *= e;
            k[t] *= e;
        }
        // rows t and t + 8 of 16 channels as a pair of right operands: channels 4 i .. 4 i + 3 of a row are two registers of lane i of it;
        // of two neighbouring channels the even one's thread takes row t of both, the odd one's row t + 8
        auto rows_out = [&](uint32_t* out, const float (&x)[CT]) {
            const bool odd = tid & 1;
            out += ((tid >> 2) & 3) * 4 + 2 * odd + ((tid >> 1) & 1);
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const float other = __shfl_xor_sync(0xffffffffu, odd ? x[t] : x[t + 8], 1);
                uint32_t part[3];
                split3<true>(part[0], part[1], part[2], odd ? other : x[t], odd ? x[t + 8] : other);
#pragma unroll
                for (int p = 0; p < 3; ++p) out[p * 128 + t * 16] = part[p];
            }
        };
        if constexpr (DELTA) {
            float w[CT];
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                float sum = 0.f;
#pragma unroll
                for (int s = 0; s <= t; ++s) sum = fmaf(Ts[t][s], k[s], sum);
                w[t] = -sum;
            }
            rows_out(operand, w);
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                float sum = q[t];
#pragma unroll
                for (int s = 0; s <= t; ++s) sum = fmaf(Bs[t][s], w[s], sum);
                q[t] = sum;
            }
        }
        rows_out(operand + (L::KINDS - 1) * L::OPERAND, q);
    }
    const int blocks = (a.vd + CB - 1) / CB;
#pragma unroll 1
    for (int j = tid; j < blocks * CB; j += DIM) {
        asm volatile("" ::: "memory");       // T and B come from shared memory again for every column: 272 values are no registers
        float v[CT], u[CT];
#pragma unroll
        for (int t = 0; t < CT; ++t) v[t] = (j < a.vd && t < len) ? a.v[(size_t)(t0 + t) * a.ld_v + h * a.vd + j] : 0.f;
        float* out = ws + L::ROWS + (size_t)(j / CB) * L::COLS;
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            if constexpr (DELTA) {
                float sum = 0.f;
#pragma unroll
                for (int s = 0; s <= t; ++s) sum = fmaf(Ts[t][s], v[s], sum);
                u[t] = sum;
                if ((t & 3) == 3) *reinterpret_cast<float4*>(out + (j % CB) * CT + t - 3) = make_float4(u[t - 3], u[t - 2], u[t - 1], u[t]);
            } else {
                u[t] = v[t];
            }
        }
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            float sum = 0.f;
#pragma unroll
            for (int s = 0; s <= t; ++s) sum = fmaf(Bs[t][s], u[s], sum);
            v[t] = sum;
            if ((t & 3) == 3) *reinterpret_cast<float4*>(out + L::O0 + (j % CB) * CT + t - 3) = make_float4(v[t - 3], v[t - 2], v[t - 1], v[t]);
        }
    }
}

// Contiguous floats (16-byte aligned, a multiple of four) into shared memory; the barrier counts the bytes.
__device__ __forceinline__ void copy_bulk(float* dst, const float* src, int floats, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(floats * 4), "r"(smem_u32(bar)) : "memory");
}

// Two 32-bit multiply-adds in one instruction (each rounded as fmaf).
__device__ __forceinline__ void fma2(float& x, float& y, float a, float b, float u) {
    asm("{ .reg .b64 p, q, r; mov.b64 p, {%0, %1}; mov.b64 q, {%2, %3}; mov.b64 r, {%4, %4}; fma.rn.f32x2 p, q, r, p; mov.b64 {%0, %1}, p; }"
        : "+f"(x), "+f"(y) : "f"(a), "f"(b), "f"(u));
}

// The operands of mma.sync m16n8k16 in three parts each, [part][register].
struct Rows3 { uint32_t r[3][4]; };
struct Cols3 { uint32_t r[3][2][2]; };       // two right operands side by side
// A times each of the two of B (16 x 16 by 16 x 8) of 32-bit numbers: the products of the parts down to 2^-16 of the largest, as three
// sums each (a chain of products waits 21 cycles for every one of two chains, 12 for one of eight). The tensor cores cut
// their sums instead of rounding them, so the largest parts' products stand alone.
__device__ __forceinline__ void product3(float (&out)[2][4], const Rows3& a, const Cols3& b) {
    float x[2][3][4];
#pragma unroll
    for (int i = 0; i < 12; ++i) (&x[0][0][0])[i] = (&x[1][0][0])[i] = 0.f;
    constexpr int PA[6] = {0, 2, 0, 1, 0, 1}, PB[6] = {0, 0, 2, 1, 1, 0}, TO[6] = {2, 0, 1, 0, 1, 0};
#pragma unroll
    for (int p = 0; p < 6; ++p)
#pragma unroll
        for (int j = 0; j < 2; ++j) mma_bf16(x[j][TO[p]], a.r[PA[p]], b.r[PB[p]][j][0], b.r[PB[p]][j][1]);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) out[j][i] = (x[j][0][i] + x[j][1][i]) + x[j][2][i];
}

template <int DIM, bool DELTA> struct Walk {
    static constexpr int WARPS = DIM / 16, READ = DELTA ? WARPS : 0, SUMS = 4, MEET = (WARPS + READ + SUMS) * 32, THREADS = MEET + 32;
    static constexpr int PART = WARPS * CT * CB;        // a product's sums over every warp's channels
    static constexpr int UP = CT + 4, US = DELTA ? 1 : 3;           // u by columns, UP floats apart (a phase's reads and stores meet few banks twice)
    static constexpr int SMEM_FLOATS = (DELTA ? 3 * PART + 2 * WARPS * 3 * 32 * 4 : 2 * PART) + US * CB * UP;
};

// What a block of the walk below does, by multiply-adds from the numbers the workspace's parts stand for: for blocks where a product of
// parts is not finite (an infinite operand's parts leave none, nor do those of the largest finite ones), once they have found that. The
// warps that meet take part; sm: DIM (CB + 1) + CT CB floats of shared memory; ws, o, v: of the first chunk; left: the portion's tokens
// from there on.
template <int DIM, bool DELTA>
__device__ __forceinline__ void walk_whole(float* sm, const float* ws, long long chunk_stride, int blk, float* st, int dim, int vd, float* o,
                                        long long o_ld, const float* v, long long ld_v, int left, int n_chunks) {
    using L = Layout<DIM, DELTA>;
    using W = Walk<DIM, DELTA>;
    auto meet = []() { asm volatile("bar.sync 1, %0;" ::"n"(W::MEET) : "memory"); };
    float *S = sm, *u = sm + DIM * (CB + 1);     // [DIM][CB + 1], [CT][CB]
    const int tid = threadIdx.x, col0 = blk * CB;
    for (int i = tid; i < DIM * CB; i += W::MEET) {
        const int r = i / CB, c = i % CB;
        S[r * (CB + 1) + c] = r < dim && col0 + c < vd ? st[(size_t)r * vd + col0 + c] : 0.f;
    }
    for (int n = 0; n < n_chunks; ++n, ws += chunk_stride, o += CT * o_ld, v += CT * ld_v, left -= CT) {
        meet();
        const float* uo = ws + L::ROWS + (size_t)blk * L::COLS;
        for (int i = tid; i < CT * CB; i += W::MEET) {
            const int t = i / CB, c = i % CB;
            const bool on = t < left && col0 + c < vd;
            auto times_S = [&](int kind) {       // row t of the right operands of this kind
                float sum = 0.f;
                for (int r = 0; r < DIM; ++r) {
                    const uint32_t* x = reinterpret_cast<const uint32_t*>(ws) + ((r >> 4) * L::KINDS + kind) * L::OPERAND +
                                        ((t & 7) * 4 + ((r >> 2) & 3)) * 4 + (t >> 3) * 2 + ((r >> 1) & 1);
                    sum = fmaf(whole_of(x[0], x[128], x[256], r & 1), S[r * (CB + 1) + c], sum);
                }
                return sum;
            };
            u[i] = DELTA ? uo[c * CT + t] + times_S(0) : on ? v[(long long)t * ld_v + c] : 0.f;
            const float y = uo[L::O0 + c * CT + t] + times_S(L::KINDS - 1);
            if (on) o[(long long)t * o_ld + c] = y;
        }
        meet();
        for (int i = tid; i < DIM * CB; i += W::MEET) {
            const int r = i / CB, c = i % CB;
            float x = S[r * (CB + 1) + c] * ws[L::DECAY + r];
            for (int t = 0; t < CT; ++t) x = fmaf(ws[L::KE + t * DIM + r], u[t * CB + c], x);
            S[r * (CB + 1) + c] = x;
        }
    }
    for (int i = tid; i < DIM * CB; i += W::MEET) {          // (the thread's own)
        const int r = i / CB, c = i % CB;
        if (r < dim && col0 + c < vd) st[(size_t)r * vd + col0 + c] = S[r * (CB + 1) + c];
    }
}

// A block carries CB columns of one (request, head)'s S through the request's chunks that are in the workspace; 16 columns make 128
// blocks of a prompt over 16 heads of 128 columns, which is nearly the GPU. Its warps by their work:
//   WARPS   hold 16 channels by 16 columns of S^T each, in the places of a left operand of mma.sync m16n8k16: S^T [-W]^T over their
//           channels, for u; then S^T <- S^T diag(E) + u^T (k E), token after token (HGRN2: u is the values)
//   READ    take the read-outs S^T Q^T over as many channels each, from copies of that left operand, beside the chain (HGRN2, whose chain
//           is short: the state's warps do, and two blocks fit an SM, which many requests need)
//   SUMS    add the warps' sums, in a fixed order, with U0 or O0 on top: u goes back by columns, o to memory
//   1       copies the chunks ahead of them all
// All numbers stay 32-bit: a product's operand enters as three bfloat16 numbers, the product as the six products of parts above 2^-24 of
// it (product3); sums over more than 16 terms are 32-bit additions. A block that has found a u or a read-out that is not finite starts again
// (walk_whole).
// Bound by the chain of a chunk, 0.95 us: products (24 of mma.sync a scheduler, 9 cycles each), the meeting of the warps, u's sums, u
// back to all of them, 64 multiply-adds of pairs a thread with their loads (which keep shared memory busy for 0.69 of the time). With multiply-adds on S in shared memory for both products
// the walk took 166 us for 2,048 tokens and 16 heads of 128 x 128, bound by shared memory's bandwidth; this form 121 (105 with both on
// the tensor cores, see the errors above). What that took: no mbarrier on the chain, loads ahead of the waits, read-outs and
// sums on warps of their own. HGRN2 with 12 heads of 64 x 128, which has no u to wait for: two prompts of 112 chunks 88 -> 58 us. Where blocks
// are many the workspace's bytes count: every block of columns reads its head's operands. HGRN2's values are fetched here, by the warps of the
// sums, two chunks ahead. Vectors and walk of 32 portions of 100 tokens over 16 heads of 128 x 128: delta rule 398 us (multiply-adds 463),
// HGRN2 205 (239); 16 portions of 1,000 tokens 1,505 (1,699) and 906 (1,026); heads of 64 x 64, 6 portions of 351 tokens, 75 (81) and 45 (53).
template <int DIM, bool DELTA>
__global__ void __launch_bounds__(Walk<DIM, DELTA>::THREADS, DIM == 128 && DELTA ? 1 : 2)
chunk_walk_kernel(float* __restrict__ o_out, float* __restrict__ state, long long slot_stride, int n_slots, const ChunkArgs a,
                  int* __restrict__ err) {
    using L = Layout<DIM, DELTA>;
    using W = Walk<DIM, DELTA>;
    constexpr int WARPS = W::WARPS, SUMS = W::SUMS;
    extern __shared__ __align__(16) float sm[];
    float* part = sm + a.stages * L::STAGE;      // [3][WARPS][CT * CB]: read-outs of even and of odd chunks, u
    float* u_part = part + 2 * W::PART;
    uint32_t* frags = reinterpret_cast<uint32_t*>(part + 3 * W::PART);        // [2][WARPS] S before even and before odd chunks
    float* u_cols = DELTA ? reinterpret_cast<float*>(frags + 2 * WARPS * L::OPERAND) : part + 2 * W::PART;        // [US][CB][UP]
    __shared__ uint64_t full[MAX_STAGES], empty[MAX_STAGES];
    __shared__ int abort_flag_, again_;
    volatile int *abort_flag = &abort_flag_, *again = &again_;
    // the column blocks of a head, its request's heads, the requests: neighbours run through the same chunks at the same time (with
    // the requests' blocks in turn, two prompts of unequal lengths took 326 us through both mixers instead of 295)
    const int blocks = (a.vd + CB - 1) / CB, blk = blockIdx.x % blocks, h = blockIdx.x / blocks % a.heads, b = blockIdx.x / blocks / a.heads;
    const int tid = threadIdx.x, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < a.stages; ++i) mbar_init(&full[i], 1), mbar_init(&empty[i], 1);
        abort_flag_ = again_ = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_trigger();
    pdl_wait();
    const int slot = a.slot_ids[b];
    if (slot < 0 || slot >= n_slots) { if (tid == 0) atomicOr(err, CELLM_DEV_BAD_SLOT); return; }
    const int start = a.cu_seqlens[b], len = a.cu_seqlens[b + 1] - start;
    if (len < a.min_len) return;
    int before = 0;                              // chunks of the requests before this one
    for (int i = lane; i < b; i += 32) before += chunks_of(a, i);
    before = __reduce_add_sync(0xffffffffu, before);
    const int c0 = max(0, a.chunk0 - before), n_chunks = min((len + CT - 1) / CT, a.chunk0 + a.chunks - before) - c0;
    if (n_chunks <= 0) return;
    __syncthreads();
    const int warp = (tid >> 5) % WARPS;
    const int g = lane >> 2, t4 = lane & 3, col0 = blk * CB;
    int at = 0;                                  // the chunk's stage
    uint32_t lap = 0;
    auto next = [&]() { if (++at == a.stages) at = 0, ++lap; };
    // the products' right operands over the warp's channels: -W (delta rule), Q
    auto right_operands = [&](Cols3& x, int kind) {
        const float* from = sm + at * L::STAGE + (size_t)(warp * L::KINDS + kind) * L::OPERAND + lane * 4;
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const uint4 y = *reinterpret_cast<const uint4*>(from + p * 128);
            x.r[p][0][0] = y.x, x.r[p][0][1] = y.y, x.r[p][1][0] = y.z, x.r[p][1][1] = y.w;
        }
    };
    auto left_operand = [&](Rows3& x, const uint32_t* from) {
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            const uint4 y = *reinterpret_cast<const uint4*>(from + (p * 32 + lane) * 4);
            x.r[p][0] = y.x, x.r[p][1] = y.y, x.r[p][2] = y.z, x.r[p][3] = y.w;
        }
    };
    float y[2][4];
    // a warp's product into its place among the warps'
    auto put = [&](float* p) {
        p += warp * (CT * CB) + lane * 4;
#pragma unroll
        for (int j = 0; j < 2; ++j)
            *reinterpret_cast<float4*>(p + 128 * j) = make_float4(y[j][0], y[j][1], y[j][2], y[j][3]);
    };
    // Once a chunk all but the copying warp meet: from then on the next chunk is there, S before this one and every warp's share of -W S
    // can be read, and so can the shares of read-outs (of the last chunk; HGRN2: of this one); the last chunk's stage is free. The state's warps of the delta rule only
    // say so and wait where u is whole. (An mbarrier costs a wait 60 cycles even where it has been passed: only the sums' warps look at
    // the copies' and tell the others.)
    auto meet = []() { asm volatile("bar.sync 1, %0;" ::"n"(W::MEET) : "memory"); };
    auto meet_later = []() { asm volatile("bar.arrive 1, %0;" ::"n"(W::MEET) : "memory"); };
    auto u_whole = []() { asm volatile("bar.arrive 2, %0;" ::"n"((WARPS + SUMS) * 32) : "memory"); };
    auto wait_u = []() { asm volatile("bar.sync 2, %0;" ::"n"((WARPS + SUMS) * 32) : "memory"); };
    float* st = state + (size_t)slot * slot_stride + (size_t)h * a.dim * a.vd;
    if (tid >= W::MEET) {        // ------------------------------------------------ copies
        if (lane != 0) return;
        const float* ws = a.ws + ((size_t)(before + c0 - a.chunk0) * a.heads + h) * a.stride;
        int issued = 0;
        for (; issued < n_chunks; ++issued, ws += (size_t)a.heads * a.stride) {
            if (lap && !mbar_wait(&empty[at], (lap - 1) & 1u, abort_flag)) break;
            mbar_expect_tx(&full[at], L::STAGE * 4);
            copy_bulk(sm + at * L::STAGE, ws, L::ROWS, &full[at]);
            copy_bulk(sm + at * L::STAGE + L::ROWS, ws + L::ROWS + (size_t)blk * L::COLS, L::COLS, &full[at]);
            next();
        }
        if (issued < n_chunks) {        // given up: the copies under way still land in this block's memory
            *abort_flag = 1;
            atomicOr(err, CELLM_DEV_WAIT_TIMEOUT);
        }
        int none = 0;
        for (int c = max(0, issued - a.stages); c < issued; ++c) mbar_wait(&full[c % a.stages], (uint32_t)(c / a.stages) & 1u, &none);
        return;
    }
    do {                                         // (one of three)
    if (tid >= (WARPS + W::READ) * 32) {                             // ------------------------------------------------ sums over the warps
        // a thread: one column of two neighbouring tokens, registers 2 half and 2 half + 1 of lane l's accumulator j
        const int r = tid - (WARPS + W::READ) * 32, l = (r >> 1) & 31, half = r & 1, j = r >> 6;
        const int col = (l >> 2) + 8 * half, token = 8 * j + 2 * (l & 3);
        auto add_up = [&](const float* p, float2 x) {
            float2 y[WARPS];
#pragma unroll
            for (int w = 0; w < WARPS; ++w) y[w] = *reinterpret_cast<const float2*>(p + w * (CT * CB) + 2 * r);
#pragma unroll
            for (int n = WARPS / 2; n >= 1; n >>= 1)
#pragma unroll
                for (int w = 0; w < n; ++w) y[w].x += y[w + n].x, y[w].y += y[w + n].y;
            return make_float2(x.x + y[0].x, x.y + y[0].y);
        };
        bool ok = true, finite = true;
        auto look = [&](float2 x) { finite = finite && fabsf(x.x + x.y) < INFINITY; };
        auto there = [&]() {
            if (mbar_wait(&full[at], lap & 1u, abort_flag)) return;
            ok = false;                          // bounded: every warp still runs through its chunks, and nothing is written
            *abort_flag = 1;
            atomicOr(err, CELLM_DEV_WAIT_TIMEOUT);
        };
        const size_t o_ld = (size_t)a.heads * a.vd;
        float* o = o_out + (size_t)(start + c0 * CT + token) * o_ld + (size_t)h * a.vd + col0 + col;
        int left = col0 + col < a.vd ? len - c0 * CT - token : 0;        // tokens from the thread's first on
        auto read_out = [&](int c, float2 x) {
            x = add_up(part + (c & 1) * W::PART, x);
            look(x);
            if (ok && left > 0) *o = x.x;
            if (ok && left > 1) o[o_ld] = x.y;
            o += CT * o_ld, left -= CT;
        };
        float2 u0 = make_float2(0.f, 0.f), o0 = u0;
        // HGRN2: u is the values, which are fetched two chunks ahead
        const float* v = a.v + (size_t)(start + c0 * CT + token) * a.ld_v + (size_t)h * a.vd + col0 + col;
        auto values = [&](int ahead) {
            const float* p = v + (size_t)ahead * CT * a.ld_v;
            const int n = left - ahead * CT;
            return make_float2(n > 0 ? p[0] : 0.f, n > 1 ? p[a.ld_v] : 0.f);
        };
        auto place = [&](int c, float2 x) { *reinterpret_cast<float2*>(u_cols + (c % W::US * CB + col) * W::UP + token) = x; };
        float2 v1 = u0, v2 = u0;
        if constexpr (!DELTA) {
            const float2 v0 = values(0);
            v1 = values(1);
            place(0, v0);
        }
        there();
        meet();
        for (int c = 0; c < n_chunks; ++c) {
            if constexpr (!DELTA) v2 = values(2), v += (size_t)CT * a.ld_v;
            const float* uo = sm + at * L::STAGE + L::ROWS + col * CT + token;
            const float2 o1 = *reinterpret_cast<const float2*>(uo + L::O0);
            if constexpr (DELTA) u0 = *reinterpret_cast<const float2*>(uo);
            const int last = at == 0 ? a.stages - 1 : at - 1;
            next();
            if constexpr (!DELTA) place(c + 1, v1), v1 = v2;
            if (c + 1 < n_chunks) there();
            meet();
            if constexpr (DELTA) {
                const float2 x = add_up(u_part, u0);
                place(c, x);
                u_whole();
                look(x);
            }
            if (c > 0 && r == 0) mbar_arrive(&empty[last]);
            // the delta rule's read-outs are formed while u's sums are: they are there a chunk later
            if constexpr (!DELTA) read_out(c, o1);
            else if (c > 0) read_out(c - 1, o0);
            o0 = o1;
        }
        meet();
        if constexpr (DELTA) read_out(n_chunks - 1, o0);
        if (!finite) *again = 1;
        meet();
        break;
    }
    Cols3 w;
    if (DELTA && tid >= WARPS * 32) {                             // ------------------------------------------------ read-outs
        meet();
        right_operands(w, L::KINDS - 1);
        for (int c = 0; c < n_chunks; ++c) {
            meet();
            Rows3 s;
            left_operand(s, frags + ((c & 1) * WARPS + warp) * L::OPERAND);
            product3(y, s, w);
            next();
            if (c + 1 < n_chunks) right_operands(w, L::KINDS - 1);
            put(part + (c & 1) * W::PART);
        }
        meet();
        meet();
        break;
    }
    // -------------------------------------------------------------------------------------------- the state
    // the lane's entries of S: accumulator j's register 2 c + e is channel row + 2 j + e, column g + 8 c of the block
    const int row = warp * 16 + t4 * 4;
    auto entry = [&](int j, int i) -> float* {
        const int r = row + 2 * j + (i & 1), c = col0 + g + 8 * (i >> 1);
        return (r < a.dim && c < a.vd) ? st + (size_t)r * a.vd + c : nullptr;
    };
    float S[2][4];
    Rows3 s;                                     // S as a left operand
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float* p = entry(j, i);
            S[j][i] = p ? *p : 0.f;
        }
    auto split_state = [&]() {
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int c = 0; c < 2; ++c) split3<false>(s.r[0][2 * j + c], s.r[1][2 * j + c], s.r[2][2 * j + c], S[j][2 * c], S[j][2 * c + 1]);
    };
    split_state();
    meet();
    right_operands(w, 0);
    for (int c = 0; c < n_chunks; ++c) {
        product3(y, s, w);
        const float* stage = sm + at * L::STAGE;
        next();
        const float4 e = *reinterpret_cast<const float4*>(stage + L::DECAY + row);
        if constexpr (DELTA) {
#pragma unroll
            for (int p = 0; p < 3; ++p)
                *reinterpret_cast<uint4*>(frags + ((c & 1) * WARPS + warp) * L::OPERAND + (p * 32 + lane) * 4) =
                    make_uint4(s.r[p][0], s.r[p][1], s.r[p][2], s.r[p][3]);
            put(u_part);
            meet_later();
        } else {
            put(part + (c & 1) * W::PART);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) S[0][i] *= i & 1 ? e.y : e.x, S[1][i] *= i & 1 ? e.w : e.z;
        float4 first[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) first[t] = *reinterpret_cast<const float4*>(stage + L::KE + t * DIM + row);
        if constexpr (DELTA) wait_u(); else meet();
        // S <- diag(E) S + (k E)^T u, token after token in 32 bits
        const float* us = u_cols + (c % W::US * CB + g) * W::UP;
        if (c + 1 < n_chunks) right_operands(w, 0);          // (beside the multiply-adds)
#pragma unroll
        for (int t = 0; t < CT; t += 4) {
            const float4 ua = *reinterpret_cast<const float4*>(us + t), ub = *reinterpret_cast<const float4*>(us + 8 * W::UP + t);
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                const float4 k = t == 0 ? first[d] : *reinterpret_cast<const float4*>(stage + L::KE + (t + d) * DIM + row);
                const float a0 = d == 0 ? ua.x : d == 1 ? ua.y : d == 2 ? ua.z : ua.w, a1 = d == 0 ? ub.x : d == 1 ? ub.y : d == 2 ? ub.z : ub.w;
                fma2(S[0][0], S[0][1], k.x, k.y, a0), fma2(S[0][2], S[0][3], k.x, k.y, a1);
                fma2(S[1][0], S[1][1], k.z, k.w, a0), fma2(S[1][2], S[1][3], k.z, k.w, a1);
            }
        }
        split_state();
    }
    meet();
    meet();
    if (*again || *abort_flag) break;            // (the copies gave up: the state stays as it was)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (float* p = entry(j, i)) *p = S[j][i];
    } while (false);
    // behind the second of the two last meetings: whether something was not finite
    if (!*again || *abort_flag) return;
    const size_t first = (size_t)start + (size_t)c0 * CT, at_col = (size_t)h * a.vd + col0;
    walk_whole<DIM, DELTA>(sm, a.ws + ((size_t)(before + c0 - a.chunk0) * a.heads + h) * a.stride, (long long)a.heads * a.stride, blk, st, a.dim, a.vd,
                           o_out + first * a.heads * a.vd + at_col, (long long)a.heads * a.vd, DELTA ? nullptr : a.v + first * a.ld_v + at_col, a.ld_v,
                           len - c0 * CT, n_chunks);
}

template <int DIM, bool DELTA> int floats_a_chunk(int vd) {
    return Layout<DIM, DELTA>::ROWS + ((vd + CB - 1) / CB) * Layout<DIM, DELTA>::COLS;
}

template <int DIM, bool DELTA>
int run(float* o_out, float* state, long long slot_stride, int n_slots, ChunkArgs a, int n_chunks, int ws_chunks, int* err, cudaStream_t stream) {
    using L = Layout<DIM, DELTA>;
    a.stride = floats_a_chunk<DIM, DELTA>(a.vd);
    const long long walk_blocks = (long long)a.B * a.heads * ((a.vd + CB - 1) / CB);
    if (walk_blocks > INT_MAX) return CELLM_ERR_SIZE;
    // The walk's blocks become resident while chunk_vectors still runs, wherever it leaves room first: without a bound two of them met
    // on one SM beside idle ones (delta rule, 128 blocks: 233 us for both kernels instead of 170). So a block asks for as
    // much shared memory as lets an SM hold no more of them than an even spread needs, and makes stages of it (more than four bring
    // nothing and keep the next kernel's blocks out: two prompts through both mixers 283 us with up to eight, 270 with four).
    const int an_sm = (int)std::min<long long>((walk_blocks + 147) / 148, 8);
    constexpr int fixed = Walk<DIM, DELTA>::SMEM_FLOATS * 4, stage = L::STAGE * 4;
    a.stages = std::max(MIN_STAGES, std::min(MAX_STAGES, (224 * 1024 / an_sm - 2048 - fixed) / stage));
    const size_t smem = std::max(a.stages * stage + fixed, 228 / (an_sm + 1) * 1024);
    cudaError_t e = cudaFuncSetAttribute(chunk_walk_kernel<DIM, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024);
    if (e != cudaSuccess) return (int)e;
    for (a.chunk0 = 0; a.chunk0 < n_chunks; a.chunk0 += ws_chunks) {
        a.chunks = std::min(ws_chunks, n_chunks - a.chunk0);
        CELLM_RUN((chunk_vectors_kernel<DIM, DELTA>), dim3(a.chunks, a.heads), DIM, 0, stream, a);
        CELLM_RUN((chunk_walk_kernel<DIM, DELTA>), (unsigned)walk_blocks, (Walk<DIM, DELTA>::THREADS), smem, stream, o_out, state,
                  slot_stride, n_slots, a, err);
    }
    return CELLM_OK;
}

bool fits(int B, int heads, int per, int dim, int vd, int n_chunks, int ws_chunks, const void* ws) {
    return B > 0 && heads > 0 && per > 0 && heads % per == 0 && dim > 0 && dim <= 128 && vd > 0 && n_chunks > 0 && ws_chunks > 0 &&
           (reinterpret_cast<uintptr_t>(ws) & 15) == 0;
}

}  // namespace

// 32-bit floats of workspace for each (chunk of 16 tokens, head); 0: sizes that are not taken (heads of more than 128 rows).
CELLM_API int cellm_state_chunks_floats(int delta, int dim, int vd) {
    if (dim <= 0 || dim > 128 || vd <= 0) return 0;
    if (dim <= 64) return delta ? floats_a_chunk<64, true>(vd) : floats_a_chunk<64, false>(vd);
    return delta ? floats_a_chunk<128, true>(vd) : floats_a_chunk<128, false>(vd);
}

// The gated delta rule over the portions of at least min_len tokens (n_chunks: the sum of their lengths / 16, each rounded up);
// the others are left alone. Arguments as cellm_delta_scan; ws: ws_chunks * heads * cellm_state_chunks_floats(1, ..) floats,
// 16-byte aligned: where it holds fewer chunks than there are, they go through it in runs (two launches each), the state
// through memory between them; the result is the same.
CELLM_API int cellm_delta_chunks(float* o_out, float* state, long long slot_stride, int n_slots, const float* qk, const float* v,
                                 const float* beta, const float* decay, const int* cu_seqlens, const int* slot_ids, int B, int n_chunks,
                                 int ws_chunks, int min_len, int heads, int kvh, int dim, int vd, float* ws, int* err, cudaStream_t stream) {
    if (kvh <= 0 || heads % kvh || !fits(B, heads, heads / kvh, dim, vd, n_chunks, ws_chunks, ws) || min_len < 1) return CELLM_ERR_SIZE;
    const long long ld = 2LL * kvh * dim;
    ChunkArgs a{qk, qk + (size_t)kvh * dim, decay, v, beta, ld, ld, (long long)heads * dim, (long long)heads * vd, heads / kvh,
                cu_seqlens, slot_ids, B, min_len, heads, dim, vd, ws, 0, 0, 0, 0};
    return dim <= 64 ? run<64, true>(o_out, state, slot_stride, n_slots, a, n_chunks, ws_chunks, err, stream)
                     : run<128, true>(o_out, state, slot_stride, n_slots, a, n_chunks, ws_chunks, err, stream);
}

// HGRN2 likewise; q and f (already silu and forget gate, as cellm_hgrn2_gates leaves them) and v are columns of proj [T, ld].
CELLM_API int cellm_hgrn2_chunks(float* o_out, float* state, long long slot_stride, int n_slots, const float* proj, long long ld, int col_q,
                                 int col_f, int col_v, const int* cu_seqlens, const int* slot_ids, int B, int n_chunks, int ws_chunks,
                                 int min_len, int heads, int dim, int vd, float* ws, int* err, cudaStream_t stream) {
    if (!fits(B, heads, 1, dim, vd, n_chunks, ws_chunks, ws) || min_len < 1) return CELLM_ERR_SIZE;
    ChunkArgs a{proj + col_q, nullptr, proj + col_f, proj + col_v, nullptr, ld, 0, ld, ld, 1, cu_seqlens, slot_ids, B, min_len, heads, dim, vd, ws, 0, 0, 0, 0};
    return dim <= 64 ? run<64, false>(o_out, state, slot_stride, n_slots, a, n_chunks, ws_chunks, err, stream)
                     : run<128, false>(o_out, state, slot_stride, n_slots, a, n_chunks, ws_chunks, err, stream);
}
