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
// Everything is 32-bit fused multiply-adds, as token by token (relative error of the read-outs against 64 bits over 2,048 tokens
// 8.9e-8, token by token 8.7e-8). One prompt of 2,048 tokens, 16 heads of 128 x 128: 938 -> 215 us (49 of them chunk_vectors).
#include <algorithm>
#include <climits>

#include "tcgen05.cuh"

namespace {

constexpr int CT = 16;          // tokens a chunk
constexpr int CB = 16;          // columns of S a block of the walk holds
constexpr int WALK_THREADS = 256;
constexpr int STAGES = 3;

struct ChunkArgs {
    const float *q, *k, *g, *v, *beta;      // k, beta: null for HGRN2
    long long ld_q, ld_k, ld_g, ld_v;
    int per;                                // heads that share a row of q and k
    const int *cu_seqlens, *slot_ids;
    int B, min_len, heads, dim, vd;
    float* ws;                              // a chunk's and head's numbers at ((chunk - chunk0) * heads + head) * stride floats
    long long stride;
    int chunk0, chunks;                     // the step's chunks that are in the workspace
};

// A (chunk, head) in the workspace: [NV][DIM] the rows of -W and Q (HGRN2: Q alone), [CT][DIM] k E(., end), [DIM] E(., end), then
// per block of CB columns [CT][CB] of U0 and [CT][CB] of O0.
template <int DIM, bool DELTA> struct Layout {
    static constexpr int NV = DELTA ? 2 * CT : CT;
    static constexpr int ROWS = (NV + CT + 1) * DIM;
    static constexpr int COLS = 2 * CT * CB;
    static constexpr int STAGE = ROWS + COLS;
};

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

// A block a (chunk, head), a thread a channel. Bound by latency and by what it writes (41 KB a block of the delta rule with
// 128 x 128).
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
    int t0 = 0, len = 0;
    for (int b = 0, c = a.chunk0 + blockIdx.x; b < a.B; ++b) {
        const int start = a.cu_seqlens[b], n = a.cu_seqlens[b + 1] - start;
        if (n < a.min_len) continue;
        const int nc = (n + CT - 1) / CT;
        if (c < nc) { t0 = start + c * CT; len = min(CT, n - c * CT); break; }
        c -= nc;
    }
    if (len == 0) return;
    float* ws = a.ws + ((size_t)blockIdx.x * a.heads + h) * a.stride;
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
            ws[(L::NV + t) * DIM + tid] = k[t] * e;
            e *= g[t];
        }
        ws[(L::NV + CT) * DIM + tid] = e;
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
        float e = 1.f, w[CT];
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            e *= g[t];
            q[t] *= e;
            k[t] *= e;
        }
        if constexpr (DELTA) {
#pragma unroll
            for (int t = 0; t < CT; ++t) {
                float sum = 0.f;
#pragma unroll
                for (int s = 0; s <= t; ++s) sum = fmaf(Ts[t][s], k[s], sum);
                w[t] = -sum;
                ws[t * DIM + tid] = -sum;
            }
        }
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            float sum = q[t];
            if constexpr (DELTA) {
#pragma unroll
                for (int s = 0; s <= t; ++s) sum = fmaf(Bs[t][s], w[s], sum);
            }
            ws[(L::NV - CT + t) * DIM + tid] = sum;
        }
    }
    const int blocks = (a.vd + CB - 1) / CB;
#pragma unroll 1
    for (int j = tid; j < blocks * CB; j += DIM) {
        asm volatile("" ::: "memory");       // T and B come from shared memory again for every column: 272 values are no registers
        float v[CT], u[CT];
#pragma unroll
        for (int t = 0; t < CT; ++t) v[t] = (j < a.vd && t < len) ? a.v[(size_t)(t0 + t) * a.ld_v + h * a.vd + j] : 0.f;
        float* out = ws + L::ROWS + (size_t)(j / CB) * L::COLS + j % CB;
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            if constexpr (DELTA) {
                float sum = 0.f;
#pragma unroll
                for (int s = 0; s <= t; ++s) sum = fmaf(Ts[t][s], v[s], sum);
                u[t] = sum;
            } else {
                u[t] = v[t];
            }
            out[t * CB] = u[t];
        }
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            float sum = 0.f;
#pragma unroll
            for (int s = 0; s <= t; ++s) sum = fmaf(Bs[t][s], u[s], sum);
            out[(CT + t) * CB] = sum;
        }
    }
}

// Two 32-bit multiply-adds in one instruction (each rounded as fmaf).
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long pair_of(float lo, float hi) {
    return (unsigned long long)__float_as_uint(hi) << 32 | __float_as_uint(lo);
}
__device__ __forceinline__ float low_of(unsigned long long x) { return __uint_as_float((unsigned)x); }
__device__ __forceinline__ float high_of(unsigned long long x) { return __uint_as_float((unsigned)(x >> 32)); }

// Contiguous floats (16-byte aligned, a multiple of four) into shared memory; the barrier counts the bytes.
__device__ __forceinline__ void copy_bulk(float* dst, const float* src, int floats, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_u32(dst)), "l"(src), "r"(floats * 4), "r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void set_barrier(int set) { asm volatile("bar.sync %0, 128;" ::"r"(set + 1) : "memory"); }

// A block carries CB columns of one (request, head)'s S through the request's chunks that are in the workspace; 16 columns make 128 blocks of a prompt
// over 16 heads of 128 columns, which is nearly the GPU. Two sets of four warps carry eight columns each, on their own barriers,
// so that one set's first product runs beside the other's second; a ninth warp copies the chunks ahead of them. S lies twice: a
// thread's own entries in registers, which the second product moves on, and all of it by columns in shared memory, which the
// first one reads.
//   first product   [-W ; Q] S: a warp takes a quarter of the rows, 16 lanes split the channels, a lane forms NV / 4 x 4 sums
//                   over its share; the lanes' shares are added so that every lane ends with its own of the sums. U0 and O0
//                   are added: u goes to shared memory, o to memory.
//   second product  S <- diag(E) S + (k E)^T u, a thread two or four rows by two columns.
// Bound by shared memory's bandwidth (every warp reads its share of the chunk's rows and the set's columns). With all eight warps
// on one barrier and every thread copying, the phases added up: 290 us a prompt of 2,048 tokens where this form takes 166.
template <int DIM, bool DELTA>
__global__ void __launch_bounds__(WALK_THREADS + 32)
chunk_walk_kernel(float* __restrict__ o_out, float* __restrict__ state, long long slot_stride, int n_slots, const ChunkArgs a,
                  int* __restrict__ err) {
    using L = Layout<DIM, DELTA>;
    constexpr int MT = L::NV / 4, SP = DIM + 4, RPT = DIM / 32;
    extern __shared__ __align__(16) float sm[];
    float* Ssh = sm + STAGES * L::STAGE;         // [CB][SP]: column by column
    float* ush = Ssh + CB * SP;                  // [2 sets][CT][CB / 2]
    __shared__ uint64_t full[STAGES], empty[STAGES];
    __shared__ int abort_flag_;
    volatile int* abort_flag = &abort_flag_;
    // the column blocks of a head, its request's heads, the requests: neighbours run through the same chunks at the same time (with
    // the requests' blocks in turn, two prompts of unequal lengths took 326 us through both mixers instead of 295)
    const int blocks = (a.vd + CB - 1) / CB, blk = blockIdx.x % blocks, h = blockIdx.x / blocks % a.heads, b = blockIdx.x / blocks / a.heads;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int i = 0; i < STAGES; ++i) mbar_init(&full[i], 1), mbar_init(&empty[i], WALK_THREADS / 32);
        abort_flag_ = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    pdl_trigger();
    pdl_wait();
    const int slot = a.slot_ids[b];
    if (slot < 0 || slot >= n_slots) { if (tid == 0) atomicOr(err, CELLM_DEV_BAD_SLOT); return; }
    const int start = a.cu_seqlens[b], len = a.cu_seqlens[b + 1] - start;
    if (len < a.min_len) return;
    int before = 0;                              // chunks of the requests before this one
    for (int i = 0; i < b; ++i) {
        const int n = a.cu_seqlens[i + 1] - a.cu_seqlens[i];
        if (n >= a.min_len) before += (n + CT - 1) / CT;
    }
    const int c0 = max(0, a.chunk0 - before), n_chunks = min((len + CT - 1) / CT, a.chunk0 + a.chunks - before) - c0;
    if (n_chunks <= 0) return;
    __syncthreads();
    if (warp == WALK_THREADS / 32) {
        if (lane != 0) return;
        const float* ws = a.ws + ((size_t)(before + c0 - a.chunk0) * a.heads + h) * a.stride;
        int issued = 0;
        for (; issued < n_chunks; ++issued, ws += (size_t)a.heads * a.stride) {
            const int st = issued % STAGES;
            if (issued >= STAGES && !mbar_wait(&empty[st], (uint32_t)(issued / STAGES - 1) & 1u, abort_flag)) break;
            mbar_expect_tx(&full[st], L::STAGE * 4);
            copy_bulk(sm + st * L::STAGE, ws, L::ROWS, &full[st]);
            copy_bulk(sm + st * L::STAGE + L::ROWS, ws + L::ROWS + (size_t)blk * L::COLS, L::COLS, &full[st]);
        }
        if (issued < n_chunks) {        // given up: the copies under way still land in this block's memory
            *abort_flag = 1;
            atomicOr(err, CELLM_DEV_WAIT_TIMEOUT);
        }
        int none = 0;
        for (int c = max(0, issued - STAGES); c < issued; ++c) mbar_wait(&full[c % STAGES], (uint32_t)(c / STAGES) & 1u, &none);
        return;
    }
    const int set = warp >> 2, vg = warp & 3, col0 = blk * CB;
    // the thread's entries of S: rows row .. row + RPT - 1, columns col, col + 1 of the block's
    const int row = vg * (DIM / 4) + (lane >> 2) * RPT, col = set * (CB / 2) + (lane & 3) * 2;
    float* st = state + (size_t)slot * slot_stride + (size_t)h * a.dim * a.vd;
    unsigned long long S[RPT / 2][2];            // [pair of rows][column]
    auto entry = [&](int r, int c) -> float* {
        return (row + r < a.dim && col0 + col + c < a.vd) ? st + (size_t)(row + r) * a.vd + col0 + col + c : nullptr;
    };
    auto publish = [&]() {
#pragma unroll
        for (int r = 0; r < RPT / 2; ++r)
#pragma unroll
            for (int c = 0; c < 2; ++c) *reinterpret_cast<unsigned long long*>(Ssh + (col + c) * SP + row + 2 * r) = S[r][c];
    };
#pragma unroll
    for (int r = 0; r < RPT / 2; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const float *lo = entry(2 * r, c), *hi = entry(2 * r + 1, c);
            S[r][c] = pair_of(lo ? *lo : 0.f, hi ? *hi : 0.f);
        }
    publish();
    const int ks = lane & 15, cols1 = set * (CB / 2) + (lane >> 4) * 4;
    float* uset = ush + set * CT * (CB / 2);
    const int left = len - c0 * CT;              // tokens from the first of these chunks on
    float* o_row = o_out + (size_t)(start + c0 * CT) * a.heads * a.vd + (size_t)h * a.vd + col0;
    bool ok = true;
    for (int c = 0; c < n_chunks; ++c) {
        const float* stage = sm + (c % STAGES) * L::STAGE;
        const float* uo = stage + L::ROWS;
        if (!mbar_wait(&full[c % STAGES], (uint32_t)(c / STAGES) & 1u, abort_flag)) {
            ok = false;
            *abort_flag = 1;
            atomicOr(err, CELLM_DEV_WAIT_TIMEOUT);
        }
        set_barrier(set);        // the set's columns of S are whole
        // sums over the even and over the odd channels of the lane's share, side by side
        unsigned long long sums[MT * 4];
#pragma unroll
        for (int i = 0; i < MT * 4; ++i) sums[i] = 0;
#pragma unroll
        for (int kk = 0; kk < DIM / 64; ++kk) {
            const int at = kk * 64 + ks * 4;
            ulonglong2 s[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) s[j] = *reinterpret_cast<const ulonglong2*>(Ssh + (cols1 + j) * SP + at);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(stage + (vg * MT + m) * DIM + at);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    fma2(sums[m * 4 + j], w.x, s[j].x);
                    fma2(sums[m * 4 + j], w.y, s[j].y);
                }
            }
        }
        float acc[MT * 4];
#pragma unroll
        for (int i = 0; i < MT * 4; ++i) acc[i] = low_of(sums[i]) + high_of(sums[i]);
        const int idx = scatter_sums<MT * 4, 8>(acc, ks);
#pragma unroll
        for (int i = 0; i < MT / 4; ++i) {
            const int v = vg * MT + (idx + i) / 4, j = cols1 + (idx + i) % 4;
            if (DELTA && v < CT) {
                uset[v * (CB / 2) + j % (CB / 2)] = acc[i] + uo[v * CB + j];
            } else {
                const int t = v - (L::NV - CT);
                if (ok && c * CT + t < left && col0 + j < a.vd) o_row[(size_t)(c * CT + t) * a.heads * a.vd + j] = acc[i] + uo[(CT + t) * CB + j];
            }
        }
        set_barrier(set);        // u is whole, and the set's columns of S have been read
        const float* ke = stage + L::NV * DIM + row;
#pragma unroll
        for (int r = 0; r < RPT / 2; ++r) {
            const unsigned long long e = *reinterpret_cast<const unsigned long long*>(ke + CT * DIM + 2 * r);
#pragma unroll
            for (int j = 0; j < 2; ++j) S[r][j] = pair_of(low_of(S[r][j]) * low_of(e), high_of(S[r][j]) * high_of(e));
        }
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            const float2 u = *reinterpret_cast<const float2*>(DELTA ? uset + t * (CB / 2) + (lane & 3) * 2 : uo + t * CB + col);
            const unsigned long long u0 = pair_of(u.x, u.x), u1 = pair_of(u.y, u.y);
            if constexpr (RPT == 4) {
                const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(ke + t * DIM);
                fma2(S[0][0], k.x, u0), fma2(S[0][1], k.x, u1);
                fma2(S[RPT / 2 - 1][0], k.y, u0), fma2(S[RPT / 2 - 1][1], k.y, u1);
            } else {
                const unsigned long long k = *reinterpret_cast<const unsigned long long*>(ke + t * DIM);
                fma2(S[0][0], k, u0), fma2(S[0][1], k, u1);
            }
        }
        publish();
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty[c % STAGES]);
    }
    if (!ok) return;             // the copies gave up: the state stays as it was
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c)
            if (float* p = entry(r, c)) *p = r & 1 ? high_of(S[r / 2][c]) : low_of(S[r / 2][c]);
}

template <int DIM, bool DELTA> int floats_a_chunk(int vd) {
    return Layout<DIM, DELTA>::ROWS + ((vd + CB - 1) / CB) * Layout<DIM, DELTA>::COLS;
}

template <int DIM, bool DELTA>
int run(float* o_out, float* state, long long slot_stride, int n_slots, ChunkArgs a, int n_chunks, int ws_chunks, int* err, cudaStream_t stream) {
    using L = Layout<DIM, DELTA>;
    a.stride = floats_a_chunk<DIM, DELTA>(a.vd);
    const size_t smem = (size_t)(STAGES * L::STAGE + CB * (DIM + 4) + CT * CB) * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(chunk_walk_kernel<DIM, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    const long long walk_blocks = (long long)a.B * a.heads * ((a.vd + CB - 1) / CB);
    if (walk_blocks > INT_MAX) return CELLM_ERR_SIZE;
    for (a.chunk0 = 0; a.chunk0 < n_chunks; a.chunk0 += ws_chunks) {
        a.chunks = std::min(ws_chunks, n_chunks - a.chunk0);
        CELLM_RUN((chunk_vectors_kernel<DIM, DELTA>), dim3(a.chunks, a.heads), DIM, 0, stream, a);
        CELLM_RUN((chunk_walk_kernel<DIM, DELTA>), (unsigned)walk_blocks, WALK_THREADS + 32, smem, stream, o_out, state,
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
                cu_seqlens, slot_ids, B, min_len, heads, dim, vd, ws, 0, 0, 0};
    return dim <= 64 ? run<64, true>(o_out, state, slot_stride, n_slots, a, n_chunks, ws_chunks, err, stream)
                     : run<128, true>(o_out, state, slot_stride, n_slots, a, n_chunks, ws_chunks, err, stream);
}

// HGRN2 likewise; q and f (already silu and forget gate, as cellm_hgrn2_gates leaves them) and v are columns of proj [T, ld].
CELLM_API int cellm_hgrn2_chunks(float* o_out, float* state, long long slot_stride, int n_slots, const float* proj, long long ld, int col_q,
                                 int col_f, int col_v, const int* cu_seqlens, const int* slot_ids, int B, int n_chunks, int ws_chunks,
                                 int min_len, int heads, int dim, int vd, float* ws, int* err, cudaStream_t stream) {
    if (!fits(B, heads, 1, dim, vd, n_chunks, ws_chunks, ws) || min_len < 1) return CELLM_ERR_SIZE;
    ChunkArgs a{proj + col_q, nullptr, proj + col_f, proj + col_v, nullptr, ld, 0, ld, ld, 1, cu_seqlens, slot_ids, B, min_len, heads, dim, vd, ws, 0, 0, 0};
    return dim <= 64 ? run<64, false>(o_out, state, slot_stride, n_slots, a, n_chunks, ws_chunks, err, stream)
                     : run<128, false>(o_out, state, slot_stride, n_slots, a, n_chunks, ws_chunks, err, stream);
}
