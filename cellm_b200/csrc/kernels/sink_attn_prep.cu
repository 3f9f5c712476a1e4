// What lies between the q, k, v projection and the attention itself for an attention whose projections pass a
// short causal convolution, are normed over the whole projection, and whose values are rotated as well as its
// queries and keys. One block a token:
//
//   1. projected value + bias, then the convolution over time (conv_taps.cuh) for every channel of q, k and v;
//   2. RMS norm of q over all its heads at once, and of k, with plain weights;
//   3. rotation of the first `rot` entries of every q and k head by pos * f_i (f from a table that may be scaled);
//   4. rotation of every value head over all its entries by pos * g_m (a table of its own);
//   5. q into the step's buffer, k and v into the token's page.
//
// All arithmetic is 32-bit; angles are pos * (hi + lo) in split arithmetic from tables made in 64-bit.
#include <algorithm>

#include "conv_taps.cuh"

template <typename TA>
__global__ void __launch_bounds__(1024)
sink_attn_prep_kernel(TA* __restrict__ q_out, TA* __restrict__ k_pool, TA* __restrict__ v_pool, ConvTaps cv,
                      const float* __restrict__ state_base, long long slot_stride, int n_slots,
                      const float* __restrict__ q_norm_w, const float* __restrict__ k_norm_w, float eps,
                      const float* __restrict__ qk_freq, int rot, const float* __restrict__ v_freq, int interleaved,
                      const int* __restrict__ positions, const int* __restrict__ seq_of_token,
                      const int* __restrict__ cu_seqlens, const int* __restrict__ slot_ids,
                      const int* __restrict__ block_table, int bt_stride, int num_pages, int page_size,
                      int nh, int nkv, int hd, int vd, const float* __restrict__ q_mult, int fours, int* __restrict__ err) {
    extern __shared__ __align__(16) float sm[];
    const int Cq = nh * hd, Ck = nkv * hd, Cv = nkv * vd, C = Cq + Ck + Cv;
    float* buf = sm;                       // [C]
    float* cq = buf + C;                   // [rot/2] cos, then [rot/2] sin
    float* sq = cq + rot / 2;
    float* cvv = sq + rot / 2;             // [vd/2] cos, then [vd/2] sin (values; only where v_freq is given)
    float* svv = cvv + vd / 2;
    __shared__ float scratch[32];
    pdl_trigger();
    const int t = blockIdx.x;
    const int pos = positions[t], b = seq_of_token[t], start = cu_seqlens[b];
    for (int p = threadIdx.x; p < rot / 2; p += blockDim.x)
        split_sincos((float)pos, qk_freq[2 * p], qk_freq[2 * p + 1], &cq[p], &sq[p]);
    if (v_freq)
        for (int p = threadIdx.x; p < vd / 2; p += blockDim.x)
            split_sincos((float)pos, v_freq[2 * p], v_freq[2 * p + 1], &cvv[p], &svv[p]);
    int slot = slot_ids[b];
    if (slot < 0 || slot >= n_slots) { if (threadIdx.x == 0) atomicOr(err, CELLM_DEV_BAD_SLOT); slot = 0; }
    cv.state = state_base + (size_t)slot * slot_stride;
    const int page = block_table[(size_t)b * bt_stride + pos / page_size];
    const bool page_ok = page >= 0 && page < num_pages;
    if (!page_ok && threadIdx.x == 0) atomicOr(err, CELLM_DEV_BAD_PAGE);
    pdl_wait();
    // (four channels a thread where the rows lie on 16-byte borders: 2,560 channels of four taps are 27 loads a thread of 256
    // instead of 90; two prompts of about 700 tokens through both mixers side by side went from 315 to 294 us with it)
    if (fours)
        for (int c = threadIdx.x * 4; c < C; c += blockDim.x * 4) *reinterpret_cast<float4*>(buf + c) = conv_taps_four(cv, t, start, c);
    else
        for (int c = threadIdx.x; c < C; c += blockDim.x) buf[c] = conv_taps_at(cv, t, start, c);
    __syncthreads();
    if (q_norm_w) {
        float s1 = 0.f, s2 = 0.f;
        for (int c = threadIdx.x; c < Cq; c += blockDim.x) s1 = fmaf(buf[c], buf[c], s1);
        for (int c = threadIdx.x; c < Ck; c += blockDim.x) s2 = fmaf(buf[Cq + c], buf[Cq + c], s2);
        s1 = block_sum(s1, scratch);
        s2 = block_sum(s2, scratch);
        const float rq = 1.f / sqrtf(s1 / (float)Cq + eps), rk = 1.f / sqrtf(s2 / (float)Ck + eps);
        for (int c = threadIdx.x; c < Cq; c += blockDim.x) buf[c] *= rq * q_norm_w[c];
        for (int c = threadIdx.x; c < Ck; c += blockDim.x) buf[Cq + c] *= rk * k_norm_w[c];
        __syncthreads();
    }
    const int half = rot / 2;
    for (int idx = threadIdx.x; idx < (nh + nkv) * half; idx += blockDim.x) {
        const int head = idx / half, i = idx % half;
        float* x = buf + head * hd;        // q heads, then k heads, all hd wide
        const int i0 = interleaved ? 2 * i : i, i1 = interleaved ? 2 * i + 1 : i + half;
        const float u = x[i0], v = x[i1];
        x[i0] = u * cq[i] - v * sq[i];
        x[i1] = v * cq[i] + u * sq[i];
    }
    if (v_freq) {
        const int vhalf = vd / 2;
        for (int idx = threadIdx.x; idx < nkv * vhalf; idx += blockDim.x) {
            const int head = idx / vhalf, m = idx % vhalf;
            float* x = buf + Cq + Ck + head * vd;
            const int i0 = interleaved ? 2 * m : m, i1 = interleaved ? 2 * m + 1 : m + vhalf;
            const float u = x[i0], v = x[i1];
            x[i0] = u * cvv[m] - v * svv[m];
            x[i1] = v * cvv[m] + u * svv[m];
        }
    }
    __syncthreads();
    // q_mult: one factor per query head (a learned temperature of the head's scores), applied in 32-bit
    for (int c = threadIdx.x; c < Cq; c += blockDim.x) q_out[(size_t)t * Cq + c] = from_float<TA>(q_mult ? buf[c] * q_mult[c / hd] : buf[c]);
    if (page_ok) {
        const int in_page = pos % page_size;
        for (int c = threadIdx.x; c < Ck; c += blockDim.x) {
            const int head = c / hd, i = c % hd;
            k_pool[(((size_t)page * nkv + head) * page_size + in_page) * hd + i] = from_float<TA>(buf[Cq + c]);
        }
        for (int c = threadIdx.x; c < Cv; c += blockDim.x) {
            const int head = c / vd, i = c % vd;
            v_pool[(((size_t)page * nkv + head) * page_size + in_page) * vd + i] = from_float<TA>(buf[Cq + Ck + c]);
        }
    }
}

// Many tokens, NT taps, everything on 16-byte borders: a block takes PREP_RUN neighbouring tokens, whose rows and taps it reads once (the
// form above reads a token's 40 KB of taps and four rows of 10 KB for every token), and all its threads share the tokens' angles. The
// convolution's sums are those of the form above; the norms' sums of squares are added in another order. A thread takes four channels,
// then four outputs of a head. Two prompts of 1,775 tokens in all, 2,560 channels of four taps: 31.8 us a block a
// token, 18.8 now.
constexpr int PREP_RUN = 4;

__device__ __forceinline__ void store4(float* dst, float4 x) { *reinterpret_cast<float4*>(dst) = x; }
__device__ __forceinline__ void store4(__nv_bfloat16* dst, float4 x) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(x.x, x.y), b = __floats2bfloat162_rn(x.z, x.w);
    *reinterpret_cast<uint2*>(dst) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

template <typename TA, int NT>
__global__ void __launch_bounds__(512)
sink_attn_prep_run_kernel(TA* __restrict__ q_out, TA* __restrict__ k_pool, TA* __restrict__ v_pool, const ConvTaps cv,
                          const float* __restrict__ state_base, long long slot_stride, int n_slots,
                          const float* __restrict__ q_norm_w, const float* __restrict__ k_norm_w, float eps,
                          const float* __restrict__ qk_freq, int rot, const float* __restrict__ v_freq, int interleaved,
                          const int* __restrict__ positions, const int* __restrict__ seq_of_token,
                          const int* __restrict__ cu_seqlens, const int* __restrict__ slot_ids,
                          const int* __restrict__ block_table, int bt_stride, int num_pages, int page_size,
                          int T, int nh, int nkv, int hd, int vd, const float* __restrict__ q_mult, int* __restrict__ err) {
    constexpr int R = PREP_RUN;
    extern __shared__ __align__(16) float sm[];
    const int Cq = nh * hd, Ck = nkv * hd, Cv = nkv * vd, C = Cq + Ck + Cv, half = rot / 2, vhalf = v_freq ? vd / 2 : 0;
    float* buf = sm;                            // [R][C]
    float* angles = buf + R * C;                // [R][half + vhalf][2]: cosine and sine, q's and k's, then the values' (each a multiple of four)
    __shared__ float part[16][2 * R];           // every warp's sums of squares, q's and k's
    __shared__ float scales[2 * R];             // 1 / rms
    __shared__ int page_of[R], in_page[R], start_of[R], slot_of[R];
    pdl_trigger();
    const int t0 = blockIdx.x * R, n = min(R, T - t0), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    if (tid < n) {
        const int t = t0 + tid, b = seq_of_token[t], pos = positions[t];
        int slot = slot_ids[b];
        if (slot < 0 || slot >= n_slots) { atomicOr(err, CELLM_DEV_BAD_SLOT); slot = 0; }
        int page = block_table[(size_t)b * bt_stride + pos / page_size];
        if (page < 0 || page >= num_pages) { atomicOr(err, CELLM_DEV_BAD_PAGE); page = -1; }
        start_of[tid] = cu_seqlens[b], slot_of[tid] = slot, page_of[tid] = page, in_page[tid] = pos % page_size;
    }
    for (int i = tid; i < n * (half + vhalf); i += blockDim.x) {
        const int r = i / (half + vhalf), p = i % (half + vhalf);
        const float* f = p < half ? qk_freq + 2 * p : v_freq + 2 * (p - half);
        split_sincos((float)positions[t0 + r], f[0], f[1], angles + 2 * i, angles + 2 * i + 1);
    }
    pdl_wait();
    __syncthreads();
    const bool together = start_of[0] == start_of[n - 1];        // the tokens are one portion's
    float ss[2 * R];
#pragma unroll
    for (int i = 0; i < 2 * R; ++i) ss[i] = 0.f;
    for (int c = tid * 4; c < C; c += blockDim.x * 4) {
        float4 y[R];
        if (together) {
            const float4 b4 = cv.bias ? *reinterpret_cast<const float4*>(cv.bias + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float* st = state_base + (size_t)slot_of[0] * slot_stride + c;
            const int start = start_of[0];
            float4 u[NT - 1 + R];
#pragma unroll
            for (int j = 0; j < NT - 1 + R; ++j) {
                const int t = t0 - (NT - 1) + j;
                if (t < start) u[j] = *reinterpret_cast<const float4*>(st + (size_t)(t - start + NT - 1) * C);
                else if (j < NT - 1 + n) {
                    const float4 x = *reinterpret_cast<const float4*>(cv.proj + (size_t)t * cv.ld + cv.col0 + c);
                    u[j] = make_float4(x.x + b4.x, x.y + b4.y, x.z + b4.z, x.w + b4.w);
                } else {
                    u[j] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
            }
            float w[4 * NT];                    // [channel][tap]
#pragma unroll
            for (int j = 0; j < NT; ++j) *reinterpret_cast<float4*>(w + 4 * j) = *reinterpret_cast<const float4*>(cv.taps + (size_t)c * NT + 4 * j);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                y[r] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    y[r].x = fmaf(w[j], u[r + j].x, y[r].x);
                    y[r].y = fmaf(w[NT + j], u[r + j].y, y[r].y);
                    y[r].z = fmaf(w[2 * NT + j], u[r + j].z, y[r].z);
                    y[r].w = fmaf(w[3 * NT + j], u[r + j].w, y[r].w);
                }
            }
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                ConvTaps one = cv;
                one.state = state_base + (size_t)slot_of[r < n ? r : 0] * slot_stride;
                y[r] = r < n ? conv_taps_four(one, t0 + r, start_of[r], c) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            *reinterpret_cast<float4*>(buf + r * C + c) = y[r];
            const float sq = fmaf(y[r].w, y[r].w, fmaf(y[r].z, y[r].z, fmaf(y[r].y, y[r].y, y[r].x * y[r].x)));
            ss[r] += c < Cq ? sq : 0.f;
            ss[R + r] += c >= Cq && c < Cq + Ck ? sq : 0.f;
        }
    }
    if (q_norm_w) {
#pragma unroll
        for (int i = 0; i < 2 * R; ++i) {
            ss[i] = warp_sum(ss[i]);
            if (lane == 0) part[warp][i] = ss[i];
        }
        __syncthreads();
        if (tid < 2 * R) {
            float sum = part[0][tid];
            for (int w = 1; w < nwarps; ++w) sum += part[w][tid];
            scales[tid] = 1.f / sqrtf(sum / (float)(tid < R ? Cq : Ck) + eps);
        }
    }
    __syncthreads();
    // four neighbouring outputs of a head, of all the block's tokens
    const int hd_shift = (hd & (hd - 1)) ? -1 : __ffs(hd) - 1, vd_shift = (vd & (vd - 1)) ? -1 : __ffs(vd) - 1;
    for (int c = tid * 4; c < C; c += blockDim.x * 4) {
        const bool is_q = c < Cq, is_v = c >= Cq + Ck;
        const int width = is_v ? vd : hd, at = is_v ? c - Cq - Ck : is_q ? c : c - Cq, shift = is_v ? vd_shift : hd_shift;
        const int head = shift >= 0 ? at >> shift : at / width, first = at - head * width, pairs = is_v ? vhalf : half;
        const bool normed = q_norm_w && !is_v, turned = first < 2 * pairs;
        // where the partners lie: in the same four, or in another four of the head
        const bool is_u = first < pairs;
        const int there = c + (interleaved ? 0 : is_u ? pairs : -pairs), angle = (is_v ? half : 0) + (interleaved ? first / 2 : is_u ? first : first - pairs);
        const float* nw = is_q ? q_norm_w : k_norm_w;
        float4 w = make_float4(1.f, 1.f, 1.f, 1.f), wo = w;
        if (normed) {
            w = *reinterpret_cast<const float4*>(nw + at);
            if (turned && !interleaved) wo = *reinterpret_cast<const float4*>(nw + at + there - c);
        }
        const float mult = is_q && q_mult ? q_mult[head] : 1.f;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (r >= n) break;
            float4 x = *reinterpret_cast<const float4*>(buf + r * C + c);
            const float scale = normed ? scales[is_q ? r : R + r] : 0.f;
            if (normed) x.x *= scale * w.x, x.y *= scale * w.y, x.z *= scale * w.z, x.w *= scale * w.w;
            if (turned) {
                const float* turn = angles + (size_t)(r * (half + vhalf) + angle) * 2;
                if (interleaved) {          // (u, v) turn to (u cos - v sin, v cos + u sin)
                    const float4 cs = *reinterpret_cast<const float4*>(turn);
                    x = make_float4(x.x * cs.x - x.y * cs.y, x.y * cs.x + x.x * cs.y, x.z * cs.z - x.w * cs.w, x.w * cs.z + x.z * cs.w);
                } else {
                    float4 o = *reinterpret_cast<const float4*>(buf + r * C + there);
                    if (normed) o.x *= scale * wo.x, o.y *= scale * wo.y, o.z *= scale * wo.z, o.w *= scale * wo.w;
                    const float4 c0 = *reinterpret_cast<const float4*>(turn), c1 = *reinterpret_cast<const float4*>(turn + 4);
                    x = is_u ? make_float4(x.x * c0.x - o.x * c0.y, x.y * c0.z - o.y * c0.w, x.z * c1.x - o.z * c1.y, x.w * c1.z - o.w * c1.w)
                             : make_float4(x.x * c0.x + o.x * c0.y, x.y * c0.z + o.y * c0.w, x.z * c1.x + o.z * c1.y, x.w * c1.z + o.w * c1.w);
                }
            }
            if (is_q) {
                if (q_mult) x.x *= mult, x.y *= mult, x.z *= mult, x.w *= mult;
                store4(q_out + (size_t)(t0 + r) * Cq + c, x);
            } else if (page_of[r] >= 0) {
                store4((is_v ? v_pool : k_pool) + (((size_t)page_of[r] * nkv + head) * page_size + in_page[r]) * width + first, x);
            }
        }
    }
}

// proj [T, ld] 32-bit: q (nh x hd), k (nkv x hd), v (nkv x vd) from col0 on; bias, taps [C, n_taps] and the state
// [slots][n_taps - 1][C] follow the same order of channels. q_norm_w / k_norm_w: null for no norm. qk_freq [rot/2][2],
// v_freq [vd/2][2] (null: values are not rotated). q_mult [nh]: a factor per query head (null: none). q_out [T, nh * hd]; pools [page][kv head][slot in page][hd | vd].
CELLM_API int cellm_sink_attn_prep(void* q_out, void* k_pool, void* v_pool, const float* proj, long long ld, int col0,
                                   const float* bias, const float* taps, int n_taps, const float* state, long long slot_stride,
                                   int n_slots, const float* q_norm_w, const float* k_norm_w, float eps, const float* qk_freq,
                                   int rot, const float* v_freq, int interleaved, const int* positions, const int* seq_of_token,
                                   const int* cu_seqlens, const int* slot_ids, const int* block_table, int bt_stride,
                                   int num_pages, int page_size, int T, int nh, int nkv, int hd, int vd, const float* q_mult,
                                   int dtype, int* err, cudaStream_t stream) {
    if (T <= 0) return CELLM_OK;
    if (nh <= 0 || nkv <= 0 || nh % nkv || hd <= 0 || vd <= 0 || rot < 0 || rot > hd || rot % 2 || (v_freq && vd % 2) ||
        n_taps > CONV_TAPS_MAX || page_size <= 0)
        return CELLM_ERR_SIZE;
    if ((n_taps > 1 && !state) || (rot > 0 && !qk_freq) || (!q_norm_w != !k_norm_w)) return CELLM_ERR_ARG;
    ConvTaps cv;
    cv.proj = proj; cv.ld = ld; cv.col0 = col0; cv.bias = bias; cv.taps = taps; cv.state = nullptr; cv.n_taps = n_taps;
    cv.C = nh * hd + nkv * hd + nkv * vd;
    const size_t smem = (size_t)(cv.C + rot + vd) * sizeof(float);
    if (smem > 200 * 1024) return CELLM_ERR_SIZE;
    // few tokens: a thread about four channels, since a step of single tokens is too few blocks to hide a thread's chain
    // of loads behind other blocks (the sums of squares are then added in another order: a rounding apart)
    const int threads = T >= 512 ? 256 : cv.C >= 4096 ? 1024 : cv.C >= 2048 ? 512 : 256;
    const int fours = conv_taps_in_fours(cv, state, slot_stride);
    // (512 tokens: below, the blocks of a token each are what fills the SMs)
    const size_t run_smem = (size_t)(PREP_RUN * (cv.C + rot + vd)) * sizeof(float);
    // (the norms' weights are read four at a time there, value by value in the form of a block a token)
    const bool borders = ((reinterpret_cast<uintptr_t>(q_out) | reinterpret_cast<uintptr_t>(k_pool) | reinterpret_cast<uintptr_t>(v_pool) |
                           reinterpret_cast<uintptr_t>(q_norm_w) | reinterpret_cast<uintptr_t>(k_norm_w)) & 15) == 0;
    if (T >= 512 && n_taps >= 2 && n_taps <= 4 && fours && borders && hd % 8 == 0 && vd % 8 == 0 && rot % 8 == 0 && run_smem <= 100 * 1024) {
        const int run_threads = std::min(512, std::max(128, (cv.C / 8 + 31) / 32 * 32));        // two pieces of four channels a thread
#define RUN_OF(TA, NT)                                                                                                        \
    do {                                                                                                                      \
        cudaError_t e = cudaFuncSetAttribute(sink_attn_prep_run_kernel<TA, NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 100 * 1024); \
        if (e != cudaSuccess) return (int)e;                                                                                  \
        CELLM_RUN((sink_attn_prep_run_kernel<TA, NT>), (T + PREP_RUN - 1) / PREP_RUN, run_threads, run_smem, stream, (TA*)q_out, (TA*)k_pool, \
                  (TA*)v_pool, cv, state, slot_stride, n_slots, q_norm_w, k_norm_w, eps, qk_freq, rot, v_freq, interleaved, positions, \
                  seq_of_token, cu_seqlens, slot_ids, block_table, bt_stride, num_pages, page_size, T, nh, nkv, hd, vd, q_mult, err); \
    } while (0)
#define RUN_OF_TAPS(TA)                                                                                                       \
    do { if (n_taps == 4) RUN_OF(TA, 4); else if (n_taps == 3) RUN_OF(TA, 3); else RUN_OF(TA, 2); return CELLM_OK; } while (0)
        if (dtype == CELLM_F32) RUN_OF_TAPS(float);
        if (dtype == CELLM_BF16) RUN_OF_TAPS(__nv_bfloat16);
        return CELLM_ERR_DTYPE;
#undef RUN_OF_TAPS
#undef RUN_OF
    }
#define PREP_RUN_TOKEN(TA)                                                                                                    \
    do {                                                                                                                      \
        if (smem > 48 * 1024) {                                                                                               \
            cudaError_t e = cudaFuncSetAttribute(sink_attn_prep_kernel<TA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
            if (e != cudaSuccess) return (int)e;                                                                              \
        }                                                                                                                     \
        CELLM_RUN(sink_attn_prep_kernel<TA>, T, threads, smem, stream, (TA*)q_out, (TA*)k_pool, (TA*)v_pool, cv, state, slot_stride, \
                  n_slots, q_norm_w, k_norm_w, eps, qk_freq, rot, v_freq, interleaved, positions, seq_of_token, cu_seqlens, \
                  slot_ids, block_table, bt_stride, num_pages, page_size, nh, nkv, hd, vd, q_mult, fours, err);                             \
    } while (0)
    if (dtype == CELLM_F32) PREP_RUN_TOKEN(float);
    else if (dtype == CELLM_BF16) PREP_RUN_TOKEN(__nv_bfloat16);
    else return CELLM_ERR_DTYPE;
#undef PREP_RUN_TOKEN
    return CELLM_OK;
}
