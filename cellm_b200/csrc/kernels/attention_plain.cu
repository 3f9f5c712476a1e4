// Plain attention over the paged cache, every earlier key of the request (or the
// last `window` of them) read through the block table: one block per (token, head),
// which takes every form (sinks, gates, values turned back, kept first keys, any
// width, bfloat16) and is the reference for the faster attention kernels; and for
// the usual form in 32 bits a block per rows of several tokens and heads
// (attention_rows_kernel).
//
// For head h the key/value head is h / (nh / nkv); scores are q.k * scale;
// softmax takes the maximum off first; all of it in 32-bit
// (crates/cellm-cache/src/kvcache.rs:753-787, :1206-1227). Keys are walked in
// chunks (128 keys, 64 by rows) that start at multiples of their size counted from key 0, so the
// order of every sum depends only on the token's position, never on how the
// sequence was cut into steps or what else is in the batch.
//
// Cache layout of one layer: [page][kv_head][slot in page][head_dim].
#include <algorithm>

#include "common.cuh"

#define ATTN_PLAIN_THREADS 128
#define ATTN_PLAIN_MAX_HD 2048

template <typename TA>
__global__ void __launch_bounds__(ATTN_PLAIN_THREADS)
attention_plain_kernel(TA* __restrict__ out, const TA* __restrict__ q, const TA* __restrict__ k_pool,
                       const TA* __restrict__ v_pool, const int* __restrict__ positions,
                       const int* __restrict__ seq_of_token, const int* __restrict__ block_table,
                       int bt_stride, int num_pages, int page_size, int nh, int nkv, int hd, int hdv, int v_row, float scale,
                       int window, const float* __restrict__ sinks, const float* __restrict__ unrot, int interleaved,
                       int keep_first, float fixed_sink, int has_fixed_sink, const float* __restrict__ gate, long long gate_ld,
                       int chunk, int* __restrict__ err) {
    constexpr int CH = ATTN_PLAIN_THREADS;
    extern __shared__ float smem[];
    float* qs = smem;             // [hd]
    float* sc = smem + hd;        // [CH]
    int* pg = (int*)(sc + CH);    // [CH] page of each key in the chunk
    __shared__ float scratch[32];
    pdl_trigger();
    pdl_wait();
    const int t = blockIdx.x / nh, h = blockIdx.x % nh;
    const int kvh = h / (nh / nkv);
    const int pos = positions[t];
    const int b = seq_of_token[t];
    // the first key this token reads: its window's, or the first of its own run of `chunk` positions
    const int lo = chunk > 0 ? pos / chunk * chunk : (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < hd; i += CH) qs[i] = to_float(q[(size_t)t * nh * hd + (size_t)h * hd + i]) * scale;
    float m = -INFINITY, l = 0.f;
    float acc[ATTN_PLAIN_MAX_HD / CH];
#pragma unroll
    for (int r = 0; r < ATTN_PLAIN_MAX_HD / CH; ++r) acc[r] = 0.f;
    const size_t page_elems = (size_t)nkv * page_size * hd, v_page_elems = (size_t)nkv * page_size * v_row;
    // with `keep_first` the first keys of the sequence stay visible behind the window: chunks are walked from key 0
    // and those that hold neither a kept key nor a key of the window are passed over
    for (int c0 = keep_first > 0 ? 0 : (lo / CH) * CH; c0 <= pos; c0 += CH) {
        if (c0 >= keep_first && c0 + CH <= lo) continue;
        __syncthreads();
        {   // page of key c0 + tid
            const int j = c0 + threadIdx.x;
            int p = -1;
            if ((j >= lo || j < keep_first) && j <= pos) {
                p = block_table[(size_t)b * bt_stride + j / page_size];
                if (p < 0 || p >= num_pages) { atomicOr(err, CELLM_DEV_BAD_PAGE); p = -1; }
            }
            pg[threadIdx.x] = p;
        }
        __syncthreads();
        for (int jj = warp; jj < CH; jj += CH / 32) {
            const int p = pg[jj];
            float s = -INFINITY;
            if (p >= 0) {
                const int j = c0 + jj;
                const TA* kr = k_pool + (size_t)p * page_elems + ((size_t)kvh * page_size + j % page_size) * hd;
                float d = 0.f;
                for (int i = lane; i < hd; i += 32) d += qs[i] * to_float(kr[i]);
                s = warp_sum(d);
            }
            if (lane == 0) sc[jj] = s;
        }
        __syncthreads();
        const float cmax = block_max(sc[threadIdx.x], scratch);
        const float m_new = fmaxf(m, cmax);
        const float s = sc[threadIdx.x];
        const float p = (s == -INFINITY) ? 0.f : expf(s - m_new);
        const float psum = block_sum(p, scratch);
        __syncthreads();
        sc[threadIdx.x] = p;
        __syncthreads();
        const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
        l = l * corr + psum;
        m = m_new;
#pragma unroll
        for (int r = 0; r < ATTN_PLAIN_MAX_HD / CH; ++r) {
            const int d = threadIdx.x + r * CH;
            if (d < hdv) {
                float a = acc[r] * corr;
                for (int jj = 0; jj < CH; ++jj) {
                    const int pgj = pg[jj];
                    if (pgj < 0) continue;
                    const int j = c0 + jj;
                    a += sc[jj] * to_float(v_pool[(size_t)pgj * v_page_elems + ((size_t)kvh * page_size + j % page_size) * v_row + d]);
                }
                acc[r] = a;
            }
        }
    }
    if (sinks || has_fixed_sink) {
        // a sink: one more term exp(sink_h) in the denominator, with no key and no value (learned per head, or one
        // fixed score for all heads)
        const float sk = sinks ? sinks[h] : fixed_sink;
        const float m_new = fmaxf(m, sk);
        const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
        l = l * corr + expf(sk - m_new);
#pragma unroll
        for (int r = 0; r < ATTN_PLAIN_MAX_HD / CH; ++r) acc[r] *= corr;
    }
    // an output gate: the head's sum times sigmoid of one number per (token, head)
    const float inv = (gate ? 1.f / (1.f + expf(-gate[(size_t)t * gate_ld + h])) : 1.f) / l;
    if (unrot) {
        // values were cached rotated by their own positions: the sum is turned back by the token's position
        // (pair m by -pos * f_m; f as [hdv/2][2] floats, high part and remainder)
        float* ov = smem;                   // the queries are not needed any more
        __syncthreads();
#pragma unroll
        for (int r = 0; r < ATTN_PLAIN_MAX_HD / CH; ++r) {
            const int d = threadIdx.x + r * CH;
            if (d < hdv) ov[d] = acc[r] * inv;
        }
        __syncthreads();
        const int half = hdv / 2;
        for (int mm = threadIdx.x; mm < half; mm += CH) {
            const float hi = unrot[2 * mm], lo = unrot[2 * mm + 1], fp = (float)pos;
            const float a = fp * hi;
            const float e = fmaf(fp, hi, -a) + fp * lo;
            float sn, cs, se, ce;
            sincosf(a, &sn, &cs);
            sincosf(e, &se, &ce);
            const float c = cs * ce - sn * se, s = sn * ce + cs * se;
            const int i0 = interleaved ? 2 * mm : mm, i1 = interleaved ? 2 * mm + 1 : mm + half;
            const float u = ov[i0], v = ov[i1];
            out[(size_t)t * nh * hdv + (size_t)h * hdv + i0] = from_float<TA>(u * c + v * s);
            out[(size_t)t * nh * hdv + (size_t)h * hdv + i1] = from_float<TA>(v * c - u * s);
        }
        return;
    }
#pragma unroll
    for (int r = 0; r < ATTN_PLAIN_MAX_HD / CH; ++r) {
        const int d = threadIdx.x + r * CH;
        if (d < hdv) out[(size_t)t * nh * hdv + (size_t)h * hdv + d] = from_float<TA>(acc[r] * inv);
    }
}

// ------------------------------------------------------------------------------------------------ the usual form in 32 bits
// Queries, keys and values of one width hd (a multiple of 4, up to 128), no sink, no gate, nothing turned back: a block takes
// RI * 8 rows, the heads of one key/value head for as many neighbouring tokens as fit, and brings every key and value of
// theirs into shared memory once, in blocks of 64 keys that start at multiples of 64 and arrive by asynchronous copies while the
// block before is worked on. (One block a (token, head) read them again for each: a layer of 24 heads of 64, three portions of
// 213 tokens in all behind 100 keys on average, its two products included, went from 998 to 231 us, 66 of them this kernel.
// Steps of single tokens gain as well, 1 to 256 requests behind 100 to 8,192 keys: 2.2 to 28 times the speed.) 16 neighbouring
// threads share a row; a thread holds RI rows by 4 keys of the scores and RI rows by 4 values of each 64 of the output. Every
// sum's order depends on the row's own position alone: a score is four sums over every fourth entry, added in pairs; a block's
// weights are summed four a thread and over the 16 threads; the output runs over the keys in order. Keys that a row does not see
// are passed over, not multiplied by zero, so what later tokens hold (infinities among it) reaches no earlier one.
#define ROWS_KEYS 64
#define ROWS_THREADS 128

struct RowsArgs {
    float* out;
    const float *q, *k_pool, *v_pool;
    const int *positions, *seq_of_token, *block_table;
    int bt_stride, num_pages, page_size, T, nh, nkv, hd, tokens;      // tokens: of a block
    float scale;
    int window;
    int* err;
};

__device__ __forceinline__ void rows_copy16(float* dst, const float* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
// Over the 16 threads that share a row.
__device__ __forceinline__ float row_max16(float x) {
#pragma unroll
    for (int d = 8; d; d >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, d));
    return x;
}
__device__ __forceinline__ float row_sum16(float x) {
#pragma unroll
    for (int d = 8; d; d >>= 1) x += __shfl_xor_sync(0xffffffffu, x, d);
    return x;
}

template <int RI, int ND>       // ND: blocks of 64 output entries (hd up to 64 ND)
__global__ void __launch_bounds__(ROWS_THREADS)
attention_rows_kernel(const RowsArgs a) {
    constexpr int R = RI * 8, PS = ROWS_KEYS + 4;
    extern __shared__ __align__(16) float rows_smem[];
    const int hd = a.hd, P = hd + 4, G = a.nh / a.nkv, kvh = blockIdx.y;
    float* qs = rows_smem;                              // [R][P]
    float* ps = qs + R * P;                             // [R][PS]
    float* kv = ps + R * PS;                            // [2 stages][K, V][ROWS_KEYS][P]
    __shared__ int pages[2][ROWS_KEYS];                 // of the keys of a stage; -1: nobody sees the key
    const int tid = threadIdx.x, x = tid & 15, y = tid >> 4;
    pdl_trigger();
    pdl_wait();
    const int t_end = min(a.T, (int)(blockIdx.x + 1) * a.tokens);
    for (int t0 = blockIdx.x * a.tokens; t0 < t_end;) {
        // the block's next tokens of one request, positions ascending (the first's and the last's bound the keys): t0 .. t0 + n - 1
        const int b = a.seq_of_token[t0];
        int n = 1;
        while (t0 + n < t_end && a.seq_of_token[t0 + n] == b && a.positions[t0 + n] >= a.positions[t0 + n - 1]) ++n;
        const int* bt = a.block_table + (size_t)b * a.bt_stride;
        const int first_pos = a.positions[t0], last_pos = a.positions[t0 + n - 1];
        const int lo_all = a.window > 0 ? max(0, first_pos - a.window + 1) : 0;
        int pos[RI], lo[RI];
        float m[RI], l[RI], acc[RI][ND][4];
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const int r = y + 8 * i;
            pos[i] = r < n * G ? a.positions[t0 + r / G] : -1;
            lo[i] = a.window > 0 ? max(0, pos[i] - a.window + 1) : 0;
            m[i] = -INFINITY;
            l[i] = 0.f;
#pragma unroll
            for (int d = 0; d < ND; ++d)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[i][d][e] = 0.f;
        }
        __syncthreads();            // the last tokens' rows and stages are done with
        for (int idx = tid; idx < R * (hd / 4); idx += ROWS_THREADS) {
            const int r = idx / (hd / 4), c = idx % (hd / 4) * 4;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < n * G) v = *reinterpret_cast<const float4*>(a.q + ((size_t)(t0 + r / G) * a.nh + kvh * G + r % G) * hd + c);
            *reinterpret_cast<float4*>(qs + r * P + c) = make_float4(v.x * a.scale, v.y * a.scale, v.z * a.scale, v.w * a.scale);
        }
        const int c_first = lo_all / ROWS_KEYS, c_last = last_pos / ROWS_KEYS;
        auto find_pages = [&](int c) {
            if (tid < ROWS_KEYS) {
                const int j = c * ROWS_KEYS + tid;
                int p = -1;
                if (j >= lo_all && j <= last_pos) {
                    p = bt[j / a.page_size];
                    if (p < 0 || p >= a.num_pages) { atomicOr(a.err, CELLM_DEV_BAD_PAGE); p = -1; }
                }
                pages[c & 1][tid] = p;
            }
        };
        auto issue = [&](int c) {
            float* dst = kv + (c & 1) * 2 * ROWS_KEYS * P;
            const int per = hd / 4;
            for (int idx = tid; idx < 2 * ROWS_KEYS * per; idx += ROWS_THREADS) {
                const int key = idx / per, col = idx % per * 4, j = key & (ROWS_KEYS - 1);
                const float* pool = key < ROWS_KEYS ? a.k_pool : a.v_pool;
                const int p = pages[c & 1][j];
                const size_t at = ((size_t)max(p, 0) * a.nkv + kvh) * a.page_size + (c * ROWS_KEYS + j) % a.page_size;
                rows_copy16(dst + key * P + col, pool + at * hd + col, p >= 0);
            }
        };
        find_pages(c_first);
        __syncthreads();
        issue(c_first);
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (int c = c_first; c <= c_last; ++c) {
            if (c < c_last) find_pages(c + 1);
            __syncthreads();        // the next block's pages are there, and its stage is free
            if (c < c_last) issue(c + 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
            const float* ks = kv + (c & 1) * 2 * ROWS_KEYS * P;
            const float* vs = ks + ROWS_KEYS * P;
            const int j0 = c * ROWS_KEYS;
            float4 s4[RI][4];
#pragma unroll
            for (int i = 0; i < RI; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s4[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int d = 0; d < hd; d += 4) {
                float4 k[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const float4*>(ks + (x + 16 * j) * P + d);
#pragma unroll
                for (int i = 0; i < RI; ++i) {
                    const float4 q = *reinterpret_cast<const float4*>(qs + (y + 8 * i) * P + d);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        s4[i][j].x = fmaf(q.x, k[j].x, s4[i][j].x);
                        s4[i][j].y = fmaf(q.y, k[j].y, s4[i][j].y);
                        s4[i][j].z = fmaf(q.z, k[j].z, s4[i][j].z);
                        s4[i][j].w = fmaf(q.w, k[j].w, s4[i][j].w);
                    }
                }
            }
            // which of the thread's keys have a page: read before the barrier, behind which a warp that is ahead may already put the
            // pages of the block after the next in this place
            unsigned paged = 0;
#pragma unroll
            for (int j = 0; j < 4; ++j) paged |= (pages[c & 1][x + 16 * j] >= 0 ? 1u : 0u) << j;
            // whether every row of the block sees every key of this block
            const bool open = __syncthreads_and(paged == 15u) && j0 + ROWS_KEYS - 1 <= first_pos && (a.window <= 0 || j0 > last_pos - a.window);
#pragma unroll
            for (int i = 0; i < RI; ++i) {
                float s[4], top = -INFINITY;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int key = j0 + x + 16 * j;
                    const bool sees = key <= pos[i] && key >= lo[i] && (paged >> j & 1u);
                    s[j] = sees ? (s4[i][j].x + s4[i][j].y) + (s4[i][j].z + s4[i][j].w) : -INFINITY;
                    top = fmaxf(top, s[j]);
                }
                const float m_new = fmaxf(m[i], row_max16(top));
                float sum = 0.f;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float p = s[j] == -INFINITY ? 0.f : expf(s[j] - m_new);
                    ps[(y + 8 * i) * PS + x + 16 * j] = p;
                    sum += p;
                }
                const float corr = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
                l[i] = l[i] * corr + row_sum16(sum);
                m[i] = m_new;
#pragma unroll
                for (int d = 0; d < ND; ++d)
#pragma unroll
                    for (int e = 0; e < 4; ++e) acc[i][d][e] *= corr;
            }
            __syncwarp();           // a row's weights come from its own half of a warp
            for (int j = 0; j < ROWS_KEYS; j += 4) {
                float4 p[RI];
#pragma unroll
                for (int i = 0; i < RI; ++i) p[i] = *reinterpret_cast<const float4*>(ps + (y + 8 * i) * PS + j);
#pragma unroll
                for (int d = 0; d < ND; ++d) {
                    const int col = d * 64 + x * 4;
                    if (col >= hd) continue;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float4 v = *reinterpret_cast<const float4*>(vs + (j + e) * P + col);
                        const int key = j0 + j + e;
#pragma unroll
                        for (int i = 0; i < RI; ++i) {
                            const float w = e == 0 ? p[i].x : e == 1 ? p[i].y : e == 2 ? p[i].z : p[i].w;
                            if (open || (key <= pos[i] && key >= lo[i])) {
                                acc[i][d][0] = fmaf(w, v.x, acc[i][d][0]);
                                acc[i][d][1] = fmaf(w, v.y, acc[i][d][1]);
                                acc[i][d][2] = fmaf(w, v.z, acc[i][d][2]);
                                acc[i][d][3] = fmaf(w, v.w, acc[i][d][3]);
                            }
                        }
                    }
                }
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
        for (int i = 0; i < RI; ++i) {
            const int r = y + 8 * i;
            if (r >= n * G) continue;
            const float inv = 1.f / l[i];
            float* o = a.out + ((size_t)(t0 + r / G) * a.nh + kvh * G + r % G) * hd;
#pragma unroll
            for (int d = 0; d < ND; ++d)
                if (d * 64 + x * 4 < hd)
                    *reinterpret_cast<float4*>(o + d * 64 + x * 4) =
                        make_float4(acc[i][d][0] * inv, acc[i][d][1] * inv, acc[i][d][2] * inv, acc[i][d][3] * inv);
        }
        t0 += n;
    }
}

template <int RI, int ND> static int attention_rows_run(const RowsArgs& a, cudaStream_t stream) {
    const size_t smem = (size_t)(RI * 8 * (a.hd + 4 + ROWS_KEYS + 4) + 4 * ROWS_KEYS * (a.hd + 4)) * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(attention_rows_kernel<RI, ND>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return (int)e;
    CELLM_RUN((attention_rows_kernel<RI, ND>), dim3((unsigned)((a.T + a.tokens - 1) / a.tokens), (unsigned)a.nkv), ROWS_THREADS, smem, stream, a);
    return CELLM_OK;
}

// q: [T, nh*hd]; out: [T, nh*hdv]; pools: one layer's keys and values; positions[t] is the
// token's place in its request (keys 0..positions[t] are read; the token's own
// key must already be in the cache). Value rows are v_row wide and a value is a row's first hdv entries.
static int attention_plain_impl(void* out, const void* q, const void* k_pool, const void* v_pool,
                                const int* positions, const int* seq_of_token, const int* block_table,
                                int bt_stride, int num_pages, int page_size, int T, int nh, int nkv,
                                int hd, int hdv, int v_row, float scale, int window, int dtype, int* err,
                                cudaStream_t stream, const float* sinks = nullptr, const float* unrot = nullptr,
                                int interleaved = 0, int keep_first = 0, float fixed_sink = 0.f, int has_fixed_sink = 0,
                                const float* gate = nullptr, long long gate_ld = 0, int chunk = 0) {
    if (T <= 0) return CELLM_OK;
    if (unrot && hdv % 2) return CELLM_ERR_SIZE;
    if (keep_first < 0 || chunk < 0 || (chunk > 0 && (window > 0 || keep_first > 0))) return CELLM_ERR_SIZE;
    if (hd > ATTN_PLAIN_MAX_HD || hd <= 0 || hdv <= 0 || hdv > v_row || hdv > ATTN_PLAIN_MAX_HD || nkv <= 0 || nh % nkv) return CELLM_ERR_SIZE;
    const int G = nh / nkv;
    if (dtype == CELLM_F32 && hdv == hd && v_row == hd && hd % 4 == 0 && hd <= 128 && G <= 32 && nkv <= 65535 && !sinks && !unrot &&
        keep_first == 0 && !has_fixed_sink && !gate && chunk == 0 &&
        (((uintptr_t)out | (uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15) == 0) {
        // tokens of a block: as many as leave two blocks an SM, and fit 32 rows
        const int most = 32 / G, tokens = (int)std::max<long long>(1, std::min<long long>(most, (long long)T * nkv / (2 * 148)));
        const RowsArgs a{(float*)out, (const float*)q, (const float*)k_pool, (const float*)v_pool, positions, seq_of_token, block_table,
                         bt_stride, num_pages, page_size, T, nh, nkv, hd, tokens, scale, window, err};
        const int rows = tokens * G;
#define ROWS_RUN(ND) (rows <= 8 ? attention_rows_run<1, ND>(a, stream) : rows <= 16 ? attention_rows_run<2, ND>(a, stream) : attention_rows_run<4, ND>(a, stream))
        return hd <= 64 ? ROWS_RUN(1) : ROWS_RUN(2);
#undef ROWS_RUN
    }
    // the first hd floats hold the query; the output is turned back in the same place (hdv floats)
    const size_t smem = (size_t)((hd > hdv ? hd : hdv) + 2 * ATTN_PLAIN_THREADS) * sizeof(float);
    const unsigned grid = (unsigned)T * (unsigned)nh;
    if (dtype == CELLM_F32)
        CELLM_RUN(attention_plain_kernel<float>, grid, ATTN_PLAIN_THREADS, smem, stream,
            (float*)out, (const float*)q, (const float*)k_pool, (const float*)v_pool, positions, seq_of_token,
            block_table, bt_stride, num_pages, page_size, nh, nkv, hd, hdv, v_row, scale, window, sinks, unrot, interleaved, keep_first, fixed_sink, has_fixed_sink, gate, gate_ld, chunk, err);
    else if (dtype == CELLM_BF16)
        CELLM_RUN(attention_plain_kernel<__nv_bfloat16>, grid, ATTN_PLAIN_THREADS, smem, stream,
            (__nv_bfloat16*)out, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k_pool,
            (const __nv_bfloat16*)v_pool, positions, seq_of_token, block_table, bt_stride, num_pages,
            page_size, nh, nkv, hd, hdv, v_row, scale, window, sinks, unrot, interleaved, keep_first, fixed_sink, has_fixed_sink, gate, gate_ld, chunk, err);
    else return CELLM_ERR_DTYPE;
    return CELLM_OK;
}

// Values in rows as wide as the keys' (hdv = hd for ordinary attention; hdv < hd with v_pool = k_pool for a cache
// whose rows serve as keys and, in their first part, as values).
CELLM_API int cellm_attention_plain(void* out, const void* q, const void* k_pool, const void* v_pool,
                                    const int* positions, const int* seq_of_token, const int* block_table,
                                    int bt_stride, int num_pages, int page_size, int T, int nh, int nkv,
                                    int hd, int hdv, float scale, int window, int dtype, int* err,
                                    cudaStream_t stream) {
    if (hdv > hd) return CELLM_ERR_SIZE;
    return attention_plain_impl(out, q, k_pool, v_pool, positions, seq_of_token, block_table, bt_stride, num_pages, page_size, T, nh, nkv,
                                hd, hdv, hd, scale, window, dtype, err, stream);
}

// Values of a width of their own: a pool of values [page][kv_head][slot][hdv] beside the keys' [..][hd].
CELLM_API int cellm_attention_plain_wide(void* out, const void* q, const void* k_pool, const void* v_pool,
                                         const int* positions, const int* seq_of_token, const int* block_table,
                                         int bt_stride, int num_pages, int page_size, int T, int nh, int nkv,
                                         int hd, int hdv, float scale, int window, int dtype, int* err,
                                         cudaStream_t stream) {
    return attention_plain_impl(out, q, k_pool, v_pool, positions, seq_of_token, block_table, bt_stride, num_pages, page_size, T, nh, nkv,
                                hd, hdv, hdv, scale, window, dtype, err, stream);
}

// The same with a learned sink per head in the softmax's denominator (`sinks` [nh], 32-bit; null: none) and with the
// output turned back by the token's position (`unrot` [hdv/2][2]: the values' frequencies; null: values were
// not rotated). Values have rows of their own width hdv.
CELLM_API int cellm_attention_plain_sink(void* out, const void* q, const void* k_pool, const void* v_pool,
                                         const int* positions, const int* seq_of_token, const int* block_table,
                                         int bt_stride, int num_pages, int page_size, int T, int nh, int nkv,
                                         int hd, int hdv, float scale, int window, const float* sinks, const float* unrot,
                                         int interleaved, int dtype, int* err, cudaStream_t stream) {
    return attention_plain_impl(out, q, k_pool, v_pool, positions, seq_of_token, block_table, bt_stride, num_pages, page_size, T, nh, nkv,
                                hd, hdv, hdv, scale, window, dtype, err, stream, sinks, unrot, interleaved);
}

// The general form: a window that keeps the sequence's first `keep_first` keys visible (from position i a key j <= i is visible when
// i - j < window or j < keep_first; window 0: every earlier key), a learned sink per head (`sinks`) or one fixed sink
// score for all heads (`has_fixed_sink`), an output gate (`gate` [T, gate_ld] 32-bit pre-activations, one per head: the
// head's output is multiplied by its sigmoid; null: none), and value rows `v_row` wide of which the first hdv entries are
// the value (v_pool may be k_pool for a cache whose rows serve as both).
CELLM_API int cellm_attention_plain_masked(void* out, const void* q, const void* k_pool, const void* v_pool,
                                           const int* positions, const int* seq_of_token, const int* block_table,
                                           int bt_stride, int num_pages, int page_size, int T, int nh, int nkv,
                                           int hd, int hdv, int v_row, float scale, int window, int keep_first,
                                           const float* sinks, float fixed_sink, int has_fixed_sink, const float* gate,
                                           long long gate_ld, int dtype, int* err, cudaStream_t stream) {
    return attention_plain_impl(out, q, k_pool, v_pool, positions, seq_of_token, block_table, bt_stride, num_pages, page_size, T, nh, nkv,
                                hd, hdv, v_row, scale, window, dtype, err, stream, sinks, nullptr, 0, keep_first, fixed_sink, has_fixed_sink,
                                gate, gate_ld);
}

// Chunked: position i reads the keys j <= i of its own run of `chunk` positions (floor(i / chunk) = floor(j / chunk), runs
// counted from position 0 of the sequence); chunk 0: every earlier key. A pool of values with rows of hdv entries.
CELLM_API int cellm_attention_plain_chunked(void* out, const void* q, const void* k_pool, const void* v_pool,
                                            const int* positions, const int* seq_of_token, const int* block_table,
                                            int bt_stride, int num_pages, int page_size, int T, int nh, int nkv,
                                            int hd, int hdv, float scale, int chunk, int dtype, int* err, cudaStream_t stream) {
    return attention_plain_impl(out, q, k_pool, v_pool, positions, seq_of_token, block_table, bt_stride, num_pages, page_size, T, nh, nkv,
                                hd, hdv, hdv, scale, 0, dtype, err, stream, nullptr, nullptr, 0, 0, 0.f, 0, nullptr, 0, chunk);
}
