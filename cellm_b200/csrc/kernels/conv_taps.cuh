// A short causal convolution over time on the channels of a projection, for kernels that apply it while they read
// the projection: y_t[c] = sum_j w[c][j] * u_(t - taps + 1 + j)[c], where u is the projected value (plus its bias).
// Rows before the portion's first token come from the request's state, which holds the last taps - 1 projected
// values of the request (zeros at its start), so a sequence cut anywhere gives the same sums in the same order.
#pragma once
#include "common.cuh"

#define CONV_TAPS_MAX 16

struct ConvTaps {
    const float* proj;      // [T, ld]: the step's projections, 32-bit
    long long ld;
    int col0;               // column of channel 0 in a row of proj
    const float* bias;      // [C] or null
    const float* taps;      // [C, n_taps]
    const float* state;     // this request's [n_taps - 1, C]
    int n_taps;             // 0: no convolution (the projected value itself)
    int C;
};

// Channel c of token t (an index into the step's rows); `start` is the first row of the token's portion.
__device__ __forceinline__ float conv_taps_at(const ConvTaps& s, int t, int start, int c) {
    const float b = s.bias ? s.bias[c] : 0.f;
    if (s.n_taps <= 0) return s.proj[(size_t)t * s.ld + s.col0 + c] + b;
    float y = 0.f;
    for (int j = 0; j < s.n_taps; ++j) {
        const int tt = t - (s.n_taps - 1) + j;
        const float u = tt >= start ? s.proj[(size_t)tt * s.ld + s.col0 + c] + b
                                    : s.state[(size_t)(tt - start + s.n_taps - 1) * s.C + c];
        y = fmaf(s.taps[(size_t)c * s.n_taps + j], u, y);
    }
    return y;
}

// The four neighbouring channels from c on (c a multiple of 4; every row, the taps and the bias on 16-byte borders), the same sums:
// the rows' loads travel together, 16 bytes a thread.
__device__ __forceinline__ float4 conv_taps_four(const ConvTaps& s, int t, int start, int c) {
    const float4 b = s.bias ? *reinterpret_cast<const float4*>(s.bias + c) : make_float4(0.f, 0.f, 0.f, 0.f);
    auto row = [&](int tt) {
        if (tt < start) return *reinterpret_cast<const float4*>(s.state + (size_t)(tt - start + s.n_taps - 1) * s.C + c);
        const float4 u = *reinterpret_cast<const float4*>(s.proj + (size_t)tt * s.ld + s.col0 + c);
        return make_float4(u.x + b.x, u.y + b.y, u.z + b.z, u.w + b.w);
    };
    if (s.n_taps <= 0) return row(t);
    float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
    const float* w = s.taps + (size_t)c * s.n_taps;
    if (s.n_taps == 4) {
        const float4 u0 = row(t - 3), u1 = row(t - 2), u2 = row(t - 1), u3 = row(t);
        const float4* w4 = reinterpret_cast<const float4*>(w);
        const float4 a = w4[0], e = w4[1], f = w4[2], g = w4[3];
        y.x = fmaf(a.w, u3.x, fmaf(a.z, u2.x, fmaf(a.y, u1.x, fmaf(a.x, u0.x, 0.f))));
        y.y = fmaf(e.w, u3.y, fmaf(e.z, u2.y, fmaf(e.y, u1.y, fmaf(e.x, u0.y, 0.f))));
        y.z = fmaf(f.w, u3.z, fmaf(f.z, u2.z, fmaf(f.y, u1.z, fmaf(f.x, u0.z, 0.f))));
        y.w = fmaf(g.w, u3.w, fmaf(g.z, u2.w, fmaf(g.y, u1.w, fmaf(g.x, u0.w, 0.f))));
        return y;
    }
    for (int j = 0; j < s.n_taps; ++j) {
        const float4 u = row(t - (s.n_taps - 1) + j);
        y.x = fmaf(w[j], u.x, y.x);
        y.y = fmaf(w[s.n_taps + j], u.y, y.y);
        y.z = fmaf(w[2 * s.n_taps + j], u.z, y.z);
        y.w = fmaf(w[3 * s.n_taps + j], u.w, y.w);
    }
    return y;
}
// Whether conv_taps_four may be used (the state's slots lie slot_stride floats apart).
inline bool conv_taps_in_fours(const ConvTaps& s, const float* state, long long slot_stride) {
    const uintptr_t p = (uintptr_t)s.proj | (uintptr_t)s.bias | (uintptr_t)s.taps | (uintptr_t)state;
    return (p & 15) == 0 && s.ld % 4 == 0 && s.col0 % 4 == 0 && s.C % 4 == 0 && slot_stride % 4 == 0;
}
