// Arithmetic of the FP32 differentiable chain (s1g_adjoint.cu) in place of
// FP64: phase factors, squared magnitudes over the whole float range, logarithm.
#pragma once

#include <cmath>
#include <mutex>

#include "s1g_df.cuh"
#include "s1g_fft_engine.h"

namespace s1g {

// cos, sin of 2 pi (hi + lo) turns, |hi + lo| <= 1/2: the angle is formed to
// 2^-46 and rounded to float once, as cis_d<float> rounds its FP64 angle, so
// the factors are those of the FP64 phases but where 2^-46 decides the
// rounding (one in 10^6 elements).
__device__ __forceinline__ cf32 cis_turn(float hi, float lo) {
    const df p = two_prod(hi, 6.283185482025146484375f);   // 2 pi as 24 bits + the rest
    const float r = p.hi + fmaf(hi, -1.74845560007449713e-7f, fmaf(lo, 6.28318530717958648f, p.lo));
    float s, c;
    __sincosf(r, &s, &c);
    return mk(c, s);
}

// An FP64 value as three floats.
struct tf {
    float a, b, c;
};
__device__ __forceinline__ tf tf_from(double x) {
    tf r;
    r.a = (float)x;
    const double y = x - (double)r.a;
    r.b = (float)y;
    r.c = (float)(y - (double)r.b);
    return r;
}

// |v|^2 2^(-2 e) as a float pair in [1, 32), v's larger part of order 2^e; zero
// gives zero.  Exact to 2^-47 for every float, whose squares leave the float
// range.
struct Norm32 {
    df I;
    int e;
};
__device__ __forceinline__ float pow2(int e) { return __int_as_float((e + 127) << 23); }   // |e| <= 126
__device__ __forceinline__ Norm32 norm32(cf32& v) {
    Norm32 r;
    float m = fmaxf(fabsf(v.x), fabsf(v.y));
    r.e = 0;
    if (m < 5.421010862427522e-20f) {   // 2^-64
        v.x *= 1.2676506002282294e30f;  // 2^100
        v.y *= 1.2676506002282294e30f;
        m *= 1.2676506002282294e30f;
        r.e = -100;
    }
    const int e = m > 0.0f ? min((__float_as_int(m) >> 23) - 127, 126) : 0;
    const float u = pow2(-e);
    v.x *= u;
    v.y *= u;
    r.e += e;
    const df a = two_prod(v.x, v.x), b = two_prod(v.y, v.y);
    r.I = two_sum(a.hi, b.hi);
    r.I.lo += a.lo + b.lo;
    r.I = quick_two_sum(r.I.hi, r.I.lo);
    return r;
}

// ln (x 2^k) of a float pair x in [1, 32) in double-float, error below 1e-12
// (an FP64 log takes ~40 operations of a pipe that does 1.9 per clock and SM):
// x = 2^e m with m in [1, 2), c = 1/m to 8 bits (table of 128 by the leading
// bits of m), r = m c - 1 exactly by one FMA (|r| < 2^-7), ln x = e ln 2 -
// ln c + log1p(r) (Tang, "Table-driven implementation of the logarithm
// function", 1990), the series' first two terms in double-float.
static __device__ float c_log_c[128];     // global, not constant: lanes read different entries
static __device__ float2 c_log_t[128];    // -ln c as hi, lo
__device__ __forceinline__ df ln32(df x, int k) {
    const unsigned int bits = (unsigned int)__float_as_int(x.hi);
    const unsigned int f = bits & 0x7fffffu;
    const int e = (int)(bits >> 23) - 127 + k;
    const float m = __int_as_float((int)(0x3f800000u | f));
    const int i = (int)(f >> 16);
    const float r = __fmaf_rn(m, __ldg(c_log_c + i), -1.0f);
    const float2 t = __ldg(c_log_t + i);
    const df r2 = two_prod(r, r);
    // r^3 (1/3 - r/4 + r^2/5 - r^3/6 + r^4/7), and the low part of x
    const float p = fmaf(r, fmaf(r, fmaf(r, fmaf(r, 1.0f / 7.0f, -1.0f / 6.0f), 0.2f), -0.25f), 1.0f / 3.0f);
    const float rest = fmaf(r2.hi * r, p, __fdividef(x.lo, x.hi));
    const float ef = (float)e;
    // e ln 2 with ln 2 = 0x1.62e4p-1 (exact products) + 1.4286068202862268e-6
    const df el = two_prod(ef, 1.42860677e-6f);
    df s = quick_two_sum(ef * 0.693145751953125f, el.hi);
    s.lo += el.lo + ef * 5.4956e-14f;
    s = df_add_abs(s, df_make(t.x, t.y));
    s = df_add_f(s, r);
    s = df_add_abs(s, df_make(-0.5f * r2.hi, -0.5f * r2.lo));
    return df_add_f(s, rest);
}
// tables of ln32, once per device
static void init_log_tables() {
    static std::mutex mu;
    static bool done[64] = {};
    int dev = 0;
    check_cuda(cudaGetDevice(&dev), "log tables");
    std::lock_guard<std::mutex> lk(mu);
    if (dev < 64 && done[dev]) return;
    float c[128];
    float2 t[128];
    for (int i = 0; i < 128; ++i) {
        const double mid = 1.0 + (i + 0.5) / 128.0;
        const double q = std::rint(256.0 / mid) / 256.0;   // 8 bits after the point, exact products with m
        c[i] = (float)q;
        const double l = -std::log(q);
        t[i].x = (float)l;
        t[i].y = (float)(l - (double)t[i].x);
    }
    upload_symbol(c_log_c, c, sizeof(c), "log tables");
    upload_symbol(c_log_t, t, sizeof(t), "log tables");
    if (dev < 64) done[dev] = true;
}

}  // namespace s1g
