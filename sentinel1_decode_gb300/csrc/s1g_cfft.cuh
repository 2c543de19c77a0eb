// Compensated FP32 FFT in shared memory (device side).
//
// Each complex value is carried as an unevaluated sum h + e of two cf32: h is
// the ordinary FP32 result and e accumulates, in FP32, the rounding error of
// every operation that produced h.  Additions use TwoSum and products use
// TwoProd (fused multiply-add) to capture their rounding errors exactly; the
// error terms themselves are propagated to first order without
// renormalisation (the compensated Cooley-Tukey scheme of Jiang, Graillat,
// Hu, Luo & Rump, "Accurate complex multiplication and FFT in floating-point
// arithmetic", restated for float pairs).  The result h + e carries about
// 1e-13 relative error, against ~2e-7 for the plain FP32 core, at roughly
// six times the arithmetic.  Twiddles are exp(-2 pi i k/n) split into float
// pairs from FP64.
//
// Butterflies of radix 2, 3 and 4 and composites of them up to 16, for the
// Doppler estimator (s1g_dcest.cu) and the ECCM notch (s1g_eccm.cu).
#pragma once

#include "s1g_df.cuh"
#include "s1g_fft.cuh"

namespace s1g {

// t = g * ns + k with 0 <= k < ns (t < 2^24)
__device__ __forceinline__ void split_idx(int t, int ns, float inv_ns, int& g, int& k) {
    g = __float2int_rz((float)t * inv_ns);
    k = t - g * ns;
    if (k < 0) {
        --g;
        k += ns;
    } else if (k >= ns) {
        ++g;
        k -= ns;
    }
}

struct CfftDesc {
    int n = 0;
    const float4* tw = nullptr;  // {cos hi, -sin hi, cos lo, -sin lo} of exp(-2 pi i k / n)
};

struct cc {
    float hx, hy, ex, ey;
};

__device__ __forceinline__ cc cc_make(cf32 h, cf32 e) { return cc{h.x, h.y, e.x, e.y}; }

__device__ __forceinline__ cc cc_add(const cc& a, const cc& b) {
    const df sx = two_sum(a.hx, b.hx);
    const df sy = two_sum(a.hy, b.hy);
    return cc{sx.hi, sy.hi, sx.lo + (a.ex + b.ex), sy.lo + (a.ey + b.ey)};
}

__device__ __forceinline__ cc cc_sub(const cc& a, const cc& b) {
    const df sx = two_sum(a.hx, -b.hx);
    const df sy = two_sum(a.hy, -b.hy);
    return cc{sx.hi, sy.hi, sx.lo + (a.ex - b.ex), sy.lo + (a.ey - b.ey)};
}

// times dir * i (exact)
__device__ __forceinline__ cc cc_mul_i(const cc& a, int dir) {
    return dir > 0 ? cc{-a.hy, a.hx, -a.ey, a.ex} : cc{a.hy, -a.hx, a.ey, -a.ex};
}

// times the float-pair complex w = (wx + wlx) + i (wy + wly)
__device__ __forceinline__ cc cc_mul(const cc& a, float wx, float wy, float wlx, float wly) {
    const df p1 = two_prod(a.hx, wx);
    const df p2 = two_prod(a.hy, wy);
    const df s = two_sum(p1.hi, -p2.hi);
    const float er = fmaf(a.ex, wx, fmaf(-a.ey, wy, fmaf(a.hx, wlx, fmaf(-a.hy, wly, s.lo + (p1.lo - p2.lo)))));
    const df q1 = two_prod(a.hx, wy);
    const df q2 = two_prod(a.hy, wx);
    const df t = two_sum(q1.hi, q2.hi);
    const float ei = fmaf(a.ex, wy, fmaf(a.ey, wx, fmaf(a.hx, wly, fmaf(a.hy, wlx, t.lo + (q1.lo + q2.lo)))));
    return cc{s.hi, t.hi, er, ei};
}

// twiddle exp(dir 2 pi i idx / n) from the table
__device__ __forceinline__ cc cc_twiddle(const cc& a, const float4* tw, int idx, int dir) {
    const float4 w = __ldg(tw + idx);
    return dir > 0 ? cc_mul(a, w.x, -w.y, w.z, -w.w) : cc_mul(a, w.x, w.y, w.z, w.w);
}

// times a real float pair (c + cl)
__device__ __forceinline__ cc cc_scale(const cc& a, float c, float cl) {
    const df px = two_prod(a.hx, c);
    const df py = two_prod(a.hy, c);
    return cc{px.hi, py.hi, px.lo + a.hx * cl + a.ex * c, py.lo + a.hy * cl + a.ey * c};
}

template <int P>
struct CBfly;

template <>
struct CBfly<2> {
    static __device__ __forceinline__ void run(cc* a, int) {
        const cc t = a[0];
        a[0] = cc_add(t, a[1]);
        a[1] = cc_sub(t, a[1]);
    }
};

template <>
struct CBfly<4> {
    static __device__ __forceinline__ void run(cc* a, int dir) {
        const cc t0 = cc_add(a[0], a[2]), t1 = cc_sub(a[0], a[2]);
        const cc t2 = cc_add(a[1], a[3]), t3 = cc_mul_i(cc_sub(a[1], a[3]), dir);
        a[0] = cc_add(t0, t2);
        a[2] = cc_sub(t0, t2);
        a[1] = cc_add(t1, t3);
        a[3] = cc_sub(t1, t3);
    }
};

template <>
struct CBfly<3> {
    // X1 = a0 - (a1 + a2)/2 + dir i (sqrt(3)/2) (a1 - a2), X2 the conjugate combination
    static __device__ __forceinline__ void run(cc* a, int dir) {
        const cc t = cc_add(a[1], a[2]);
        const cc d = cc_sub(a[1], a[2]);
        const cc x0 = cc_add(a[0], t);
        const cc half = cc{0.5f * t.hx, 0.5f * t.hy, 0.5f * t.ex, 0.5f * t.ey};
        const cc m = cc_sub(a[0], half);
        const cc r = cc_mul_i(cc_scale(d, 0.866025388240814209f, 1.55436250537377420e-08f), dir);
        a[0] = x0;
        a[1] = cc_add(m, r);
        a[2] = cc_sub(m, r);
    }
};

// times exp(DIR 2 pi i NUM / 48) for the composite radices below
template <int NUM, int DIR>
__device__ __forceinline__ cc cc_root48(const cc& a) {
    static_assert(NUM >= 0 && NUM < 48, "");
    if constexpr (NUM == 0) return a;
    else if constexpr (NUM == 24) return cc{-a.hx, -a.hy, -a.ex, -a.ey};
    else if constexpr (NUM > 24) {
        const cc t = cc_root48<NUM - 24, DIR>(a);
        return cc{-t.hx, -t.hy, -t.ex, -t.ey};
    } else if constexpr (NUM >= 12) return cc_mul_i(cc_root48<NUM - 12, DIR>(a), DIR);
    else if constexpr (NUM == 6) {
        // (1 + DIR i) / sqrt 2
        const df x = two_sum(a.hx, DIR > 0 ? -a.hy : a.hy), y = two_sum(a.hy, DIR > 0 ? a.hx : -a.hx);
        const cc z{x.hi, y.hi, x.lo + (DIR > 0 ? a.ex - a.ey : a.ex + a.ey), y.lo + (DIR > 0 ? a.ey + a.ex : a.ey - a.ex)};
        constexpr float c = (float)0.70710678118654752440;
        return cc_scale(z, c, (float)(0.70710678118654752440 - (double)c));
    } else {
        // cos, sin of 22.5, 30, 60 and 67.5 degrees
        static_assert(NUM == 3 || NUM == 4 || NUM == 8 || NUM == 9, "");
        constexpr double cd = NUM == 3 ? 0.92387953251128675613 : NUM == 4 ? 0.86602540378443864676
                            : NUM == 8 ? 0.5 : 0.38268343236508977173;
        constexpr double sd = NUM == 3 ? 0.38268343236508977173 : NUM == 4 ? 0.5
                            : NUM == 8 ? 0.86602540378443864676 : 0.92387953251128675613;
        constexpr float c = (float)cd, s = (float)(DIR * sd);
        return cc_mul(a, c, s, (float)(cd - (double)c), (float)(DIR * sd - (double)s));
    }
}

// A x B points in registers, j = b + B a in, s + A q out: A-point butterflies
// over a, twiddles exp(DIR 2 pi i b s / (A B)), B-point butterflies over b.
template <int A, int B, int DIR>
__device__ __forceinline__ void cc_composite(cc* x) {
    constexpr int U = 48 / (A * B);
    cc y[A * B];   // [b][s]
#pragma unroll
    for (int b = 0; b < B; ++b) {
        cc t[A];
#pragma unroll
        for (int a = 0; a < A; ++a) t[a] = x[b + B * a];
        CBfly<A>::run(t, DIR);
#pragma unroll
        for (int s = 0; s < A; ++s) y[b * A + s] = t[s];
    }
    if constexpr (B > 1) {
        if constexpr (A > 1) y[A + 1] = cc_root48<(U * 1) % 48, DIR>(y[A + 1]);
        if constexpr (A > 2) y[A + 2] = cc_root48<(U * 2) % 48, DIR>(y[A + 2]);
        if constexpr (A > 3) y[A + 3] = cc_root48<(U * 3) % 48, DIR>(y[A + 3]);
    }
    if constexpr (B > 2) {
        if constexpr (A > 1) y[2 * A + 1] = cc_root48<(U * 2) % 48, DIR>(y[2 * A + 1]);
        if constexpr (A > 2) y[2 * A + 2] = cc_root48<(U * 4) % 48, DIR>(y[2 * A + 2]);
        if constexpr (A > 3) y[2 * A + 3] = cc_root48<(U * 6) % 48, DIR>(y[2 * A + 3]);
    }
    if constexpr (B > 3) {
        if constexpr (A > 1) y[3 * A + 1] = cc_root48<(U * 3) % 48, DIR>(y[3 * A + 1]);
        if constexpr (A > 2) y[3 * A + 2] = cc_root48<(U * 6) % 48, DIR>(y[3 * A + 2]);
        if constexpr (A > 3) y[3 * A + 3] = cc_root48<(U * 9) % 48, DIR>(y[3 * A + 3]);
    }
#pragma unroll
    for (int s = 0; s < A; ++s) {
        cc t[B];
#pragma unroll
        for (int b = 0; b < B; ++b) t[b] = y[b * A + s];
        CBfly<B>::run(t, DIR);
#pragma unroll
        for (int q = 0; q < B; ++q) x[s + A * q] = t[q];
    }
}
template <int P, int DIR>
__device__ __forceinline__ void cc_fft(cc* x) {
    static_assert(P == 4 || P == 6 || P == 8 || P == 12 || P == 16, "");
    if constexpr (P == 4) CBfly<4>::run(x, DIR);
    else if constexpr (P == 6) cc_composite<2, 3, DIR>(x);
    else if constexpr (P == 8) cc_composite<2, 4, DIR>(x);
    else if constexpr (P == 12) cc_composite<4, 3, DIR>(x);
    else cc_composite<4, 4, DIR>(x);
}

}  // namespace s1g
