// Index arithmetic of the time unfolding's axes (s1g_tufr.cu).
#pragma once

#include <cuda_runtime.h>

namespace s1g {

// Knot intervals of the TS-point deramp axis (K_a resampled S -> TS,
// linear_resample): sample u lies in interval floor(u (S - 1) / (TS - 1))
// (the last sample in interval S - 2), and interval iv starts at
// ceil(iv (TS - 1) / (S - 1)).  Both from float estimates (within one of the
// answer for TS < 2^24) corrected with exact integer products, which keeps
// 64-bit divisions off the sample path.
// The interval of sample u and its step from the interval's first sample.
// The remainder num = u (S - 1) - q (TS - 1) is below 2 TS in magnitude, so
// 32-bit products that wrap give it exactly; the step is floor(num / (S - 1)).
__device__ __forceinline__ int knot_of_near(int u, int S, int TS, float gk, float inv_s1, int& d) {
    int q = __float2int_rz((float)u * gk);
    int num = (int)((unsigned int)u * (unsigned int)(S - 1) - (unsigned int)q * (unsigned int)(TS - 1));
    if (num < 0) {
        --q;
        num += TS - 1;
    } else if (num >= TS - 1) {
        ++q;
        num -= TS - 1;
    }
    if (q > S - 2) {
        q = S - 2;
        num += TS - 1;
    }
    d = __float2int_rz(((float)num + 0.5f) * inv_s1);
    return q;
}
__device__ __forceinline__ int knot_first_near(int iv, int S, long long TS, float rt) {
    const long long num = (long long)iv * (TS - 1);
    int n = __float2int_ru((float)iv * rt);
    if ((long long)n * (S - 1) < num) ++n;
    else if ((long long)(n - 1) * (S - 1) >= num) --n;
    return n;
}

// Smallest n with m2 n >= A, and largest n with m2 n <= B (m2 > 0), for
// A = a TS, B = b TS: the float estimate a TS / m2 (two exact float factors,
// |a|, TS < 2^24) is within one of the answer, the loops correct it with
// exact integer products.  No 64-bit conversions (FP64 pipe on this part).
__device__ __forceinline__ int first_at_or_above(int a, int TS, int m2, float inv_m2) {
    const long long A = (long long)a * TS;
    int n = (int)ceilf((float)a * (float)TS * inv_m2);
    while ((long long)m2 * n < A) ++n;
    while ((long long)m2 * (n - 1) >= A) --n;
    return n;
}

}  // namespace s1g
