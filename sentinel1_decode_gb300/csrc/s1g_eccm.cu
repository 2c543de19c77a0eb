// The ECCM notch of the FP32 pipelines in compensated FP32 arithmetic.
//
// eccm() (signal_processing.cpp:914-1004) zeroes the bins of 128-point
// short-time spectra whose central-difference gradient magnitude reaches the
// mitigation threshold.  Those are hard decisions, and the notched lines feed
// the Doppler-centroid estimate, whose sums turn ~2e-7 relative noise into
// SLC errors beyond 1e-4; the FP32 pipelines therefore need the notch to the
// accuracy of the FP64 one.  Here every sample is carried as h + e (two
// complex<float>, s1g_cfft.cuh: TwoSum / TwoProd error terms propagated to
// first order, ~1e-13 relative), taken from the FP64 decoded samples, so the
// gradient decisions are the FP64 path's (up to bins within ~1e-12 of the
// threshold) and the notched samples round to the same floats, at FP32
// arithmetic speed rather than FP64's.  GB300 does 1.9 FP64 operations or
// conversions per clock and SM, so what runs per value stays off that pipe:
// the samples are split by their bits, a gradient is formed in FP32 and in
// FP64 only within 1e-5 of the threshold.  1500 lines of 12000 samples: the
// notch 0.90 ms (1.32 with a trip through shared memory per radix-4 stage, 3.70
// with FP64 splits, gradients and output sums too), the detection 0.06 ms (0.56
// with FP64 magnitudes).
//
// One block per flagged line (flags from k_eccm_detect_mixed below), windows
// of 128 samples at stride 64 in batches of kEccmBatch: forward transform,
// gradient and decision from h + e, zeroing, inverse transform, 1/128, and
// each sample written from the last window that covers it (later windows
// overwrite earlier ones).
#include <stdexcept>

#include "s1g_dcest.h"
#include "s1g_fft_engine.h"
#include "s1g_kernels.h"

namespace s1g {

namespace {

constexpr int kEccmFft = 128;
constexpr int kEccmBatch = 16;                       // windows per pass
constexpr int kEccmThreads = 128;
constexpr int kEccmRow = kEccmFft + kEccmFft / 8;    // float4 of a window, one of padding in 8

__device__ __forceinline__ cc at_cc(const float4* S, int i) {
    const float4 v = S[i];
    return cc{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ double2 cc_value(const cc& v) {
    return make_double2((double)v.hx + (double)v.ex, (double)v.hy + (double)v.ey);
}

}  // namespace

// A window is 16 x 8 points: radix-16 butterflies (one per thread) over the
// samples k + 8 r, read from the line and written to it by the same passes,
// and radix-8 ones over positions 8 s0 + s1, which then hold frequency
// s0 + 16 s1.
__global__ void __launch_bounds__(kEccmThreads, 4) k_eccm_notch_cc(const cf64* __restrict__ in, long long ip,
                                                                   cf32* __restrict__ out, long long op, int n_r,
                                                                   const int* __restrict__ flags, double mit, CfftDesc d,
                                                                   int num_ffts) {
    __shared__ float4 S[kEccmBatch * kEccmRow];
    __shared__ unsigned char zero[kEccmBatch * kEccmFft];
    const long long row = blockIdx.x;
    if (!flags[row]) return;
    const cf64* line = in + row * ip;
    cf32* o = out + row * op;
    // FP32 gradients decide for thresholds whose square is well inside the
    // float range; big_max < 0 sends every bin to FP64
    const float mit2 = (float)(mit * mit);
    const float big_max = mit > 1e-9 && mit < 1e12 ? (float)mit * 1e5f : -1.0f;
    const int wa = threadIdx.x >> 3, k = threadIdx.x & 7;
    float4* Sa = S + wa * kEccmRow + k;
    for (int w0 = 0; w0 < num_ffts; w0 += kEccmBatch) {
        const int nw = min(kEccmBatch, num_ffts - w0);
        // the original line's window, zero-filled past its (cut) end
        const int s0 = (w0 + wa) * 64;
        int end = s0 + kEccmFft;
        if (end > n_r) end = n_r - 1;
        if (wa < nw) {
            cc v[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                df x = df_make(0.f, 0.f), y = x;
                const int j = s0 + k + 8 * r;
                if (j < end) {
                    const double2 z = __ldg(reinterpret_cast<const double2*>(line) + j);
                    x = df_split(z.x);
                    y = df_split(z.y);
                }
                v[r] = cc{x.hi, y.hi, x.lo, y.lo};
            }
            cc_fft<16, -1>(v);
#pragma unroll
            for (int s = 0; s < 16; ++s) {
                if (s > 0) v[s] = cc_twiddle(v[s], d.tw, s * k, -1);
                Sa[9 * s] = make_float4(v[s].hx, v[s].hy, v[s].ex, v[s].ey);
            }
        }
        __syncthreads();
        for (int t = threadIdx.x; t < nw * 16; t += kEccmThreads) {
            float4* b = S + (t >> 4) * kEccmRow + 9 * (t & 15);
            cc v[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) v[r] = at_cc(b, r);
            cc_fft<8, -1>(v);
#pragma unroll
            for (int s = 0; s < 8; ++s) b[s] = make_float4(v[s].hx, v[s].hy, v[s].ex, v[s].ey);
        }
        __syncthreads();
        // central-difference gradient along frequency (one-sided at the ends)
        for (int t = threadIdx.x; t < nw * kEccmFft; t += kEccmThreads) {
            const int w = t >> 7, q = t & 127;
            const float4* b = S + w * kEccmRow;
            // (X[up] - X[dn]) scale; in FP32 where that decides: its error is
            // below 2^-22 of itself and 2^-40 of the values
            const int up = min(q + 1, kEccmFft - 1), dn = max(q - 1, 0);
            const float scale = q != 0 && q != kEccmFft - 1 ? 0.5f : 1.0f;
            const cc u = at_cc(b, 9 * (up & 15) + (up >> 4)), v = at_cc(b, 9 * (dn & 15) + (dn >> 4));
            const float gx = scale * ((u.hx - v.hx) + (u.ex - v.ex)), gy = scale * ((u.hy - v.hy) + (u.ey - v.ey));
            const float g2 = fmaf(gx, gx, gy * gy);
            const float big = fmaxf(fmaxf(fabsf(u.hx), fabsf(u.hy)), fmaxf(fabsf(v.hx), fabsf(v.hy)));
            if (fabsf(g2 - mit2) > 1e-5f * mit2 && big < big_max) {
                zero[t] = g2 < mit2 ? 0 : 1;
            } else {
                const double2 a = cc_value(u), c = cc_value(v);
                const double x = (a.x - c.x) * scale, y = (a.y - c.y) * scale;
                zero[t] = (hypot(x, y) < mit) ? 0 : 1;
            }
        }
        __syncthreads();
        for (int t = threadIdx.x; t < nw * 16; t += kEccmThreads) {
            const int w = t >> 4, s = t & 15;
            float4* b = S + w * kEccmRow + 9 * s;
            cc v[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                v[r] = at_cc(b, r);
                if (zero[w * kEccmFft + s + 16 * r]) v[r] = cc{0.f, 0.f, 0.f, 0.f};
            }
            cc_fft<8, 1>(v);
#pragma unroll
            for (int r = 0; r < 8; ++r) b[r] = make_float4(v[r].hx, v[r].hy, v[r].ex, v[r].ey);
        }
        __syncthreads();
        if (wa < nw) {
            cc v[16];
#pragma unroll
            for (int s = 0; s < 16; ++s) {
                v[s] = at_cc(Sa, 9 * s);
                if (s > 0) v[s] = cc_twiddle(v[s], d.tw, s * k, +1);
            }
            cc_fft<16, 1>(v);
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const int wi = w0 + wa, j = s0 + k + 8 * r;
                if (j >= end) continue;
                // a later window that covers j overwrites it: the next one
                // covers the second half of this one
                if (8 * r + k >= 64 && wi + 1 < num_ffts) {
                    int ce = (wi + 1) * 64 + kEccmFft;
                    if (ce > n_r) ce = n_r - 1;
                    if (j < ce) continue;
                }
                o[j] = mk((v[r].hx + v[r].ex) * (1.0f / 128.0f), (v[r].hy + v[r].ey) * (1.0f / 128.0f));
            }
        }
        __syncthreads();
    }
}

// ---- line detection from an FP32 spectrum, FP64 where it is close
// A line is flagged when max_k |X_k| >= det.  From the FP32 spectrum of the
// line (FP32 samples and FFT: every |X_k| good to ~1e-6 of det whenever the
// maximum is near det) the decision is certain unless the maximum lies within
// kDetMargin (relative) of det; such a line is decided from the exact FP64
// DFT of its FP64 samples at the bins that could reach det (FP32 magnitude
// >= det (1 - kDetMargin)), one bin at a time by the whole block, stopping at
// the first bin that reaches det.
constexpr double kDetMargin = 1e-4;

__global__ void k_roots64(cf64* __restrict__ roots, int n) {
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < n; m += gridDim.x * blockDim.x) {
        double sn, cs;
        sincospi(-2.0 * (double)m / (double)n, &sn, &cs);
        cf64 r;
        r.x = cs;
        r.y = sn;
        roots[m] = r;
    }
}

__device__ __forceinline__ double block_sum256(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < 8; ++w) t += red[w];
    return t;   // thread 0
}

__global__ void __launch_bounds__(256) k_eccm_detect_mixed(const cf32* __restrict__ X, long long xp, int n, double det,
                                                           const cf64* __restrict__ x64, long long p64,
                                                           const cf64* __restrict__ roots, int* __restrict__ flags) {
    __shared__ double red[256];
    __shared__ int cand[256];
    __shared__ int ncand, hit;
    const long long row = blockIdx.x;
    const cf32* Xr = X + row * xp;
    // the FP32 magnitude (3e-7) is inside the margin
    float mf = 0.0f;
    for (int k = threadIdx.x; k < n; k += 256) {
        const cf32 v = Xr[k];
        mf = fmaxf(mf, hypotf(v.x, v.y));
    }
    double mx = (double)mf;
    red[threadIdx.x] = mx;
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + s]);
        __syncthreads();
    }
    mx = red[0];
    __syncthreads();
    if (mx < det * (1.0 - kDetMargin) || mx >= det * (1.0 + kDetMargin)) {
        if (threadIdx.x == 0) flags[row] = (mx < det) ? 0 : 1;
        return;
    }
    const cf64* line = x64 + row * p64;
    const double lo = det * (1.0 - kDetMargin);
    if (threadIdx.x == 0) hit = 0;
    for (int base = 0; base < n; base += 256) {
        if (threadIdx.x == 0) ncand = 0;
        __syncthreads();
        const int k = base + threadIdx.x;
        if (k < n) {
            const cf32 v = Xr[k];
            if (hypot((double)v.x, (double)v.y) >= lo) cand[atomicAdd(&ncand, 1)] = k;
        }
        __syncthreads();
        const int nc = ncand;
        for (int c = 0; c < nc; ++c) {
            const long long kk = cand[c];
            long long m = (kk * threadIdx.x) % n;
            const long long step = (kk * 256) % n;
            double re = 0.0, im = 0.0;
            for (int j = threadIdx.x; j < n; j += 256) {
                const cf64 v = line[j], w = roots[m];
                re = fma(v.x, w.x, fma(-v.y, w.y, re));
                im = fma(v.x, w.y, fma(v.y, w.x, im));
                m += step;
                if (m >= n) m -= n;
            }
            re = block_sum256(re, red);
            im = block_sum256(im, red + 8);
            if (threadIdx.x == 0 && !(hypot(re, im) < det)) hit = 1;
            __syncthreads();
            if (hit) break;
        }
        __syncthreads();
        if (hit) break;
    }
    if (threadIdx.x == 0) flags[row] = hit;
}

void eccm_detect_mixed(const cf32* X32, long long xp, int n, long long rows, double det, const cf64* x64,
                       long long p64, cf64* roots, int* flags, cudaStream_t st) {
    if (rows <= 0 || n <= 0) return;
    note_launch(), k_roots64<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(roots, n);
    note_launch(), k_eccm_detect_mixed<<<(unsigned)rows, 256, 0, st>>>(X32, xp, n, det, x64, p64, roots, flags);
}

void eccm_notch_cc(const cf64* in, long long ip, cf32* out, long long op, int n_r, long long rows, const int* flags,
                   double mit, const CfftDesc& d128, cudaStream_t st) {
    if (d128.n != kEccmFft) throw std::runtime_error("eccm: the twiddles must be those of 128 points");
    const int num_ffts = eccm_num_windows(n_r);
    if (rows > 0 && num_ffts > 0)
        note_launch(), k_eccm_notch_cc<<<(unsigned)rows, kEccmThreads, 0, st>>>(in, ip, out, op, n_r, flags, mit, d128,
                                                                        num_ffts);
}

}  // namespace s1g
