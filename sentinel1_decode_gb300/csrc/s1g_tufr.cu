// Time unfolding, quadratic resampling and re-ramp of the TOPS chain
// (image_formation.cpp:222-388): the band of the length-(T*S) DFT and its
// evaluation at the resampling stencils as two non-uniform FFTs on one grid.
#include <algorithm>
#include <cmath>
#include <map>
#include <mutex>
#include <stdexcept>

#include "s1g_czt.cuh"
#include "s1g_tufr_index.cuh"

namespace s1g {

// ------------------------------------------------------------------ time unfolding

// Knot of the deramp / re-ramp phase at azimuth row rw of a range bin:
// pi K_t and the deramp time -f_dc/K_a.
struct Knot {
    df pkt, dct;
};
__device__ __forceinline__ Knot knot_at(const RowDf& rw, df Q, df fdc, df ilr, const TufrArgs& a) {
    const df F = df_add_abs(rw.fa, fdc);
    const df vq = df_mul(rw.P, df_add_abs(rw.A, df_neg(Q)));
    const df x = df_div2(df_mul(a.lam2_4, df_mul(F, F)), vq);
    // 1 / K_a with K_a = -2 v^2 D^3 / (lambda R), D = sqrt(1 - x); then
    // K_t = -K_a r / (r - K_a) = 1 / (1 / r - 1 / K_a)
    const df w = df_mul(df_mul(vq, df_pow32_1m(x)), ilr);
    const df iu = df_div2(df_make(-0.5f, 0.f), w);
    Knot k;
    k.dct = df_neg(df_mul(fdc, iu));                          // -f_dc / K_a
    k.pkt = df_div2(a.pi_, df_add_abs(a.inv_rate, df_neg(iu)));
    return k;
}

// Re-ramp phase of azimuth_time_ufr (image_formation.cpp:365-373) at time tau
// between two knots (fraction al).  With t = dct + tau and K_a dct = -f_dc
// the reference's pi kt t^2 - 2 pi (kt + K_a) dct t equals
// pi kt (tau^2 - dct^2) + 2 pi f_dc (tau + dct), evaluated here as
// (tau + dct) [pi kt (tau - dct) + 2 pi f_dc]; the deramp phase
// (image_formation.cpp:305-313) is its negative (DerampPoly).
__device__ __forceinline__ float reramp_phase(Knot k0, Knot k1, float al, df tau, df tpf) {
    const df pkt = df_add_f(k0.pkt, ((k1.pkt.hi - k0.pkt.hi) + (k1.pkt.lo - k0.pkt.lo)) * al);
    const df dct = df_add_f(k0.dct, ((k1.dct.hi - k0.dct.hi) + (k1.dct.lo - k0.dct.lo)) * al);
    const df a = df_add_abs(tau, dct);
    const df b = df_add_abs(tau, df_neg(dct));
    return df_wrap(df_mul(a, df_add_abs(df_mul(pkt, b), tpf)));
}

// ---- deramp phase of a knot interval as a polynomial in the sample step
// Over the samples n = n_a + d of one knot interval iv (K_a resampled from
// knots iv, iv + 1, fraction al = al_a + d (S - 1) / (TS - 1)), pi K_t and
// -f_dc/K_a are linear in d and so is az_time, and the deramp argument
// th = (tau + dct) [pi kt (tau - dct) + 2 pi f_dc] (reramp_phase) is the cubic
//   th(d) = H0 + G1 d + G2 d^2 + (A1 C2 d^3, below 1e-8 rad over an interval)
// H0 and G1 in double-float, reduced to fractions of a turn in 32-bit fixed
// point; the phase -th / (2 pi) - n k_s / TS then wraps by integer overflow.
struct DerampPoly {
    unsigned int base, slope;   // -H0, -G1 in turns x 2^32 (mod 2^32)
    float curv;                 // -G2 in turns x 2^32
};

// frac(x / (2 pi)) x 2^32 (mod 2^32) of a double-float x (|x| < ~1e6)
__device__ __forceinline__ unsigned int turns_fx(df x, df i2p) {
    const df t = df_mul(x, i2p);
    const float k = rintf(t.hi);
    // |t.hi - k| <= 1/2: x 2^32 saturates only at exactly +2^31 (one unit off)
    return (unsigned int)__float2int_rn((t.hi - k) * 4294967296.0f) + (unsigned int)__float2int_rn(t.lo * 4294967296.0f);
}

__device__ __forceinline__ DerampPoly deramp_poly(Knot k0, Knot k1, float al, df tau, df tpf, df dt, float gk, df i2p) {
    const float dpk = (k1.pkt.hi - k0.pkt.hi) + (k1.pkt.lo - k0.pkt.lo);
    const float ddc = (k1.dct.hi - k0.dct.hi) + (k1.dct.lo - k0.dct.lo);
    const df P = df_add_f(k0.pkt, dpk * al);
    const df D = df_add_f(k0.dct, ddc * al);
    const float Pd = dpk * gk, Dd = ddc * gk;   // per-sample steps of P and D
    const df A0 = df_add_abs(tau, D), B0 = df_add_abs(tau, df_neg(D));
    const df C0 = df_add_abs(df_mul(P, B0), tpf);
    const df H0 = df_mul(A0, C0);
    // th'(0) = A1 C0 + A0 C1 with A1 = dt + Dd, B1 = dt - Dd, C1 = P B1 + Pd B0:
    //   dt (C0 + A0 P) + Dd (C0 - A0 P) + A0 Pd B0
    // the first term (~1 rad per sample) in double-float, the others (~1e-3)
    // in float
    const df Q = df_mul(A0, P);
    const float small = fmaf(Dd, C0.hi - Q.hi, A0.hi * Pd * B0.hi);
    const df G1 = df_add_f(df_mul(dt, df_add_abs(C0, Q)), small);
    // th''(0) / 2 = A0 C2 + A1 C1 with C2 = Pd B1 (~1e-5 rad): float
    const float B1 = dt.hi - Dd, A1 = dt.hi + Dd;
    const float C1 = fmaf(P.hi, B1, Pd * B0.hi);
    const float G2 = fmaf(A0.hi, Pd * B1, A1 * C1);
    DerampPoly r;
    r.base = 0u - turns_fx(H0, i2p);
    r.slope = 0u - turns_fx(G1, i2p);
    r.curv = -G2 * 683565275.57643158f;   // 2^32 / (2 pi)
    return r;
}

// exp(i 2 pi (phase in turns)) at step d of the interval, band shift pm
__device__ __forceinline__ cf32 deramp_rot(unsigned int base, unsigned int slope, float curv, int d, float d2,
                                           unsigned int pm) {
    const unsigned int ph = base + slope * (unsigned int)d + (unsigned int)__float2int_rn(curv * d2) - pm;
    float sn, cs;
    __sincosf((float)(int)ph * 1.46291807926715968e-9f, &sn, &cs);   // 2 pi / 2^32
    return mk(cs, sn);
}

// Deramp polynomials of every knot interval and range bin: a warp forms 32
// adjacent knots of a bin, each lane the interval to the next one.  Bound by
// instruction issue (86 % of it; double-float arithmetic, 430 instructions a
// knot): 1.06 ms for 12000 bins of 6900 knots, 1.67 with df_div / df_sqrt
// instead of two-digit quotients and series, about 2.4 inside the spreading
// kernel, between its barriers.
__global__ void __launch_bounds__(256) k_tufr_knots(TufrArgs a) {
    if (!a.P->ok) return;
    const int S = a.S;
    const int TS = a.P->q.num_tiles * S;
    const int lane = threadIdx.x & 31;
    const int iv0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * 31;
    if (iv0 >= S - 1) return;
    const int j = blockIdx.y;
    const int iv = iv0 + lane;
    const df fdc = a.fdc[j];
    const Knot k0 = knot_at(a.rows[min(iv, S - 1)], a.cols[j].Q, fdc, a.inv_lamR[j], a);
    Knot k1;
    k1.pkt = df_make(__shfl_down_sync(0xffffffffu, k0.pkt.hi, 1), __shfl_down_sync(0xffffffffu, k0.pkt.lo, 1));
    k1.dct = df_make(__shfl_down_sync(0xffffffffu, k0.dct.hi, 1), __shfl_down_sync(0xffffffffu, k0.dct.lo, 1));
    if (lane == 31 || iv >= S - 1) return;
    const df dt = a.P->dt, dtau = a.P->dtau, tau0 = a.P->tau0;
    const float gk = a.P->gk;
    const df i2p = df_from(0.15915494309189533577);
    const int na = knot_first_near(iv, S, TS, a.P->rt);
    // knot fraction and az_time of the anchor, as the reference's
    // linear_resample and linspace give them
    const float al = (float)(int)((long long)na * (S - 1) - (long long)iv * (TS - 1)) / (float)(TS - 1);
    const df tau = df_add_abs(tau0, df_mul_f(dtau, (float)na));
    const DerampPoly p = deramp_poly(k0, k1, al, tau, df_mul(a.two_pi_, fdc), dt, gk, i2p);
    const long long o = (long long)j * S + iv;
    a.poly[o] = make_uint2(p.base, p.slope);
    a.curv[o] = p.curv;
}

// exp(i re-ramp phase) of every output row and range bin (image_formation.cpp:355-378).
__global__ void __launch_bounds__(256) k_tufr_ramp(TufrArgs a) {
    if (!a.P->ok) return;
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n_out) return;
    const int j = blockIdx.y;
    const float4 rr = __ldg(a.tab.rer + p);
    const int ir = __float_as_int(rr.x);
    const df fdc = a.fdc[j], Q = a.cols[j].Q, ilr = a.inv_lamR[j];
    const Knot k0 = knot_at(a.rows[ir], Q, fdc, ilr, a), k1 = knot_at(a.rows[ir + 1], Q, fdc, ilr, a);
    a.ramp[(long long)j * a.n_out + p] =
        cexpf_fast(reramp_phase(k0, k1, rr.y, df_make(rr.z, rr.w), df_mul(a.two_pi_, fdc)));
}

// Band of the length-TS DFT (image_formation.cpp:315-333), type-1 non-uniform
// FFT: spread y[n] exp(-2 pi i n k_s / TS), the deramped tiled line
// y[s + S t] = A[s] exp(-i deramp(s + S t)), onto the grid (grid point l
// gathers the samples within W/2 of x_n = n M / TS; n is taken modulo TS).
//
// A CTA takes kTufrGroup = 4 range bins and a run of lc grid points: it stages
// the deramped samples around them in shared memory (two float4 planes, two
// bins each), then each thread gathers 4 adjacent grid points of all four
// bins: per sample two 16-byte shared loads, one 16-byte load of the four
// weights and 32 FMAs.  The weights do not depend on the range bin: a table
// per burst in the order the threads read it (2.7 MB, from L2).  The threads
// of a warp take point groups `perm` apart, which puts the 8 lanes of a
// quarter-warp load on different banks for the sample spacing at hand
// (perm = 1 put all 8 on one where 4 TS / M is near a multiple of 8).
// Three CTAs of 128 threads per SM, so one's staging (latency of L2 loads)
// runs under another's gather (FMA).
//
// 12000 bins of 41400 samples onto 10240 points: 2.09 ms (2.72 with one or two
// samples' loads in flight in the staging instead of three).  The kernel
// before took two bins and two points per thread, formed each weight from its
// square root and exponential (special-function bound), and spread,
// transformed and evaluated in one CTA: 8.75 ms, now 4.37 for the four kernels.
constexpr int kSpreadThreads = 128;

__global__ void __launch_bounds__(kSpreadThreads, 3) k_tufr_spread(TufrArgs a, int launch_chunks) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    static_assert(kTufrGroup == 4, "two planes of range-bin pairs");
    const TufrDev& dev = *a.P;
    const TufrParams q = dev.q;
    const int T = q.num_tiles;
    const int S = a.S, M = a.dnu.n;
    const int bw = q.end - q.start;
    // outside the launch plan (tile count, band, chunk): flag, do nothing
    if (!dev.ok || bw > a.bwmax || dev.chunks > launch_chunks) {
        if (blockIdx.x == 0 && threadIdx.x == 0) *a.status = 1;
        return;
    }
    const int chunk = blockIdx.x % launch_chunks;
    if (chunk >= dev.chunks) return;
    const int j0 = (int)(blockIdx.x / launch_chunks) * kTufrGroup;
    const int rc = min(kTufrGroup, a.n_r - j0);
    const int TS = T * S;
    const int m2 = 2 * M;
    const float inv_m2 = 1.0f / (float)m2;
    const int lc = dev.lc, kw = dev.kw;
    const int l0 = chunk * lc;
    const int l1 = min(M, l0 + lc);
    float4* pa = reinterpret_cast<float4*>(smem_raw);
    float4* pb = pa + a.ycap;
    // samples nA .. nA + len of the windows of groups l0 .. l1 - 4
    const int nA = first_at_or_above(2 * l0 - kNuW, TS, m2, inv_m2);
    const int len = first_at_or_above(2 * (l1 - 4) - kNuW, TS, m2, inv_m2) + kw - nA;
    {
        const float gk = dev.gk;
        const float inv_s = 1.0f / (float)S, inv_s1 = 1.0f / (float)(S - 1);
        const unsigned long long KS64 = dev.ks64;
        const cf32* in[kTufrGroup];
        const uint2* po[kTufrGroup];
        const float* cu[kTufrGroup];
#pragma unroll
        for (int r = 0; r < kTufrGroup; ++r) {
            const long long o = (long long)(j0 + min(r, rc - 1)) * S;
            in[r] = a.in + o;
            po[r] = a.poly + o;
            cu[r] = a.curv + o;
        }
        // kBatch samples' loads in flight before the first is used
        constexpr int kBatch = 3;
        for (int i0 = threadIdx.x; i0 < len; i0 += kBatch * kSpreadThreads) {
            cf32 v[kBatch][kTufrGroup];
            uint2 p[kBatch][kTufrGroup];
            float c[kBatch][kTufrGroup];
            unsigned int pm[kBatch];
            int d[kBatch];
#pragma unroll
            for (int b = 0; b < kBatch; ++b) {
                int u = nA + min(i0 + b * kSpreadThreads, len - 1);
                while (u < 0) u += TS;
                while (u >= TS) u -= TS;
                int si = u - S * __float2int_rz((float)u * inv_s);
                if (si < 0) si += S;
                else if (si >= S) si -= S;
                const unsigned int iv = knot_of_near(u, S, TS, gk, inv_s1, d[b]);
                pm[b] = (unsigned int)(((unsigned long long)u * KS64) >> 32);
#pragma unroll
                for (int r = 0; r < kTufrGroup; ++r) {
                    v[b][r] = ldg(in[r] + (unsigned int)si);
                    p[b][r] = __ldg(po[r] + iv);
                    c[b][r] = __ldg(cu[r] + iv);
                }
            }
#pragma unroll
            for (int b = 0; b < kBatch; ++b) {
                const int i = i0 + b * kSpreadThreads;
                const float d2 = (float)(d[b] * d[b]);
                cf32 o[kTufrGroup];
#pragma unroll
                for (int r = 0; r < kTufrGroup; ++r)
                    o[r] = v[b][r] * deramp_rot(p[b][r].x, p[b][r].y, c[b][r], d[b], d2, pm[b]);
                if (i < len) {
                    pa[i] = make_float4(o[0].x, o[0].y, o[1].x, o[1].y);
                    pb[i] = make_float4(o[2].x, o[2].y, o[3].x, o[3].y);
                }
            }
        }
    }
    __syncthreads();
    const int ng = lc >> 2;
    const int l = l0 + 4 * (int)((unsigned int)(threadIdx.x * dev.perm) % (unsigned int)ng);
    if (threadIdx.x >= ng || l >= M) return;
    const int lo = first_at_or_above(2 * l - kNuW, TS, m2, inv_m2) - nA;
    const float4* wt = a.tab.wt + (long long)chunk * kw * kSpreadThreads + threadIdx.x;
    float4 g[4][2];
#pragma unroll
    for (int c = 0; c < 4; ++c) g[c][0] = g[c][1] = make_float4(0.f, 0.f, 0.f, 0.f);
    auto step = [&](int k, float4 w) {
        const float4 x = pa[lo + k], y = pb[lo + k];
        const float wc[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            g[c][0].x = fmaf(wc[c], x.x, g[c][0].x);
            g[c][0].y = fmaf(wc[c], x.y, g[c][0].y);
            g[c][0].z = fmaf(wc[c], x.z, g[c][0].z);
            g[c][0].w = fmaf(wc[c], x.w, g[c][0].w);
            g[c][1].x = fmaf(wc[c], y.x, g[c][1].x);
            g[c][1].y = fmaf(wc[c], y.y, g[c][1].y);
            g[c][1].z = fmaf(wc[c], y.z, g[c][1].z);
            g[c][1].w = fmaf(wc[c], y.w, g[c][1].w);
        }
    };
    // the next four weights are on their way while four are used (the table
    // is four entries of a row longer than it is read)
    float4 w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __ldg(wt + i * kSpreadThreads);
    int k = 0;
    for (; k + 4 <= kw; k += 4) {
        float4 nx[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) nx[i] = __ldg(wt + (k + 4 + i) * kSpreadThreads);
#pragma unroll
        for (int i = 0; i < 4; ++i) step(k + i, w[i]);
#pragma unroll
        for (int i = 0; i < 4; ++i) w[i] = nx[i];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
        if (k + i < kw) step(k + i, w[i]);
#pragma unroll
    for (int r = 0; r < kTufrGroup; ++r) {
        if (r >= rc) break;
        float4* o = reinterpret_cast<float4*>(a.G + (long long)(j0 + r) * M + l);
        const int h = r >> 1;
        if (r & 1) {
            o[0] = make_float4(g[0][h].z, g[0][h].w, g[1][h].z, g[1][h].w);
            o[1] = make_float4(g[2][h].z, g[2][h].w, g[3][h].z, g[3][h].w);
        } else {
            o[0] = make_float4(g[0][h].x, g[0][h].y, g[1][h].x, g[1][h].y);
            o[1] = make_float4(g[2][h].x, g[2][h].y, g[3][h].x, g[3][h].y);
        }
    }
}

// Grid FFT of a range bin (bin p then holds Z[K0 + p] Phi(p / M) on the band),
// band mask and both deconvolutions, inverse grid FFT of the type-2
// evaluation, kNuTaps-tap interpolation at the output rows (weights fold the
// Lagrange stencil, the centring phase and 1/TS) and the re-ramp.
template <int NT, int MB>
__global__ void __launch_bounds__(NT, MB) k_tufr_grid(TufrArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (!a.P->ok) return;
    cf32* buf = reinterpret_cast<cf32*>(smem_raw);
    const int M = a.dnu.n;
    const cf32* G = a.G + (long long)blockIdx.x * M;
    fft4_head(buf, a.dnu, [&](int l) { return ldg(G + l); });
    fft4_mid(buf, a.dnu, [&](int m, cf32 v) { return v * __ldg(a.tab.band + m); });
    fft4_tail(buf, a.dnu, [&](int l, cf32 v) { buf[pad16(l)] = v; });
    __syncthreads();
    cf32* out = a.out + (long long)blockIdx.x * a.n_out;
    const cf32* ramp = a.ramp + (long long)blockIdx.x * a.n_out;
    for (int p = threadIdx.x; p < a.n_out; p += NT) {
        int l = __ldg(a.tab.nu_l0 + p) % M;
        if (l < 0) l += M;
        const cf32* w = a.tab.nu_w + p;   // tap t at w[t n_out]: lanes read consecutive words
        cf32 acc = mk(0.f, 0.f);
#pragma unroll
        for (int t = 0; t < kNuTaps; ++t) {
            acc = acc + buf[pad16(l)] * ldg(w + (long long)t * a.n_out);
            if (++l == M) l = 0;
        }
        out[p] = acc * ldg(ramp + p);
    }
}

// Exponential-of-semicircle kernel of width kNuW (support |t| < kNuW / 2, t in
// grid units) and its Fourier transform by Gauss-Legendre quadrature.
__device__ __forceinline__ double nu_kernel(double t, double beta) {
    const double z = 2.0 * t / kNuW;
    return fabs(z) < 1.0 ? exp(beta * (sqrt(1.0 - z * z) - 1.0)) : 0.0;
}

// Per-burst tables of the time unfolding (see TufrTables), one thread per entry.
// Band mask / Phi(p / M)^2 at the grid bins, a warp per bin: Phi by the
// Gauss-Legendre rule, whose nodes come in pairs +-x (two pairs per lane).
__global__ void __launch_bounds__(256) k_tufr_band(const TufrDev* __restrict__ P, int M, const int* __restrict__ mid,
                                                   TufrTables t) {
    if (!P->ok) return;
    const int p = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (p >= M) return;
    const int bw = P->q.end - P->q.start;
    const int K0 = bw / 2;
    if (!(p < bw - K0 || p >= M - K0)) {
        if (lane == 0) t.band[mid[p]] = 0.0f;
        return;
    }
    // oversampling M / bw >= 1.25 and the kernel's beta for it
    const double sigma = (double)M / (double)bw;
    const double beta = 0.97 * 3.141592653589793 * kNuW * (1.0 - 1.0 / (2.0 * sigma));
    const double xi = (double)(p < bw - K0 ? p : p - M) / (double)M;
    double acc = 0.0;
    for (int q = lane; q < kNuQuad / 2; q += 32) {
        const double tq = 0.5 * kNuW * t.gl_x[q];
        acc += 2.0 * t.gl_w[q] * nu_kernel(tq, beta) * cospi(2.0 * xi * tq);
    }
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
        const double inv_phi = 1.0 / (0.5 * kNuW * acc);
        t.band[mid[p]] = (float)(inv_phi * inv_phi);
    }
}

__global__ void k_tufr_tables(const TufrDev* __restrict__ P, int S, int n_out, int s0, int M, TufrTables t) {
    const TufrParams q = P->q;
    const int T = q.num_tiles;
    if (!P->ok) return;
    const long long TS = (long long)T * S;
    const double ft = q.focused_time;
    const int bw = q.end - q.start;
    const int K0 = bw / 2;
    // oversampling M / bw >= 1.25 and the kernel's beta for it
    const double sigma = (double)M / (double)bw;
    const double beta = 0.97 * 3.141592653589793 * kNuW * (1.0 - 1.0 / (2.0 * sigma));
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long tid = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    for (long long p = tid; p < n_out; p += stride) {
        const long long qo = s0 + p;
        // quadratic resampling TS -> down: stencil n = i-1, i, i+1 (signal_processing.cpp:109-155)
        const long long num = qo * (TS - 1);
        long long i = num / (q.down - 1);
        double xi = (double)(num - i * (q.down - 1)) / (double)(q.down - 1);
        if (i > TS - 2) {
            xi += (double)(i - (TS - 2));
            i = TS - 2;
        }
        const double L[3] = {0.5 * xi * (xi - 1.0), -(xi + 1.0) * (xi - 1.0), 0.5 * (xi + 1.0) * xi};
        // grid positions x = M n / TS of the three stencil points (n modulo TS)
        double xs[3], ph_c[3], ph_s[3];
        for (int k = 0; k < 3; ++k) {
            const long long n = (((i - 1 + k) % TS) + TS) % TS;
            xs[k] = (double)M * (double)n / (double)TS;
            sincospi(2.0 * (double)(((long long)K0 * n) % TS) / (double)TS, &ph_s[k], &ph_c[k]);
        }
        const long long l0 = (long long)ceil(xs[0] - 0.5 * kNuW);
        t.nu_l0[p] = (int)l0;
        for (int jt = 0; jt < kNuTaps; ++jt) {
            double wr = 0.0, wi = 0.0;
            for (int k = 0; k < 3; ++k) {
                // a stencil point at the top of the TS period wraps to the grid's start
                double d = xs[k] - (double)(l0 + jt);
                if (d > 0.5 * M) d -= M;
                if (d < -0.5 * M) d += M;
                const double f = L[k] * nu_kernel(d, beta) / (double)TS;
                wr += f * ph_c[k];
                wi += f * ph_s[k];
            }
            t.nu_w[(long long)jt * n_out + p] = mk((float)wr, (float)wi);
        }
        // re-ramp: az_times = linspace(n_ref - ft/2, n_ref + ft/2, down); K_a resampled S -> down
        const long long nr = qo * (S - 1);
        int ir = (int)(nr / (q.down - 1));
        float alr = (float)(nr - (long long)ir * (q.down - 1)) / (float)(q.down - 1);
        if (ir >= S - 1) {
            ir = S - 2;
            alr = 1.0f;
        }
        const df taur = df_from((q.n_ref - ft / 2) + qo * (((q.n_ref + ft / 2) - (q.n_ref - ft / 2)) / (double)(q.down - 1)));
        t.rer[p] = make_float4(__int_as_float(ir), alr, taur.hi, taur.lo);
    }
}


// Spreading weights in the order k_tufr_spread reads them: entry
// [chunk][k][thread] holds the weights of the thread's sample k for its four
// grid points (0 outside the kernel's support).
__global__ void k_tufr_weights(const TufrDev* __restrict__ P, int S, int M, float4* __restrict__ wt) {
    const TufrDev& dev = *P;
    if (!dev.ok) return;
    const long long TS = (long long)dev.q.num_tiles * S;
    const double sigma = (double)M / (double)(dev.q.end - dev.q.start);
    const double beta = 0.97 * 3.141592653589793 * kNuW * (1.0 - 1.0 / (2.0 * sigma));
    const int ng = dev.lc >> 2;
    const double zs = 2.0 / ((double)kNuW * (double)TS);
    const long long total = (long long)dev.chunks * dev.kw * kSpreadThreads;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const int t = (int)(e % kSpreadThreads);
        const int k = (int)(e / kSpreadThreads % dev.kw);
        const int chunk = (int)(e / kSpreadThreads / dev.kw);
        const long long l = (long long)chunk * dev.lc + 4 * (int)((unsigned int)(t * dev.perm) % (unsigned int)ng);
        const long long num0 = (2 * l - kNuW) * TS, den = 2LL * M;
        const long long lo = num0 >= 0 ? (num0 + den - 1) / den : -((-num0) / den);   // ceil
        float w[4];
        for (int c = 0; c < 4; ++c) {
            const double z = (double)((lo + k) * M - (l + c) * TS) * zs;
            w[c] = fabs(z) < 1.0 ? (float)exp(beta * (sqrt(1.0 - z * z) - 1.0)) : 0.0f;
        }
        wt[e] = make_float4(w[0], w[1], w[2], w[3]);
    }
}

// Samples a spreading CTA can hold (two float4 each) with three CTAs per SM;
// where a group of four grid points alone spans more (tile counts far above
// the band's, no burst of the IW geometry), what one CTA can.
static int spread_cap(int S, int tmax, int M) {
    const double ratio = (double)tmax * S / M;
    return (kNuW + 3) * ratio * 4 < 2392 ? 2392 : (kFft4SmemBytes - 1024) / 32;
}
// Upper bounds of the chunk count and of the weight table for any tile count
// up to tmax (the device picks the chunk length from its own).
static int spread_chunks(int S, int tmax, int M, int cap) {
    int most = 0;
    for (int T = 1; T <= tmax; ++T) {
        const TufrSplit sp = tufr_split((long long)T * S, M, cap);
        most = std::max(most, sp.lc >= 4 ? sp.chunks : 0);
    }
    return std::max(most, 1);
}
TufrLaunch tufr_launch(int S, int tmax, int M) {
    TufrLaunch L;
    L.ycap = spread_cap(S, tmax, M);
    L.chunks = spread_chunks(S, tmax, M, L.ycap);
    L.weights = 0;
    for (int T = 1; T <= tmax; ++T) {
        const TufrSplit sp = tufr_split((long long)T * S, M, L.ycap);
        if (sp.lc >= 4) L.weights = std::max<long long>(L.weights, (long long)sp.chunks * sp.kw * kSpreadThreads);
    }
    L.weights = std::max<long long>(L.weights, 1) + 8 * kSpreadThreads;   // read ahead
    return L;
}

void tufr_tables(const TufrArgs& a, cudaStream_t st) {
    note_launch(), k_tufr_band<<<(a.dnu.n + 7) / 8, 256, 0, st>>>(a.P, a.dnu.n, a.dnu.mid, a.tab);
    note_launch(), k_tufr_tables<<<(a.n_out + 63) / 64, 64, 0, st>>>(a.P, a.S, a.n_out, a.s0, a.dnu.n, a.tab);
    note_launch(), k_tufr_weights<<<152 * 8, 256, 0, st>>>(a.P, a.S, a.dnu.n, a.tab.wt);
}

void tufr_fused(const TufrArgs& a, const TufrLaunch& L, cudaStream_t st) {
    const dim3 gk((a.S - 1 + 31 * 8 - 1) / (31 * 8), a.n_r);
    note_launch(), k_tufr_knots<<<gk, 256, 0, st>>>(a);
    note_launch(), k_tufr_ramp<<<dim3((a.n_out + 255) / 256, a.n_r), 256, 0, st>>>(a);
    const size_t sm = sizeof(float4) * 2 * (size_t)L.ycap;
    allow_smem(k_tufr_spread);
    const long long blocks = (long long)((a.n_r + kTufrGroup - 1) / kTufrGroup) * L.chunks;
    note_launch(), k_tufr_spread<<<(unsigned)blocks, kSpreadThreads, sm, st>>>(a, L.chunks);
    const size_t smem = fft4_smem(a.dnu.n);
    fft4_launch(smem, [&](auto nt, auto mb) {
        auto kernel = k_tufr_grid<decltype(nt)::value, decltype(mb)::value>;
        allow_smem(kernel);
        note_launch(), kernel<<<a.n_r, decltype(nt)::value, smem, st>>>(a);
    });
}

// Scalars of azimuth_time_ufr (tile count, band, output crop), FP64, one block.
// K_a is evaluated analytically (the reference's az_fm_rate table).
// K_a of azimuth row i at range bin j (get_effective_velocities and the
// s1_decoder.cpp:667-676 expression), FP64.
__device__ __forceinline__ double ka_at(const RowParam* rows, const double* slant, const double* f_dc, int i, int j) {
    const double wl = 299792458.0 / 5.405000454334350e+9;
    const RowParam rp = rows[i];
    const double R = slant[j];
    const double num = rp.re * rp.re + rp.h * rp.h - R * R;
    const double beta = num / (2 * rp.re * rp.h);
    const double vg = rp.re * rp.v * beta / rp.h;
    const double v = sqrt(rp.v * vg);
    const double fa = rp.fa + f_dc[j];
    const double D = sqrt(1 - ((wl * wl) * (fa * fa)) / (4 * v * v));
    return (-2 * (v * v) * (D * D * D)) / (wl * R);
}

// K_a along the first range bin, all azimuth rows in parallel.
__global__ void k_ka_row0(const RowParam* rows, const double* slant, const double* f_dc, int S, double* ka0) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < S) ka0[i] = ka_at(rows, slant, f_dc, i, 0);
}

__global__ void k_tufr_params_fast(const RowParam* rows, const double* slant, const double* f_dc, int S, int n_r,
                                   double rate, double T, double prf, double bd, int swath_number,
                                   const double* ka0, int M, int ycap, int tmax, TufrDev* out) {
    __shared__ double part[256];
    // ordered blocked sum of K_a over the first range bin (contiguous runs per thread)
    const int per = (S + blockDim.x - 1) / blockDim.x;
    double acc = 0.0;
    for (int i = threadIdx.x * per; i < min(S, (int)(threadIdx.x + 1) * per); ++i) acc += ka0[i];
    part[threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.x != 0) return;
    double partial = 0.0;
    for (int k = 0; k < (int)blockDim.x; ++k) partial += part[k];
    auto ka_at_ = [&](int i, int j) { return ka_at(rows, slant, f_dc, i, j); };
    TufrDev d;
    TufrParams& q = d.q;
    const int num_az = S, num_rng = n_r;
    const double num_replicas = fabs(rate * T / prf);
    q.bandwidth = (num_replicas * prf) - bd;
    q.ka_mean = fabs(partial) / num_az;
    double ft = T + ((q.bandwidth - (2 * bd)) / q.ka_mean);
    double ka_ref;
    if (num_az / 2 < num_rng && num_rng / 2 < num_az) ka_ref = ka_at_(num_rng / 2, num_az / 2);
    else ka_ref = ka_at_(num_az / 2, num_rng / 2);
    q.n_ref = f_dc[num_rng / 2] / ka_ref;
    ft *= (swath_number != 11) ? 0.9 : 1.05;
    q.focused_time = ft;
    const int pos = (int)ceil((q.n_ref + ft / 2) / T);
    const int neg = (int)floor((q.n_ref - ft / 2) / T);
    q.num_tiles = pos - neg;
    const int ext = swath_number == 11 ? (int)floor(bd * 1.15) : (int)floor(bd * 0.26);
    q.output_shape = (int)floor(prf * T);
    q.down = q.output_shape + ext;
    q.shape = q.num_tiles * num_az;
    const int mid = q.shape / 2;
    q.start = (int)(mid - q.bandwidth / 2);
    q.end = (int)(mid + q.bandwidth / 2);
    q.ok = (q.num_tiles >= 1 && q.num_tiles <= 64 && q.start >= 0 && q.end <= q.shape && q.down >= 3) ? 1 : 0;
    // spreading split and the checks of the launch plan that need the tile count
    d.ok = 0;
    const long long TS = (long long)q.num_tiles * S;
    const int bw = q.end - q.start;
    if (q.ok && q.num_tiles <= tmax && S >= 8 && TS < (1LL << 24) && 5LL * bw <= 4LL * M) {
        const TufrSplit sp = tufr_split(TS, M, ycap);
        d.lc = sp.lc;
        d.kw = sp.kw;
        d.chunks = sp.chunks;
        d.perm = 1;
        // az_times = linspace(-ft/2, ft/2, TS): first time, step, sample
        // spacing; knot positions per sample and samples per knot
        const double f = q.focused_time;
        d.tau0 = df_from(-f / 2);
        d.dtau = df_from((f / 2 - (-f / 2)) / (double)(TS - 1));
        d.dt = df_from(f / (double)(TS - 1));
        d.gk = (float)((double)(S - 1) / (double)(TS - 1));
        d.rt = (float)((double)(TS - 1) / (double)(S - 1));
        // band shift k_s / TS (k_s the band centre bin) as a 64-bit fraction of a turn
        const unsigned long long kk = (unsigned long long)((((long long)q.start + bw / 2) % TS + TS) % TS);
        const unsigned long long hi = (kk << 32) / (unsigned long long)TS;
        const unsigned long long rem = (kk << 32) - hi * (unsigned long long)TS;
        d.ks64 = (hi << 32) | ((rem << 32) / (unsigned long long)TS);
        if (sp.lc >= 4) {
            d.ok = 1;
            // groups this far apart put the 16-byte loads of 8 lanes on
            // different bank quads, as far as their sample spacing allows
            const double step = 4.0 * (double)TS / (double)M;
            const int ng = sp.lc / 4;
            int best = 1 << 30;
            for (int D = 1; D < 16; ++D) {
                int x = D, y = ng;
                while (y) { const int r = x % y; x = y; y = r; }
                if (x != 1) continue;
                int cost = 0;
                for (int f = 0; f < 4; ++f) {
                    int hit[8] = {0, 0, 0, 0, 0, 0, 0, 0}, worst = 0;
                    for (int i = 0; i < 8; ++i) worst = max(worst, ++hit[(long long)(step * D * i + 0.25 * f) & 7]);
                    cost += worst;
                }
                if (cost < best) {
                    best = cost;
                    d.perm = D;
                }
            }
        }
    }
    *out = d;
}

void tufr_params_fast(const RowParam* rows, const double* slant, const double* f_dc, int S, int n_r, double rate,
                      double T, double prf, double bd, int swath_number, double* ka0, int M, int ycap, int tmax,
                      TufrDev* out, cudaStream_t st) {
    note_launch(), k_ka_row0<<<(S + 127) / 128, 128, 0, st>>>(rows, slant, f_dc, S, ka0);
    note_launch(), k_tufr_params_fast<<<1, 256, 0, st>>>(rows, slant, f_dc, S, n_r, rate, T, prf, bd, swath_number,
                                                        ka0, M, ycap, tmax, out);
}

}  // namespace s1g
