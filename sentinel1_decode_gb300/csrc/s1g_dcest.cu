// Doppler-centroid estimator input of the FP32 path: the lag-1 azimuth sums
// of doppler.cpp:4-39,98-143 formed from a compensated (double-float
// accurate) range compression.
//
// The TOPS time unfolding turns the centroid into a deramp time -f_dc/K_a,
// and the burst SLC moves by ~7e-5 (relative L2) per 1e-5 Hz of centroid
// change.  Range-compressed lines carrying FP32 rounding noise (~2e-7) shift
// the centroid by up to ~1e-5 Hz on low-coherence scenes, so the sums are
// formed from a second range compression in compensated arithmetic
// (s1g_cfft.cuh) whose result is accurate to ~1e-13, as the reference's
// FP64 range compression is.
//
// The correlation out[k] = (1/E) sum_t x~[k - h + t] conj(c[t]) (x~ the
// zero-padded line indexed modulo M, s1_decoder.cpp:459-509 with the shift h
// of the fused FP32 kernel) is evaluated by overlap-save with blocks of B
// points: block b produces the U = B - L + 1 outputs [b U, b U + U).
#include <algorithm>
#include <cmath>
#include <memory>
#include <stdexcept>
#include <vector>

#include "s1g_dcest.h"
#include "s1g_fft_engine.h"

namespace s1g {

// One block of one line.  Passes of radix 4 to 16 in registers (16 values of
// four floats are 64 registers): the first reads the line, the last of the
// forward transform multiplies by the filter and starts the inverse one, the
// last writes the result, so a block of 8192 crosses shared memory six times.
// Decimation in frequency forward, its mirror image back.  FP32 arithmetic
// bounds it (26 operations per value and radix-2 level, 32 per twiddle; the
// 140 KB of a block leave 16 warps per SM).  1500 lines of 12000 samples:
// 0.99 ms; 1.67 with a trip through shared memory per radix-4 stage, twiddles
// strided through one table and separate loads, filter and output loops.
template <int P>
__device__ __forceinline__ void dc_twiddles(cc* a, const float4* tw, int Ns, int k, bool inverse) {
#pragma unroll
    for (int s = 1; s < P; ++s) {
        const float4 w = __ldg(tw + (s - 1) * Ns + k);
        a[s] = inverse ? cc_mul(a[s], w.x, -w.y, w.z, -w.w) : cc_mul(a[s], w.x, w.y, w.z, w.w);
    }
}
__device__ __forceinline__ cc dc_get(const float4* S, int sh, int i) {
    const float4 v = S[i + (i >> sh)];
    return cc{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ void dc_put(float4* S, int sh, int i, const cc& v) {
    S[i + (i >> sh)] = make_float4(v.hx, v.hy, v.ex, v.ey);
}
template <int P>
__device__ __forceinline__ void dc_first(const DcEstArgs& a, float4* S, const cf32* x, int i0) {
    const int Ns = a.d.n / P, sh = a.d.sh;
    for (int k = threadIdx.x; k < Ns; k += blockDim.x) {
        cc v[P];
#pragma unroll
        for (int r = 0; r < P; ++r) {
            int i = i0 + k + r * Ns;
            while (i >= a.M) i -= a.M;
            v[r] = cc_make(i < a.n_r ? ldg(x + i) : mk(0.f, 0.f), mk(0.f, 0.f));
        }
        cc_fft<P, -1>(v);
        dc_twiddles<P>(v, a.d.tw[0], Ns, k, false);
#pragma unroll
        for (int s = 0; s < P; ++s) dc_put(S, sh, k + s * Ns, v[s]);
    }
}
template <int P, int DIR>
__device__ __forceinline__ void dc_mid(const DcEstArgs& a, float4* S, const float4* tw, int Ns) {
    const int nb = a.d.n / P, sh = a.d.sh;
    const float inv = 1.0f / (float)Ns;
    for (int t = threadIdx.x; t < nb; t += blockDim.x) {
        int g, k;
        split_idx(t, Ns, inv, g, k);
        const int base = g * (Ns * P) + k;
        cc v[P];
#pragma unroll
        for (int r = 0; r < P; ++r) v[r] = dc_get(S, sh, base + r * Ns);
        if (DIR > 0) dc_twiddles<P>(v, tw, Ns, k, true);
        cc_fft<P, DIR>(v);
        if (DIR < 0) dc_twiddles<P>(v, tw, Ns, k, false);
#pragma unroll
        for (int s = 0; s < P; ++s) dc_put(S, sh, base + s * Ns, v[s]);
    }
}
template <int P>
__device__ __forceinline__ void dc_join(const DcEstArgs& a, float4* S) {
    const int nb = a.d.n / P, sh = a.d.sh;
    for (int t = threadIdx.x; t < nb; t += blockDim.x) {
        cc v[P];
#pragma unroll
        for (int r = 0; r < P; ++r) v[r] = dc_get(S, sh, t * P + r);
        cc_fft<P, -1>(v);
#pragma unroll
        for (int s = 0; s < P; ++s) {
            const float4 w = __ldg(a.H + s * nb + t);
            v[s] = cc_mul(v[s], w.x, w.y, w.z, w.w);
        }
        cc_fft<P, 1>(v);
#pragma unroll
        for (int r = 0; r < P; ++r) dc_put(S, sh, t * P + r, v[r]);
    }
}
template <int P>
__device__ __forceinline__ void dc_last(const DcEstArgs& a, const float4* S, float4* y, int count) {
    const int Ns = a.d.n / P, sh = a.d.sh;
    for (int k = threadIdx.x; k < Ns; k += blockDim.x) {
        cc v[P];
#pragma unroll
        for (int s = 0; s < P; ++s) v[s] = dc_get(S, sh, k + s * Ns);
        dc_twiddles<P>(v, a.d.tw[0], Ns, k, true);
        cc_fft<P, 1>(v);
#pragma unroll
        for (int r = 0; r < P; ++r) {
            const int u = k + r * Ns;
            if (u < count) {
                const df re = two_sum(v[r].hx, v[r].ex), im = two_sum(v[r].hy, v[r].ey);
                y[u] = make_float4(re.hi, im.hi, re.lo, im.lo);
            }
        }
    }
}
#define DC_RADIX(r, CALL)                  \
    switch (r) {                           \
        case 4: { constexpr int P = 4; CALL; break; }   \
        case 6: { constexpr int P = 6; CALL; break; }   \
        case 8: { constexpr int P = 8; CALL; break; }   \
        case 12: { constexpr int P = 12; CALL; break; } \
        default: { constexpr int P = 16; CALL; break; } \
    }

__global__ void __launch_bounds__(512) k_rc_dc(const __grid_constant__ DcEstArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float4* S = reinterpret_cast<float4*>(smem_raw);
    const int line = blockIdx.x / a.nb;
    const int k0 = (blockIdx.x - line * a.nb) * a.U;
    const cf32* x = a.raw + (long long)line * a.n_r;
    int i0 = (k0 - a.h) % a.M;
    if (i0 < 0) i0 += a.M;
    const int np = a.d.np;
    DC_RADIX(a.d.radix[0], dc_first<P>(a, S, x, i0));
    __syncthreads();
    int Ns = a.d.n / a.d.radix[0];
    for (int p = 1; p < np - 1; ++p) {
        Ns /= a.d.radix[p];
        const float4* tw = p == 1 ? a.d.tw[1] : a.d.tw[2];
        DC_RADIX(a.d.radix[p], (dc_mid<P, -1>(a, S, tw, Ns)));
        __syncthreads();
    }
    if (a.d.radix[np - 1] == 4) dc_join<4>(a, S);
    else if (a.d.radix[np - 1] == 8) dc_join<8>(a, S);
    else dc_join<16>(a, S);
    __syncthreads();
    for (int p = np - 2; p > 0; --p) {
        const float4* tw = p == 1 ? a.d.tw[1] : a.d.tw[2];
        DC_RADIX(a.d.radix[p], (dc_mid<P, 1>(a, S, tw, Ns)));
        __syncthreads();
        Ns *= a.d.radix[p];
    }
    float4* y = a.rcd + (long long)line * a.n_r + k0;
    const int count = min(a.U, a.n_r - k0);
    DC_RADIX(a.d.radix[0], dc_last<P>(a, S, y, count));
}

__device__ __forceinline__ void ld_pair(const float4& v, df& re, df& im) {
    re = df_make(v.x, v.z);
    im = df_make(v.y, v.w);
}

// part[c][j] = sum over the pairs t of chunk c of rc[t][j] conj(rc[t+1][j]) g[t]
__global__ void __launch_bounds__(128) k_dc_lag1(DcEstArgs a) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= a.n_r) return;
    const int pairs = a.n_a - 1;
    const int per = (pairs + a.nchunk - 1) / a.nchunk;
    const int t0 = blockIdx.y * per;
    const int t1 = min(t0 + per, pairs);
    df sr = df_make(0.f, 0.f), si = df_make(0.f, 0.f);
    if (t0 < t1) {
        df xr, xi;
        ld_pair(a.rcd[(long long)t0 * a.n_r + j], xr, xi);
        for (int t = t0; t < t1; ++t) {
            df yr, yi;
            ld_pair(a.rcd[(long long)(t + 1) * a.n_r + j], yr, yi);
            const df pr = df_add(df_mul(xr, yr), df_mul(xi, yi));
            const df pi_ = df_sub(df_mul(xi, yr), df_mul(xr, yi));
            const float4 g = __ldg(a.g + t);
            const df gr = df_make(g.x, g.z), gi = df_make(g.y, g.w);
            sr = df_add(sr, df_sub(df_mul(pr, gr), df_mul(pi_, gi)));
            si = df_add(si, df_add(df_mul(pr, gi), df_mul(pi_, gr)));
            xr = yr;
            xi = yi;
        }
    }
    a.part[(long long)blockIdx.y * a.n_r + j] = mk(df_to_double(sr), df_to_double(si));
}

static size_t dc_smem(int n, int sh) { return sizeof(float4) * (size_t)(n + (n >> sh)); }

void dc_lag1_sums(const DcEstArgs& a, cudaStream_t st) {
    allow_dynamic_smem<k_rc_dc>(kSmemBytes);
    const size_t smem = dc_smem(a.d.n, a.d.sh);
    if (smem > (size_t)kSmemBytes) throw std::runtime_error("Doppler estimator: shared memory");
    const long long blocks = (long long)a.n_a * a.nb;
    if (blocks > 0x7fffffffLL) throw std::runtime_error("Doppler estimator: grid");
    note_launch(), k_rc_dc<<<(unsigned)blocks, a.d.nt, smem, st>>>(a);
    dim3 grid((a.n_r + 127) / 128, a.nchunk);
    note_launch(), k_dc_lag1<<<grid, 128, 0, st>>>(a);
}

// ------------------------------------------------------------------ host tables
CfftPlan::~CfftPlan() {
    for (void* p : owned) cudaFree(p);
}

std::shared_ptr<CfftPlan> make_cfft_plan(int n) {
    auto p = std::make_shared<CfftPlan>();
    p->d.n = n;
    std::vector<float4> tw(n);
    for (int i = 0; i < n; ++i) {
        const double ang = 2.0 * M_PI * ((double)i / (double)n);
        const df c = df_from(std::cos(ang)), s = df_from(-std::sin(ang));
        tw[i] = make_float4(c.hi, s.hi, c.lo, s.lo);
    }
    void* dt = nullptr;
    check_cuda(cudaMalloc(&dt, sizeof(float4) * n), "cfft tw");
    p->owned.push_back(dt);
    upload_table(dt, tw.data(), sizeof(float4) * n, "cfft tw up");
    p->d.tw = (const float4*)dt;
    return p;
}

// Passes of a block of n points, empty if there are none: the cheapest
// sequence of two to four radices with a power of two last, where a pass costs
// its arithmetic and a trip through shared memory, and threads without a
// butterfly in its last round count as busy.
static DcFft dc_passes(int n) {
    DcFft best;
    double bc = 0;
    std::vector<int> cur;
    auto take = [&] {
        const int last = cur.back();
        const int sh = last == 4 ? 2 : last == 8 ? 3 : 4;
        const size_t smem = dc_smem(n, sh);
        if (cur.size() < 2 || last == 6 || last == 12 || smem > (size_t)kSmemBytes) return;
        const int ctas = std::max(1, std::min(4, (int)((size_t)kFft4SmemBytes / (smem + 1024))));
        for (int nt = 128; nt * ctas <= 512; nt += 64) {
            double c = 0;
            for (size_t p = 0; p < cur.size(); ++p) {
                const int bf = n / cur[p];
                const double busy = (double)((bf + nt - 1) / nt) * nt / bf;
                c += (p + 1 < cur.size() ? 2 : 1.4) * busy * (std::log2((double)cur[p]) + 1.5);
            }
            c *= 1 + 0.1 * (512 - nt * ctas) / 512.0;   // fewer warps to hide latency
            if (best.n == 0 || c < bc) {
                bc = c;
                best.n = n;
                best.np = (int)cur.size();
                best.nt = nt;
                best.sh = sh;
                for (size_t p = 0; p < cur.size(); ++p) best.radix[p] = cur[p];
            }
        }
    };
    auto walk = [&](auto&& self, int m) -> void {
        if (m == 1) take();
        else if (cur.size() < 4)
            for (int r : {16, 12, 8, 6, 4})
                if (m % r == 0) {
                    cur.push_back(r);
                    self(self, m / r);
                    cur.pop_back();
                }
    };
    walk(walk, n);
    return best;
}

DcFftPlan::~DcFftPlan() {
    for (void* p : owned) cudaFree(p);
}

std::shared_ptr<DcFftPlan> make_dc_plan(int n) {
    auto plan = std::make_shared<DcFftPlan>();
    DcFft& d = plan->d;
    d = dc_passes(n);
    if (d.n != n) throw std::runtime_error("Doppler estimator: block length");
    int span = n;
    Uploads uploads;
    for (int p = 0; p + 1 < d.np; ++p) {
        const int P = d.radix[p], Ns = span / P;
        std::vector<float4> tw((size_t)(P - 1) * Ns);
        for (int s = 1; s < P; ++s)
            for (int k = 0; k < Ns; ++k) {
                const double ang = 2.0 * M_PI * ((double)((long long)s * k % span) / (double)span);
                const df c = df_from(std::cos(ang)), sn = df_from(-std::sin(ang));
                tw[(size_t)(s - 1) * Ns + k] = make_float4(c.hi, sn.hi, c.lo, sn.lo);
            }
        void* v = nullptr;
        check_cuda(cudaMalloc(&v, sizeof(float4) * tw.size()), "dc twiddles");
        plan->owned.push_back(v);
        uploads.table(v, tw.data(), sizeof(float4) * tw.size(), "dc twiddles up");
        d.tw[p] = (const float4*)v;
        span = Ns;
    }
    // position t P + s of the last pass holds frequency f = s_0 + r_0 s_1 + ...
    const int P = d.radix[d.np - 1], nb = n / P;
    plan->at.resize(n);
    for (int f = 0; f < n; ++f) {
        int m = f, rest = n, pos = 0;
        for (int p = 0; p < d.np; ++p) {
            rest /= d.radix[p];
            pos += (m % d.radix[p]) * rest;
            m /= d.radix[p];
        }
        plan->at[f] = (pos % P) * nb + pos / P;
    }
    return plan;
}

bool choose_dc_block(int n_r, int L, int& B, int& U, int& nb) {
    double best = 0;
    B = 0;
    for (int p3 = 1; p3 <= 27; p3 *= 3) {
        for (long long b = p3; b <= 1 << 16; b *= 2) {
            if (b < 64 || b < L + 32) continue;
            if (b > 1 << 14 || dc_passes((int)b).n == 0) continue;
            const int u = (int)b - L + 1;
            const int nbl = (n_r + u - 1) / u;
            const double cost = (double)nbl * (double)b * (std::log2((double)b) + 2.0);
            if (B == 0 || cost < best * 0.999 || (cost < best * 1.001 && b < B)) {
                best = cost;
                B = (int)b;
                U = u;
                nb = nbl;
            }
        }
    }
    return B != 0;
}

}  // namespace s1g
