// Row pass of the azimuth chains, one azimuth row per CTA: range FFT, secondary
// range compression, range IFFT, scale, RCMC and azimuth filter
// (s1_decoder.cpp:616-677), and the sinc RCMC option.
#include "s1g_czt.cuh"
#include "s1g_sinc.cuh"

namespace s1g {

// ------------------------------------------------------------------ row pass


// SRC phase, image_formation.cpp:422-455: -pi f_r^2 / K_src with
// K_src = 2 v^2 f_c^3 D^2 / (c R F^2).
__device__ __forceinline__ float src_phase(const RowDf& r, df Q, float csrc, df fdc, float lam2_4) {
    const float F = r.fa.hi + fdc.hi + (r.fa.lo + fdc.lo);
    const float vq = r.P.hi * ((r.A.hi - Q.hi) + (r.A.lo - Q.lo));
    const float F2 = F * F;
    return -csrc * F2 / (vq - lam2_4 * F2);   // v^2 D^2 = v^2 - lambda^2 F^2 / 4
}

// Scale, RCMC and azimuth filter factor (s1_decoder.cpp:643-676).
__device__ __forceinline__ cf32 post_factor(const RowDf& r, const ColDf& c, df fdc, df lam2_4, int tops) {
    const df F = df_add_abs(r.fa, fdc);
    const df vq = df_mul(r.P, df_add_abs(r.A, df_neg(c.Q)));
    const df omd = df_one_minus_sqrt1m(df_div2(df_mul(lam2_4, df_mul(F, F)), vq));   // 1 - D
    const df th = df_add_abs(df_neg(df_mul(c.k4r, omd)), df_mul(c.tau2pi, F));
    float theta = df_wrap(th);
    if (tops) theta -= c.crcmc * __fdividef(omd.hi, 1.0f - omd.hi);
    return cexpf_fast(theta) * c.az0 * c.rscale;
}

// What the SRC phase takes of the range columns, in the order of the
// transform's factor table (the direct row pass reads it there).
__global__ void k_rowpass_src_table(const ColDf* __restrict__ cols, const df* __restrict__ fdc,
                                    const int* __restrict__ mid, int n_r, float4* __restrict__ src,
                                    float* __restrict__ src_lo) {
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= n_r) return;
    const int m = mid[f];
    src[m] = make_float4(cols[f].Q.hi, cols[f].Q.lo, cols[f].csrc, fdc[f].hi);
    src_lo[m] = fdc[f].lo;
}

void rowpass_src_table(const ColDf* cols, const df* fdc, const int* mid, int n_r, float4* src, float* src_lo,
                       cudaStream_t st) {
    note_launch(), k_rowpass_src_table<<<(n_r + 255) / 256, 256, 0, st>>>(cols, fdc, mid, n_r, src, src_lo);
}

template <int NT, int MB>
__global__ void __launch_bounds__(NT, MB) k_rowpass_fused(RowArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cf32* buf = reinterpret_cast<cf32*>(smem_raw);
    const int i = blockIdx.x;
    const RowDf rp = a.rows[i];
    cf32* row = a.data + (long long)i * a.n_r;
    const float l24 = a.lam2_4.hi;
    auto src = [&](int j) { return cexpf_fast(src_phase(rp, a.cols[j].Q, a.cols[j].csrc, a.fdc[j], l24)); };
    auto put = [&](int j, cf32 v) {
        row[j] = a.post ? v * post_factor(rp, a.cols[j], a.fdc[j], a.lam2_4, a.tops) : v;
    };
    if (a.smooth) {
        if (a.tops) {
            fft4_head(buf, a.d, [&](int j) { return row[j]; });
            fft4_mid(buf, a.d, [&](int m, cf32 v) {
                const float4 c = __ldg(a.src + m);
                return v * cexpf_fast(src_phase(rp, df_make(c.x, c.y), c.z, df_make(c.w, __ldg(a.src_lo + m)), l24));
            });
            fft4_tail<true>(buf, a.d, put);
        } else {
            // stripmap: the SRC phase is applied to the range-time samples;
            // the inverse transform is the forward one of the conjugates
            for (int j = threadIdx.x; j < a.n_r; j += blockDim.x) row[j] = row[j] * src(j);
            __syncthreads();
            fft4_head(buf, a.d, [&](int j) { return conj(row[j]); });
            fft4_spectrum(buf, a.d);
            for (int j = threadIdx.x; j < a.n_r; j += blockDim.x) put(j, conj(buf[pad16(__ldg(a.d.pos + j))]));
        }
    } else if (a.tops) {
        fft4_head(buf, a.cz.dm, [&](int q) { return czt_in(a.cz, -1, q, [&](int k) { return row[k]; }); });
        czt_mid(buf, a.cz);
        // range frequency k: SRC, then input k of the inverse transform
        fft4_join(buf, a.cz.dm, [&](int k, cf32 v) {
            if (k >= a.n_r) return mk(0.f, 0.f);
            return conj(czt_out(a.cz, -1, k, v) * src(k)) * ldg(a.cz.chirp + k);
        });
        czt_mid(buf, a.cz);
        fft4_tail<true>(buf, a.cz.dm, [&](int k, cf32 v) {
            if (k < a.n_r) put(k, czt_out(a.cz, +1, k, v));
        });
    } else {
        // stripmap: SRC on the range-time samples, inverse transform
        for (int j = threadIdx.x; j < a.n_r; j += blockDim.x) row[j] = row[j] * src(j);
        __syncthreads();
        czt_run<true>(buf, a.cz, +1, [&](int q) { return row[q]; }, put);
    }
}

void rowpass_fused(const RowArgs& a, cudaStream_t st) {
    const size_t smem = fft4_smem(a.smooth ? a.d.n : a.cz.dm.n);
    fft4_launch(smem, [&](auto nt, auto mb) {
        auto kernel = k_rowpass_fused<decltype(nt)::value, decltype(mb)::value>;
        allow_smem(kernel);
        note_launch(), kernel<<<a.S, decltype(nt)::value, smem, st>>>(a);
    });
}

// Sinc RCMC: a warp forms 32 consecutive range bins of one azimuth row.  The
// migration of bin j is rmig_j (1 - D) / D samples (D of post_factor, a few
// samples at the band edges), so the 32 positions advance about one sample
// per lane and their taps come from two samples per lane by warp shuffles.
__global__ void __launch_bounds__(256) k_rcmc_sinc(RcmcArgs a) {
    const int lane = threadIdx.x & 31;
    const int wpr = (a.n_r + 31) / 32;
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (gw >= (long long)a.S * wpr) return;   // whole warps leave together
    const int i = (int)(gw / wpr);
    const int j = (int)(gw % wpr) * 32 + lane;
    const bool act = j < a.n_r;
    const RowDf rp = a.rows[i];
    const int jj = act ? j : a.n_r - 1;
    const ColDf c = a.cols[jj];
    const df fdc = a.fdc[jj];
    const df F = df_add_abs(rp.fa, fdc);
    const df vq = df_mul(rp.P, df_add_abs(rp.A, df_neg(c.Q)));
    const df omd = df_one_minus_sqrt1m(df_div2(df_mul(a.lam2_4, df_mul(F, F)), vq));   // 1 - D
    const double t = (double)j + (double)(c.rmig * (omd.hi / (1.0f - omd.hi)));
    const cf32 v = sinc_warp<float>(a.in + (long long)i * a.n_r, a.n_r, t, a.L, act);
    if (act) a.out[(long long)i * a.n_r + j] = v * post_factor(rp, c, fdc, a.lam2_4, 0);
}

void rcmc_sinc(const RcmcArgs& a, cudaStream_t st) {
    const long long warps = (long long)a.S * ((a.n_r + 31) / 32);
    note_launch(), k_rcmc_sinc<<<(unsigned)((warps * 32 + 255) / 256), 256, 0, st>>>(a);
}

}  // namespace s1g
