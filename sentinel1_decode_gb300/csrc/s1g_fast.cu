// Fused FP32 kernels of the fast path.  Each stage of the reference's
// _range_compress / _azimuth_compress runs as one kernel that keeps its
// working line in shared memory:
//   k_rc_fused      range compression (pad, FFT, matched filter, IFFT, shift/crop)
//   k_fufr_fused    azimuth FFT + frequency unfolding,
//                   the two length-S DFTs done as band-limited chirp-z transforms
//   k_czt_rows      azimuth IFFT (length S, chirp-z) per range bin
// here, k_rowpass_fused (range FFT, SRC, range IFFT, scaling, RCMC, azimuth
// filter) in s1g_rowpass.cu and the k_tufr_* kernels (time unfolding, resampling
// and re-ramp) in s1g_tufr.cu.  The Doppler lag-1 sums come from s1g_dcest.cu.
// Phase arguments are formed in double-float (s1g_df.cuh); no FP64
// arithmetic runs per sample.
#include <algorithm>
#include <cmath>
#include <stdexcept>

#include "s1g_czt.cuh"

namespace s1g {

// Row-wise CZT: out[row][k] = scale * X_row[k] (used for the azimuth IFFT of
// the time unfolding, length S, dir +1).  Bound by instruction issue and
// shared-memory latency, as every kernel over the FFT core: 11838
// rows of 6702 points 2.56 ms with the previous core (8 more sweeps of shared
// memory), 1.13 now.
template <int NT, int MB>
__global__ void __launch_bounds__(NT, MB)
    k_czt_rows(const cf32* __restrict__ in, long long ip, cf32* __restrict__ out, long long op, CztDev c, int dir,
               float scale) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cf32* buf = reinterpret_cast<cf32*>(smem_raw);
    const cf32* x = in + (long long)blockIdx.x * ip;
    cf32* y = out + (long long)blockIdx.x * op;
    czt_run(buf, c, dir, [&](int q) { return x[q]; }, [&](int k, cf32 v) { y[k] = v * scale; });
}

void czt_rows(const cf32* in, long long ip, cf32* out, long long op, long long rows, const CztDev& c, int dir,
              float scale, cudaStream_t st) {
    const size_t smem = fft4_smem(c.dm.n);
    fft4_launch(smem, [&](auto nt, auto mb) {
        auto kernel = k_czt_rows<decltype(nt)::value, decltype(mb)::value>;
        allow_smem(kernel);
        note_launch(), kernel<<<(unsigned)rows, decltype(nt)::value, smem, st>>>(in, ip, out, op, c, dir, scale);
    });
}

__device__ __forceinline__ void cp_async4(int* shared, const int* global) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(shared)), "l"(global) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// ------------------------------------------------------------------ range compression
// ref: the matched filter's spectrum at d.mid.
template <int NT, int MB>
__global__ void __launch_bounds__(NT, MB)
    k_rc_fused(const cf32* __restrict__ raw, cf32* __restrict__ rc, int n_r, int h, Fft4Desc d,
               const cf32* __restrict__ ref, Failed failed) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cf32* buf = reinterpret_cast<cf32*>(smem_raw);
    const cf32* x = raw + (long long)blockIdx.x * n_r;
    cf32* y = rc + (long long)blockIdx.x * n_r;
    // the failure word travels to the buffer's last element, which holds no
    // point, while the line does (a branch on it here cost 1.4 of 69 us for 64
    // lines, a register held through the passes 4 of 532 us for 1481)
    int* word = reinterpret_cast<int*>(buf + padded16_len(d.n) - 1);
    if (threadIdx.x == 0) {
        if (failed.a) cp_async4(word, failed.a);
        else *word = 0;
    }
    fft4_head(buf, d, [&](int q) { return q < n_r ? x[q] : mk(0.f, 0.f); });
    if (threadIdx.x == 0) cp_async_wait();
    fft4_mid(buf, d, [&](int m, cf32 v) { return v * ldg(ref + m); });
    fft4_back(buf, d);
    const int bad = *word;
    fft4_last(buf, d, [&](int q, cf32 v) {
        int k = q + h;
        if (k >= d.n) k -= d.n;
        if (k < n_r && !bad) y[k] = v;
    });
}

void rc_fused(const cf32* raw, cf32* rc, int n_a, int n_r, int h, const Fft4Desc& d, const cf32* ref,
              cudaStream_t st, Failed failed) {
    const size_t smem = fft4_smem(d.n);
    fft4_launch(smem, [&](auto nt, auto mb) {
        auto kernel = k_rc_fused<decltype(nt)::value, decltype(mb)::value>;
        allow_smem(kernel);
        note_launch(), kernel<<<n_a, decltype(nt)::value, smem, st>>>(raw, rc, n_r, h, d, ref, failed);
    });
}

// ------------------------------------------------------------------ frequency unfolding
// Shared memory: the transforms' buffer and X, the azimuth spectrum (n_a,
// natural order).  At 80 registers (fft4_launch) the functors of the tiling and
// of the joined transforms leave 176 bytes of spill stores and 156 of loads per
// thread.  12000 bins of 1500 lines unfolded to 6908: 1.69 ms.
static int fufr_big(const FufrArgs& a) {
    return std::max(padded16_len(a.cf.dm.n), padded16_len(a.na_smooth ? a.dna.n : a.cna.dm.n));
}

template <int NT, int MB>
__global__ void __launch_bounds__(NT, MB) k_fufr_fused(FufrArgs a, int big_len) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cf32* big = reinterpret_cast<cf32*>(smem_raw);
    cf32* X = big + big_len;
    const int j = blockIdx.x;
    const int n_a = a.n_a;
    const cf32* row = a.rcT + (long long)j * n_a;
    // azimuth FFT (length n_a) into X
    if (a.na_smooth) {
        fft4_head(big, a.dna, [&](int q) { return row[q]; });
        fft4_spectrum(big, a.dna);
        for (int k = threadIdx.x; k < n_a; k += blockDim.x) X[k] = big[pad16(__ldg(a.dna.pos + k))];
    } else {
        czt_run(big, a.cna, -1, [&](int q) { return row[q]; }, [&](int k, cf32 v) { X[k] = v; });
    }
    __syncthreads();
    // tile (after the azimuth fftshift), deramp, band-limited forward DFT_S
    fft4_head(big, a.cf.dm, [&](int s) {
        return czt_in(a.cf, -1, s, [&](int q) {
            if (q >= a.tile_len) return mk(0.f, 0.f);
            int k = (q % n_a) - n_a / 2;
            if (k < 0) k += n_a;
            return X[k] * ldg(a.dfwd + q);
        });
    });
    czt_mid(big, a.cf);
    // the band moved to the front: input of the inverse DFT_S, of the same
    // convolution length
    fft4_join(big, a.cf.dm, [&](int k, cf32 v) {
        if (k >= a.bw) return mk(0.f, 0.f);
        return conj(czt_out(a.cf, -1, k, v)) * ldg(a.ci.chirp + k);
    });
    czt_mid(big, a.ci);
    // re-ramp, 1/S
    cf32* out = a.out + (long long)j * a.S;
    fft4_tail(big, a.ci.dm, [&](int k, cf32 v) {
        if (k < a.S) out[k] = czt_out(a.ci, +1, k, v) * ldg(a.reramp + k);
    });
}

void fufr_fused(const FufrArgs& a, cudaStream_t st) {
    const int big = fufr_big(a);
    const size_t smem = sizeof(cf32) * ((size_t)big + a.n_a);
    if (smem > (size_t)kFft4SmemBytes) throw std::runtime_error("frequency unfolding: shared memory");
    fft4_launch(smem, [&](auto nt, auto mb) {
        auto kernel = k_fufr_fused<decltype(nt)::value, decltype(mb)::value>;
        allow_smem(kernel);
        note_launch(), kernel<<<a.n_r, decltype(nt)::value, smem, st>>>(a, big);
    });
}

// ------------------------------------------------------------------ Doppler fit
// FP64 on one pipe-bound SM: what can be spread over threads or blocks is.
constexpr double kPIref = 3.14159265358979;
constexpr int kFitBlocks = 64;    // num_blocks at most

// Wrapped per-bin centroid -prf arg(sum) / (2 pi) (doppler.cpp:4-39), all bins in parallel.
__global__ void k_dc_wrapped(const cf64* __restrict__ part, int nchunk, int n, double prf, double* __restrict__ f_dc) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double sr = 0.0, si = 0.0;
    for (int c = 0; c < nchunk; ++c) {
        sr += part[(long long)c * n + j].x;
        si += part[(long long)c * n + j].y;
    }
    f_dc[j] = -prf * atan2(si, sr) / (2 * kPIref);
}

// Block means, unwrap (doppler.cpp:42-95) and the quadratic fit's three
// coefficients: a warp per block mean, a thread per bin of the dense DFT (its
// roots from a table: one SM does 1.9 FP64 operations a clock) and per block
// of the unwrap.  69 us (84 with the kernels before and after it), where 256
// threads with serial means and one thread for the unwrap took 288 (and the FP64
// pipeline's all-serial fit 19.8 ms).
__global__ void __launch_bounds__(1024) k_dc_fit(const double* __restrict__ f_dc, DcFitArgs a, double* __restrict__ poly) {
    __shared__ double fine[kFitBlocks], fval[kFitBlocks], un[kFitBlocks];
    __shared__ double mag2[8 * kFitBlocks], fre[8 * kFitBlocks], fim[8 * kFitBlocks];
    __shared__ double wre[8 * kFitBlocks], wim[8 * kFitBlocks];
    __shared__ double line[2];
    const int n = a.n_rng, nb = a.num_blocks, m = nb * 8;
    const int bs = n / nb;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int b = warp; b < nb; b += (int)(blockDim.x >> 5)) {
        const int s = b * bs;
        const int e = (s + bs < n) ? s + bs : n - 1;
        double acc = 0.0;
        for (int j = s + lane; j < e; j += 32) acc += f_dc[j];
        for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) {
            fine[b] = acc / ((double)e - (double)s);
            double sn, cs;
            sincos((2.0 * kPIref) * fine[b] / a.prf, &sn, &cs);
            fval[b] = floor(hypot(cs, sn));
        }
    }
    for (int k = threadIdx.x; k < m; k += blockDim.x) sincospi(-2.0 * (double)k / (double)m, &wim[k], &wre[k]);
    __syncthreads();
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
        double re = 0.0, im = 0.0;
        for (int j = 0; j < nb; ++j) {
            if (fval[j] == 0.0) continue;
            const int q = (int)((long long)j * k % m);
            re += fval[j] * wre[q];
            im += fval[j] * wim[q];
        }
        const double mg = hypot(re, im);
        mag2[k] = mg * mg;
        fre[k] = re;
        fim[k] = im;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int bi = 0;
        for (int k = 1; k < m; ++k)
            if (mag2[k] > mag2[bi]) bi = k;
        const float dt = (float)(a.rt[1] - a.rt[0]);
        const double val = 1.0 / (m * (double)dt);
        const int N = (m - 1) / 2 + 1;
        const double v = bi < N ? bi * val : (bi - m) * val;
        line[0] = v / (double)dt;
        line[1] = atan2(fim[bi], fre[bi]) / (2.0 * kPIref);
    }
    __syncthreads();
    if (threadIdx.x < nb) {
        const int j = threadIdx.x;
        const double aa = line[0], bb = line[1];
        double s1, c1, s2, c2;
        sincos((2.0 * kPIref) * fine[j] / a.prf, &s1, &c1);
        sincos(-1.0 * (aa * a.rt[j] + bb), &s2, &c2);
        const double pr = c1 * c2 - s1 * s2, pi_ = c1 * s2 + s1 * c2;
        un[j] = (aa * a.rt[j] + bb + atan2(pi_, pr) / (2.0 * kPIref)) * a.prf;
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    // polyfit, degree 2 (signal_processing.cpp:159-214)
    double Sx[5] = {0, 0, 0, 0, 0}, Sy[3] = {0, 0, 0};
    for (int i = 0; i < nb; ++i) {
        double xi = 1.0;
        for (int jj = 0; jj <= 4; ++jj) {
            if (jj <= 2) Sy[jj] += xi * un[i];
            Sx[jj] += xi;
            xi *= a.rt[i];
        }
    }
    double A[3][3] = {{Sx[0], Sx[1], Sx[2]}, {Sx[1], Sx[2], Sx[3]}, {Sx[2], Sx[3], Sx[4]}};
    double B[3] = {Sy[0], Sy[1], Sy[2]};
    for (int i = 0; i < 3; ++i) {
        for (int k = i + 1; k < 3; ++k)
            if (fabs(A[k][i]) > fabs(A[i][i])) {
                for (int jj = 0; jj < 3; ++jj) {
                    const double t = A[i][jj];
                    A[i][jj] = A[k][jj];
                    A[k][jj] = t;
                }
                const double t = B[i];
                B[i] = B[k];
                B[k] = t;
            }
        for (int k = i + 1; k < 3; ++k) {
            const double f = A[k][i] / A[i][i];
            for (int jj = i; jj < 3; ++jj) A[k][jj] -= f * A[i][jj];
            B[k] -= f * B[i];
        }
    }
    double c[3];
    for (int i = 2; i >= 0; --i) {
        c[i] = B[i];
        for (int jj = i + 1; jj < 3; ++jj) c[i] -= A[i][jj] * c[jj];
        c[i] /= A[i][i];
    }
    poly[0] = c[0];
    poly[1] = c[1];
    poly[2] = c[2];
}

// The fitted centroid of every range bin (f_dc_df may be null).
__global__ void k_dc_eval(const double* __restrict__ poly, DcFitArgs a, double* __restrict__ f_dc, df* __restrict__ f_dc_df) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= a.n_rng) return;
    const double step = (a.far - a.near) / (a.n_rng - 1);
    const double t = (a.near + j * step) - a.near;
    const double v = (poly[0] + poly[1] * t + poly[2] * t * t);
    f_dc[j] = v;
    if (f_dc_df) f_dc_df[j] = df_from(v);
}

void dc_fit(const cf64* part, int nchunk, const DcFitArgs& a, double* poly, double* f_dc, df* f_dc_df, cudaStream_t st) {
    if (a.num_blocks > kFitBlocks) throw std::runtime_error("Doppler fit: too many blocks");
    const int grid = (a.n_rng + 127) / 128;
    note_launch(), k_dc_wrapped<<<grid, 128, 0, st>>>(part, nchunk, a.n_rng, a.prf, f_dc);
    note_launch(), k_dc_fit<<<1, 1024, 0, st>>>(f_dc, a, poly);
    note_launch(), k_dc_eval<<<grid, 128, 0, st>>>(poly, a, f_dc, f_dc_df);
}

}  // namespace s1g
