// Batched row-FFT engine: plans, kernels and launchers (see s1g_fft_engine.h).
#include "s1g_fft_engine.h"
#include "s1g_tma.h"

#include <algorithm>
#include <iterator>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <stdexcept>
#include <string>

namespace s1g {

void check_cuda(cudaError_t e, const char* what) {
    if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

int device_sms() {
    static std::atomic<int> known[64];
    int dev = 0, n = 0;
    check_cuda(cudaGetDevice(&dev), "device");
    if (dev < 64) n = known[dev].load(std::memory_order_relaxed);
    if (n == 0) {
        check_cuda(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev), "device");
        if (dev < 64) known[dev].store(n, std::memory_order_relaxed);
    }
    return n;
}

static std::atomic<long long> g_launches{0};
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
long long launch_count() { return g_launches.load(); }
void note_launches(long long n) { g_launches.fetch_add(n, std::memory_order_relaxed); }

bool is_smooth7(long long n) {
    if (n < 1) return false;
    for (int p : {2, 3, 5, 7})
        while (n % p == 0) n /= p;
    return n == 1;
}

long long next_smooth7(long long n) {
    if (n < 1) n = 1;
    while (!is_smooth7(n)) ++n;
    return n;
}

// Modelled instructions per point of a pass of the fused kernels' core.
static double pass_cost(int r) {
    switch (r) {
        case 2: return 9;
        case 3: return 11;
        case 4: return 11;
        case 5: return 14;
        case 6: return 15;
        case 7: return 19;
        case 8: return 13.5;
        case 9: return 18;
        case 10: return 18;
        case 12: return 17;
        case 15: return 24;
        default: return 16;
    }
}

static const int kRadices[] = {16, 15, 12, 10, 9, 8, 7, 6, 5, 4, 3, 2};

// factorisations of n into the radices (largest first), at most `left` of them
static void factorisations(long long n, size_t first, int left, std::vector<int>& cur,
                           std::vector<std::vector<int>>& out) {
    if (n == 1) {
        out.push_back(cur);
        return;
    }
    if (left == 0) return;
    for (size_t i = first; i < sizeof(kRadices) / sizeof(int); ++i)
        if (n % kRadices[i] == 0) {
            cur.push_back(kRadices[i]);
            factorisations(n / kRadices[i], i, left - 1, cur, out);
            cur.pop_back();
        }
}

static double order_cost(const std::vector<int>& r) {
    double c = 0;
    for (int x : r) c += pass_cost(x);
    // the last inverse pass reads 32 bytes of twiddles per butterfly
    return c + 8.0 / r.front();
}

std::vector<std::vector<int>> fft4_orders(long long n, size_t most) {
    std::vector<std::pair<double, std::vector<int>>> c;
    std::vector<std::vector<int>> f;
    std::vector<int> cur;
    if (n < 2 || !is_smooth7(n)) return {};
    if (n % 16 == 0) {
        // affine: radix 16 last, a radix of the functor passes first
        factorisations(n / 16, 0, kFft4Passes - 1, cur, f);
        for (auto v : f) {
            if (v.empty()) continue;
            std::sort(v.begin(), v.end());
            do {
                if (!fft4_end_radix(v[0])) continue;
                std::vector<int> o = v;
                o.push_back(16);
                c.push_back({order_cost(o), o});
            } while (std::next_permutation(v.begin(), v.end()));
        }
    }
    if (c.empty()) {
        f.clear();
        factorisations(n, 0, kFft4Passes, cur, f);
        for (auto& v : f) c.push_back({order_cost(v), v});
    }
    std::stable_sort(c.begin(), c.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
    std::vector<std::vector<int>> out;
    for (size_t i = 0; i < c.size() && out.size() < most; ++i) out.push_back(c[i].second);
    return out;
}

std::vector<int> fft4_order64(long long n) {
    // FP64 instructions per point of a pass with its twiddles
    static const std::pair<int, double> cost[] = {{8, 9.4}, {7, 20}, {6, 13.5}, {5, 11}, {4, 6.3}, {3, 7.5}, {2, 3.2}};
    std::vector<std::vector<int>> f;
    std::vector<int> cur;
    if (n < 2 || !is_smooth7(n)) return {};
    factorisations(n, 5, kFft4Passes, cur, f);   // radices from 8 down
    std::vector<int> best;
    double bc = 1e30;
    for (const auto& v : f) {
        double c = 0.3 * v.size();
        for (int r : v)
            for (const auto& k : cost)
                if (k.first == r) c += k.second;
        if (c < bc) {
            bc = c;
            best = v;
        }
    }
    return best;
}

std::vector<long long> fft4_lengths(long long minlen, size_t most) {
    std::vector<std::pair<double, long long>> c;
    const long long hi = std::max(64LL, (long long)(minlen * 1.25) + 16);
    // past hi where there is none below it (the first is 96)
    for (long long m = std::max(64LL, (minlen + 15) / 16 * 16); m <= hi || c.empty(); m += 16) {
        if ((long long)sizeof(cf32) * padded16_len((int)m) > kFft4SmemBytes) break;
        const auto o = fft4_orders(m, 1);
        if (o.empty() || o[0].back() != 16 || !fft4_end_radix(o[0][0])) continue;
        c.push_back({(double)m * (order_cost(o[0]) + 12.0), m});
    }
    std::stable_sort(c.begin(), c.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
    std::vector<long long> out;
    for (size_t i = 0; i < c.size() && out.size() < most; ++i) out.push_back(c[i].second);
    return out;
}

long long fast_len(long long minlen) {
    const auto c = fft4_lengths(minlen, 1);
    return c.empty() ? -1 : c[0];
}

DeviceArena::~DeviceArena() {
    if (ptr) cudaFree(ptr);
}

void* DeviceArena::get(size_t bytes) {
    if (bytes > size) {
        if (ptr) {
            cudaDeviceSynchronize();
            cudaFree(ptr);
            if (moves) ++*moves;
        }
        ptr = nullptr;
        size = 0;
        check_cuda(cudaMalloc(&ptr, bytes), "scratch cudaMalloc");
        size = bytes;
    }
    return ptr;
}

// ------------------------------------------------------------------ kernels
// Launch shape of the row kernels.  FP64 is bound by its pipe (1.9 FMAs per
// clock and SM): 512 threads per SM keep it busy and leave radix 8 its
// registers (256 where one CTA fits: 6.09 ms for 3002 rows of 10k points, 5.86
// with 512).
template <typename R, class F>
static void rows4_launch(size_t smem, F f) {
    using std::integral_constant;
    if constexpr (sizeof(R) == 4) {
        fft4_launch(smem, f);
    } else {
        if (2 * (smem + 1024) <= 228 * 1024) f(integral_constant<int, 256>(), integral_constant<int, 2>());
        else f(integral_constant<int, 512>(), integral_constant<int, 1>());
    }
}

// Where the rows of a launch lie.  Split rows: row r takes every a-th element
// of line r / a from element r % a on, and its output k is multiplied by
// exp(dir 2 pi i (r % a) k / n) (tw, n entries).
template <typename R>
struct RowsIo {
    const cpx<R>* in;
    long long ip;
    cpx<R>* out;
    long long op;
    int a;               // 1: plain rows
    const cpx<R>* tw;
    int dir;
    int n, roll;         // points of a row, where output 0 goes
    R scale;
    int valid, count;    // inputs given (zeros follow), outputs wanted (of the rolled row)
    const cpx<R>* mul;   // factor of output k (before the roll), or null
};
template <typename R>
__device__ __forceinline__ void rows_put(const RowsIo<R>& io, cpx<R>* y, int k, int off, cpx<R> v) {
    if (io.dir > 0) v = conj(v);
    if (io.a > 1) {
        cpx<R> w = ldg(io.tw + (long long)off * k);
        if (io.dir > 0) w = conj(w);
        v = cmul4(v, w);
    }
    v = v * io.scale;
    if (io.mul) v = v * ldg(io.mul + k);
    k += io.roll;
    if (k >= io.n) k -= io.n;
    if (k < io.count) y[k] = v;
}

// Rows of a 7-smooth length: out[k] = sum_j in[j] exp(dir 2 pi i j k / n).
// The core transforms forward; dir = +1 conjugates both ends.
template <typename R, int NT, int MB>
__global__ void __launch_bounds__(NT, MB) k_rows_smooth(RowsIo<R> io, Fft4DescT<R> d) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cpx<R>* buf = reinterpret_cast<cpx<R>*>(smem_raw);
    const long long line = blockIdx.x / io.a;
    const int off = (int)(blockIdx.x - line * io.a);
    const cpx<R>* x = io.in + line * io.ip + off;
    cpx<R>* y = io.out + (long long)blockIdx.x * io.op;
    fft4_head(buf, d, [&](int j) {
        if (j >= io.valid) return mk((R)0, (R)0);
        const cpx<R> v = x[(long long)j * io.a];
        return io.dir > 0 ? conj(v) : v;
    });
    fft4_spectrum(buf, d);
    for (int k = threadIdx.x; k < d.n; k += NT) rows_put(io, y, k, off, buf[pad16(__ldg(d.pos + k))]);
}

// Rows of any length n by Bluestein's identity over a convolution of d.n.  In
// FP32 80 registers leave 44 bytes of spill stores per thread.
template <typename R, int NT, int MB>
__global__ void __launch_bounds__(NT, MB) k_rows_blue(RowsIo<R> io, Fft4DescT<R> d, int n,
                                                      const cpx<R>* __restrict__ chirp,
                                                      const cpx<R>* __restrict__ kern) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cpx<R>* buf = reinterpret_cast<cpx<R>*>(smem_raw);
    const long long line = blockIdx.x / io.a;
    const int off = (int)(blockIdx.x - line * io.a);
    const cpx<R>* x = io.in + line * io.ip + off;
    cpx<R>* y = io.out + (long long)blockIdx.x * io.op;
    fft4_head(buf, d, [&](int j) {
        if (j >= io.valid) return mk((R)0, (R)0);
        const cpx<R> v = x[(long long)j * io.a];
        return cmul4(io.dir > 0 ? conj(v) : v, ldg(chirp + j));
    });
    fft4_mid(buf, d, [&](int m, cpx<R> v) { return cmul4(v, ldg(kern + m)); });
    fft4_tail(buf, d, [&](int k, cpx<R> v) {
        if (k < n) rows_put(io, y, k, off, cmul4(v, ldg(chirp + k)));
    });
}

// Band transforms (FftEngine::to_band, from_band), FP64, a CTA for several rows.
// n (k0 + k) = n k0 + (n^2 + k^2 - (k - n)^2) / 2 makes them convolutions with
// a chirp.  The side with all P points goes through shared memory in nb runs
// of L points, each against its own shift of the chirp; the other side is one
// run, so the products of all runs add up as spectra (in W, a few hundred KB
// per CTA that stay in L2) before one inverse transform, or are formed from
// one spectrum.  FP64 arithmetic bounds it (1.9 FMAs per clock and SM), so
// what counts is the sum of the transform lengths: nb + 1 of L + width - 1
// points against 2 of 2 P - 1, or 12 of 2 (P / 6) - 1 where those split.  3002
// rows of 4987 points, a band of 600: 2.5 ms forward and 2.4 back, whole
// transforms 6.1 each way; of 29922 = 6 x 4987 points: 28.9 and 28.3, 36.1
// split.
struct BandArgs {
    const cf64* in;
    long long ip;
    cf64* out;
    long long op;
    long long rows;
    Fft4DescT<double> d;
    int P, width, L, nb;
    const cf64 *pre, *chirp, *H;
    cf64* W;
    double scale;
};
template <int NT, int MB>
__global__ void __launch_bounds__(NT, MB) k_to_band(const __grid_constant__ BandArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cf64* buf = reinterpret_cast<cf64*>(smem_raw);
    const Fft4DescT<double>& d = a.d;
    const int last = d.radix[d.np - 1];
    cf64* W = a.W + (long long)blockIdx.x * d.n;
    for (long long row = blockIdx.x; row < a.rows; row += gridDim.x) {
        const cf64* x = a.in + row * a.ip;
        cf64* y = a.out + row * a.op;
        for (int b = 0; b < a.nb; ++b) {
            const int n0 = b * a.L;
            fft4_head(buf, d, [&](int j) {
                if (j >= a.L || n0 + j >= a.P) return mk(0.0, 0.0);
                return cmul4(x[n0 + j], ldg(a.pre + n0 + j));
            });
            pass4_any<-1>(buf, d, last, 1, d.fw[d.np - 1]);
            __syncthreads();
            const cf64* H = a.H + (long long)b * d.n;
            for (int i = threadIdx.x; i < d.n; i += NT) {
                cf64 v = cmul4(buf[pad16(i)], ldg(H + i));
                if (b > 0) v = v + W[i];
                if (b + 1 < a.nb) W[i] = v;
                else buf[pad16(i)] = v;
            }
            __syncthreads();
        }
        pass4_any<+1>(buf, d, last, 1, d.iv[d.np - 1]);
        __syncthreads();
        fft4_tail(buf, d, [&](int k, cf64 v) {
            if (k < a.width) y[k] = cmul4(v, ldg(a.chirp + k));
        });
        __syncthreads();
    }
}
template <int NT, int MB>
__global__ void __launch_bounds__(NT, MB) k_from_band(const __grid_constant__ BandArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cf64* buf = reinterpret_cast<cf64*>(smem_raw);
    const Fft4DescT<double>& d = a.d;
    const int last = d.radix[d.np - 1];
    cf64* W = a.W + (long long)blockIdx.x * d.n;
    for (long long row = blockIdx.x; row < a.rows; row += gridDim.x) {
        const cf64* x = a.in + row * a.ip;
        cf64* y = a.out + row * a.op;
        fft4_head(buf, d, [&](int k) { return k < a.width ? cmul4(conj(x[k]), ldg(a.chirp + k)) : mk(0.0, 0.0); });
        pass4_any<-1>(buf, d, last, 1, d.fw[d.np - 1]);
        __syncthreads();
        for (int b = 0; b < a.nb; ++b) {
            const int n0 = b * a.L;
            const cf64* H = a.H + (long long)b * d.n;
            for (int i = threadIdx.x; i < d.n; i += NT) {
                const cf64 v = b > 0 ? W[i] : buf[pad16(i)];
                if (b == 0 && a.nb > 1) W[i] = v;
                buf[pad16(i)] = cmul4(v, ldg(H + i));
            }
            __syncthreads();
            pass4_any<+1>(buf, d, last, 1, d.iv[d.np - 1]);
            __syncthreads();
            fft4_tail(buf, d, [&](int j, cf64 v) {
                if (j < a.L && n0 + j < a.P) y[n0 + j] = conj(cmul4(v, ldg(a.pre + n0 + j))) * a.scale;
            });
            __syncthreads();
        }
    }
}

// a-point transforms across the a split rows of a line: out[k + b k1].
template <typename R, int A>
__device__ __forceinline__ void split_out(const cpx<R>* y, cpx<R>* out, int b, int k, int dir, int roll, R scale) {
    cpx<R> v[A];
#pragma unroll
    for (int r = 0; r < A; ++r) v[r] = y[(long long)r * b + k];
    if (dir > 0) Dft<R, A, +1>::run(v);
    else Dft<R, A, -1>::run(v);
#pragma unroll
    for (int j = 0; j < A; ++j) {
        const int i = k + j * b + roll;
        out[i < A * b ? i : i - A * b] = v[j] * scale;
    }
}
template <typename R>
__global__ void __launch_bounds__(256) k_split_out(const cpx<R>* __restrict__ y, cpx<R>* __restrict__ out,
                                                   long long op, int a, int b, int dir, int roll, R scale) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= b) return;
    y += (long long)blockIdx.y * a * b;
    out += (long long)blockIdx.y * op;
    switch (a) {
        case 2: split_out<R, 2>(y, out, b, k, dir, roll, scale); break;
        case 3: split_out<R, 3>(y, out, b, k, dir, roll, scale); break;
        case 4: split_out<R, 4>(y, out, b, k, dir, roll, scale); break;
        case 5: split_out<R, 5>(y, out, b, k, dir, roll, scale); break;
        case 6: split_out<R, 6>(y, out, b, k, dir, roll, scale); break;
        case 7: split_out<R, 7>(y, out, b, k, dir, roll, scale); break;
        case 8: split_out<R, 8>(y, out, b, k, dir, roll, scale); break;
        case 9: split_out<R, 9>(y, out, b, k, dir, roll, scale); break;
        case 10: split_out<R, 10>(y, out, b, k, dir, roll, scale); break;
        case 12: split_out<R, 12>(y, out, b, k, dir, roll, scale); break;
        case 15: split_out<R, 15>(y, out, b, k, dir, roll, scale); break;
        default: split_out<R, 16>(y, out, b, k, dir, roll, scale); break;
    }
}

// The radix-8 plans' kernels (plan8), one CTA per row, decimation in time from
// digit-reversed positions.  The first and the last stage take and give the
// row itself: consecutive threads read elements j, j + n / P, ... that the
// first butterfly wants.  The arithmetic and its order are those of fft_dit
// (s1g_fft.cuh).  4.2 M points in rows of 1024 or 4096: 38 us (71 with separate
// loops for loading and storing, unpadded shared memory and 512 threads at
// every length): a chain of dependent shared-memory stages.
// The chirp-z rows stay with separate loops: joined in the same manner they
// fuse other products and sums, and the gradients move (see plan8).
constexpr int kFftThreads = 512;
struct Rows8 {
    const cf32* in;
    long long ip;
    cf32* out;
    long long op;
    int n, roll;             // as RowsIo
    float scale;
    int valid, count;
    const cf32* mul;
    int dir;
    int mask;                // -1: padded shared memory, 0: not
    FftDesc<float> d;        // length n, or of the chirp-z convolution
    const cf32* chirp;       // n
    const cf32* kern;        // d.n
};
__host__ __device__ __forceinline__ int pad8(int i, int mask) { return i + (((i >> 3) + (i >> 6) + (i >> 9)) & mask); }
// t = g Ns + k
__device__ __forceinline__ int rows8_base(int t, int Ns, int P, float inv, int& k) {
    int g = __float2int_rz((float)t * inv);
    k = t - g * Ns;
    if (k < 0) {
        --g;
        k += Ns;
    } else if (k >= Ns) {
        ++g;
        k -= Ns;
    }
    return g * Ns * P + k;
}
template <int P, class Load>
__device__ __forceinline__ void rows8_in(cf32* buf, const FftDesc<float>& d, int dir, int mask, Load load) {
    const int nb = d.n / P;
    for (int j = threadIdx.x; j < nb; j += blockDim.x) {
        cf32 a[P];
#pragma unroll
        for (int r = 0; r < P; ++r) a[r] = load(j + r * nb);
        Bfly<float, P>::run(a, dir);
        const int pos = __ldg(d.perm + j);
#pragma unroll
        for (int s = 0; s < P; ++s) buf[pad8(pos + s, mask)] = a[s];
    }
}
template <int P>
__device__ __forceinline__ void rows8_dit(cf32* buf, const FftDesc<float>& d, int Ns, int dir, int mask) {
    const int nb = d.n / P, step = nb / Ns;
    const float inv = 1.0f / (float)Ns;
    for (int t = threadIdx.x; t < nb; t += blockDim.x) {
        int k;
        const int base = rows8_base(t, Ns, P, inv, k);
        cf32 a[P];
        a[0] = buf[pad8(base, mask)];
#pragma unroll
        for (int r = 1; r < P; ++r) a[r] = buf[pad8(base + r * Ns, mask)] * twid(d, r * k * step, dir);
        Bfly<float, P>::run(a, dir);
#pragma unroll
        for (int s = 0; s < P; ++s) buf[pad8(base + s * Ns, mask)] = a[s];
    }
}
template <int P, class Store>
__device__ __forceinline__ void rows8_out(const cf32* buf, const FftDesc<float>& d, int dir, int mask, Store store) {
    const int nb = d.n / P;
    for (int k = threadIdx.x; k < nb; k += blockDim.x) {
        cf32 a[P];
        a[0] = buf[pad8(k, mask)];
#pragma unroll
        for (int r = 1; r < P; ++r) a[r] = buf[pad8(k + r * nb, mask)] * twid(d, r * k, dir);
        Bfly<float, P>::run(a, dir);
#pragma unroll
        for (int s = 0; s < P; ++s) store(k + s * nb, a[s]);
    }
}
#define ROWS8_RADIX(r, CALL)                              \
    switch (r) {                                          \
        case 2: { constexpr int P = 2; CALL; break; }     \
        case 3: { constexpr int P = 3; CALL; break; }     \
        case 4: { constexpr int P = 4; CALL; break; }     \
        case 5: { constexpr int P = 5; CALL; break; }     \
        case 7: { constexpr int P = 7; CALL; break; }     \
        default: { constexpr int P = 8; CALL; break; }    \
    }
__device__ __forceinline__ void rows8_put(const Rows8& a, cf32* y, int k, cf32 v) {
    v = v * a.scale;
    if (a.mul) {
        // rounded as the product of a pass of its own
        const cf32 m = ldg(a.mul + k);
        v = mk(__fmaf_rn(v.x, m.x, -__fmul_rn(v.y, m.y)), __fmaf_rn(v.y, m.x, __fmul_rn(v.x, m.y)));
    }
    k += a.roll;
    if (k >= a.n) k -= a.n;
    if (k < a.count) y[k] = v;
}

__global__ void __launch_bounds__(kFftThreads, 2) k_rows8_smooth(const __grid_constant__ Rows8 a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cf32* buf = reinterpret_cast<cf32*>(smem_raw);
    const FftDesc<float>& d = a.d;
    const cf32* x = a.in + (long long)blockIdx.x * a.ip;
    cf32* y = a.out + (long long)blockIdx.x * a.op;
    auto put = [&](int k, cf32 v) { rows8_put(a, y, k, v); };
    if (d.nstages < 2) {
        // n is 1 or a radix: one thread
        if (threadIdx.x > 0) return;
        cf32 v[8];
        for (int j = 0; j < d.n; ++j) v[j] = j < a.valid ? x[j] : mk(0.0f, 0.0f);
        if (d.nstages == 1) ROWS8_RADIX(d.radix[0], (Bfly<float, P>::run(v, a.dir)));
        for (int j = 0; j < d.n; ++j) put(j, v[j]);
        return;
    }
    ROWS8_RADIX(d.radix[0], (rows8_in<P>(buf, d, a.dir, a.mask, [&](int j) { return j < a.valid ? x[j] : mk(0.0f, 0.0f); })));
    __syncthreads();
    int Ns = d.radix[0];
    for (int st = 1; st + 1 < d.nstages; ++st) {
        const int p = d.radix[st];
        ROWS8_RADIX(p, (rows8_dit<P>(buf, d, Ns, a.dir, a.mask)));
        __syncthreads();
        Ns *= p;
    }
    ROWS8_RADIX(d.radix[d.nstages - 1], (rows8_out<P>(buf, d, a.dir, a.mask, put)));
}

__global__ void __launch_bounds__(kFftThreads) k_rows8_blue(const __grid_constant__ Rows8 a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cf32* buf = reinterpret_cast<cf32*>(smem_raw);
    const long long row = blockIdx.x;
    const cf32* x = a.in + row * a.ip;
    const int m = a.d.n;
    for (int q = threadIdx.x; q < m; q += blockDim.x) {
        cf32 v = mk(0.0f, 0.0f);
        if (q < a.valid) {
            cf32 xv = x[q];
            if (a.dir > 0) xv = conj(xv);
            v = xv * ldg(a.chirp + q);
        }
        buf[__ldg(a.d.perm + q)] = v;
    }
    __syncthreads();
    fft_dit(buf, a.d, -1);
    for (int q = threadIdx.x; q < m; q += blockDim.x) buf[q] = buf[q] * ldg(a.kern + q);
    __syncthreads();
    fft_dif(buf, a.d, +1);
    cf32* y = a.out + row * a.op;
    for (int k = threadIdx.x; k < a.n; k += blockDim.x) {
        cf32 v = ldg(a.chirp + k) * buf[__ldg(a.d.perm + k)];
        rows8_put(a, y, k, a.dir > 0 ? conj(v) : v);
    }
}

// 32x32 tiled transpose of a batch of matrices.
template <typename R>
__global__ void k_transpose(const cpx<R>* __restrict__ in, long long irp, long long ibp, cpx<R>* __restrict__ out,
                            long long orp, long long obp, int rows, int cols, Failed failed) {
    __shared__ cpx<R> tile[32][33];
    if (failed.first() | failed.second()) return;
    const long long b = blockIdx.z;
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    const cpx<R>* src = in + b * ibp;
    cpx<R>* dst = out + b * obp;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int r = r0 + i, c = c0 + threadIdx.x;
        if (r < rows && c < cols) tile[i][threadIdx.x] = src[(long long)r * irp + c];
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int c = c0 + i, r = r0 + threadIdx.x;
        if (r < rows && c < cols) dst[(long long)c * orp + r] = tile[threadIdx.x][i];
    }
}

// four-step twiddle: data [B][n2][n1], element (j2, k1) *= w_n^(dir j2 k1)
template <typename R>
__global__ void k_twiddle4(cpx<R>* __restrict__ a, long long total, int n1, int n2, const cpx<R>* __restrict__ tw,
                           int n, int dir) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int k1 = (int)(i % n1);
        const int j2 = (int)((i / n1) % n2);
        const int idx = (int)(((long long)j2 * k1) % n);
        cpx<R> w = tw[idx];
        if (dir > 0) w = conj(w);
        a[i] = a[i] * w;
    }
}

template <typename R>
__global__ void k_blue_pre(const cpx<R>* __restrict__ in, long long in_pitch, cpx<R>* __restrict__ a, int n, int m,
                           long long batch, const cpx<R>* __restrict__ chirp, int dir) {
    const long long total = batch * m;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int q = (int)(i % m);
        const long long b = i / m;
        cpx<R> v = mk((R)0, (R)0);
        if (q < n) {
            cpx<R> xv = in[b * in_pitch + q];
            if (dir > 0) xv = conj(xv);
            v = xv * chirp[q];
        }
        a[i] = v;
    }
}

template <typename R>
__global__ void k_mul_rows(cpx<R>* __restrict__ a, long long total, int m, const cpx<R>* __restrict__ k) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x)
        a[i] = a[i] * k[i % m];
}

template <typename R>
__global__ void k_blue_post(const cpx<R>* __restrict__ a, int m, cpx<R>* __restrict__ out, long long out_pitch, int n,
                            long long batch, const cpx<R>* __restrict__ chirp, int dir) {
    const long long total = batch * n;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int k = (int)(i % n);
        const long long b = i / n;
        cpx<R> v = chirp[k] * a[b * m + k];
        out[b * out_pitch + k] = dir > 0 ? conj(v) : v;
    }
}

// out[at[i]] = in[i] scale (at null: out[i])
template <typename R>
__global__ void k_cvt64(const cpx<double>* __restrict__ in, cpx<R>* __restrict__ out, long long n, double scale,
                        const int* __restrict__ at) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        out[at ? at[i] : i] = mk((R)(in[i].x * scale), (R)(in[i].y * scale));
}

template <typename R>
__global__ void k_roll_scale(const cpx<R>* __restrict__ in, cpx<R>* __restrict__ out, long long op, int n, long long rows,
                             int roll, R scale) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < rows * n; i += (long long)gridDim.x * blockDim.x) {
        const long long r = i / n;
        const int k = (int)(i - r * n) + roll;
        out[r * op + (k < n ? k : k - n)] = in[i] * scale;
    }
}

// exp(-pi i t / P), t reduced mod 2 P exactly
__device__ __forceinline__ cf64 half_root(long long t, int P) {
    t %= 2LL * P;
    if (t < 0) t += 2LL * P;
    double c, s;
    sincospi((double)t / (double)P, &s, &c);
    return mk(c, -s);
}
// Tables of a BandPlan; h: nb rows of m, the conjugate chirp at t + step b for
// t in (-before, after), the negative ones at the row's end.
__global__ void k_band_tables(int P, int k0, int width, int m, int nb, int step, int before, int after,
                              cf64* __restrict__ pre, cf64* __restrict__ chirp, cf64* __restrict__ h) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < max((long long)P, (long long)m * nb);
         i += (long long)gridDim.x * blockDim.x) {
        if (i < P) pre[i] = half_root(2 * i * k0 + i * i, P);
        if (i < width) chirp[i] = half_root(i * i, P);
        if (i < (long long)m * nb) {
            const int b = (int)(i / m), q = (int)(i - (long long)b * m);
            const long long t = q < after ? q : q - m, u = t + (long long)step * b;
            h[i] = q < after || q - m > -before ? conj(half_root(u * u, P)) : mk(0.0, 0.0);
        }
    }
}

static int grid_for(long long total, int threads = 256) {
    long long g = (total + threads - 1) / threads;
    if (g > 152 * 32) g = 152 * 32;
    if (g < 1) g = 1;
    return (int)g;
}

// ------------------------------------------------------------------ plans
template <typename R>
FftPlan<R>::~FftPlan() {
    for (void* p : owned) cudaFree(p);
}

static void radices_for(int n, std::vector<int>& out) {
    int c2 = 0, c3 = 0, c5 = 0, c7 = 0;
    while (n % 2 == 0) { n /= 2; ++c2; }
    while (n % 3 == 0) { n /= 3; ++c3; }
    while (n % 5 == 0) { n /= 5; ++c5; }
    while (n % 7 == 0) { n /= 7; ++c7; }
    while (c2 >= 3) { out.push_back(8); c2 -= 3; }
    if (c2 == 2) out.push_back(4);
    if (c2 == 1) out.push_back(2);
    for (int i = 0; i < c5; ++i) out.push_back(5);
    for (int i = 0; i < c3; ++i) out.push_back(3);
    for (int i = 0; i < c7; ++i) out.push_back(7);
}

template <typename R>
static void* upload(FftPlan<R>& p, const void* host, size_t bytes, Uploads& up) {
    void* d = nullptr;
    check_cuda(cudaMalloc(&d, bytes), "plan cudaMalloc");
    p.owned.push_back(d);
    up.table(d, host, bytes, "plan upload");
    return d;
}

// exp(-2 pi i num/den) in FP64 with the argument reduced exactly first.
static inline void unit_root(long long num, long long den, double& c, double& s) {
    num %= den;
    if (num < 0) num += den;
    const double a = 2.0 * M_PI * ((double)num / (double)den);
    c = std::cos(a);
    s = -std::sin(a);
}

FftDescTables::~FftDescTables() {
    for (void* p : owned) cudaFree(p);
}

template <typename R>
static void fill_desc(FftDescTables& t, FftDesc<R>& d, int n) {
    std::vector<int> rad;
    radices_for(n, rad);
    if ((int)rad.size() > kMaxStages) throw std::runtime_error("fft: too many stages");
    d.n = n;
    d.nstages = (int)rad.size();
    for (size_t i = 0; i < rad.size(); ++i) d.radix[i] = (int8_t)rad[i];
    std::vector<cpx<R>> tw(n);
    for (int i = 0; i < n; ++i) {
        double c, s;
        unit_root(i, n, c, s);
        tw[i] = mk((R)c, (R)s);
    }
    std::vector<int> perm(n);
    for (int j = 0; j < n; ++j) {
        int jj = j, size = n, pos = 0;
        for (int st = d.nstages - 1; st >= 0; --st) {
            const int r = jj % rad[st];
            jj /= rad[st];
            size /= rad[st];
            pos += r * size;
        }
        perm[j] = pos;
    }
    Uploads uploads;
    auto up = [&](const void* src, size_t bytes) {
        void* v = nullptr;
        check_cuda(cudaMalloc(&v, bytes), "desc table");
        t.owned.push_back(v);
        uploads.table(v, src, bytes, "desc upload");
        return v;
    };
    d.tw = (const cpx<R>*)up(tw.data(), sizeof(cpx<R>) * n);
    d.perm = (const int*)up(perm.data(), sizeof(int) * n);
}

static void split_four(int n, int cap, int& n1, int& n2) {
    int best = -1;
    for (int a = 2; a <= cap && a < n; ++a) {
        if (n % a) continue;
        const int b = n / a;
        if (b > cap) continue;
        if (best < 0 || std::abs(a - b) < std::abs(best - n / best)) best = a;
    }
    if (best < 0) throw std::runtime_error("fft: no four-step split for n=" + std::to_string(n));
    n1 = best;
    n2 = n / best;
}

FftEngine::FftEngine(cudaStream_t s) : stream(s) {}
FftEngine::~FftEngine() = default;

template <typename R>
static std::map<int, std::shared_ptr<FftPlan<R>>>& plan_map(FftEngine& e, bool radix8);
template <>
std::map<int, std::shared_ptr<FftPlan<float>>>& plan_map<float>(FftEngine& e, bool radix8) {
    return radix8 ? e.plans8 : e.plans32;
}
template <>
std::map<int, std::shared_ptr<FftPlan<double>>>& plan_map<double>(FftEngine& e, bool) { return e.plans64; }

template <typename R>
static Tw4<R> twiddle_entry(long long num, long long den, int sign) {
    cpx<R> w[4];
    for (int b = 0; b < 4; ++b) {
        double c, s;
        unit_root(num * (1 << b), den, c, s);   // exp(-)
        w[b] = mk((R)c, (R)(sign > 0 ? -s : s));
    }
    return Tw4<R>{w[0], w[1], w[2], w[3]};
}

template <typename R>
std::shared_ptr<Fft4PlanT<R>> build_plan4(int n, const std::vector<int>& rad) {
    if (rad.empty() || (int)rad.size() > kFft4Passes || sizeof(cpx<R>) * padded16_len(n) > (size_t)kFft4SmemBytes)
        throw std::runtime_error("plan4: length " + std::to_string(n) + " not smooth/small");
    long long prod = 1;
    for (int r : rad) {
        if (std::find(std::begin(kRadices), std::end(kRadices), r) == std::end(kRadices))
            throw std::runtime_error("plan4: radix");
        prod *= r;
    }
    if (prod != n) throw std::runtime_error("plan4: radices do not multiply to the length");
    auto p = std::make_shared<Fft4PlanT<R>>();
    Fft4DescT<R>& d = p->d;
    d.n = n;
    d.np = (int)rad.size();
    d.affine = sizeof(R) == 4 && d.np >= 2 && rad.back() == 16 && fft4_end_radix(rad[0]);
    // block g of a pass holds the input modulo x^len - exp(-2 pi i F[g] / N)
    std::vector<long long> F{0};
    std::vector<Tw4<R>> tab;
    size_t fo[kFft4Passes], io[kFft4Passes];
    long long N = 1;
    int Ns = n;
    for (int q = 0; q < d.np; ++q) {
        const int r = rad[q];
        d.radix[q] = r;
        Ns /= r;
        fo[q] = tab.size();
        for (long long f : F) tab.push_back(twiddle_entry<R>(f, N * r, -1));
        io[q] = tab.size();
        for (int k = 0; k < Ns; ++k) tab.push_back(twiddle_entry<R>(k, (long long)Ns * r, +1));
        std::vector<long long> G;
        G.reserve(F.size() * r);
        for (long long f : F)
            for (int j = 0; j < r; ++j) G.push_back(f + j * N);
        F.swap(G);
        N *= r;
    }
    std::vector<int> pos(n);
    p->mid.resize(n);
    const int last = rad.back();
    for (int i = 0; i < n; ++i) {
        pos[F[i]] = i;
        p->mid[F[i]] = (i % last) * (n / last) + i / last;
    }
    Uploads uploads;
    auto up = [&](const void* src, size_t bytes) {
        void* v = nullptr;
        check_cuda(cudaMalloc(&v, bytes), "plan4 table");
        p->owned.push_back(v);
        uploads.table(v, src, bytes, "plan4 upload");
        return v;
    };
    const Tw4<R>* t = (const Tw4<R>*)up(tab.data(), sizeof(Tw4<R>) * tab.size());
    for (int q = 0; q < d.np; ++q) {
        d.fw[q] = t + fo[q];
        d.iv[q] = t + io[q];
    }
    d.pos = (const int*)up(pos.data(), sizeof(int) * n);
    d.mid = (const int*)up(p->mid.data(), sizeof(int) * n);
    return p;
}

template std::shared_ptr<Fft4PlanT<float>> build_plan4<float>(int, const std::vector<int>&);
template std::shared_ptr<Fft4PlanT<double>> build_plan4<double>(int, const std::vector<int>&);

// Factors of SPLIT (k_split_out).
static const int kSplits[] = {2, 3, 4, 5, 6, 7, 8, 9, 10, 12, 15, 16};

// Lengths of the core in FP64 with their modelled instructions, ascending.
static const std::vector<std::pair<int, double>>& lengths64() {
    static const auto all = [] {
        std::vector<std::pair<int, double>> v;
        for (int n = 2; n <= fft4_capacity<double>(); ++n) {
            const auto r = fft4_order64(n);
            if (r.empty()) continue;
            double c = 5.0;
            for (int x : r) c += (x & (x - 1)) == 0 ? 3.1 * std::log2((double)x) : 4.2 * std::log2((double)x);
            v.push_back({n, c * n});
        }
        return v;
    }();
    return all;
}
static double cost64(long long n) {
    const auto& v = lengths64();
    const auto it = std::lower_bound(v.begin(), v.end(), std::make_pair((int)n, 0.0));
    return it != v.end() && it->first == n ? it->second : 1e30;
}
// The cheapest length >= least of the core in FP64, -1 if none fits.
static long long length64(long long least) {
    const auto& v = lengths64();
    long long best = -1;
    double bc = 1e30;
    for (auto it = std::lower_bound(v.begin(), v.end(), std::make_pair((int)std::min(least, 1LL << 30), 0.0));
         it != v.end() && it->first <= least * 5 / 4 + 8; ++it)
        if (it->second < bc) {
            bc = it->second;
            best = it->first;
        }
    return best;
}

template <typename R>
static std::shared_ptr<FftPlan<R>> make_plan(FftEngine& e, int n, bool radix8) {
    auto& mp = plan_map<R>(e, radix8);
    auto it = mp.find(n);
    if (it != mp.end()) return it->second;
    cudaStream_t stream = e.stream;
    auto p = std::make_shared<FftPlan<R>>();
    p->n = n;
    const int cap = radix8 ? smem_capacity<R>() : fft4_capacity<R>();
    // convolution length of a Bluestein transform of b points: the cheapest
    // that fits, -1 if none does
    auto conv_len = [&](long long b) -> long long {
        if (radix8) {
            const long long m = next_smooth7(2 * b - 1);
            return m <= cap ? m : -1;
        }
        if constexpr (sizeof(R) == 4) {
            return 2 * b - 1 <= cap ? fast_len(2 * b - 1) : -1;
        } else {
            return length64(2 * b - 1);
        }
    };
    auto core = [&](int len) {
        if constexpr (sizeof(R) == 4) return build_plan4<R>(len, fft4_orders(len, 1).at(0));
        else return build_plan4<R>(len, fft4_order64(len));
    };
    auto desc = [&](int len) {
        for (auto k : {(const void*)k_rows8_smooth, (const void*)k_rows8_blue})
            check_cuda(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes), "smem attr");
        auto t = std::make_shared<FftDescTables>();
        if constexpr (sizeof(R) == 4) fill_desc<R>(*t, t->d32, len);
        else fill_desc<R>(*t, t->d64, len);
        return t;
    };
    const bool fits = radix8 ? is_smooth7(n) && n <= cap :
                      n >= 2 && is_smooth7(n) && n <= cap &&
                      (sizeof(R) == 4 ? !fft4_orders(n, 1).empty() : !fft4_order64(n).empty());
    const long long mc = fits ? 0 : conv_len(n);
    int a = 0;   // split n = a b with b of the one-kernel kinds
    if (!fits && mc < 0 && !radix8)
        for (int x : kSplits)
            if (n % x == 0) {
                const auto sub = make_plan<R>(e, n / x, radix8);
                if (sub->kind == FFT_SMEM || sub->kind == FFT_BLUE) {
                    a = x;
                    break;
                }
            }
    auto roots = [&] {
        std::vector<cpx<R>> tw(n);
        for (int i = 0; i < n; ++i) {
            double c, s;
            unit_root(i, n, c, s);
            tw[i] = mk((R)c, (R)s);
        }
        Uploads up;
        return (cpx<R>*)upload(*p, tw.data(), sizeof(cpx<R>) * n, up);
    };
    if (fits) {
        p->kind = FFT_SMEM;
        if (radix8) p->desc = desc(n);
        else p->core = core(n);
    } else if (a) {
        p->kind = FFT_SPLIT;
        p->n1 = a;
        p->n2 = n / a;
        p->p2 = make_plan<R>(e, p->n2, radix8);
        p->tw4 = roots();
    } else if (mc < 0 && is_smooth7(n)) {
        p->kind = FFT_FOUR;
        split_four(n, cap, p->n1, p->n2);
        p->p1 = make_plan<R>(e, p->n1, radix8);
        p->p2 = make_plan<R>(e, p->n2, radix8);
        p->tw4 = roots();
    } else {
        const long long m = mc >= 0 ? mc : next_smooth7(2LL * n - 1);
        p->m = (int)m;
        if (mc >= 0) {
            p->kind = FFT_BLUE;
            if (radix8) p->desc = desc((int)m);
            else p->core = core((int)m);
        } else {
            p->kind = FFT_BLUE4;
            p->pm = make_plan<R>(e, (int)m, radix8);
        }
        // chirp w[k] = exp(-i pi k^2/n) = exp(-2 pi i (k^2 mod 2n)/(2n))
        std::vector<cpx<R>> w(n);
        std::vector<cpx<double>> b((size_t)m, mk(0.0, 0.0));
        for (int k = 0; k < n; ++k) {
            double c, s;
            unit_root((long long)k * k % (2LL * n), 2LL * n, c, s);
            w[k] = mk((R)c, (R)s);
            b[k] = mk(c, -s);  // conj(w)
            if (k > 0) b[m - k] = mk(c, -s);
        }
        Uploads up;
        p->chirp = (cpx<R>*)upload(*p, w.data(), sizeof(cpx<R>) * n, up);
        // kernel spectrum computed in FP64 on the device, scaled by 1/m
        auto p64 = make_plan<double>(e, (int)m, false);
        cpx<double>* d64 = nullptr;
        check_cuda(cudaMalloc(&d64, sizeof(cpx<double>) * m), "blue tmp");
        up.table(d64, b.data(), sizeof(cpx<double>) * m, "blue up");
        up.done();
        e.rows<double>(*p64, d64, m, d64, m, 1, -1);
        cpx<R>* kd = nullptr;
        check_cuda(cudaMalloc(&kd, sizeof(cpx<R>) * m), "blue kern");
        p->owned.push_back(kd);
        note_launch(), k_cvt64<R><<<grid_for(m), 256, 0, stream>>>(d64, kd, m, 1.0 / (double)m,
                                                                     p->core ? p->core->d.mid : nullptr);
        check_cuda(cudaStreamSynchronize(stream), "blue kern sync");
        cudaFree(d64);
        p->kern = kd;
    }
    mp[n] = p;
    return p;
}

template <typename R>
std::shared_ptr<FftPlan<R>> FftEngine::plan(int n) { return make_plan<R>(*this, n, false); }
std::shared_ptr<FftPlan<float>> FftEngine::plan8(int n) { return make_plan<float>(*this, n, true); }

// The same of a row transform of n points as make_plan chooses it.
static double row_cost64(long long n) {
    const double c = cost64(n);
    if (c < 1e29) return c;
    const long long m = length64(2 * n - 1);
    if (m >= 0) return 2 * cost64(m);
    for (int x : kSplits)
        if (n % x == 0 && (cost64(n / x) < 1e29 || length64(2 * (n / x) - 1) >= 0)) return x * row_cost64(n / x) + 4.0 * n;
    return 1e29;
}

BandPlan::~BandPlan() {
    for (void* q : owned) cudaFree(q);
}

// Bands follow a burst's Doppler rate: four plans a burst, up to 2 MB each.
constexpr size_t kBandPlans = 40;

std::shared_ptr<BandPlan> FftEngine::band_plan(int P, int k0, int width, bool inverse) {
    const std::vector<int> key{P, k0, width, (int)inverse};
    const auto it = bands.find(key);
    if (it != bands.end()) return it->second;
    auto p = std::make_shared<BandPlan>();
    p->P = P;
    p->k0 = k0;
    p->width = width;
    p->inverse = inverse;
    // runs of L points: nb + 1 transforms, against the plain one of P
    double best = P > 0 && width > 0 ? row_cost64(P) : 0.0;
    long long m = 0;
    for (int nb = 1; nb <= 16; ++nb) {
        const int L = (P + nb - 1) / nb;
        const long long q = length64((long long)L + width - 1);
        if (q < 0) continue;
        const double c = (nb + 1) * cost64(q);
        if (c < 0.95 * best) {
            best = c;
            m = q;
            p->nb = nb;
            p->L = L;
        }
    }
    if (p->nb) {
        const auto pm = plan<double>((int)m);   // a length of the core
        p->core = pm->core;
        auto table = [&](size_t n) {
            void* q = nullptr;
            check_cuda(cudaMalloc(&q, sizeof(cf64) * n), "band table");
            p->owned.push_back(q);
            return (cf64*)q;
        };
        p->pre = table(P);
        p->chirp = table(width);
        p->H = table((size_t)m * p->nb);
        cf64* tmp = (cf64*)scratch_band.get(sizeof(cf64) * (size_t)m * p->nb);
        const int before = inverse ? width : p->L, after = inverse ? p->L : width;
        note_launch(), k_band_tables<<<grid_for(std::max<long long>(P, m * p->nb)), 256, 0, stream>>>(
            P, k0, width, (int)m, p->nb, inverse ? p->L : -p->L, before, after, p->pre, p->chirp, tmp);
        rows<double>(*pm, tmp, m, tmp, m, p->nb, -1);
        for (int b = 0; b < p->nb; ++b)
            note_launch(), k_cvt64<double><<<grid_for(m), 256, 0, stream>>>(tmp + b * m, p->H + b * m, m, 1.0 / (double)m,
                                                                            p->core->d.pos);
    }
    if (bands.size() >= kBandPlans) bands.clear();
    bands[key] = p;
    return p;
}

static void launch_band(FftEngine& e, const BandPlan& p, BandArgs a) {
    if (a.rows <= 0) return;
    a.d = p.core->d;
    a.P = p.P;
    a.width = p.width;
    a.L = p.L;
    a.nb = p.nb;
    a.pre = p.pre;
    a.chirp = p.chirp;
    a.H = p.H;
    const size_t smem = sizeof(cf64) * (size_t)padded16_len(a.d.n);
    rows4_launch<double>(smem, [&](auto nt, auto mb) {
        constexpr int NT = decltype(nt)::value, MB = decltype(mb)::value;
        const int grid = (int)std::min<long long>(a.rows, (long long)device_sms() * MB);
        a.W = (cf64*)e.scratch_band.get(sizeof(cf64) * (size_t)grid * a.d.n);
        auto kernel = p.inverse ? k_from_band<NT, MB> : k_to_band<NT, MB>;
        check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFft4SmemBytes), "attr");
        note_launch(), kernel<<<grid, NT, smem, e.stream>>>(a);
    });
    check_cuda(cudaGetLastError(), "band launch");
}
void FftEngine::to_band(const BandPlan& p, const cf64* in, long long ip, cf64* out, long long op, long long rows) {
    BandArgs a{};
    a.in = in;
    a.ip = ip;
    a.out = out;
    a.op = op;
    a.rows = rows;
    launch_band(*this, p, a);
}
void FftEngine::from_band(const BandPlan& p, const cf64* in, long long ip, cf64* out, long long op, long long rows,
                          double scale) {
    BandArgs a{};
    a.in = in;
    a.ip = ip;
    a.out = out;
    a.op = op;
    a.rows = rows;
    a.scale = scale;
    launch_band(*this, p, a);
}

std::shared_ptr<Fft4Plan> FftEngine::plan4(int n) {
    auto it = plans4.find(n);
    if (it != plans4.end()) return it->second;
    auto p = build_plan4<float>(n, tuned_radices(n, stream));
    plans4[n] = p;
    return p;
}

long long FftEngine::tuned_len(long long minlen) { return tuned_length(minlen, stream); }

template <typename R>
FftDesc<R> FftEngine::smem_desc(int n) {
    if (!is_smooth7(n) || n > smem_capacity<R>())
        throw std::runtime_error("smem_desc: length not smooth/small: " + std::to_string(n));
    auto& t = (sizeof(R) == 4 ? descs32 : descs64)[n];
    if (!t) {
        t = std::make_shared<FftDescTables>();
        if constexpr (sizeof(R) == 4) fill_desc<R>(*t, t->d32, n);
        else fill_desc<R>(*t, t->d64, n);
    }
    if constexpr (sizeof(R) == 4) return t->d32;
    else return t->d64;
}

template <typename R>
void transpose_batched(const cpx<R>* in, long long irp, long long ibp, cpx<R>* out, long long orp, long long obp,
                       int rows, int cols, long long batch, cudaStream_t s, Failed failed) {
    if constexpr (sizeof(R) == 4) {
        // single complex<float> matrices go through the TMA-staged corner turn
        if (batch == 1 && transpose_tma(in, irp, out, orp, rows, cols, s, failed)) return;
    }
    dim3 grid((cols + 31) / 32, (rows + 31) / 32, (unsigned)batch);
    note_launch(), k_transpose<R><<<grid, dim3(32, 8), 0, s>>>(in, irp, ibp, out, orp, obp, rows, cols, failed);
}

// rows of a plan of one of the one-kernel kinds
template <typename R>
static void launch_rows(const FftPlan<R>& p, const RowsIo<R>& io, long long rows, cudaStream_t st) {
    if constexpr (sizeof(R) == 4) {
        if (p.desc) {
            const FftDesc<float>& d = p.desc->d32;
            const int padded = pad8(d.n, -1);
            const bool smooth = p.kind == FFT_SMEM, fits = smooth && sizeof(cf32) * (size_t)padded <= (size_t)kSmemBytes;
            const int nt = smooth ? std::min(kFftThreads, std::max(64, (d.n / 8 + 31) / 32 * 32)) : kFftThreads;
            const size_t smem = sizeof(cf32) * (size_t)(fits ? padded : d.n);
            const Rows8 q{io.in, io.ip, io.out, io.op, p.n, io.roll, io.scale, io.valid, io.count, io.mul, io.dir, fits ? -1 : 0, d, p.chirp, p.kern};
            if (smooth) note_launch(), k_rows8_smooth<<<(unsigned)rows, nt, smem, st>>>(q);
            else note_launch(), k_rows8_blue<<<(unsigned)rows, nt, smem, st>>>(q);
            return;
        }
    }
    const Fft4DescT<R>& d = p.core->d;
    const size_t smem = sizeof(cpx<R>) * (size_t)padded16_len(d.n);
    rows4_launch<R>(smem, [&](auto nt, auto mb) {
        constexpr int NT = decltype(nt)::value, MB = decltype(mb)::value;
        if (p.kind == FFT_SMEM) {
            auto kernel = k_rows_smooth<R, NT, MB>;
            check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFft4SmemBytes), "attr");
            note_launch(), kernel<<<(unsigned)rows, NT, smem, st>>>(io, d);
        } else {
            auto kernel = k_rows_blue<R, NT, MB>;
            check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFft4SmemBytes), "attr");
            note_launch(), kernel<<<(unsigned)rows, NT, smem, st>>>(io, d, p.n, p.chirp, p.kern);
        }
    });
}

template <typename R>
void FftEngine::rows(const FftPlan<R>& p, const cpx<R>* in, long long in_pitch, cpx<R>* out, long long out_pitch,
                     long long batch, int dir, int roll, double scale, const RowEnds<R>* ends) {
    if (batch <= 0) return;
    const int n = p.n;
    if (ends && !one_kernel(p)) throw std::runtime_error("fft: partial rows of a length over one CTA");
    switch (p.kind) {
        case FFT_SMEM:
        case FFT_BLUE: launch_rows<R>(p, RowsIo<R>{in, in_pitch, out, out_pitch, 1, nullptr, dir, n, roll, (R)scale,
                                                ends ? ends->valid : n, ends ? ends->count : n,
                                                ends ? ends->mul : nullptr}, batch, stream);
            return;
        case FFT_SPLIT: {
            const long long limit = (1LL << 30) / (long long)sizeof(cpx<R>);
            const long long chunk = std::max(1LL, std::min(std::min(batch, limit / n), 65535LL));
            cpx<R>* Y = (cpx<R>*)scratch_a.get(sizeof(cpx<R>) * chunk * n);
            for (long long b0 = 0; b0 < batch; b0 += chunk) {
                const long long nb = std::min(chunk, batch - b0);
                launch_rows<R>(*p.p2, RowsIo<R>{in + b0 * in_pitch, in_pitch, Y, p.n2, p.n1, p.tw4, dir, p.n2, 0, (R)1, p.n2, p.n2,
                                                   nullptr}, nb * p.n1, stream);
                note_launch(), k_split_out<R><<<dim3((p.n2 + 255) / 256, (unsigned)nb), 256, 0, stream>>>(
                    Y, out + b0 * out_pitch, out_pitch, p.n1, p.n2, dir, roll, (R)scale);
            }
            return;
        }
        case FFT_FOUR: {
            const int n1 = p.n1, n2 = p.n2;
            const long long limit = (256LL << 20) / (long long)sizeof(cpx<R>);
            const long long chunk = std::max(1LL, std::min(batch, limit / n));
            cpx<R>* A = (cpx<R>*)scratch_a.get(sizeof(cpx<R>) * chunk * n);
            cpx<R>* B = (cpx<R>*)scratch_b.get(sizeof(cpx<R>) * chunk * n);
            for (long long b0 = 0; b0 < batch; b0 += chunk) {
                const long long nb = std::min(chunk, batch - b0);
                // [nb][n1][n2] -> A [nb][n2][n1]
                transpose_batched<R>(in + b0 * in_pitch, n2, in_pitch, A, n1, n, n1, n2, nb, stream);
                rows<R>(*p.p1, A, n1, A, n1, nb * n2, dir);
                note_launch(), k_twiddle4<R><<<grid_for(nb * n), 256, 0, stream>>>(A, nb * n, n1, n2, p.tw4, n, dir);
                // A [nb][n2][n1] -> B [nb][n1][n2]
                transpose_batched<R>(A, n1, n, B, n2, n, n2, n1, nb, stream);
                rows<R>(*p.p2, B, n2, B, n2, nb * n1, dir);
                // B [nb][n1(k1)][n2(k2)] -> out [nb][n2][n1]: index k1 + n1 k2
                transpose_batched<R>(B, n2, n, out + b0 * out_pitch, n1, out_pitch, n1, n2, nb, stream);
            }
            break;
        }
        case FFT_BLUE4: {
            const int m = p.m;
            const long long limit = (256LL << 20) / (long long)sizeof(cpx<R>);
            const long long chunk = std::max(1LL, std::min(batch, limit / m));
            // this level's buffer must not alias the four-step scratch (a, b)
            cpx<R>* A = (cpx<R>*)scratch_c.get(sizeof(cpx<R>) * chunk * m);
            for (long long b0 = 0; b0 < batch; b0 += chunk) {
                const long long nb = std::min(chunk, batch - b0);
                note_launch(), k_blue_pre<R><<<grid_for(nb * m), 256, 0, stream>>>(in + b0 * in_pitch, in_pitch, A, n, m, nb,
                                                                    p.chirp, dir);
                rows<R>(*p.pm, A, m, A, m, nb, -1);
                note_launch(), k_mul_rows<R><<<grid_for(nb * m), 256, 0, stream>>>(A, nb * m, m, p.kern);
                rows<R>(*p.pm, A, m, A, m, nb, +1);
                note_launch(), k_blue_post<R><<<grid_for(nb * n), 256, 0, stream>>>(A, m, out + b0 * out_pitch, out_pitch, n, nb,
                                                                     p.chirp, dir);
            }
            break;
        }
    }
    // lengths over one CTA: roll and scale are passes of their own
    if (roll || scale != 1.0) {
        const long long chunk = std::max(1LL, std::min(batch, (256LL << 20) / (long long)sizeof(cpx<R>) / n));
        cpx<R>* A = (cpx<R>*)scratch_a.get(sizeof(cpx<R>) * chunk * n);
        for (long long b0 = 0; b0 < batch; b0 += chunk) {
            const long long nb = std::min(chunk, batch - b0);
            check_cuda(cudaMemcpy2DAsync(A, sizeof(cpx<R>) * n, out + b0 * out_pitch, sizeof(cpx<R>) * out_pitch,
                                         sizeof(cpx<R>) * n, nb, cudaMemcpyDeviceToDevice, stream), "fft copy");
            note_launch(), k_roll_scale<R><<<grid_for(nb * n), 256, 0, stream>>>(A, out + b0 * out_pitch, out_pitch, n, nb,
                                                                                 roll, (R)scale);
        }
    }
    check_cuda(cudaGetLastError(), "fft launch");
}

template std::shared_ptr<FftPlan<float>> FftEngine::plan<float>(int);
template std::shared_ptr<FftPlan<double>> FftEngine::plan<double>(int);
template void FftEngine::rows<float>(const FftPlan<float>&, const cpx<float>*, long long, cpx<float>*, long long,
                                     long long, int, int, double, const RowEnds<float>*);
template void FftEngine::rows<double>(const FftPlan<double>&, const cpx<double>*, long long, cpx<double>*, long long,
                                      long long, int, int, double, const RowEnds<double>*);
template FftDesc<float> FftEngine::smem_desc<float>(int);
template FftDesc<double> FftEngine::smem_desc<double>(int);
template void transpose_batched<float>(const cpx<float>*, long long, long long, cpx<float>*, long long, long long,
                                       int, int, long long, cudaStream_t, Failed);
template void transpose_batched<double>(const cpx<double>*, long long, long long, cpx<double>*, long long,
                                        long long, int, int, long long, cudaStream_t, Failed);
template struct FftPlan<float>;
template struct FftPlan<double>;

}  // namespace s1g
