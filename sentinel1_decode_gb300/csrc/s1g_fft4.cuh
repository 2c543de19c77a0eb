// Shared-memory FFT core of the fused kernels (FP32) and of the row engine
// (FP32 and FP64): forward transform,
// pointwise factor, inverse transform, with the ends of the chain in
// registers.
//
// A transform of n = R0 R1 .. points runs one pass per radix, in place:
//   forward (exp(-)), natural order in, digit-reversed out: pass p splits
//     every block of r0 .. r_{p-1} blocks into R_p; the elements of a
//     butterfly lie Ns = n / (R0 .. Rp) apart and take the twiddles of their
//     block (the residue of the input modulo x^(Ns Rp) - c_block);
//   inverse (exp(+)), digit-reversed in, natural out: the passes in the
//     opposite order, twiddles by the position within the block.
// Both put the twiddles before the butterfly, where a radix-2 step
// x +- w y takes six FMAs (s = x + w y, then 2 x - s).
// The first forward pass takes its inputs from a functor (global memory) and
// the last inverse pass gives its outputs to one, and the last forward pass,
// the factor and the first inverse pass are one pass over shared memory: a
// forward / inverse pair of P passes sweeps shared memory 2 P - 2 times,
// with as many barriers.
//
// Twiddles: w, w^2, w^4, w^8 of each block or position as one entry in global
// memory (32 bytes in FP32), rounded from FP64 (read through L1 / L2, coalesced where they
// differ from lane to lane); other powers are products of at most three.
//
// Layout: one element of padding per 16.  With Ns a multiple of 16 (a plan
// whose last radix is 16) the elements of a butterfly lie at a constant
// stride and no pass has bank conflicts: the passes with Ns >= 16 read runs
// of 16 consecutive elements, the last one elements 17 apart.
#pragma once

#include <type_traits>

#include "s1g_fft.cuh"

namespace s1g {

constexpr int kFft4Passes = 6;

// Launch shape of a kernel over this core: 768 threads per SM at 80 registers,
// as three CTAs of 256, two of 384 or one of 768 by what their shared memory
// leaves room for (an SM holds 228 KB, 1 KB of it reserved per CTA).  Chirp-z
// transforms of 8192 points took 8.3 us per row and SM as three CTAs, 9.3 as
// two of 384 or 512 threads, 9.9 as two of 256; of 24576 points 27.8 with 768
// threads, 30.2 with 512 or 1024 (64 registers: spills).
template <class F>
inline void fft4_launch(size_t smem, F f) {
    using std::integral_constant;
    if (3 * (smem + 1024) <= 228 * 1024) f(integral_constant<int, 256>(), integral_constant<int, 3>());
    else if (2 * (smem + 1024) <= 228 * 1024) f(integral_constant<int, 384>(), integral_constant<int, 2>());
    else f(integral_constant<int, 768>(), integral_constant<int, 1>());
}

template <typename R>
struct alignas(16) Tw4 {
    cpx<R> w1, w2, w4, w8;
};

template <typename R>
struct Fft4DescT {
    int n = 0;
    int np = 0;
    int affine = 0;                    // last radix 16 and a first radix of the fused kernels' set (FP32 only)
    int radix[kFft4Passes] = {};
    const Tw4<R>* fw[kFft4Passes] = {};   // forward pass p: an entry per block
    const Tw4<R>* iv[kFft4Passes] = {};   // inverse pass p: an entry per position
    const int* pos = nullptr;          // digit-reversed position of frequency f
    const int* mid = nullptr;          // where the factor of frequency f lies: j (n / R) + g
};
using Fft4Desc = Fft4DescT<float>;

__device__ __forceinline__ Tw4<float> ldg_tw(const Tw4<float>* p) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    return Tw4<float>{mk(a.x, a.y), mk(a.z, a.w), mk(b.x, b.y), mk(b.z, b.w)};
}
__device__ __forceinline__ Tw4<double> ldg_tw(const Tw4<double>* p) {
    return Tw4<double>{ldg(&p->w1), ldg(&p->w2), ldg(&p->w4), ldg(&p->w8)};
}

__host__ __device__ inline int pad16(int i) { return i + (i >> 4); }
__host__ __device__ inline int padded16_len(int n) { return n + (n >> 4) + 1; }

// t = g * ns + k with 0 <= k < ns (t < 2^24)
__device__ __forceinline__ void split4(int t, int ns, float inv_ns, int& g, int& k) {
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

// ---------------------------------------------------------------- butterflies
__device__ __forceinline__ float fma_(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fma_(double a, double b, double c) { return fma(a, b, c); }
// x, y -> x + w y, x - w y
template <typename T>
__device__ __forceinline__ void pm4(cpx<T>& x, cpx<T>& y, cpx<T> w) {
    const cpx<T> s = mk(fma_(w.x, y.x, fma_(-w.y, y.y, x.x)), fma_(w.x, y.y, fma_(w.y, y.x, x.y)));
    y = mk(fma_((T)2, x.x, -s.x), fma_((T)2, x.y, -s.y));
    x = s;
}
template <typename T>
__device__ __forceinline__ cpx<T> cmul4(cpx<T> a, cpx<T> b) {
    return mk(fma_(a.x, b.x, -a.y * b.y), fma_(a.x, b.y, a.y * b.x));
}
// times exp(DIR i pi m / 8) for m = 0..3
template <int DIR, int M, typename T>
__device__ __forceinline__ cpx<T> rot16(cpx<T> w) {
    constexpr T c[4] = {(T)1.0, (T)0.92387953251128675613, (T)0.70710678118654752440, (T)0.38268343236508977173};
    constexpr T s[4] = {(T)0.0, (T)0.38268343236508977173, (T)0.70710678118654752440, (T)0.92387953251128675613};
    if (M == 0) return w;
    return mk(fma_(c[M], w.x, -DIR * s[M] * w.y), fma_(c[M], w.y, DIR * s[M] * w.x));
}
template <int DIR, typename T>
__device__ __forceinline__ cpx<T> muli4(cpx<T> w) { return DIR > 0 ? mk(-w.y, w.x) : mk(w.y, -w.x); }

// out[j] = sum_r a[r] w^r exp(DIR 2 pi i r j / R), R = 2, 4, 8, 16 with the
// powers w1 = w, w2 = w^2, w4, w8; out[j] lies at a[slot(j)].
template <typename T, int R, int DIR>
struct Tw2 {
    // a[slot]: out index of slot s is the bit reversal of s
    static __device__ __forceinline__ void run(cpx<T>* a, cpx<T> w1, cpx<T> w2, cpx<T> w4, cpx<T> w8) {
        if (R == 16) {
#pragma unroll
            for (int r = 0; r < 8; ++r) pm4(a[r], a[r + 8], w8);
        }
        if (R >= 8) {
            const cpx<T> u = muli4<DIR>(w4);
#pragma unroll
            for (int b = 0; b < R / 8; ++b)
#pragma unroll
                for (int r = 0; r < 4; ++r) pm4(a[8 * b + r], a[8 * b + r + 4], b ? u : w4);
        }
        if (R >= 4) {
            const cpx<T> v1 = R >= 16 ? rot16<DIR, 2>(w2) : w2;   // w2 exp(DIR i pi / 4): only with 16
            const cpx<T> i0 = muli4<DIR>(w2), i1 = muli4<DIR>(v1);
            // out index bits so far of block b (bit-reversed): R = 16: 0, 2, 1, 3; R = 8: 0, 1; R = 4: 0
            const cpx<T> w[4] = {w2, i0, v1, i1};
#pragma unroll
            for (int b = 0; b < R / 4; ++b)
#pragma unroll
                for (int r = 0; r < 2; ++r) pm4(a[4 * b + r], a[4 * b + r + 2], w[b]);
        }
        {
            // factors exp(DIR 2 pi i j / R) of the out index bits of block b
            const cpx<T> e1 = R >= 16 ? rot16<DIR, 1>(w1) : w1, e3 = R >= 16 ? rot16<DIR, 3>(w1) : w1;
            const cpx<T> e2 = R >= 8 ? rot16<DIR, 2>(w1) : w1;
            const cpx<T> f[8] = {w1, muli4<DIR>(w1), e2, muli4<DIR>(e2), e1, muli4<DIR>(e1), e3, muli4<DIR>(e3)};
#pragma unroll
            for (int b = 0; b < R / 2; ++b) pm4(a[2 * b], a[2 * b + 1], f[b]);
        }
    }
    static __device__ __forceinline__ constexpr int out_of(int s) {
        int j = 0;
        for (int b = 1, c = R / 2; b < R; b <<= 1, c >>= 1)
            if (s & b) j |= c;
        return j;
    }
};

// plain DFTs of the other radices, out[j] at a[j]
template <typename T, int R, int DIR>
struct Dft {
    static __device__ __forceinline__ void run(cpx<T>* a) { Bfly<T, R>::run(a, DIR); }
};
template <typename T, int DIR>
struct Dft<T, 2, DIR> {
    static __device__ __forceinline__ void run(cpx<T>* a) {
        const cpx<T> t = a[0];
        a[0] = t + a[1];
        a[1] = t - a[1];
    }
};
template <typename T, int DIR>
struct Dft<T, 16, DIR> {
    static __device__ __forceinline__ void run(cpx<T>* a) {
        // r = r0 + 4 r1, j = j0 + 4 j1, inner twiddles exp(DIR 2 pi i r0 j0 / 16)
        cpx<T> b[4][4];
#pragma unroll
        for (int r0 = 0; r0 < 4; ++r0) {
            cpx<T> v[4] = {a[r0], a[r0 + 4], a[r0 + 8], a[r0 + 12]};
            Bfly<T, 4>::run(v, DIR);
#pragma unroll
            for (int j0 = 0; j0 < 4; ++j0) b[r0][j0] = v[j0];
        }
        b[1][1] = rot16<DIR, 1>(b[1][1]);
        b[1][2] = rot16<DIR, 2>(b[1][2]);
        b[1][3] = rot16<DIR, 3>(b[1][3]);
        b[2][1] = rot16<DIR, 2>(b[2][1]);
        b[2][2] = muli4<DIR>(b[2][2]);
        b[2][3] = muli4<DIR>(rot16<DIR, 2>(b[2][3]));
        b[3][1] = rot16<DIR, 3>(b[3][1]);
        b[3][2] = muli4<DIR>(rot16<DIR, 2>(b[3][2]));
        b[3][3] = muli4<DIR>(muli4<DIR>(rot16<DIR, 1>(b[3][3])));
#pragma unroll
        for (int j0 = 0; j0 < 4; ++j0) {
            cpx<T> v[4] = {b[0][j0], b[1][j0], b[2][j0], b[3][j0]};
            Bfly<T, 4>::run(v, DIR);
#pragma unroll
            for (int j1 = 0; j1 < 4; ++j1) a[j0 + 4 * j1] = v[j1];
        }
    }
};
// coprime factors A x B (Good-Thomas): r = (B r1 + A r2) mod R, and the out
// index j with j = j1 mod A, j = j2 mod B
template <int A, int B, int DIR, typename T>
__device__ __forceinline__ void good_thomas(cpx<T>* a) {
    constexpr int R = A * B;
    cpx<T> t[A][B];
#pragma unroll
    for (int r1 = 0; r1 < A; ++r1)
#pragma unroll
        for (int r2 = 0; r2 < B; ++r2) t[r1][r2] = a[(B * r1 + A * r2) % R];
#pragma unroll
    for (int r1 = 0; r1 < A; ++r1) Dft<T, B, DIR>::run(t[r1]);
#pragma unroll
    for (int r2 = 0; r2 < B; ++r2) {
        cpx<T> c[A];
#pragma unroll
        for (int r1 = 0; r1 < A; ++r1) c[r1] = t[r1][r2];
        Dft<T, A, DIR>::run(c);
#pragma unroll
        for (int j1 = 0; j1 < A; ++j1) {
            // (B r1 + A r2) j / R = r1 j / A + r2 j / B
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (j % A == j1 && j % B == r2) a[j] = c[j1];
        }
    }
}
template <typename T, int DIR>
struct Dft<T, 6, DIR> {
    static __device__ __forceinline__ void run(cpx<T>* a) { good_thomas<2, 3, DIR>(a); }
};
template <typename T, int DIR>
struct Dft<T, 10, DIR> {
    static __device__ __forceinline__ void run(cpx<T>* a) { good_thomas<2, 5, DIR>(a); }
};
template <typename T, int DIR>
struct Dft<T, 12, DIR> {
    static __device__ __forceinline__ void run(cpx<T>* a) { good_thomas<4, 3, DIR>(a); }
};
template <typename T, int DIR>
struct Dft<T, 15, DIR> {
    static __device__ __forceinline__ void run(cpx<T>* a) { good_thomas<3, 5, DIR>(a); }
};
template <typename T, int DIR>
struct Dft<T, 9, DIR> {
    static __device__ __forceinline__ void run(cpx<T>* a) {
        // r = 3 r1 + r2, j = j1 + 3 j2, inner twiddles exp(DIR 2 pi i r2 j1 / 9)
        constexpr T c1 = (T)0.76604444311897803520, s1 = (T)0.64278760968653932632;
        constexpr T c2 = (T)0.17364817766693034885, s2 = (T)0.98480775301220805937;
        constexpr T c4 = (T)-0.93969262078590838405, s4 = (T)0.34202014332566873304;
        cpx<T> t[3][3];
#pragma unroll
        for (int r2 = 0; r2 < 3; ++r2) {
            cpx<T> v[3] = {a[r2], a[3 + r2], a[6 + r2]};
            Dft<T, 3, DIR>::run(v);
            for (int j1 = 0; j1 < 3; ++j1) t[r2][j1] = v[j1];
        }
        t[1][1] = cmul4(t[1][1], mk(c1, DIR * s1));
        t[1][2] = cmul4(t[1][2], mk(c2, DIR * s2));
        t[2][1] = cmul4(t[2][1], mk(c2, DIR * s2));
        t[2][2] = cmul4(t[2][2], mk(c4, DIR * s4));
#pragma unroll
        for (int j1 = 0; j1 < 3; ++j1) {
            cpx<T> v[3] = {t[0][j1], t[1][j1], t[2][j1]};
            Dft<T, 3, DIR>::run(v);
            for (int j2 = 0; j2 < 3; ++j2) a[j1 + 3 * j2] = v[j2];
        }
    }
};

__host__ __device__ constexpr bool pow2r(int r) { return r == 2 || r == 4 || r == 8 || r == 16; }

// a[r] <- sum_r a[r] w^r exp(DIR 2 pi i r j / R) at a[j]
template <int R, int DIR, typename T>
__device__ __forceinline__ void bfly4_tw(cpx<T>* a, const Tw4<T>& e) {
    if constexpr (pow2r(R)) {
        Tw2<T, R, DIR>::run(a, e.w1, e.w2, e.w4, e.w8);
        cpx<T> t[R];
#pragma unroll
        for (int s = 0; s < R; ++s) t[Tw2<T, R, DIR>::out_of(s)] = a[s];
#pragma unroll
        for (int s = 0; s < R; ++s) a[s] = t[s];
    } else {
        const cpx<T> w[4] = {e.w1, e.w2, e.w4, e.w8};
#pragma unroll
        for (int r = 1; r < R; ++r) {
            cpx<T> f = mk((T)1, (T)0);
            bool first = true;
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if (r & (1 << b)) {
                    f = first ? w[b] : cmul4(f, w[b]);
                    first = false;
                }
            a[r] = cmul4(a[r], f);
        }
        Dft<T, R, DIR>::run(a);
    }
}
template <int R, int DIR, typename T>
__device__ __forceinline__ void bfly4(cpx<T>* a) {
    Dft<T, R, DIR>::run(a);
}

// ---------------------------------------------------------------- passes
// Padded position of element r of a butterfly: constant stride when AFF.
template <bool AFF>
struct At4 {
    int b, s;
    __device__ __forceinline__ At4(int base, int Ns) : b(AFF ? pad16(base) : base), s(AFF ? Ns + (Ns >> 4) : Ns) {}
    __device__ __forceinline__ int operator()(int r) const { return AFF ? b + r * s : pad16(b + r * s); }
};

template <int R, int DIR, bool AFF, typename T>
__device__ __forceinline__ void pass4_r(cpx<T>* buf, int n, int Ns, const Tw4<T>* __restrict__ tw) {
    const int nb = n / R;
    const float inv = 1.0f / (float)Ns;
    for (int t = threadIdx.x; t < nb; t += blockDim.x) {
        int g, k;
        split4(t, Ns, inv, g, k);
        // forward: the block's entry; inverse: the position's
        const Tw4<T> e = ldg_tw(tw + (DIR < 0 ? g : k));
        const At4<AFF> at(g * Ns * R + k, Ns);
        cpx<T> a[R];
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = buf[at(r)];
        bfly4_tw<R, DIR>(a, e);
#pragma unroll
        for (int r = 0; r < R; ++r) buf[at(r)] = a[r];
    }
}

// One pass with twiddles over shared memory (caller synchronises).
template <int DIR, bool AFF, typename T>
__device__ __noinline__ void pass4(unsigned int smem, int R, int n, int Ns, const Tw4<T>* tw) {
    // behind the call a pointer would be generic: the shared-space address
    // keeps the accesses LDS / STS
    cpx<T>* buf = reinterpret_cast<cpx<T>*>(__cvta_shared_to_generic(smem));
    switch (R) {
        case 2: pass4_r<2, DIR, AFF>(buf, n, Ns, tw); break;
        case 3: pass4_r<3, DIR, AFF>(buf, n, Ns, tw); break;
        case 4: pass4_r<4, DIR, AFF>(buf, n, Ns, tw); break;
        case 5: pass4_r<5, DIR, AFF>(buf, n, Ns, tw); break;
        case 6: pass4_r<6, DIR, AFF>(buf, n, Ns, tw); break;
        case 7: pass4_r<7, DIR, AFF>(buf, n, Ns, tw); break;
        case 8: pass4_r<8, DIR, AFF>(buf, n, Ns, tw); break;
        default:
            // FP64 plans stop at radix 8 (registers)
            if constexpr (sizeof(T) == 4) {
                switch (R) {
                    case 9: pass4_r<9, DIR, AFF>(buf, n, Ns, tw); break;
                    case 10: pass4_r<10, DIR, AFF>(buf, n, Ns, tw); break;
                    case 12: pass4_r<12, DIR, AFF>(buf, n, Ns, tw); break;
                    case 15: pass4_r<15, DIR, AFF>(buf, n, Ns, tw); break;
                    default: pass4_r<16, DIR, AFF>(buf, n, Ns, tw); break;
                }
            }
    }
}

template <int DIR, typename T>
__device__ __forceinline__ void pass4_any(cpx<T>* buf, const Fft4DescT<T>& d, int R, int Ns, const Tw4<T>* tw) {
    if constexpr (sizeof(T) == 4) {
        if (d.affine) {
            pass4<DIR, true, T>((unsigned int)__cvta_generic_to_shared(buf), R, d.n, Ns, tw);
            return;
        }
    }
    pass4<DIR, false, T>((unsigned int)__cvta_generic_to_shared(buf), R, d.n, Ns, tw);
}

template <int R, typename T, class LoadF>
__device__ __forceinline__ void first4_r(cpx<T>* buf, int n, LoadF load) {
    const int Ns = n / R;
    for (int t = threadIdx.x; t < Ns; t += blockDim.x) {
        const At4<true> at(t, Ns);
        cpx<T> a[R];
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = load(t + r * Ns);
        bfly4<R, -1>(a);
#pragma unroll
        for (int r = 0; r < R; ++r) buf[at(r)] = a[r];
    }
}
// ROLL: the outputs go back to the thread's own slots and to the functor from
// a loop, for functors too long to be unrolled R times.
template <int R, bool ROLL, typename T, class StoreF>
__device__ __forceinline__ void last4_r(cpx<T>* buf, int n, const Tw4<T>* __restrict__ tw, StoreF store) {
    const int Ns = n / R;
    for (int t = threadIdx.x; t < Ns; t += blockDim.x) {
        const Tw4<T> e = ldg_tw(tw + t);
        const At4<true> at(t, Ns);
        cpx<T> a[R];
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = buf[at(r)];
        bfly4_tw<R, +1>(a, e);
        if (ROLL) {
#pragma unroll
            for (int r = 0; r < R; ++r) buf[at(r)] = a[r];
#pragma unroll 2
            for (int r = 0; r < R; ++r) store(t + r * Ns, buf[at(r)]);
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) store(t + r * Ns, a[r]);
        }
    }
}

// Radices of the passes with functors (a plan's first radix).
__host__ __device__ constexpr bool fft4_end_radix(int r) {
    return r == 6 || r == 8 || r == 10 || r == 12 || r == 16;
}

// Forward passes of d up to the last: load(i) gives input i.  Ends with a
// barrier; buf may be read by other threads until the call.
template <typename T, class LoadF>
__device__ __forceinline__ void fft4_head(cpx<T>* buf, const Fft4DescT<T>& d, LoadF load) {
    int Ns = d.n;
    int p = 0;
    bool done = false;
    if constexpr (sizeof(T) == 4) if (d.affine) {
        done = true;
        switch (d.radix[0]) {
            case 6: first4_r<6>(buf, d.n, load); break;
            case 8: first4_r<8>(buf, d.n, load); break;
            case 10: first4_r<10>(buf, d.n, load); break;
            case 12: first4_r<12>(buf, d.n, load); break;
            default: first4_r<16>(buf, d.n, load); break;
        }
        Ns /= d.radix[0];
        p = 1;
    }
    if (!done) {
        for (int i = threadIdx.x; i < d.n; i += blockDim.x) buf[pad16(i)] = load(i);
    }
    __syncthreads();
    for (; p + 1 < d.np; ++p) {
        Ns /= d.radix[p];
        pass4_any<-1>(buf, d, d.radix[p], Ns, d.fw[p]);
        __syncthreads();
    }
}

// The last forward pass (Ns = 1), mid(m, v) at every frequency with m its
// place in the factor table, and the first inverse pass.  Barrier at the end.
template <int R, bool AFF, typename T, class MidF>
__device__ __forceinline__ void mid4_r(cpx<T>* buf, const Fft4DescT<T>& d, MidF mid) {
    const int nb = d.n / R;
    const Tw4<T>* __restrict__ tw = d.fw[d.np - 1];
    for (int g = threadIdx.x; g < nb; g += blockDim.x) {
        const Tw4<T> e = ldg_tw(tw + g);
        cpx<T> a[R];
        const int b = AFF ? 17 * g : R * g;
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = buf[AFF ? b + r : pad16(b + r)];
        bfly4_tw<R, -1>(a, e);
#pragma unroll
        for (int j = 0; j < R; ++j) a[j] = mid(j * nb + g, a[j]);
        bfly4<R, +1>(a);
#pragma unroll
        for (int r = 0; r < R; ++r) buf[AFF ? b + r : pad16(b + r)] = a[r];
    }
}
template <typename T, class MidF>
__device__ __forceinline__ void fft4_mid(cpx<T>* buf, const Fft4DescT<T>& d, MidF mid) {
    bool done = false;
    if constexpr (sizeof(T) == 4) if (d.affine) {
        done = true;
        mid4_r<16, true>(buf, d, mid);
    }
    if (!done) {
        // the last pass, the factor and the first inverse pass (no twiddles) apart
        const int R = d.radix[d.np - 1], nb = d.n / R;
        pass4_any<-1>(buf, d, R, 1, d.fw[d.np - 1]);
        __syncthreads();
        for (int i = threadIdx.x; i < d.n; i += blockDim.x) {
            const int g = i / R;
            buf[pad16(i)] = mid((i - g * R) * nb + g, buf[pad16(i)]);
        }
        __syncthreads();
        pass4_any<+1>(buf, d, R, 1, d.iv[d.np - 1]);
    }
    __syncthreads();
}

// The remaining inverse passes but the last (functor) one.
template <typename T>
__device__ __forceinline__ void fft4_back(cpx<T>* buf, const Fft4DescT<T>& d) {
    int Ns = d.radix[d.np - 1];
    for (int p = d.np - 2; p >= (sizeof(T) == 4 && d.affine ? 1 : 0); --p) {
        pass4_any<+1>(buf, d, d.radix[p], Ns, d.iv[p]);
        Ns *= d.radix[p];
        __syncthreads();
    }
}

// The last inverse pass: store(i, v) gets output i.  No barrier at the end.
template <bool ROLL = false, typename T, class StoreF>
__device__ __forceinline__ void fft4_last(cpx<T>* buf, const Fft4DescT<T>& d, StoreF store) {
    bool done = false;
    if constexpr (sizeof(T) == 4) if (d.affine) {
        done = true;
        switch (d.radix[0]) {
            case 6: last4_r<6, ROLL>(buf, d.n, d.iv[0], store); break;
            case 8: last4_r<8, ROLL>(buf, d.n, d.iv[0], store); break;
            case 10: last4_r<10, ROLL>(buf, d.n, d.iv[0], store); break;
            case 12: last4_r<12, ROLL>(buf, d.n, d.iv[0], store); break;
            default: last4_r<16, ROLL>(buf, d.n, d.iv[0], store); break;
        }
    }
    if (!done) {
        for (int i = threadIdx.x; i < d.n; i += blockDim.x) store(i, buf[pad16(i)]);
    }
}

// The inverse passes after fft4_mid.
template <bool ROLL = false, typename T, class StoreF>
__device__ __forceinline__ void fft4_tail(cpx<T>* buf, const Fft4DescT<T>& d, StoreF store) {
    fft4_back(buf, d);
    fft4_last<ROLL>(buf, d, store);
}

// fft4_tail and fft4_head of the next transform of the same plan in one:
// f(i, v) takes output i to input i of the next (in registers: the last
// inverse and the first forward pass have the same butterflies).  Ends with a
// barrier, as fft4_head.
template <int R, typename T, class JoinF>
__device__ __forceinline__ void join4_r(cpx<T>* buf, int n, const Tw4<T>* __restrict__ tw, JoinF f) {
    const int Ns = n / R;
    for (int t = threadIdx.x; t < Ns; t += blockDim.x) {
        const Tw4<T> e = ldg_tw(tw + t);
        const At4<true> at(t, Ns);
        cpx<T> a[R];
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = buf[at(r)];
        bfly4_tw<R, +1>(a, e);
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = f(t + r * Ns, a[r]);
        bfly4<R, -1>(a);
#pragma unroll
        for (int r = 0; r < R; ++r) buf[at(r)] = a[r];
    }
}
template <typename T, class JoinF>
__device__ __forceinline__ void fft4_join(cpx<T>* buf, const Fft4DescT<T>& d, JoinF f) {
    fft4_back(buf, d);
    int Ns = d.n, p = 0;
    bool done = false;
    if constexpr (sizeof(T) == 4) if (d.affine) {
        done = true;
        switch (d.radix[0]) {
            case 6: join4_r<6>(buf, d.n, d.iv[0], f); break;
            case 8: join4_r<8>(buf, d.n, d.iv[0], f); break;
            case 10: join4_r<10>(buf, d.n, d.iv[0], f); break;
            case 12: join4_r<12>(buf, d.n, d.iv[0], f); break;
            default: join4_r<16>(buf, d.n, d.iv[0], f); break;
        }
        Ns /= d.radix[0];
        p = 1;
    }
    if (!done) {
        for (int i = threadIdx.x; i < d.n; i += blockDim.x) buf[pad16(i)] = f(i, buf[pad16(i)]);
    }
    __syncthreads();
    for (; p + 1 < d.np; ++p) {
        Ns /= d.radix[p];
        pass4_any<-1>(buf, d, d.radix[p], Ns, d.fw[p]);
        __syncthreads();
    }
}

// The last forward pass alone: frequency f then lies at buf[pad16(d.pos[f])].
// Barrier at the end.
template <typename T>
__device__ __forceinline__ void fft4_spectrum(cpx<T>* buf, const Fft4DescT<T>& d) {
    pass4_any<-1>(buf, d, d.radix[d.np - 1], 1, d.fw[d.np - 1]);
    __syncthreads();
}

}  // namespace s1g
