// FP32 shared-memory FFT core of the fused kernels: forward transform,
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
// Twiddles: w, w^2, w^4, w^8 of each block or position as 32 bytes in global
// memory, rounded from FP64 (read through L1 / L2, coalesced where they
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

struct Fft4Desc {
    int n = 0;
    int np = 0;
    int affine = 0;                    // last radix 16 and a first radix of the fused kernels' set
    int radix[kFft4Passes] = {};
    const float4* fw[kFft4Passes] = {};   // forward pass p: 2 float4 per block
    const float4* iv[kFft4Passes] = {};   // inverse pass p: 2 float4 per position
    const int* pos = nullptr;          // digit-reversed position of frequency f
    const int* mid = nullptr;          // where the factor of frequency f lies: j (n / R) + g
};

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
// x, y -> x + w y, x - w y
__device__ __forceinline__ void pm4(cf32& x, cf32& y, cf32 w) {
    const cf32 s = mk(fmaf(w.x, y.x, fmaf(-w.y, y.y, x.x)), fmaf(w.x, y.y, fmaf(w.y, y.x, x.y)));
    y = mk(fmaf(2.0f, x.x, -s.x), fmaf(2.0f, x.y, -s.y));
    x = s;
}
__device__ __forceinline__ cf32 cmul4(cf32 a, cf32 b) {
    return mk(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// times exp(DIR i pi m / 8) for m = 0..3
template <int DIR, int M>
__device__ __forceinline__ cf32 rot16(cf32 w) {
    constexpr float c[4] = {1.0f, 0.92387953251128675613f, 0.70710678118654752440f, 0.38268343236508977173f};
    constexpr float s[4] = {0.0f, 0.38268343236508977173f, 0.70710678118654752440f, 0.92387953251128675613f};
    if (M == 0) return w;
    return mk(fmaf(c[M], w.x, -DIR * s[M] * w.y), fmaf(c[M], w.y, DIR * s[M] * w.x));
}
template <int DIR>
__device__ __forceinline__ cf32 muli4(cf32 w) { return DIR > 0 ? mk(-w.y, w.x) : mk(w.y, -w.x); }

// out[j] = sum_r a[r] w^r exp(DIR 2 pi i r j / R), R = 2, 4, 8, 16 with the
// powers w1 = w, w2 = w^2, w4, w8; out[j] lies at a[slot(j)].
template <int R, int DIR>
struct Tw2 {
    // a[slot]: out index of slot s is the bit reversal of s
    static __device__ __forceinline__ void run(cf32* a, cf32 w1, cf32 w2, cf32 w4, cf32 w8) {
        if (R == 16) {
#pragma unroll
            for (int r = 0; r < 8; ++r) pm4(a[r], a[r + 8], w8);
        }
        if (R >= 8) {
            const cf32 u = muli4<DIR>(w4);
#pragma unroll
            for (int b = 0; b < R / 8; ++b)
#pragma unroll
                for (int r = 0; r < 4; ++r) pm4(a[8 * b + r], a[8 * b + r + 4], b ? u : w4);
        }
        if (R >= 4) {
            const cf32 v1 = R >= 16 ? rot16<DIR, 2>(w2) : w2;   // w2 exp(DIR i pi / 4): only with 16
            const cf32 i0 = muli4<DIR>(w2), i1 = muli4<DIR>(v1);
            // out index bits so far of block b (bit-reversed): R = 16: 0, 2, 1, 3; R = 8: 0, 1; R = 4: 0
            const cf32 w[4] = {w2, i0, v1, i1};
#pragma unroll
            for (int b = 0; b < R / 4; ++b)
#pragma unroll
                for (int r = 0; r < 2; ++r) pm4(a[4 * b + r], a[4 * b + r + 2], w[b]);
        }
        {
            // factors exp(DIR 2 pi i j / R) of the out index bits of block b
            const cf32 e1 = R >= 16 ? rot16<DIR, 1>(w1) : w1, e3 = R >= 16 ? rot16<DIR, 3>(w1) : w1;
            const cf32 e2 = R >= 8 ? rot16<DIR, 2>(w1) : w1;
            const cf32 f[8] = {w1, muli4<DIR>(w1), e2, muli4<DIR>(e2), e1, muli4<DIR>(e1), e3, muli4<DIR>(e3)};
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
template <int R, int DIR>
struct Dft {
    static __device__ __forceinline__ void run(cf32* a) { Bfly<float, R>::run(a, DIR); }
};
template <int DIR>
struct Dft<2, DIR> {
    static __device__ __forceinline__ void run(cf32* a) {
        const cf32 t = a[0];
        a[0] = t + a[1];
        a[1] = t - a[1];
    }
};
template <int DIR>
struct Dft<16, DIR> {
    static __device__ __forceinline__ void run(cf32* a) {
        // r = r0 + 4 r1, j = j0 + 4 j1, inner twiddles exp(DIR 2 pi i r0 j0 / 16)
        cf32 b[4][4];
#pragma unroll
        for (int r0 = 0; r0 < 4; ++r0) {
            cf32 v[4] = {a[r0], a[r0 + 4], a[r0 + 8], a[r0 + 12]};
            Bfly<float, 4>::run(v, DIR);
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
            cf32 v[4] = {b[0][j0], b[1][j0], b[2][j0], b[3][j0]};
            Bfly<float, 4>::run(v, DIR);
#pragma unroll
            for (int j1 = 0; j1 < 4; ++j1) a[j0 + 4 * j1] = v[j1];
        }
    }
};
// coprime factors A x B (Good-Thomas): r = (B r1 + A r2) mod R, and the out
// index j with j = j1 mod A, j = j2 mod B
template <int A, int B, int DIR>
__device__ __forceinline__ void good_thomas(cf32* a) {
    constexpr int R = A * B;
    cf32 t[A][B];
#pragma unroll
    for (int r1 = 0; r1 < A; ++r1)
#pragma unroll
        for (int r2 = 0; r2 < B; ++r2) t[r1][r2] = a[(B * r1 + A * r2) % R];
#pragma unroll
    for (int r1 = 0; r1 < A; ++r1) Dft<B, DIR>::run(t[r1]);
#pragma unroll
    for (int r2 = 0; r2 < B; ++r2) {
        cf32 c[A];
#pragma unroll
        for (int r1 = 0; r1 < A; ++r1) c[r1] = t[r1][r2];
        Dft<A, DIR>::run(c);
#pragma unroll
        for (int j1 = 0; j1 < A; ++j1) {
            // (B r1 + A r2) j / R = r1 j / A + r2 j / B
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (j % A == j1 && j % B == r2) a[j] = c[j1];
        }
    }
}
template <int DIR>
struct Dft<6, DIR> {
    static __device__ __forceinline__ void run(cf32* a) { good_thomas<2, 3, DIR>(a); }
};
template <int DIR>
struct Dft<10, DIR> {
    static __device__ __forceinline__ void run(cf32* a) { good_thomas<2, 5, DIR>(a); }
};
template <int DIR>
struct Dft<12, DIR> {
    static __device__ __forceinline__ void run(cf32* a) { good_thomas<4, 3, DIR>(a); }
};
template <int DIR>
struct Dft<15, DIR> {
    static __device__ __forceinline__ void run(cf32* a) { good_thomas<3, 5, DIR>(a); }
};
template <int DIR>
struct Dft<9, DIR> {
    static __device__ __forceinline__ void run(cf32* a) {
        // r = 3 r1 + r2, j = j1 + 3 j2, inner twiddles exp(DIR 2 pi i r2 j1 / 9)
        constexpr float c1 = 0.76604444311897803520f, s1 = 0.64278760968653932632f;
        constexpr float c2 = 0.17364817766693034885f, s2 = 0.98480775301220805937f;
        constexpr float c4 = -0.93969262078590838405f, s4 = 0.34202014332566873304f;
        cf32 t[3][3];
#pragma unroll
        for (int r2 = 0; r2 < 3; ++r2) {
            cf32 v[3] = {a[r2], a[3 + r2], a[6 + r2]};
            Dft<3, DIR>::run(v);
            for (int j1 = 0; j1 < 3; ++j1) t[r2][j1] = v[j1];
        }
        t[1][1] = cmul4(t[1][1], mk(c1, DIR * s1));
        t[1][2] = cmul4(t[1][2], mk(c2, DIR * s2));
        t[2][1] = cmul4(t[2][1], mk(c2, DIR * s2));
        t[2][2] = cmul4(t[2][2], mk(c4, DIR * s4));
#pragma unroll
        for (int j1 = 0; j1 < 3; ++j1) {
            cf32 v[3] = {t[0][j1], t[1][j1], t[2][j1]};
            Dft<3, DIR>::run(v);
            for (int j2 = 0; j2 < 3; ++j2) a[j1 + 3 * j2] = v[j2];
        }
    }
};

__host__ __device__ constexpr bool pow2r(int r) { return r == 2 || r == 4 || r == 8 || r == 16; }

// a[r] <- sum_r a[r] w^r exp(DIR 2 pi i r j / R) at a[j] for the twiddle entry
// (w, w^2) (w^4, w^8)
template <int R, int DIR>
__device__ __forceinline__ void bfly4_tw(cf32* a, float4 p, float4 q) {
    const cf32 w1 = mk(p.x, p.y), w2 = mk(p.z, p.w), w4 = mk(q.x, q.y), w8 = mk(q.z, q.w);
    if constexpr (pow2r(R)) {
        Tw2<R, DIR>::run(a, w1, w2, w4, w8);
        cf32 t[R];
#pragma unroll
        for (int s = 0; s < R; ++s) t[Tw2<R, DIR>::out_of(s)] = a[s];
#pragma unroll
        for (int s = 0; s < R; ++s) a[s] = t[s];
    } else {
        const cf32 w[4] = {w1, w2, w4, w8};
#pragma unroll
        for (int r = 1; r < R; ++r) {
            cf32 f = mk(1.f, 0.f);
            bool first = true;
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if (r & (1 << b)) {
                    f = first ? w[b] : cmul4(f, w[b]);
                    first = false;
                }
            a[r] = cmul4(a[r], f);
        }
        Dft<R, DIR>::run(a);
    }
}
template <int R, int DIR>
__device__ __forceinline__ void bfly4(cf32* a) {
    Dft<R, DIR>::run(a);
}

// ---------------------------------------------------------------- passes
// Padded position of element r of a butterfly: constant stride when AFF.
template <bool AFF>
struct At4 {
    int b, s;
    __device__ __forceinline__ At4(int base, int Ns) : b(AFF ? pad16(base) : base), s(AFF ? Ns + (Ns >> 4) : Ns) {}
    __device__ __forceinline__ int operator()(int r) const { return AFF ? b + r * s : pad16(b + r * s); }
};

template <int R, int DIR, bool AFF>
__device__ __forceinline__ void pass4_r(cf32* buf, int n, int Ns, const float4* __restrict__ tw) {
    const int nb = n / R;
    const float inv = 1.0f / (float)Ns;
    for (int t = threadIdx.x; t < nb; t += blockDim.x) {
        int g, k;
        split4(t, Ns, inv, g, k);
        // forward: the block's entry; inverse: the position's
        const int e = DIR < 0 ? g : k;
        const float4 p = __ldg(tw + 2 * e), q = __ldg(tw + 2 * e + 1);
        const At4<AFF> at(g * Ns * R + k, Ns);
        cf32 a[R];
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = buf[at(r)];
        bfly4_tw<R, DIR>(a, p, q);
#pragma unroll
        for (int r = 0; r < R; ++r) buf[at(r)] = a[r];
    }
}

// One pass with twiddles over shared memory (caller synchronises).
template <int DIR, bool AFF>
__device__ __noinline__ void pass4(cf32* buf, int R, int n, int Ns, const float4* tw) {
    switch (R) {
        case 2: pass4_r<2, DIR, AFF>(buf, n, Ns, tw); break;
        case 3: pass4_r<3, DIR, AFF>(buf, n, Ns, tw); break;
        case 4: pass4_r<4, DIR, AFF>(buf, n, Ns, tw); break;
        case 5: pass4_r<5, DIR, AFF>(buf, n, Ns, tw); break;
        case 6: pass4_r<6, DIR, AFF>(buf, n, Ns, tw); break;
        case 7: pass4_r<7, DIR, AFF>(buf, n, Ns, tw); break;
        case 8: pass4_r<8, DIR, AFF>(buf, n, Ns, tw); break;
        case 9: pass4_r<9, DIR, AFF>(buf, n, Ns, tw); break;
        case 10: pass4_r<10, DIR, AFF>(buf, n, Ns, tw); break;
        case 12: pass4_r<12, DIR, AFF>(buf, n, Ns, tw); break;
        case 15: pass4_r<15, DIR, AFF>(buf, n, Ns, tw); break;
        default: pass4_r<16, DIR, AFF>(buf, n, Ns, tw); break;
    }
}

template <int R, class LoadF>
__device__ __forceinline__ void first4_r(cf32* buf, int n, LoadF load) {
    const int Ns = n / R;
    for (int t = threadIdx.x; t < Ns; t += blockDim.x) {
        const At4<true> at(t, Ns);
        cf32 a[R];
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = load(t + r * Ns);
        bfly4<R, -1>(a);
#pragma unroll
        for (int r = 0; r < R; ++r) buf[at(r)] = a[r];
    }
}
// ROLL: the outputs go back to the thread's own slots and to the functor from
// a loop, for functors too long to be unrolled R times.
template <int R, bool ROLL, class StoreF>
__device__ __forceinline__ void last4_r(cf32* buf, int n, const float4* __restrict__ tw, StoreF store) {
    const int Ns = n / R;
    for (int t = threadIdx.x; t < Ns; t += blockDim.x) {
        const float4 p = __ldg(tw + 2 * t), q = __ldg(tw + 2 * t + 1);
        const At4<true> at(t, Ns);
        cf32 a[R];
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = buf[at(r)];
        bfly4_tw<R, +1>(a, p, q);
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
template <class LoadF>
__device__ __forceinline__ void fft4_head(cf32* buf, const Fft4Desc& d, LoadF load) {
    int Ns = d.n;
    int p = 0;
    if (d.affine) {
        switch (d.radix[0]) {
            case 6: first4_r<6>(buf, d.n, load); break;
            case 8: first4_r<8>(buf, d.n, load); break;
            case 10: first4_r<10>(buf, d.n, load); break;
            case 12: first4_r<12>(buf, d.n, load); break;
            default: first4_r<16>(buf, d.n, load); break;
        }
        Ns /= d.radix[0];
        p = 1;
    } else {
        for (int i = threadIdx.x; i < d.n; i += blockDim.x) buf[pad16(i)] = load(i);
    }
    __syncthreads();
    for (; p + 1 < d.np; ++p) {
        Ns /= d.radix[p];
        if (d.affine) pass4<-1, true>(buf, d.radix[p], d.n, Ns, d.fw[p]);
        else pass4<-1, false>(buf, d.radix[p], d.n, Ns, d.fw[p]);
        __syncthreads();
    }
}

// The last forward pass (Ns = 1), mid(m, v) at every frequency with m its
// place in the factor table, and the first inverse pass.  Barrier at the end.
template <int R, bool AFF, class MidF>
__device__ __forceinline__ void mid4_r(cf32* buf, const Fft4Desc& d, MidF mid) {
    const int nb = d.n / R;
    const float4* __restrict__ tw = d.fw[d.np - 1];
    for (int g = threadIdx.x; g < nb; g += blockDim.x) {
        const float4 p = __ldg(tw + 2 * g), q = __ldg(tw + 2 * g + 1);
        cf32 a[R];
        const int b = AFF ? 17 * g : R * g;
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = buf[AFF ? b + r : pad16(b + r)];
        bfly4_tw<R, -1>(a, p, q);
#pragma unroll
        for (int j = 0; j < R; ++j) a[j] = mid(j * nb + g, a[j]);
        bfly4<R, +1>(a);
#pragma unroll
        for (int r = 0; r < R; ++r) buf[AFF ? b + r : pad16(b + r)] = a[r];
    }
}
template <class MidF>
__device__ __forceinline__ void fft4_mid(cf32* buf, const Fft4Desc& d, MidF mid) {
    if (d.affine) {
        mid4_r<16, true>(buf, d, mid);
    } else {
        // the last pass, the factor and the first inverse pass (no twiddles) apart
        const int R = d.radix[d.np - 1], nb = d.n / R;
        pass4<-1, false>(buf, R, d.n, 1, d.fw[d.np - 1]);
        __syncthreads();
        for (int i = threadIdx.x; i < d.n; i += blockDim.x) {
            const int g = i / R;
            buf[pad16(i)] = mid((i - g * R) * nb + g, buf[pad16(i)]);
        }
        __syncthreads();
        pass4<+1, false>(buf, R, d.n, 1, d.iv[d.np - 1]);
    }
    __syncthreads();
}

// The remaining inverse passes but the last (functor) one.
__device__ __forceinline__ void fft4_back(cf32* buf, const Fft4Desc& d) {
    int Ns = d.radix[d.np - 1];
    for (int p = d.np - 2; p >= (d.affine ? 1 : 0); --p) {
        if (d.affine) pass4<+1, true>(buf, d.radix[p], d.n, Ns, d.iv[p]);
        else pass4<+1, false>(buf, d.radix[p], d.n, Ns, d.iv[p]);
        Ns *= d.radix[p];
        __syncthreads();
    }
}

// The other inverse passes: store(i, v) gets output i.  No barrier at the end.
template <bool ROLL = false, class StoreF>
__device__ __forceinline__ void fft4_tail(cf32* buf, const Fft4Desc& d, StoreF store) {
    fft4_back(buf, d);
    if (d.affine) {
        switch (d.radix[0]) {
            case 6: last4_r<6, ROLL>(buf, d.n, d.iv[0], store); break;
            case 8: last4_r<8, ROLL>(buf, d.n, d.iv[0], store); break;
            case 10: last4_r<10, ROLL>(buf, d.n, d.iv[0], store); break;
            case 12: last4_r<12, ROLL>(buf, d.n, d.iv[0], store); break;
            default: last4_r<16, ROLL>(buf, d.n, d.iv[0], store); break;
        }
    } else {
        for (int i = threadIdx.x; i < d.n; i += blockDim.x) store(i, buf[pad16(i)]);
    }
}

// fft4_tail and fft4_head of the next transform of the same plan in one:
// f(i, v) takes output i to input i of the next (in registers: the last
// inverse and the first forward pass have the same butterflies).  Ends with a
// barrier, as fft4_head.
template <int R, class JoinF>
__device__ __forceinline__ void join4_r(cf32* buf, int n, const float4* __restrict__ tw, JoinF f) {
    const int Ns = n / R;
    for (int t = threadIdx.x; t < Ns; t += blockDim.x) {
        const float4 p = __ldg(tw + 2 * t), q = __ldg(tw + 2 * t + 1);
        const At4<true> at(t, Ns);
        cf32 a[R];
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = buf[at(r)];
        bfly4_tw<R, +1>(a, p, q);
#pragma unroll
        for (int r = 0; r < R; ++r) a[r] = f(t + r * Ns, a[r]);
        bfly4<R, -1>(a);
#pragma unroll
        for (int r = 0; r < R; ++r) buf[at(r)] = a[r];
    }
}
template <class JoinF>
__device__ __forceinline__ void fft4_join(cf32* buf, const Fft4Desc& d, JoinF f) {
    fft4_back(buf, d);
    int Ns = d.n, p = 0;
    if (d.affine) {
        switch (d.radix[0]) {
            case 6: join4_r<6>(buf, d.n, d.iv[0], f); break;
            case 8: join4_r<8>(buf, d.n, d.iv[0], f); break;
            case 10: join4_r<10>(buf, d.n, d.iv[0], f); break;
            case 12: join4_r<12>(buf, d.n, d.iv[0], f); break;
            default: join4_r<16>(buf, d.n, d.iv[0], f); break;
        }
        Ns /= d.radix[0];
        p = 1;
    } else {
        for (int i = threadIdx.x; i < d.n; i += blockDim.x) buf[pad16(i)] = f(i, buf[pad16(i)]);
    }
    __syncthreads();
    for (; p + 1 < d.np; ++p) {
        Ns /= d.radix[p];
        if (d.affine) pass4<-1, true>(buf, d.radix[p], d.n, Ns, d.fw[p]);
        else pass4<-1, false>(buf, d.radix[p], d.n, Ns, d.fw[p]);
        __syncthreads();
    }
}

// The last forward pass alone: frequency f then lies at buf[pad16(d.pos[f])].
// Barrier at the end.
__device__ __forceinline__ void fft4_spectrum(cf32* buf, const Fft4Desc& d) {
    if (d.affine) pass4<-1, true>(buf, 16, d.n, 1, d.fw[d.np - 1]);
    else pass4<-1, false>(buf, d.radix[d.np - 1], d.n, 1, d.fw[d.np - 1]);
    __syncthreads();
}

}  // namespace s1g
