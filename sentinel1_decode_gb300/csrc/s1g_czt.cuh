// Chirp-z transforms over the fused kernels' FFT core, and what else the fused
// kernels' translation units share.
#pragma once

#include "s1g_fast.cuh"

namespace s1g {

__device__ __forceinline__ cf32 cexpf_fast(float th) {
    float s, c;
    __sincosf(th, &s, &c);
    return mk(c, s);
}

template <class K>
static void allow_smem(K kernel) {
    check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFft4SmemBytes), "attr");
}

static size_t fft4_smem(int n) { return sizeof(cf32) * (size_t)padded16_len(n); }

// CZT: X[k] = sum_{s<nin} x[s] exp(dir 2 pi i s k / P) (k < nout), the input
// from load(s), the output to store(k, X[k]).  dir = +1 conjugates both ends.
template <class LoadF>
__device__ __forceinline__ cf32 czt_in(const CztDev& c, int dir, int q, LoadF load) {
    if (q >= c.nin) return mk(0.f, 0.f);
    cf32 x = load(q);
    if (dir > 0) x = conj(x);
    return x * ldg(c.chirp + q);
}
__device__ __forceinline__ cf32 czt_out(const CztDev& c, int dir, int k, cf32 v) {
    v = ldg(c.chirp + k) * v;
    return dir > 0 ? conj(v) : v;
}
__device__ __forceinline__ void czt_mid(cf32* buf, const CztDev& c) {
    fft4_mid(buf, c.dm, [&](int m, cf32 v) { return v * ldg(c.kern + m); });
}
template <bool ROLL = false, class LoadF, class StoreF>
__device__ __forceinline__ void czt_run(cf32* buf, const CztDev& c, int dir, LoadF load, StoreF store) {
    fft4_head(buf, c.dm, [&](int q) { return czt_in(c, dir, q, load); });
    czt_mid(buf, c);
    fft4_tail<ROLL>(buf, c.dm, [&](int k, cf32 v) {
        if (k < c.nout) store(k, czt_out(c, dir, k, v));
    });
}

}  // namespace s1g
