// The library's device arithmetic applied to arrays (tests/test_device_math.py):
// the functions themselves, from the headers that the kernels include.
#include "s1g_adjoint_math.cuh"
#include "s1g_df.cuh"
#include "s1g_tufr_index.cuh"

using namespace s1g;

// what: 0 df_div2(x, y), 1 df_one_minus_sqrt1m(x), 2 df_pow32_1m(x): doubles in,
// double out, the operands rounded to float pairs first (x, y give them back)
__global__ void k_pairs(int what, double* x, double* y, double* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const df a = df_from(x[i]), b = df_from(y[i]);
    x[i] = df_to_double(a);
    y[i] = df_to_double(b);
    out[i] = df_to_double(what == 0 ? df_div2(a, b) : what == 1 ? df_one_minus_sqrt1m(a) : df_pow32_1m(a));
}
__global__ void k_split(const double* x, double* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const df a = df_split(x[i]);
    out[2 * i] = (double)a.hi;
    out[2 * i + 1] = (double)a.lo;
}
// |v|^2 as pair and exponent, its logarithm as a pair
__global__ void k_norm_log(const float2* v, double* out, int* e, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    cf32 z = mk(v[i].x, v[i].y);
    const Norm32 q = norm32(z);
    const df l = ln32(q.I, 2 * q.e);
    e[i] = q.e;
    out[4 * i] = (double)q.I.hi;
    out[4 * i + 1] = (double)q.I.lo;
    out[4 * i + 2] = (double)l.hi;
    out[4 * i + 3] = (double)l.lo;
}
__global__ void k_cis(const float2* t, float2* out, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const cf32 z = cis_turn(t[i].x, t[i].y);
    out[i] = make_float2(z.x, z.y);
}
// knot interval, step, first sample of the interval; first n with m2 n >= a TS
__global__ void k_index(const int* u, int* out, int n, int S, int TS, int m2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gk = (float)((double)(S - 1) / (double)(TS - 1)), rt = (float)((double)(TS - 1) / (double)(S - 1));
    int d;
    const int iv = knot_of_near(u[i], S, TS, gk, 1.0f / (float)(S - 1), d);
    out[4 * i] = iv;
    out[4 * i + 1] = d;
    out[4 * i + 2] = knot_first_near(iv, S, TS, rt);
    out[4 * i + 3] = first_at_or_above(u[i] % m2 - 13, TS, m2, 1.0f / (float)m2);
}

// device copies of host arrays, copied back by finish()
struct Arrays {
    struct A {
        void *host, *dev;
        size_t bytes;
    } a[4];
    int n = 0;
    template <class T>
    T* add(T* host, size_t count) {
        A& x = a[n++];
        x = {host, nullptr, sizeof(T) * count};
        check_cuda(cudaMalloc(&x.dev, x.bytes), "alloc");
        check_cuda(cudaMemcpy(x.dev, host, x.bytes, cudaMemcpyHostToDevice), "up");
        check_cuda(cudaDeviceSynchronize(), "up");
        return (T*)x.dev;
    }
    void finish() {
        check_cuda(cudaDeviceSynchronize(), "run");
        for (int i = 0; i < n; ++i) {
            check_cuda(cudaMemcpy(a[i].host, a[i].dev, a[i].bytes, cudaMemcpyDeviceToHost), "down");
            cudaFree(a[i].dev);
        }
    }
};
static int blocks(int n) { return (n + 255) / 256; }

extern "C" {
void dm_pairs(int what, double* x, double* y, double* out, int n) {
    Arrays m;
    double *dx = m.add(x, n), *dy = m.add(y, n), *d = m.add(out, n);
    k_pairs<<<blocks(n), 256>>>(what, dx, dy, d, n);
    m.finish();
}
void dm_split(double* x, double* out, int n) {
    Arrays m;
    double *dx = m.add(x, n), *d = m.add(out, 2 * (size_t)n);
    k_split<<<blocks(n), 256>>>(dx, d, n);
    m.finish();
}
void dm_norm_log(float2* v, double* out, int* e, int n) {
    init_log_tables();
    Arrays m;
    float2* dv = m.add(v, n);
    double* d = m.add(out, 4 * (size_t)n);
    int* de = m.add(e, n);
    k_norm_log<<<blocks(n), 256>>>(dv, d, de, n);
    m.finish();
}
void dm_cis(float2* t, float2* out, int n) {
    Arrays m;
    float2 *dt = m.add(t, n), *d = m.add(out, n);
    k_cis<<<blocks(n), 256>>>(dt, d, n);
    m.finish();
}
void dm_index(int* u, int* out, int n, int S, int TS, int m2) {
    Arrays m;
    int *du = m.add(u, n), *d = m.add(out, 4 * (size_t)n);
    k_index<<<blocks(n), 256>>>(du, d, n, S, TS, m2);
    m.finish();
}
}
