// Batched row-FFT engine of arbitrary length (host-side plans).
//
// Plan kinds, chosen by length n and precision:
//   SMEM      n is 7-smooth and fits one CTA's shared memory: one kernel, one
//             CTA per row, over the core of s1g_fft4.cuh;
//   BLUE      n has a prime factor > 7: Bluestein chirp-z through a 7-smooth
//             convolution length m >= 2n-1 that fits shared memory;
//   SPLIT     n = a b too long for either, a <= 16 and b of the first two
//             kinds: a kernel of the b-point transforms of every a-th element
//             with the twiddles of the split, and one of the a-point ones;
//   FOUR      n is 7-smooth but too long: four-step (n = n1*n2) through global
//             memory with batched transposes;
//   BLUE4     Bluestein whose convolution length needs SPLIT or FOUR.
// Every transform is unnormalised; dir=-1 forward, dir=+1 backward.
//
// plan8 gives FP32 plans (SMEM, BLUE, FOUR, BLUE4) over the radix-8 core of
// s1g_fft.cuh instead.  The plain FP32 pipelines and the differentiable chains
// use them: a focus gradient is a sum that cancels to 1e-4 of its terms, so it
// moves by up to 1e-4 with the rounding of the transforms, and so do decisions
// of the plain pipelines at their thresholds.  Those paths keep one arithmetic
// (a 1024 x 4096 evaluation's ten transforms: 0.38 ms, 0.42 over the other
// core).
#pragma once

#include <atomic>
#include <cstdint>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "s1g_fft.cuh"
#include "s1g_fft4.cuh"

namespace s1g {

enum FftKind { FFT_SMEM = 0, FFT_BLUE = 1, FFT_FOUR = 2, FFT_BLUE4 = 3, FFT_SPLIT = 4 };

// Largest shared-memory buffer a CTA may use (bytes).
constexpr int kSmemBytes = 220 * 1024;

bool is_smooth7(long long n);
long long next_smooth7(long long n);
// Shared memory of the fused kernels (the most a CTA can have).
constexpr int kFft4SmemBytes = 227 * 1024;
// Transform length >= minlen for the fused kernels' core: the affine length
// (16 x radices, s1g_fft4.cuh) in [minlen, 1.25 minlen] of least modelled
// cost that fits shared memory, -1 if there is none.
long long fast_len(long long minlen);
template <typename R>
inline int smem_capacity() { return kSmemBytes / (int)sizeof(cpx<R>); }
// Longest transform of the core that fits a CTA.
template <typename R>
inline int fft4_capacity() { return (kFft4SmemBytes / (int)sizeof(cpx<R>) - 1) * 16 / 17; }

// Device memory arena owned by a processing context: grow-only scratch.
// moves: the owner's count of arenas given up for larger ones.
struct DeviceArena {
    uint64_t* moves = nullptr;
    void* ptr = nullptr;
    size_t size = 0;
    ~DeviceArena();
    void* get(size_t bytes);
};

// Device tables of the core (s1g_fft4.cuh) for one length.
template <typename R>
struct Fft4PlanT {
    Fft4DescT<R> d;
    std::vector<int> mid;         // host copy of d.mid
    std::vector<void*> owned;
    ~Fft4PlanT() {
        for (void* p : owned) cudaFree(p);
    }
};
using Fft4Plan = Fft4PlanT<float>;

// Tables of a FftDesc (s1g_fft.cuh).
struct FftDescTables {
    FftDesc<float> d32;
    FftDesc<double> d64;
    std::vector<void*> owned;
    ~FftDescTables();
};

template <typename R>
struct FftPlan {
    int n = 0;
    FftKind kind = FFT_SMEM;
    std::shared_ptr<Fft4PlanT<R>> core;   // SMEM: length n; BLUE: length m
    std::shared_ptr<FftDescTables> desc;  // the same of a plan8 (no core)
    int m = 0;                    // Bluestein convolution length
    cpx<R>* chirp = nullptr;      // w[k] = exp(-i pi k^2 / n), k < n
    cpx<R>* kern = nullptr;       // FFT_m of conj chirp, scaled by 1/m (BLUE: at core->d.mid)
    int n1 = 0, n2 = 0;           // split of n: FOUR n1 x n2, SPLIT n1 = a, n2 = b
    std::shared_ptr<FftPlan<R>> p1, p2, pm;   // sub-plans (SPLIT: p2 of length b)
    cpx<R>* tw4 = nullptr;        // exp(-2 pi i k / n) of the split, length n
    std::vector<void*> owned;     // device allocations
    ~FftPlan();
};

// A row transform of which part is given or wanted: inputs from `valid` on are
// zero and not read, output k is multiplied by mul[k] (null: not) before the
// roll, rolled outputs from `count` on are not written.
template <typename R>
struct RowEnds {
    int valid, count;
    const cpx<R>* mul;
};

// FP64 transforms of P points of which only a band of the spectrum is wanted
// or given (to_band, from_band), as chirp-z transforms of runs of L points
// that share one transform of length m on the band's side: nb + 1 of them.
struct BandPlan {
    int P = 0, k0 = 0, width = 0, L = 0, nb = 0;   // nb = 0: the plain transform is cheaper
    bool inverse = false;
    std::shared_ptr<Fft4PlanT<double>> core;       // length m
    cf64* pre = nullptr;    // P: exp(-2 pi i n k0 / P - pi i n^2 / P)
    cf64* chirp = nullptr;  // width: exp(-pi i k^2 / P)
    cf64* H = nullptr;      // nb x m: spectra of the shifted conjugate chirps, at core->d.pos
    std::vector<void*> owned;
    ~BandPlan();
};

// One per processing context (device + stream).
struct FftEngine {
    explicit FftEngine(cudaStream_t s);
    ~FftEngine();
    cudaStream_t stream;
    std::map<int, std::shared_ptr<FftPlan<float>>> plans32;
    std::map<int, std::shared_ptr<FftPlan<double>>> plans64;
    std::map<int, std::shared_ptr<FftPlan<float>>> plans8;
    std::map<std::vector<int>, std::shared_ptr<BandPlan>> bands;   // at most kBandPlans
    std::map<int, std::shared_ptr<FftDescTables>> descs32, descs64;   // smem_desc
    std::map<int, std::shared_ptr<Fft4Plan>> plans4;
    uint64_t moves = 0;
    DeviceArena scratch_a{&moves}, scratch_b{&moves}, scratch_c{&moves}, scratch_band{&moves};

    template <typename R>
    std::shared_ptr<FftPlan<R>> plan(int n);
    std::shared_ptr<FftPlan<float>> plan8(int n);

    // out[b*out_pitch + (k + roll) % n] = scale sum_j in[b*in_pitch + j] exp(dir 2 pi i jk/n),
    // 0 <= roll < n.  in may equal out.  Works for any n >= 1.
    template <typename R>
    void rows(const FftPlan<R>& p, const cpx<R>* in, long long in_pitch, cpx<R>* out,
              long long out_pitch, long long batch, int dir, int roll = 0, double scale = 1.0,
              const RowEnds<R>* ends = nullptr);
    // whether a plan takes RowEnds
    template <typename R>
    static bool one_kernel(const FftPlan<R>& p) { return p.kind == FFT_SMEM || p.kind == FFT_BLUE; }

    // to_band: out[k] = sum_n in[n] exp(-2 pi i n (k0 + k) / P), k < width, rows
    // of P points; from_band: out[n] = scale sum_k in[k] exp(2 pi i n k / P),
    // n < P, rows of width points (k0 = 0).  in and out are different.
    std::shared_ptr<BandPlan> band_plan(int P, int k0, int width, bool inverse);
    void to_band(const BandPlan& p, const cf64* in, long long ip, cf64* out, long long op, long long rows);
    void from_band(const BandPlan& p, const cf64* in, long long ip, cf64* out, long long op, long long rows, double scale);

    // Smooth descriptor for device-side fused kernels (throws if n is not
    // 7-smooth or does not fit shared memory).
    template <typename R>
    FftDesc<R> smem_desc(int n);

    // Plan of the fused kernels' core (n 7-smooth, fits shared memory); the
    // radix order comes from the autotuner (s1g_tune.cu) when it is on.
    std::shared_ptr<Fft4Plan> plan4(int n);
    // Transform length >= minlen for the fused kernels: the autotuner's pick
    // among the cheapest candidates, or fast_len.
    long long tuned_len(long long minlen);
};

// Radix orders for length n in the order of their modelled cost (at most
// `most`; affine ones where there are any); empty if n is not 7-smooth.
std::vector<std::vector<int>> fft4_orders(long long n, size_t most);
// The order of the row engine's FP64 transforms (radices up to 8: registers).
std::vector<int> fft4_order64(long long n);
// The cheapest affine lengths >= minlen that fit shared memory.
std::vector<long long> fft4_lengths(long long minlen, size_t most);
template <typename R>
std::shared_ptr<Fft4PlanT<R>> build_plan4(int n, const std::vector<int>& radices);
// Radix order for length n: the fastest measured candidate when tuning is on
// (S1G_AUTOTUNE unset or not "0"), else the model's.  Measurements run on
// `st` (skipped while st is being captured) and persist in a text file
// (S1G_FFT_TUNE_FILE, default fft_tune.txt beside the library).
std::vector<int> tuned_radices(int n, cudaStream_t st);
long long tuned_length(long long minlen, cudaStream_t st);
// "n:r1.r2..;..." of the radix orders and "minlen>M;..." of the lengths
// chosen so far in this process.
std::string tuning_report();

// Device words (null: none) of which any but 0 says that the chain has failed:
// its last kernel then leaves its output, which is a caller's buffer, as it is.
// Kernels fetch them beside other loads and look at them when they store.
struct Failed {
    const int *a = nullptr, *b = nullptr;
    __device__ __forceinline__ int first() const { return a ? *a : 0; }
    __device__ __forceinline__ int second() const { return b ? *b : 0; }
};

// batched transpose: in [B][rows][cols] (pitches in elements) -> out [B][cols][rows]
template <typename R>
void transpose_batched(const cpx<R>* in, long long in_row_pitch, long long in_batch_pitch, cpx<R>* out,
                       long long out_row_pitch, long long out_batch_pitch, int rows, int cols, long long batch,
                       cudaStream_t s, Failed failed = {});

void check_cuda(cudaError_t e, const char* what);
// Copies of host tables to device memory, there for every stream when this goes.
// A copy of pageable memory by cudaMemcpy may return before the device has it,
// and the handles' streams do not wait for the legacy stream, so that one is
// waited for (not the handle's, whose kernels may run on meanwhile); an
// asynchronous copy might read the host's memory after it has returned.
struct Uploads {
    bool open = false;
    Uploads() = default;
    Uploads(const Uploads&) = delete;
    void table(void* dst, const void* src, size_t bytes, const char* what) {
        open = true;
        check_cuda(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice), what);
    }
    void done() {
        if (open) check_cuda(cudaStreamSynchronize(cudaStreamLegacy), "uploads");
        open = false;
    }
    ~Uploads() {
        if (open) cudaStreamSynchronize(cudaStreamLegacy);
    }
};
// One of them.
inline void upload_table(void* dst, const void* src, size_t bytes, const char* what) {
    Uploads u;
    u.table(dst, src, bytes, what);
    u.done();
}
// Copy a host table to a device variable that every stream may read from now on.
template <class T>
inline void upload_symbol(T& symbol, const void* src, size_t bytes, const char* what) {
    check_cuda(cudaMemcpyToSymbol(symbol, src, bytes), what);
    check_cuda(cudaStreamSynchronize(cudaStreamLegacy), what);
}
// Multiprocessors of the current device.
int device_sms();
// Allow a kernel `bytes` (the same at every call) of dynamic shared memory on
// the current device: the limit belongs to a device, so one flag per process
// would leave the second device without it.
template <auto kernel>
inline void allow_dynamic_smem(int bytes) {
    static std::atomic<bool> done[64];
    int dev = 0;
    check_cuda(cudaGetDevice(&dev), "attr");
    if (dev < 64 && done[dev].load(std::memory_order_relaxed)) return;
    check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes), "attr");
    if (dev < 64) done[dev].store(true, std::memory_order_relaxed);
}

// Count of kernels this library has launched (reported by the benchmark).
void note_launch();
// Add n (may be negative) to the launch count (graph replays and captures).
void note_launches(long long n);
long long launch_count();

}  // namespace s1g
