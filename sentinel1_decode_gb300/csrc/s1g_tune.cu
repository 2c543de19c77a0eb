// Autotuner of the fused kernels' FFT core (s1g_fft4.cuh): for each transform
// length the fused kernels need, it times the modelled cheapest radix orders
// and, where the length is free (chirp-z convolutions, zero-padded range
// lines, the non-uniform FFT grid), the cheapest affine lengths, on this GPU
// with the kernels' own launch shape (fft4_launch), and keeps the fastest.
//
// A measurement is a launch of one CTA per slot of every SM, each running a
// forward transform, a factor and an inverse transform four times; the
// minimum of three timed launches after one warm-up counts.  Results persist
// in a text file so every process on a machine makes the same choices (the
// FP32 results depend on them at the rounding level):
//   R <n> <r1> <r2> ...        radix order of length n
//   L <minlen> <M>             length chosen for a request
// Entries that are not among the candidates (a file written by another
// version) are ignored.  S1G_AUTOTUNE=0 turns tuning off (the model's
// choices); S1G_FFT_TUNE_FILE names the file (default fft_tune.txt in the
// directory of this library).
#include <dlfcn.h>
#include <unistd.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <mutex>
#include <set>
#include <sstream>
#include <stdexcept>

#include "s1g_fft_engine.h"

namespace s1g {

template <int NT, int MB>
__global__ void __launch_bounds__(NT, MB) k_fft_tune(Fft4Desc d, int reps, float* sink) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    cf32* buf = reinterpret_cast<cf32*>(smem_raw);
    float acc = 0.f;
    for (int r = 0; r < reps; ++r) {
        fft4_head(buf, d, [&](int i) { return mk((float)((i * 7 + blockIdx.x) & 15), 1.0f); });
        fft4_mid(buf, d, [&](int m, cf32 v) { return v * (1.0f + (float)(m & 1)); });
        fft4_tail(buf, d, [&](int i, cf32 v) { acc += v.x; });
        __syncthreads();
    }
    if (acc == 12345.678f) sink[blockIdx.x] = acc;
}

// candidates of a length's radix order / of a request's length
constexpr size_t kOrders = 5, kLengths = 3;

namespace {

struct Tuner {
    std::mutex mu;
    bool on = true;
    std::string path;
    std::map<int, std::vector<int>> rad;
    std::map<long long, long long> len;
    int sms = 0;
    float* sink = nullptr;

    Tuner() {
        const char* e = std::getenv("S1G_AUTOTUNE");
        on = !(e && std::string(e) == "0");
        const char* f = std::getenv("S1G_FFT_TUNE_FILE");
        if (f && *f) {
            path = f;
        } else {
            Dl_info info;
            if (dladdr(reinterpret_cast<void*>(&tuning_report), &info) && info.dli_fname) {
                std::string so = info.dli_fname;
                const size_t k = so.rfind('/');
                path = (k == std::string::npos ? std::string(".") : so.substr(0, k)) + "/fft_tune.txt";
            }
        }
    }

    // (re)read the file: another process may have tuned lengths since
    void load() {
        if (path.empty()) return;
        std::ifstream in(path);
        std::string line;
        while (std::getline(in, line)) {
            std::istringstream is(line);
            std::string tag;
            is >> tag;
            if (tag == "R") {
                int n = 0, r = 0;
                std::vector<int> v;
                is >> n;
                long long prod = 1;
                while (is >> r) {
                    v.push_back(r);
                    prod *= r;
                }
                if (n > 0 && prod == n && !rad.count(n)) {
                    const auto c = fft4_orders(n, kOrders);
                    if (std::find(c.begin(), c.end(), v) != c.end()) rad[n] = v;
                }
            } else if (tag == "L") {
                long long a = 0, m = 0, more = 0;
                if ((is >> a >> m) && !(is >> more) && !len.count(a)) {
                    const auto c = fft4_lengths(a, kLengths);
                    if (std::find(c.begin(), c.end(), m) != c.end()) len[a] = m;
                }
            }
        }
    }

    void save() {
        if (path.empty()) return;
        const std::string tmp = path + ".tmp" + std::to_string((long long)getpid());
        {
            std::ofstream out(tmp);
            if (!out) return;
            for (const auto& kv : rad) {
                out << "R " << kv.first;
                for (int r : kv.second) out << " " << r;
                out << "\n";
            }
            for (const auto& kv : len) out << "L " << kv.first << " " << kv.second << "\n";
        }
        std::rename(tmp.c_str(), path.c_str());
    }

    static bool capturing(cudaStream_t st) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        return cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone;
    }

    // time of one launch (microseconds) of the forward / inverse pair, x4
    double time_plan(const Fft4Desc& d, cudaStream_t st) {
        if (!sms) {
            int dev = 0;
            check_cuda(cudaGetDevice(&dev), "tune device");
            check_cuda(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "tune sms");
            check_cuda(cudaMalloc(&sink, sizeof(float) * 4096), "tune sink");
        }
        const size_t smem = sizeof(cf32) * (size_t)padded16_len(d.n);
        double best = 1e30;
        fft4_launch(smem, [&](auto nt, auto mb) {
            auto kernel = k_fft_tune<decltype(nt)::value, decltype(mb)::value>;
            check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFft4SmemBytes),
                       "tune attr");
            const int grid = std::min(sms * (int)decltype(mb)::value, 4096);
            cudaEvent_t e0, e1;
            check_cuda(cudaEventCreate(&e0), "tune event");
            check_cuda(cudaEventCreate(&e1), "tune event");
            for (int it = 0; it < 4; ++it) {
                check_cuda(cudaEventRecord(e0, st), "tune record");
                note_launch(), kernel<<<grid, decltype(nt)::value, smem, st>>>(d, 4, sink);
                check_cuda(cudaGetLastError(), "tune launch");
                check_cuda(cudaEventRecord(e1, st), "tune record");
                check_cuda(cudaEventSynchronize(e1), "tune sync");
                float ms = 0;
                check_cuda(cudaEventElapsedTime(&ms, e0, e1), "tune elapsed");
                if (it > 0) best = std::min(best, 1e3 * (double)ms / decltype(mb)::value);
            }
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
        });
        return best;
    }

    std::vector<int> radices_locked(int n, cudaStream_t st) {
        auto it = rad.find(n);
        if (it != rad.end()) return it->second;
        load();
        it = rad.find(n);
        if (it != rad.end()) return it->second;
        const auto cand = fft4_orders(n, kOrders);
        if (cand.empty()) throw std::runtime_error("fused FFT: length " + std::to_string(n) + " is not 7-smooth");
        if (!on || capturing(st) || cand.size() == 1) return cand[0];
        // the first candidate is the model's; another replaces it only
        // when it is more than 2 % faster
        std::vector<int> best;
        double bt = 1e30;
        for (const auto& c : cand) {
            auto plan = build_plan4<float>(n, c);
            const double t = time_plan(plan->d, st);
            if (best.empty() || t < bt * 0.98) {
                bt = t;
                best = c;
            }
        }
        rad[n] = best;
        save();
        return best;
    }
};

Tuner& tuner() {
    static Tuner t;
    return t;
}

}  // namespace

std::vector<int> tuned_radices(int n, cudaStream_t st) {
    Tuner& t = tuner();
    std::lock_guard<std::mutex> lk(t.mu);
    return t.radices_locked(n, st);
}

long long tuned_length(long long minlen, cudaStream_t st) {
    Tuner& t = tuner();
    std::lock_guard<std::mutex> lk(t.mu);
    auto it = t.len.find(minlen);
    if (it != t.len.end()) return it->second;
    t.load();
    it = t.len.find(minlen);
    if (it != t.len.end()) return it->second;
    const auto c = fft4_lengths(minlen, kLengths);
    if (c.empty()) return -1;
    if (!t.on || Tuner::capturing(st)) return c[0];
    long long best = c[0];
    double bt = 1e30;
    for (const long long m : c) {
        auto plan = build_plan4<float>((int)m, t.radices_locked((int)m, st));
        const double us = t.time_plan(plan->d, st);
        if (us < bt * 0.98) {
            bt = us;
            best = m;
        }
    }
    t.len[minlen] = best;
    t.save();
    return best;
}

std::string tuning_report() {
    Tuner& t = tuner();
    std::lock_guard<std::mutex> lk(t.mu);
    std::ostringstream o;
    o << (t.on ? "on" : "off") << " radices";
    for (const auto& kv : t.rad) {
        o << " " << kv.first << ":";
        for (size_t i = 0; i < kv.second.size(); ++i) o << (i ? "." : "") << kv.second[i];
    }
    o << " lengths";
    for (const auto& kv : t.len) o << " " << kv.first << ">" << kv.second;
    return o.str();
}

}  // namespace s1g
