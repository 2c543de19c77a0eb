// Packet indexer and FDBAQ (type D) decoder kernels.
//
// Indexer: the space-packet chain is sequential (next = cur + 7 +
// packet_data_length, packet.cpp:850-879), so the stream is cut into chunks
// and one warp per chunk finds the first packet start in its chunk (ballot
// over the secondary-header sync marker 0x352EF853 at byte 12 of a packet)
// and walks the chain to the chunk end.  A single block then checks that
// every chunk's speculative entry equals the previous chunk's exit (re-walking
// sequentially only where it does not), and exclusive-scans the per-chunk
// packet counts.  A last pass writes every packet offset at its global index.
//
// Decoder: one warp per packet reproduces the bitstream walk of
// _set_quad_type_d / _get_h_code_type_d / huffman_decode (packet.cpp:755-818,
// decoding_utils.cpp:44-77): the lanes walk short pieces of a block's bits
// from guessed starts until the pieces fit together (see k_decode_fdbaq), and
// the reconstruction of _get_s_values_type_d (packet.cpp:678-693) and the
// IE/IO/QE/QO interleave of _get_signal_type_d (packet.cpp:696-752) happen in
// the same kernel.  Errors become per-packet status codes instead of
// exceptions.
#include <cstring>
#include <stdexcept>

#include "s1g_kernels.h"

namespace s1g {

// ------------------------------------------------------------------ tables
__constant__ double c_simple[5][17] = {
    {3.0000, 3.0000, 3.1600, 3.5300},
    {4.0000, 4.0000, 4.0800, 4.3700},
    {6.0000, 6.0000, 6.0000, 6.1500, 6.5000, 6.8800},
    {9.0000, 9.0000, 9.0000, 9.0000, 9.3600, 9.5000, 10.1000},
    {15.0000, 15.0000, 15.0000, 15.0000, 15.0000, 15.0000, 15.2200, 15.5000, 16.0600},
};
__constant__ double c_norm[5][16] = {
    {0.3637, 1.0915, 1.8208, 2.6406},
    {0.3042, 0.9127, 1.5216, 2.1313, 2.8426},
    {0.2305, 0.6916, 1.1528, 1.6140, 2.0754, 2.5369, 3.1191},
    {0.1702, 0.5107, 0.8511, 1.1916, 1.5321, 1.8726, 2.2131, 2.5536, 2.8942, 3.3744},
    {0.1130, 0.3389, 0.5649, 0.7908, 1.0167, 1.2428, 1.4687, 1.6947, 1.9206, 2.1466, 2.3725,
     2.5985, 2.8244, 3.0504, 3.2764, 3.6623},
};
__constant__ double c_sf[256] = {
    0.00, 0.63, 1.25, 1.88, 2.51, 3.13, 3.76, 4.39, 5.01, 5.64, 6.27, 6.89, 7.52, 8.15, 8.77,
    9.40, 10.03, 10.65, 11.28, 11.91, 12.53, 13.16, 13.79, 14.41, 15.04, 15.67, 16.29, 16.92,
    17.55, 18.17, 18.80, 19.43, 20.06, 20.68, 21.31, 21.93, 22.56, 23.19, 23.81, 24.44, 25.06,
    25.69, 26.32, 26.94, 27.57, 28.20, 28.83, 29.45, 30.08, 30.71, 31.33, 31.96, 32.59, 33.21,
    33.84, 34.47, 35.09, 35.72, 36.35, 36.97, 37.60, 38.23, 38.85, 39.48, 40.11, 40.73, 41.36,
    41.99, 42.61, 43.24, 43.87, 44.49, 45.12, 45.75, 46.37, 47.00, 47.63, 48.25, 48.88, 49.51,
    50.13, 50.76, 51.39, 52.01, 52.64, 53.27, 53.89, 54.52, 55.15, 55.77, 56.40, 57.03, 57.65,
    58.28, 58.91, 59.54, 60.16, 60.79, 61.41, 62.04, 62.98, 64.24, 65.49, 66.74, 68.00, 69.25,
    70.50, 71.76, 73.01, 74.26, 75.52, 76.77, 78.02, 79.28, 80.53, 81.78, 83.04, 84.29, 85.54,
    86.80, 88.05, 89.30, 90.56, 91.81, 93.07, 94.32, 95.57, 96.83, 98.08, 99.33, 100.58,
    101.84, 103.09, 104.34, 105.60, 106.85, 108.10, 109.36, 110.61, 111.86, 113.11, 114.37,
    115.62, 116.87, 118.13, 119.38, 120.63, 121.89, 123.14, 124.39, 125.65, 126.90, 128.15,
    129.41, 130.66, 131.91, 133.17, 134.42, 135.67, 136.93, 138.18, 139.43, 140.69, 141.94,
    143.19, 144.45, 145.70, 146.95, 148.21, 149.46, 150.71, 151.97, 153.22, 154.47, 155.73,
    156.98, 158.23, 159.49, 160.74, 161.99, 163.25, 164.50, 165.75, 167.01, 168.26, 169.51,
    170.77, 172.02, 173.27, 174.53, 175.78, 177.03, 178.29, 179.54, 180.79, 182.05, 183.30,
    184.55, 185.81, 187.06, 188.31, 189.57, 190.82, 192.07, 193.33, 194.58, 195.83, 197.09,
    198.34, 199.59, 200.85, 202.10, 203.35, 204.61, 205.86, 207.11, 208.37, 209.62, 210.87,
    212.13, 213.38, 214.63, 215.89, 217.14, 218.39, 219.65, 220.90, 222.15, 223.41, 224.66,
    225.91, 227.17, 228.42, 229.67, 230.93, 232.18, 233.43, 234.69, 235.94, 237.19, 238.45,
    239.70, 240.95, 242.21, 243.46, 244.71, 245.97, 247.22, 248.47, 249.73, 250.98, 252.23,
    253.49, 254.74, 255.99,
};
__constant__ int c_brc_thidx[5] = {3, 3, 5, 6, 8};
__constant__ int c_brc_mcode[5] = {3, 4, 6, 9, 15};

// Huffman lookup: for BRC b and the next 10 bits w (MSB = next bit: the
// sample's sign, then its code; no code is longer than 9 bits), the value-keyed
// walk of huffman_decode is resolved into the symbol byte sign<<7 | mcode (low
// byte) and the bits the sample takes with its sign, 2..10 (high byte).  The
// table is built on the host by running that walk on every window; every
// window starts with a code, so "Max bit length exceeded" cannot happen.
typedef uint16_t HuffEntry;
constexpr int kHuffWindow = 1024;

// ------------------------------------------------------------------ indexer
constexpr uint32_t kSync = 0x352EF853u;

__device__ __forceinline__ bool is_packet_start(const uint8_t* s, long long n, long long p) {
    if (p + 68 > n) return false;
    const uint8_t b0 = s[p];
    if ((b0 >> 5) != 0) return false;          // packet version 0
    if (((b0 >> 3) & 1) != 1) return false;    // secondary header flag
    const uint32_t sync = ((uint32_t)s[p + 12] << 24) | ((uint32_t)s[p + 13] << 16) |
                          ((uint32_t)s[p + 14] << 8) | (uint32_t)s[p + 15];
    return sync == kSync;
}

__device__ __forceinline__ long long packet_next(const uint8_t* s, long long p) {
    const uint32_t pdl = ((uint32_t)s[p + 4] << 8) | s[p + 5];
    return p + 7 + (long long)pdl;
}

// One warp per chunk: entry = first position in [chunk begin, chunk end) that
// looks like a packet start (or -1); the walk from there counts chain
// positions p with p < chunk end and p + 6 <= n (the reference stops when a
// 6-byte primary header can no longer be read); exit = where the walk left.
__global__ void k_index_chunks(const uint8_t* __restrict__ s, long long n, long long chunk, int nchunks,
                               long long* __restrict__ entry, long long* __restrict__ exitp, int* __restrict__ count) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (warp >= nchunks) return;
    const long long c0 = (long long)warp * chunk;
    const long long c1 = min(n, c0 + chunk);
    long long found = -1;
    for (long long base = c0; base < c1 && found < 0; base += 32) {
        const long long p = base + lane;
        const bool hit = p < c1 && is_packet_start(s, n, p);
        const unsigned m = __ballot_sync(0xffffffffu, hit);
        if (m) found = base + __ffs(m) - 1;
    }
    if (lane == 0) {
        int cnt = 0;
        long long p = found;
        if (found >= 0) {
            while (p < c1 && p + 6 <= n) {
                ++cnt;
                p = packet_next(s, p);
            }
        }
        entry[warp] = found;
        count[warp] = cnt;
        exitp[warp] = p;
    }
}

// Block-wide inclusive scan helpers (1024 threads, one value per thread).
__device__ int block_scan_max(int v, int* sh) {
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int off = 1; off < blockDim.x; off <<= 1) {
        const int t = threadIdx.x >= off ? sh[threadIdx.x - off] : -1;
        __syncthreads();
        sh[threadIdx.x] = max(sh[threadIdx.x], t);
        __syncthreads();
    }
    return sh[threadIdx.x];
}

__device__ int block_scan_sum(int v, int* sh) {
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int off = 1; off < blockDim.x; off <<= 1) {
        const int t = threadIdx.x >= off ? sh[threadIdx.x - off] : 0;
        __syncthreads();
        sh[threadIdx.x] += t;
        __syncthreads();
    }
    return sh[threadIdx.x];
}

// Single block of 1024 threads.  The chain reaches chunk k at T_k = exit of
// the last non-empty chunk before k (0 for the first).  Chunk k is consistent
// if the chain skips it and its walk found nothing, or if its speculative
// entry is T_k.  If every chunk is consistent the per-chunk counts are the
// chain's; otherwise thread 0 re-walks the chain sequentially.
__global__ void k_index_fix(const uint8_t* __restrict__ s, long long n, long long chunk, int nchunks,
                            long long* __restrict__ entry, long long* __restrict__ exitp, int* __restrict__ count,
                            int* __restrict__ base, int* __restrict__ total) {
    __shared__ int sh[1024];
    __shared__ int bad;
    const int per = (nchunks + blockDim.x - 1) / blockDim.x;
    const int k0 = threadIdx.x * per;
    const int k1 = min(nchunks, k0 + per);
    if (threadIdx.x == 0) bad = 0;
    // last non-empty chunk index at or before each position (segment-local, then block scan)
    int last = -1;
    for (int k = k0; k < k1; ++k)
        if (count[k] > 0) last = k;
    const int incl = block_scan_max(last, sh);
    int prev = (threadIdx.x > 0) ? sh[threadIdx.x - 1] : -1;
    (void)incl;
    __syncthreads();
    for (int k = k0; k < k1; ++k) {
        const long long T = (prev < 0) ? 0 : exitp[prev];
        const long long c1 = min(n, (long long)k * chunk + chunk);
        const bool ok = (T >= c1) ? (count[k] == 0) : (entry[k] == T);
        if (!ok) atomicAdd(&bad, 1);
        if (count[k] > 0) prev = k;
    }
    __syncthreads();
    if (bad) {
        if (threadIdx.x == 0) {
            long long p = 0;
            int acc = 0;
            for (int k = 0; k < nchunks; ++k) {
                const long long c1 = min(n, (long long)k * chunk + chunk);
                entry[k] = p;
                int cnt = 0;
                while (p < c1 && p + 6 <= n) {
                    ++cnt;
                    p = packet_next(s, p);
                }
                count[k] = cnt;
                exitp[k] = p;
                base[k] = acc;
                acc += cnt;
            }
            *total = acc;
        }
        return;
    }
    int local = 0;
    for (int k = k0; k < k1; ++k) local += count[k];
    const int inc = block_scan_sum(local, sh);
    int acc = inc - local;
    for (int k = k0; k < k1; ++k) {
        base[k] = acc;
        acc += count[k];
    }
    if (threadIdx.x == blockDim.x - 1) *total = inc;
}

__global__ void k_index_write(const uint8_t* __restrict__ s, long long n, long long chunk, int nchunks,
                              const long long* __restrict__ entry, const int* __restrict__ count,
                              const int* __restrict__ base, long long* __restrict__ offsets, int max_out) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nchunks) return;
    long long p = entry[k];
    for (int i = 0; i < count[k]; ++i) {
        const int idx = base[k] + i;
        if (idx < max_out) offsets[idx] = p;
        p = packet_next(s, p);
    }
}

int index_packets(const uint8_t* d_stream, long long n, long long* d_offsets, int max_packets, IndexScratch& sc,
                  cudaStream_t st, bool sync_count, int* h_count) {
    const long long chunk = 1 << 14;
    const int nchunks = (int)((n + chunk - 1) / chunk);
    if (nchunks <= 0) {
        // an empty stream holds no packets; launch nothing (the scratch
        // arrays, the count word included, are not allocated for 0 chunks)
        if (h_count) *h_count = 0;
        return 0;
    }
    sc.reserve(nchunks);
    const int threads = 256;
    const int warps_per_block = threads / 32;
    note_launch(), k_index_chunks<<<(nchunks + warps_per_block - 1) / warps_per_block, threads, 0, st>>>(
        d_stream, n, chunk, nchunks, sc.entry, sc.exitp, sc.count);
    note_launch(), k_index_fix<<<1, 1024, 0, st>>>(d_stream, n, chunk, nchunks, sc.entry, sc.exitp, sc.count, sc.base, sc.total);
    note_launch(), k_index_write<<<(nchunks + 127) / 128, 128, 0, st>>>(d_stream, n, chunk, nchunks, sc.entry, sc.count, sc.base,
                                                         d_offsets, max_packets);
    if (sync_count && h_count) {
        check_cuda(cudaMemcpyAsync(h_count, sc.total, sizeof(int), cudaMemcpyDeviceToHost, st), "index count");
        check_cuda(cudaStreamSynchronize(st), "index sync");
        return *h_count;
    }
    return -1;
}

void IndexScratch::reserve(int nchunks) {
    if (nchunks <= cap) return;
    release();
    check_cuda(cudaMalloc(&entry, sizeof(long long) * nchunks), "index scratch");
    check_cuda(cudaMalloc(&exitp, sizeof(long long) * nchunks), "index scratch");
    check_cuda(cudaMalloc(&count, sizeof(int) * nchunks), "index scratch");
    check_cuda(cudaMalloc(&base, sizeof(int) * nchunks), "index scratch");
    check_cuda(cudaMalloc(&total, sizeof(int)), "index scratch");
    cap = nchunks;
}

void IndexScratch::release() {
    if (entry) cudaFree(entry);
    if (exitp) cudaFree(exitp);
    if (count) cudaFree(count);
    if (base) cudaFree(base);
    if (total) cudaFree(total);
    entry = exitp = nullptr;
    count = base = total = nullptr;
    cap = 0;
}

// Gather the 68 header bytes of each packet (for host-side segmentation).
__global__ void k_gather_headers(const uint8_t* __restrict__ s, long long n, const long long* __restrict__ off,
                                 int npk, uint8_t* __restrict__ hdr) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)npk * 68) return;
    const int p = (int)(i / 68), b = (int)(i % 68);
    const long long at = off[p] + b;
    hdr[i] = at < n ? s[at] : 0;
}

void gather_headers(const uint8_t* d_stream, long long n, const long long* d_off, int npk, uint8_t* d_hdr,
                    cudaStream_t st) {
    const long long tot = (long long)npk * 68;
    if (tot == 0) return;
    note_launch(), k_gather_headers<<<(unsigned)((tot + 255) / 256), 256, 0, st>>>(d_stream, n, d_off, npk, d_hdr);
}

// ------------------------------------------------------------------ decoder
// Where packet j of a decode goes.  Job-table mode (jobs != nullptr): any mix
// of bursts and row lengths in one launch.  Uniform mode: packets p0 + j (or
// pk_idx[j]) of one burst, nq quads each, rows j * pitch.
struct DecodeSpec {
    const DecodeJob* jobs;
    int njobs;
    const int* pk_idx;
    int p0;
    int nq;
    long long pitch;
};

__device__ __forceinline__ DecodeJob job_at(const DecodeSpec& d, int j) {
    if (d.jobs) return d.jobs[j];
    DecodeJob o;
    o.pk = d.pk_idx ? d.pk_idx[j] : d.p0 + j;
    o.nq = d.nq;
    o.out = (long long)j * d.pitch;
    return o;
}

// ---- FDBAQ walk and reconstruction, one warp per packet
//
// A packet's codes are a serial chain (a code starts where the previous one
// ends), and a thread that follows it takes ~170 cycles a code: 2.0 ms for
// the 24000 codes of a 12000-sample packet, with 1500 such threads on a chip
// that runs 300000.  Here a warp takes a block of 128 codes at a time: lane l
// walks the piece of `seg` bits that starts at bit l * seg.  Codes
// resynchronise within a few codes from a wrong start, so a lane first walks
// the `pre` bits before its piece, from the block's start where that lies
// inside them and else from an arbitrary bit, and takes the bit where it
// arrives as its start.  Then every lane hands the bit where its last code
// ended to the next, and lanes whose start was another walk again until none
// is: lane 0 is right, so each round fixes at least one more lane, and 0.1
// (BRC 0-2) to 2 (BRC 4) rounds are enough on average.  A prefix sum over the
// lanes' code counts then places every symbol.  The pieces hold at most 7
// codes (the shortest take 2 bits for BRC 0-2, 3 for BRC 3-4) and 32 of them
// about one block: seg = 12, 12, 14, 16, 18 bits for BRC 0..4.  Where a block
// takes more than 32 pieces the rest of it follows the same way.
//
// The reconstruction runs as soon as a channel pair is there: the even
// samples are (IE, QE) and the odd ones (IO, QO), so only the symbols of IE
// and IO wait in shared memory (2 bytes a quad) and no symbol goes through
// global memory.  Values come from a 16-entry table per block (the products
// of the reconstruction level and the sigma factor, formed in FP64).
//
// Bound by the latency of this chain: ~520 instructions and ~3300 cycles a
// block with 2.4 warps per scheduler in a 1500-packet burst.  1500 packets of
// 12000 samples: 0.30 ms, where a thread per packet and a second kernel for
// the values took 2.0 + 0.22 ms (6.2 ms through the allocation-free call, in
// three chunks of a fixed scratch array).  The walk with branches in place of
// selects took 0.39 ms, without the run-up 0.43, and a table of jumps over 16
// codes from every bit (no guesses, but 250 shared-memory accesses a block)
// 0.99.
constexpr int kDecodeWarps = 4;
constexpr int kRingWords = 256;      // the packet's words around the walk (1 KB per warp)
constexpr int kMaxBlocks = 512;      // nq <= 65535

// shared memory of one warp, before its 2 * sym_pitch(nq) symbol bytes
struct DecodeWarp {
    double tab64[16];
    float tab32[16];
    uint32_t ring[kRingWords];
    uint8_t stage[128];
    uint8_t brc[kMaxBlocks];
    uint8_t thidx[kMaxBlocks];
};
struct DecodeShared {
    double norm[5][16];
    HuffEntry lut[5 * kHuffWindow];
};
static_assert(sizeof(DecodeWarp) % 16 == 0 && sizeof(DecodeShared) % 16 == 0, "16-byte rows");

__host__ __device__ inline size_t decode_warp_bytes(int nq) {
    return sizeof(DecodeWarp) + (((size_t)2 * sym_pitch(nq) + 15) & ~(size_t)15);
}
static size_t decode_smem(int nq, int warps) { return sizeof(DecodeShared) + warps * decode_warp_bytes(nq); }

// The packet's user data as big-endian bits.  Bit positions count from the
// aligned 32-bit word that holds the first byte.  Words stream into the ring
// by cp.async, 32 per step and at least three steps ahead of the walk; only
// aligned words that end inside the data are copied (the first may begin up
// to 3 bytes before it, inside the packet header), the others are assembled
// byte by byte with zeros past `avail`: nothing past the data is read.
struct PacketBits {
    const uint8_t* u;
    int avail;
    int mis;                 // bytes from the aligned word to u
    const uint32_t* wbase;
    uint32_t* ring;
    int filled;              // words asked for so far

    // make words [.., upto) readable by every lane
    __device__ __forceinline__ void fill(int upto, int lane) {
        __syncwarp();        // the slots written next have been read
        while (filled < upto + 96) {
            const int kw = filled + lane;
            uint32_t* slot = ring + (kw & (kRingWords - 1));
            const int end = 4 * kw + 4 - mis;   // bytes of u up to the end of word kw
            if (end <= avail) {
                const unsigned sa = (unsigned)__cvta_generic_to_shared(slot);
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(wbase + kw) : "memory");
            } else {
                uint32_t v = 0;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int at = end - 4 + i;
                    if (at >= 0 && at < avail) v |= (uint32_t)u[at] << (8 * i);
                }
                *slot = v;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            filled += 32;
        }
        asm volatile("cp.async.wait_group 3;" ::: "memory");
        __syncwarp();
    }
    __device__ __forceinline__ uint32_t word(int k) const {
        return __byte_perm(ring[k & (kRingWords - 1)], 0, 0x0123);
    }
    __device__ __forceinline__ uint32_t top32(int bit) const {
        return __funnelshift_l(word((bit >> 5) + 1), word(bit >> 5), bit & 31);
    }
};

// Rows of out32 (F32) and out64 (F64): out[2k] = IE_k + i QE_k,
// out[2k+1] = IO_k + i QO_k; a packet that failed gets a zero row.
template <bool F32, bool F64>
__global__ void __launch_bounds__(32 * kDecodeWarps) k_decode_fdbaq(const uint8_t* __restrict__ s, long long n,
                                                        const long long* __restrict__ offsets, DecodeSpec spec,
                                                        cf32* __restrict__ out32, cf64* __restrict__ out64,
                                                        int* __restrict__ status, int nq_max,
                                                        const HuffEntry* __restrict__ lut_g, int* __restrict__ any) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    DecodeShared& sh = *reinterpret_cast<DecodeShared*>(smem_raw);
    for (int i = threadIdx.x; i < 5 * kHuffWindow / 2; i += blockDim.x)
        reinterpret_cast<uint32_t*>(sh.lut)[i] = reinterpret_cast<const uint32_t*>(lut_g)[i];
    for (int i = threadIdx.x; i < 80; i += blockDim.x) sh.norm[i >> 4][i & 15] = c_norm[i >> 4][i & 15];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j = blockIdx.x * (blockDim.x >> 5) + warp;
    if (j >= spec.njobs) return;
    DecodeWarp& w = *reinterpret_cast<DecodeWarp*>(smem_raw + sizeof(DecodeShared) + warp * decode_warp_bytes(nq_max));
    uint8_t* sym = reinterpret_cast<uint8_t*>(&w + 1);
    const DecodeJob jb = job_at(spec, j);
    const int nq = jb.nq;
    const long long off = offsets[jb.pk];
    int st = 0;
    // the 68 header bytes must lie inside the stream before any is read
    // (offsets can come from the caller, not only from the indexer)
    const bool inside = off >= 0 && off <= n - 68;
    const uint8_t* hdr = s + (inside ? off : 0);
    long long ulen = -1;
    if (inside) {
        ulen = (((long long)hdr[4] << 8) | hdr[5]) + 1 - 62;
        const int pnq = (hdr[6 + 59] << 8) | hdr[6 + 60];
        if (ulen < 0) st = S1G_E_PACKET_LENGTH;
        else if (pnq != nq) st = S1G_E_RAGGED_BURST;
    } else {
        st = S1G_E_PACKET_LENGTH;
    }
    if (!st) {
        const int nb = (2 * nq + 255) / 256;
        const int sp = sym_pitch(nq);
        PacketBits pb;
        pb.u = hdr + 68;
        // bytes actually present (a truncated last packet reads as zeros)
        pb.avail = (int)max(0LL, min(ulen, n - (off + 68)));
        pb.mis = (int)((uintptr_t)pb.u & 3);
        pb.wbase = reinterpret_cast<const uint32_t*>((uintptr_t)pb.u & ~(uintptr_t)3);
        pb.ring = w.ring;
        pb.filled = 0;
        const int bit0 = 8 * pb.mis;
        const int uend = bit0 + (int)ulen * 8;   // user data: below 65536 bytes
        int bit = bit0;
        for (int ch = 0; ch < 4 && !st; ++ch) {
            for (int b = 0; b < nb && !st; ++b) {
                // the largest head (8 bits), 32 pieces of 18 bits and the window of the last one
                pb.fill(((bit + 8 + 32 * 18) >> 5) + 4, lane);
                int brc;
                if (ch == 0) {
                    if (bit + 3 > uend) { st = S1G_E_READ_PAST_END; break; }
                    brc = (int)(pb.top32(bit) >> 29);
                    if (brc > 4) { st = S1G_E_BAD_BRC; break; }
                    if (lane == 0) w.brc[b] = (uint8_t)brc;
                    bit += 3;
                } else {
                    brc = w.brc[b];
                    if (ch == 2) {
                        if (bit + 8 > uend) { st = S1G_E_READ_PAST_END; break; }
                        if (lane == 0) w.thidx[b] = (uint8_t)(pb.top32(bit) >> 24);
                        bit += 8;
                    }
                }
                const HuffEntry* L = sh.lut + brc * kHuffWindow;
                const int seg = brc <= 1 ? 12 : brc == 2 ? 14 : brc == 3 ? 16 : 18;
                const int pre = brc <= 2 ? seg : 24;
                const int cnt = (b == nb - 1) ? nq - 128 * (nb - 1) : 128;
                uint8_t* dst = ch < 2 ? sym + ch * sp + 128 * b : w.stage;
                int done = 0;
                while (done < cnt) {
                    if (done) pb.fill(((bit + 32 * 18) >> 5) + 4, lane);
                    const int p = bit + lane * seg;
                    const uint32_t w0 = pb.word(p >> 5), w1 = pb.word((p >> 5) + 1), w2 = pb.word((p >> 5) + 2);
                    const uint32_t hi = __funnelshift_l(w1, w0, p & 31), lo = __funnelshift_l(w2, w1, p & 31);
                    int start = 0;
                    {
                        // the bits before the piece; a lane whose run-up begins at
                        // or before the block's first bit starts there
                        const int r = p - pre;
                        const uint32_t v0 = pb.word(r >> 5);
                        const uint32_t v1 = (r >> 5) + 1 == (p >> 5) ? w0 : w1;
                        const uint32_t v2 = (r >> 5) + 1 == (p >> 5) ? w1 : w2;
                        const uint32_t ph = __funnelshift_l(v1, v0, r & 31), pl = __funnelshift_l(v2, v1, r & 31);
                        int o = max(0, pre - lane * seg);
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int step = L[__funnelshift_l(pl, ph, o) >> 22] >> 8;
                            o += o < pre ? step : 0;
                        }
                        start = lane == 0 ? 0 : o - pre;
                    }
                    // symbols and code ends of the piece, a byte each; what follows
                    // its c codes is not used
                    uint32_t sa = 0, sb = 0, ea = 0, eb = 0;
                    int c;
                    auto walk = [&](int o) {
                        c = 0;
#pragma unroll
                        for (int i = 0; i < 7; ++i) {
                            const uint32_t e = L[__funnelshift_l(lo, hi, o) >> 22];
                            const bool on = o < seg;
                            o += on ? (int)(e >> 8) : 0;
                            c += on ? 1 : 0;
                            // byte i & 3 of the pair of words
                            const int at = 4 * (i & 3);
                            const int sel = (0x3210 & ~(15 << at)) | (4 << at);
                            uint32_t& sy = i < 4 ? sa : sb;
                            uint32_t& en = i < 4 ? ea : eb;
                            sy = __byte_perm(sy, e, sel);
                            en = __byte_perm(en, (uint32_t)o, sel);
                        }
                        return o - seg;
                    };
                    int left = walk(start);
                    for (int round = 0; round < 32; ++round) {
                        int ns = __shfl_up_sync(0xffffffffu, left, 1);
                        if (lane == 0) ns = 0;
                        if (__all_sync(0xffffffffu, ns == start)) break;
                        start = ns;
                        left = walk(ns);
                    }
                    // codes before the piece and in all of them (1 to 7 each: three bits)
                    const unsigned c0 = __ballot_sync(0xffffffffu, c & 1), c1 = __ballot_sync(0xffffffffu, c & 2),
                                   c2 = __ballot_sync(0xffffffffu, c & 4), lt = (1u << lane) - 1;
                    const int excl = __popc(c0 & lt) + 2 * __popc(c1 & lt) + 4 * __popc(c2 & lt);
                    const int total = __popc(c0) + 2 * __popc(c1) + 4 * __popc(c2);
                    const int rem = cnt - done;
                    const int lim = min(c, rem - excl);   // codes of this piece that belong to the block
                    uint8_t* to = dst + done + excl;
#pragma unroll
                    for (int i = 0; i < 7; ++i)
                        if (i < lim) to[i] = (uint8_t)((i < 4 ? sa : sb) >> (8 * (i & 3)));
                    // the bit behind the last of them
                    const int k = max(lim - 1, 0);
                    const int end = lane * seg + (int)(((k < 4 ? ea : eb) >> (8 * (k & 3))) & 255u);
                    bit += __reduce_max_sync(0xffffffffu, lim > 0 ? end : 0);
                    done += min(total, rem);
                }
                // the reference reads the codes one width at a time, all inside
                // the user data (decoding_utils.cpp:107-119)
                if (bit > uend) { st = S1G_E_READ_PAST_END; break; }
                if (ch >= 2) {
                    __syncwarp();
                    const int th = w.thidx[b];
                    if (lane < 16) {
                        // m <= the BRC's comparison flag for every code of its tree
                        double v;
                        if (th <= c_brc_thidx[brc]) v = lane == c_brc_mcode[brc] ? c_simple[brc][th] : (double)lane;
                        else v = sh.norm[brc][lane] * c_sf[th];
                        if (F64) w.tab64[lane] = v;
                        if (F32) w.tab32[lane] = (float)v;
                    }
                    __syncwarp();
                    const uint8_t* re = sym + (ch - 2) * sp + 128 * b;
                    const long long at = jb.out + 256LL * b + (ch - 2);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int q = lane + 32 * i;
                        if (q < cnt) {
                            const int x = re[q], y = w.stage[q];
                            if (F32) {
                                const float a = w.tab32[x & 15], c = w.tab32[y & 15];
                                out32[at + 2 * q] = mk(x & 128 ? -a : a, y & 128 ? -c : c);
                            }
                            if (F64) {
                                const double a = w.tab64[x & 15], c = w.tab64[y & 15];
                                out64[at + 2 * q] = mk(x & 128 ? -a : a, y & 128 ? -c : c);
                            }
                        }
                    }
                }
                __syncwarp();
            }
            bit += -(bit - bit0) & 15;   // channels end on 16-bit words
        }
        asm volatile("cp.async.wait_all;" ::: "memory");   // no copy outlives the walk
    }
    if (st)
        for (int k = lane; k < 2 * nq; k += 32) {
            if (F32) out32[jb.out + k] = mk(0.f, 0.f);
            if (F64) out64[jb.out + k] = mk(0.0, 0.0);
        }
    if (lane == 0) {
        status[j] = st;
        if (st && any) *any = 1;
    }
}

static void launch_fdbaq(const uint8_t* d_stream, long long n, const long long* d_offsets, const DecodeSpec& spec,
                         cf32* out32, cf64* out64, int* d_status, int nq_max, const void* d_lut, cudaStream_t st,
                         int* any = nullptr) {
    // one warp per CTA where the symbols of kDecodeWarps packets do not fit (nq above ~25000)
    const int warps = decode_smem(nq_max, kDecodeWarps) <= (size_t)kSmemBytes ? kDecodeWarps : 1;
    const size_t smem = decode_smem(nq_max, warps);
    auto go = [&](auto kernel) {
        if (smem > 48 * 1024)
            check_cuda(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes), "attr");
        note_launch(), kernel<<<(spec.njobs + warps - 1) / warps, 32 * warps, smem, st>>>(
            d_stream, n, d_offsets, spec, out32, out64, d_status, nq_max, (const HuffEntry*)d_lut, any);
    };
    if (out32 && out64) go(k_decode_fdbaq<true, true>);
    else if (out64) go(k_decode_fdbaq<false, true>);
    else go(k_decode_fdbaq<true, false>);
}

// ------------------------------------------------------------------ formats A, B, C
// Bypass (formats A/B, baq_mode 0) and BAQ (format C, baq_mode 3/4/5)
// packets have fixed-length fields, so every sample is found by arithmetic:
// one block per packet, one thread per quad.
//   A/B: channel c (IE, IO, QE, QO) at c * W, W = 10 nq rounded up to 16;
//        sample q = sign bit + 9-bit magnitude at 10 q (packet.cpp:519-538).
//   C:   sample = sign bit + (M-1)-bit code, M = baq_mode, in blocks of 128
//        quads; every QE block starts with an 8-bit THIDX; channels padded to
//        16 bits (packet.cpp:622-666); reconstruction _get_s_values_type_c
//        (packet.cpp:548-564) with the BAQ rows of the tables.
// With `fields` == 0 the output is the reference's: its decoders append the
// codes to containers that already hold zero entries (H_CODE() with 128,
// H_CODE(n) with n, QUAD(key, n) with n default blocks) and then read the
// leading entries, so for A/B quad q carries the codes of quad q - 128 (zero
// below 128) and for C every sample of a block is the reconstruction of
// sign 0, code 0 at that block's THIDX.  With `fields` == 1 every sample is
// decoded from its own bits.  Either way the packet must hold every bit the
// reference reads, else S1G_E_READ_PAST_END.  FDBAQ rows are left alone.
__constant__ double c_baq_simple[3][17] = {
    {3.00, 3.00, 3.12, 3.55},
    {7.00, 7.00, 7.00, 7.17, 7.40, 7.76},
    {15.00, 15.00, 15.00, 15.00, 15.00, 15.00, 15.44, 15.56, 16.11, 16.38, 16.65},
};
__constant__ double c_baq_norm[3][16] = {
    {0.2490, 0.7680, 1.3655, 2.1864},
    {0.1290, 0.3900, 0.6601, 0.9471, 1.2623, 1.6261, 2.0793, 2.7467},
    {0.0660, 0.1985, 0.3320, 0.4677, 0.6061, 0.7487, 0.8964, 1.0510, 1.2143, 1.3896, 1.5800, 1.7914, 2.0329,
     2.3234, 2.6971, 3.2692},
};
__constant__ int c_baq_thidx[3] = {3, 7, 15};
__constant__ int c_baq_mcode[3] = {3, 5, 10};

// n <= 25 bits at bit position `bit` of u (bytes at or past `avail` read as 0)
__device__ __forceinline__ uint32_t read_field(const uint8_t* u, long long avail, long long bit, int n) {
    const long long by = bit >> 3;
    uint32_t w = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) w = (w << 8) | (by + i < avail ? (uint32_t)u[by + i] : 0u);
    return (w << (bit & 7)) >> (32 - n);
}

__device__ __forceinline__ long long align16(long long b) { return (b + 15) & ~15LL; }

template <typename R>
__global__ void __launch_bounds__(256) k_decode_fixed(const uint8_t* __restrict__ s, long long n,
                                                      const long long* __restrict__ offsets, DecodeSpec spec,
                                                      cpx<R>* __restrict__ out, int* __restrict__ status, int fields) {
    __shared__ int bad;
    const int j = blockIdx.x;
    const DecodeJob jb = job_at(spec, j);
    const long long off = offsets[jb.pk];
    if (off < 0 || off > n - 68) {           // header outside the stream
        if (threadIdx.x == 0) status[j] = S1G_E_PACKET_LENGTH;
        for (int k = threadIdx.x; k < 2 * jb.nq; k += blockDim.x) out[jb.out + k] = mk((R)0, (R)0);
        return;
    }
    const uint8_t* hdr = s + off;
    const int baq = hdr[37] & 31;            // baq_mode: bits 299..303 of the header
    if (baq >= 12 && baq <= 14) return;      // FDBAQ: the type-D decoder's row
    const int nq = jb.nq;
    cpx<R>* row = out + jb.out;
    const long long pdl = ((long long)hdr[4] << 8) | hdr[5];
    const long long ulen = pdl + 1 - 62;
    long long avail = n - (off + 68);
    if (avail > ulen) avail = ulen;
    if (avail < 0) avail = 0;
    const int pnq = (hdr[6 + 59] << 8) | hdr[6 + 60];
    const int M = baq;
    const int nb = (2 * nq + 255) / 256;
    // bit offsets of the channels and the last bit the reference reads
    long long w = 0, cw = 0, qe = 0, need = 0;
    int st = 0;
    if (ulen < 0) st = S1G_E_PACKET_LENGTH;
    else if (pnq != nq) st = S1G_E_RAGGED_BURST;
    else if (baq == 0) {
        w = align16(10LL * nq);
        need = 3 * w + 10LL * nq;
    } else if (baq >= 3 && baq <= 5) {
        cw = align16((long long)M * nq);
        qe = align16(8LL * nb + (long long)M * nq);
        need = 2 * cw + qe + (long long)M * nq;
    } else {
        st = S1G_E_BAD_FORMAT;
    }
    if (!st && need > 8 * ulen) st = S1G_E_READ_PAST_END;
    if (threadIdx.x == 0) bad = st;
    __syncthreads();
    const uint8_t* u = hdr + 68;
    if (bad == 0) {
        for (int q = threadIdx.x; q < nq; q += blockDim.x) {
            double v[4] = {0.0, 0.0, 0.0, 0.0};
            bool err = false;
            if (baq == 0) {
                const int src = fields ? q : q - 128;
                if (src >= 0) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t x = read_field(u, avail, c * w + 10LL * src, 10);
                        v[c] = ((x >> 9) ? -1.0 : 1.0) * (double)(x & 511u);
                    }
                }
            } else {
                const int b = q >> 7;
                const int th = (int)read_field(u, avail, 2 * cw + (long long)b * (8 + 128 * M), 8);
                const int lim = c_baq_thidx[M - 3], flag = c_baq_mcode[M - 3];
                if (!fields) {
                    const double x = th <= lim ? 0.0 : c_baq_norm[M - 3][0] * c_sf[th];
                    v[0] = v[1] = v[2] = v[3] = x;
                } else {
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const long long start = c == 0 ? 0 : c == 1 ? cw : c == 2 ? 2 * cw : 2 * cw + qe;
                        const long long pos = start + (c == 2 ? 8LL * (b + 1) : 0) + (long long)M * q;
                        const uint32_t x = read_field(u, avail, pos, M);
                        const double sg = (x >> (M - 1)) ? -1.0 : 1.0;
                        const int m = (int)(x & ((1u << (M - 1)) - 1));
                        if (th <= lim) {
                            if (m < flag) v[c] = sg * (double)m;
                            else if (m == flag) v[c] = sg * c_baq_simple[M - 3][th];
                            else err = true;
                        } else {
                            v[c] = sg * c_baq_norm[M - 3][m] * c_sf[th];
                        }
                    }
                }
            }
            if (err) atomicExch(&bad, S1G_E_MCODE);
            row[2 * q] = mk((R)v[0], (R)v[2]);
            row[2 * q + 1] = mk((R)v[1], (R)v[3]);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) status[j] = bad;
    if (bad != 0)
        for (int k = threadIdx.x; k < 2 * nq; k += blockDim.x) row[k] = mk((R)0, (R)0);
}

static void build_lut(std::vector<HuffEntry>& lut) {
    // value-keyed maps of structs.h:170-227 (key value -> mcode) and the
    // start lengths of structs.h:170; the walk of decoding_utils.cpp:44-77
    static const int keys[5][16][2] = {
        {{0, 0}, {2, 1}, {6, 2}, {7, 3}},
        {{0, 0}, {2, 1}, {6, 2}, {14, 3}, {15, 4}},
        {{0, 0}, {2, 1}, {6, 2}, {14, 3}, {30, 4}, {62, 5}, {63, 6}},
        {{0, 0}, {1, 1}, {2, 2}, {6, 3}, {14, 4}, {30, 5}, {62, 6}, {126, 7}, {254, 8}, {255, 9}},
        {{0, 0}, {2, 1}, {3, 2}, {4, 3}, {5, 4}, {12, 5}, {13, 6}, {14, 7}, {30, 8}, {62, 9},
         {252, 10}, {253, 11}, {508, 12}, {509, 13}, {510, 14}, {511, 15}},
    };
    static const int nkeys[5] = {4, 5, 7, 10, 16};
    static const int start[5] = {1, 1, 1, 2, 2};
    lut.assign(5 * kHuffWindow, 0);
    for (int brc = 0; brc < 5; ++brc) {
        for (int w = 0; w < kHuffWindow / 2; ++w) {
            auto bits = [&](int len) { return (w >> (9 - len)) & ((1 << len) - 1); };
            int len = start[brc];
            int mcode = 0, clen = 0;
            if (brc == 4 && bits(2) == 0) {
                clen = 2;
            } else {
                if (brc == 4) len += 1;
                for (; len <= 9 && !clen; ++len) {
                    const int v = bits(len);
                    for (int k = 0; k < nkeys[brc]; ++k)
                        if (keys[brc][k][0] == v) {
                            mcode = keys[brc][k][1];
                            clen = len;
                        }
                }
            }
            if (!clen) throw std::runtime_error("FDBAQ table: a bit window without a code");
            for (int sign = 0; sign < 2; ++sign)
                lut[brc * kHuffWindow + (sign << 9) + w] = (HuffEntry)(((1 + clen) << 8) | (sign << 7) | mcode);
        }
    }
}

size_t huffman_lut_bytes() { return sizeof(HuffEntry) * 5 * kHuffWindow; }

void huffman_lut_fill(void* host_dst) {
    std::vector<HuffEntry> h;
    build_lut(h);
    memcpy(host_dst, h.data(), sizeof(HuffEntry) * h.size());
}

// Decode npk packets (offsets d_offsets[0 .. npk)) into FP32 rows with a device
// copy of the Huffman table; allocates nothing and uses no global scratch.
void decode_fp32_uniform(const uint8_t* d_stream, long long n, const long long* d_offsets, int npk, int nq, cf32* out,
                         long long pitch, int* d_status, const void* d_lut, cudaStream_t st) {
    const DecodeSpec spec{nullptr, npk, nullptr, 0, nq, pitch};
    launch_fdbaq(d_stream, n, d_offsets, spec, out, nullptr, d_status, nq, d_lut, st);
}

DecodeTables::~DecodeTables() {
    if (lut) cudaFree(lut);
}

void DecodeTables::init() {
    if (lut) return;
    std::vector<HuffEntry> h;
    build_lut(h);
    check_cuda(cudaMalloc(&lut, sizeof(HuffEntry) * h.size()), "lut");
    upload_table(lut, h.data(), sizeof(HuffEntry) * h.size(), "lut up");
}

template <typename R>
void decode_burst(const uint8_t* d_stream, long long n, const long long* d_offsets, const int* d_pkidx, int p0,
                  int npk, int nq, cpx<R>* out, long long pitch, int* d_status, const DecodeTables& tabs,
                  cudaStream_t st, int* any) {
    const DecodeSpec spec{nullptr, npk, d_pkidx, p0, nq, pitch};
    if constexpr (sizeof(R) == 4) launch_fdbaq(d_stream, n, d_offsets, spec, out, nullptr, d_status, nq, tabs.lut, st, any);
    else launch_fdbaq(d_stream, n, d_offsets, spec, nullptr, out, d_status, nq, tabs.lut, st, any);
}

__global__ void k_any_status(const int* __restrict__ status, int n, int* __restrict__ any) {
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (status[i]) *any = 1;
}
void any_status(const int* d_status, int n, int* any, cudaStream_t st) {
    note_launch(), k_any_status<<<1, 256, 0, st>>>(d_status, n, any);
}

void decode_jobs(const uint8_t* d_stream, long long n, const long long* d_offsets, const DecodeJob* d_jobs, int njobs,
                 int nq_max, cf32* out32, cf64* out64, int* d_status, const DecodeTables& tabs, cudaStream_t st) {
    if (njobs <= 0) return;
    const DecodeSpec spec{d_jobs, njobs, nullptr, 0, 0, 0};
    launch_fdbaq(d_stream, n, d_offsets, spec, out32, out64, d_status, nq_max, tabs.lut, st);
}

template <typename R>
void decode_fixed_burst(const uint8_t* d_stream, long long n, const long long* d_offsets, const int* d_pkidx, int p0,
                        int npk, int nq, cpx<R>* out, long long pitch, int* d_status, int fields, cudaStream_t st) {
    if (npk <= 0) return;
    const DecodeSpec spec{nullptr, npk, d_pkidx, p0, nq, pitch};
    note_launch(), k_decode_fixed<R><<<npk, 256, 0, st>>>(d_stream, n, d_offsets, spec, out, d_status, fields);
}

template <typename R>
void decode_fixed_jobs(const uint8_t* d_stream, long long n, const long long* d_offsets, const DecodeJob* d_jobs,
                       int njobs, cpx<R>* out, int* d_status, int fields, cudaStream_t st) {
    if (njobs <= 0) return;
    const DecodeSpec spec{d_jobs, njobs, nullptr, 0, 0, 0};
    note_launch(), k_decode_fixed<R><<<njobs, 256, 0, st>>>(d_stream, n, d_offsets, spec, out, d_status, fields);
}

template void decode_fixed_burst<float>(const uint8_t*, long long, const long long*, const int*, int, int, int,
                                        cpx<float>*, long long, int*, int, cudaStream_t);
template void decode_fixed_burst<double>(const uint8_t*, long long, const long long*, const int*, int, int, int,
                                         cpx<double>*, long long, int*, int, cudaStream_t);
template void decode_fixed_jobs<float>(const uint8_t*, long long, const long long*, const DecodeJob*, int,
                                       cpx<float>*, int*, int, cudaStream_t);
template void decode_fixed_jobs<double>(const uint8_t*, long long, const long long*, const DecodeJob*, int,
                                        cpx<double>*, int*, int, cudaStream_t);

template void decode_burst<float>(const uint8_t*, long long, const long long*, const int*, int, int, int, cpx<float>*,
                                  long long, int*, const DecodeTables&, cudaStream_t, int*);
template void decode_burst<double>(const uint8_t*, long long, const long long*, const int*, int, int, int,
                                   cpx<double>*, long long, int*, const DecodeTables&, cudaStream_t, int*);

}  // namespace s1g
