// Records (canonical key, 8 multiplicities) in key order on the device, for
// the copies of a graph to the host that ask for it. Hand-written: one block
// orders up to kOne records in shared memory in one launch; more take a
// stable least-significant-digit radix sort, 8 bits a pass over the 2k bits
// of a key. Bound by memory: a pass reads the keys twice and the records
// once and writes them once (40 bytes a record), and by launches below about
// a million records.
#include <cuda_runtime.h>

#include <algorithm>

#include "dev_util.cuh"
#include "kmer_dev.cuh"
#include "swg_internal.h"
#include "text_dev.cuh"

namespace swg {
namespace {

constexpr uint32_t kOne = 4096;         // records one block orders
constexpr int kDigits = 256;
constexpr int kItems = 16;              // records per thread of a pass
constexpr uint32_t kTile = 256 * kItems;

// Bitonic sort of the keys with their index; the multiplicities follow the
// index. Padded with the largest key.
__global__ void __launch_bounds__(1024) k_sort_one(const unsigned long long *__restrict__ keys,
                                                   const unsigned long long *__restrict__ mult, uint32_t n,
                                                   unsigned long long *__restrict__ okeys,
                                                   unsigned long long *__restrict__ omult) {
    __shared__ unsigned long long sk[kOne];
    __shared__ unsigned short si[kOne];
    uint32_t m = 32;
    while (m < n) m <<= 1;
    for (uint32_t i = threadIdx.x; i < m; i += 1024) {
        sk[i] = i < n ? keys[i] : ~0ull;
        si[i] = (unsigned short)i;
    }
    for (uint32_t k = 2; k <= m; k <<= 1)
        for (uint32_t j = k >> 1; j; j >>= 1) {
            __syncthreads();
            for (uint32_t t = threadIdx.x; t < m / 2; t += 1024) {
                const uint32_t a = 2 * t - (t & (j - 1)), b = a + j;  // the pair's lower and upper place
                const unsigned long long x = sk[a], y = sk[b];
                if ((x > y) == ((a & k) == 0)) {
                    sk[a] = y;
                    sk[b] = x;
                    const unsigned short u = si[a];
                    si[a] = si[b];
                    si[b] = u;
                }
            }
        }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += 1024) {
        okeys[i] = sk[i];
        omult[i] = mult[si[i]];
    }
}

// Records per digit of every tile, digit-major.
__global__ void __launch_bounds__(256) k_sort_hist(const unsigned long long *__restrict__ keys, uint64_t n, int shift,
                                                   uint64_t tiles, uint64_t *__restrict__ counts) {
    __shared__ unsigned hist[kDigits];
    hist[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t base = (uint64_t)blockIdx.x * kTile;
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        const uint64_t r = base + (uint64_t)i * 256 + threadIdx.x;
        if (r < n) atomicAdd(&hist[(unsigned)(keys[r] >> shift) & (kDigits - 1)], 1u);
    }
    __syncthreads();
    counts[(uint64_t)threadIdx.x * tiles + blockIdx.x] = hist[threadIdx.x];
}

// One pass: each warp ranks its 512 consecutive records within their digits
// (match.any, so that equal digits keep their order), the block orders its
// tile by digit in shared memory and writes one run per digit.
constexpr size_t kPassSmem = (size_t)kTile * 16;
__global__ void __launch_bounds__(256) k_sort_pass(const unsigned long long *__restrict__ keys,
                                                   const unsigned long long *__restrict__ mult, uint64_t n, int shift,
                                                   uint64_t tiles, const uint64_t *__restrict__ base,
                                                   unsigned long long *__restrict__ okeys,
                                                   unsigned long long *__restrict__ omult) {
    extern __shared__ __align__(16) unsigned char dyn[];
    unsigned long long *sk = reinterpret_cast<unsigned long long *>(dyn), *sm = sk + kTile;
    __shared__ unsigned wc[8][kDigits];  // records per warp and digit, then where the warp's start
    __shared__ uint64_t gbase[kDigits];  // where the tile's run of a digit goes, less its start in the tile
    __shared__ uint64_t wb[8];
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
#pragma unroll
    for (int w = 0; w < 8; ++w) wc[w][threadIdx.x] = 0;
    __syncthreads();
    const uint64_t r0 = (uint64_t)blockIdx.x * kTile + (uint64_t)wp * (32 * kItems) + lane;
    unsigned long long kv[kItems], mv[kItems];
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        const uint64_t r = r0 + 32 * i;
        kv[i] = r < n ? keys[r] : 0ull;
        mv[i] = r < n ? mult[r] : 0ull;
    }
    unsigned rank[kItems];
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        const bool in = r0 + 32 * i < n;
        const unsigned d = in ? (unsigned)(kv[i] >> shift) & (kDigits - 1) : kDigits;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const unsigned before = in ? wc[wp][d] : 0;
        __syncwarp();
        if (in && lane == __ffs(peers) - 1) wc[wp][d] = before + __popc(peers);
        __syncwarp();
        rank[i] = before + __popc(peers & ((1u << lane) - 1));
    }
    __syncthreads();
    unsigned total = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        const unsigned c = wc[w][threadIdx.x];
        wc[w][threadIdx.x] = total;
        total += c;
    }
    const unsigned start = (unsigned)block_exclusive_scan<256>((uint64_t)total, wb, nullptr);
#pragma unroll
    for (int w = 0; w < 8; ++w) wc[w][threadIdx.x] += start;
    gbase[threadIdx.x] = base[(uint64_t)threadIdx.x * tiles + blockIdx.x] - start;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
        if (r0 + 32 * i < n) {
            const unsigned p = wc[wp][(unsigned)(kv[i] >> shift) & (kDigits - 1)] + rank[i];
            sk[p] = kv[i];
            sm[p] = mv[i];
        }
    }
    __syncthreads();
    const uint32_t m = (uint32_t)(n - (uint64_t)blockIdx.x * kTile < kTile ? n - (uint64_t)blockIdx.x * kTile : kTile);
    for (uint32_t j = threadIdx.x; j < m; j += 256) {
        const unsigned long long key = sk[j];
        const uint64_t to = gbase[(unsigned)(key >> shift) & (kDigits - 1)] + j;
        okeys[to] = key;
        omult[to] = sm[j];
    }
}

}  // namespace

uint64_t sort_scratch_bytes(uint64_t n) {
    if (n <= kOne) return 16 * n;
    const uint64_t nc = (n + kTile - 1) / kTile * kDigits;
    return 32 * n + 8 * (nc + gscan_scratch(nc) + 1);
}

// ws: sort_scratch_bytes(n) of device scratch, 8-byte aligned. The inputs are
// not touched.
swg_status copy_records_sorted(const unsigned long long *d_keys, const unsigned long long *d_mult, uint64_t n, int bits,
                               cudaStream_t s, void *ws, uint64_t *keys, uint8_t *mult) {
    if (!n) return SWG_OK;
    unsigned long long *k[2], *m[2];
    k[0] = static_cast<unsigned long long *>(ws);
    m[0] = k[0] + n;
    int at = 0;
    if (n <= kOne) {
        k_sort_one<<<1, 1024, 0, s>>>(d_keys, d_mult, (uint32_t)n, k[0], m[0]);
    } else {
        k[1] = m[0] + n;
        m[1] = k[1] + n;
        const uint64_t tiles = (n + kTile - 1) / kTile, nc = tiles * kDigits;
        uint64_t *counts = reinterpret_cast<uint64_t *>(m[1] + n), *tmp = counts + nc, *total = tmp + gscan_scratch(nc);
        allow_smem(k_sort_pass, kPassSmem);
        for (int p = 0; p < (bits + 7) / 8; ++p) {
            const unsigned long long *ik = p ? k[(p - 1) & 1] : d_keys, *im = p ? m[(p - 1) & 1] : d_mult;
            at = p & 1;
            k_sort_hist<<<(unsigned)tiles, 256, 0, s>>>(ik, n, 8 * p, tiles, counts);
            launch_gscan(counts, counts, nc, tmp, total, s);
            k_sort_pass<<<(unsigned)tiles, 256, kPassSmem, s>>>(ik, im, n, 8 * p, tiles, counts, k[at], m[at]);
        }
    }
    EMIT_CUDA(cudaGetLastError(), "sort kernels");
    if (keys) EMIT_CUDA(cudaMemcpyAsync(keys, k[at], n * 8, cudaMemcpyDeviceToHost, s), "copy keys");
    if (mult) EMIT_CUDA(cudaMemcpyAsync(mult, m[at], n * 8, cudaMemcpyDeviceToHost, s), "copy multiplicities");
    EMIT_CUDA(cudaStreamSynchronize(s), "sorted copy");
    return SWG_OK;
}

}  // namespace swg
