// Records (canonical key, 8 multiplicities) in key order on the device, for
// the copies of a graph to the host that ask for it, and for the merge's lines.
// Hand-written, by size: one block orders up to kOne records in one launch; up
// to kSplitMost are scattered to buckets between sampled splitters and ordered
// by a block a bucket, in three launches; more, or a bucket that outgrows its
// region, take a stable least-significant-digit radix sort, 8 bits a pass over
// the 2k bits of a key. The first two are bound by launches and a block's steps,
// a radix pass by memory: it reads the keys twice and the records once and
// writes them once (40 bytes a record).
#include <cuda_runtime.h>

#include <algorithm>

#include "dev_util.cuh"
#include "kmer_dev.cuh"
#include "swg_internal.h"
#include "text_dev.cuh"

namespace swg {
namespace {

constexpr uint32_t kOne = 1024;         // records one block orders alone
constexpr uint32_t kRoom = 4096;        // records one block can order
constexpr int kDigits = 256;
constexpr int kItems = 16;              // records per thread of a pass
constexpr uint32_t kTile = 256 * kItems;

// Bitonic sort of m (a power of two, at most 1024 R) keys by 1024 threads;
// thread t holds keys R t .. R t + R - 1, with an index each. Partners at a
// distance below R are in the thread, below 32 R in the warp (shuffles), the
// others go through shared memory (a sort of 4096 has 15 such steps of 78; all
// 78 through shared memory took 40 us, the launch included).
template <int R, bool kIdx>
__device__ __forceinline__ void bitonic(unsigned long long (&v)[R], unsigned (&ix)[R], unsigned long long *sk,
                                        unsigned short *si, uint32_t m) {
    const uint32_t t = threadIdx.x, e0 = t * R;
    for (uint32_t k = 2; k <= m; k <<= 1)
        for (uint32_t j = k >> 1; j; j >>= 1) {
            if (j < R) {
#pragma unroll
                for (int jj = R / 2; jj; jj >>= 1) {
                    if (j != (uint32_t)jj) continue;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        if (r & jj) continue;
                        if ((v[r] > v[r | jj]) == (((e0 + r) & k) == 0)) {
                            const unsigned long long x = v[r];
                            v[r] = v[r | jj];
                            v[r | jj] = x;
                            const unsigned u = ix[r];
                            ix[r] = ix[r | jj];
                            ix[r | jj] = u;
                        }
                    }
                }
                continue;
            }
            const uint32_t d = j / R;
            const bool least = ((e0 & k) == 0) == ((t & d) == 0);  // this side keeps the smaller key
            if (d >= 32) {
                __syncthreads();
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    sk[r * 1024 + t] = v[r];
                    if (kIdx) si[r * 1024 + t] = (unsigned short)ix[r];
                }
                __syncthreads();
            }
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const unsigned long long y = d < 32 ? __shfl_xor_sync(0xffffffffu, v[r], d) : sk[r * 1024 + (t ^ d)];
                const unsigned u = !kIdx ? 0 : (d < 32 ? __shfl_xor_sync(0xffffffffu, ix[r], d) : si[r * 1024 + (t ^ d)]);
                if ((v[r] > y) == least) {
                    v[r] = y;
                    ix[r] = u;
                }
            }
        }
}

// n <= kRoom records ordered by one block: the keys with their index, the
// multiplicities after it. Padded with the largest key.
template <int R>
__device__ __forceinline__ void sort_block_of(unsigned long long *sk, unsigned short *si,
                                              const unsigned long long *__restrict__ keys,
                                              const unsigned long long *__restrict__ mult, uint32_t n, uint32_t m,
                                              unsigned long long *__restrict__ okeys,
                                              unsigned long long *__restrict__ omult) {
    unsigned long long v[R];
    unsigned ix[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        ix[r] = threadIdx.x * R + r;
        v[r] = ix[r] < n ? keys[ix[r]] : ~0ull;
    }
    bitonic<R, true>(v, ix, sk, si, m);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t i = threadIdx.x * R + r;
        if (i < n) {
            okeys[i] = v[r];
            omult[i] = mult[ix[r]];
        }
    }
}

// As few keys a thread as hold them all: the steps' latency counts here.
__device__ __forceinline__ void sort_block(unsigned long long *sk, unsigned short *si,
                                           const unsigned long long *__restrict__ keys,
                                           const unsigned long long *__restrict__ mult, uint32_t n,
                                           unsigned long long *__restrict__ okeys,
                                           unsigned long long *__restrict__ omult) {
    uint32_t m = 32;
    while (m < n) m <<= 1;
    if (m <= 1024) sort_block_of<1>(sk, si, keys, mult, n, m, okeys, omult);
    else if (m <= 2048) sort_block_of<2>(sk, si, keys, mult, n, m, okeys, omult);
    else sort_block_of<kRoom / 1024>(sk, si, keys, mult, n, m, okeys, omult);
}

__global__ void __launch_bounds__(1024) k_sort_one(const unsigned long long *__restrict__ keys,
                                                   const unsigned long long *__restrict__ mult, uint32_t n,
                                                   unsigned long long *__restrict__ okeys,
                                                   unsigned long long *__restrict__ omult) {
    __shared__ unsigned long long sk[kRoom];
    __shared__ unsigned short si[kRoom];
    sort_block(sk, si, keys, mult, n, okeys, omult);
}

// ---- splitters: nb buckets of kMean records on average (a block's sort of
// twice as many takes three times as long: its steps are bound by shuffles),
// from a sample of kOver keys a bucket at even strides (the keys are distinct,
// so that the quantiles of any distribution are splitters; at 4 sampled keys a
// bucket one of 8 times the mean, which would not fit its region, has odds of
// 1e-10). Such a bucket sets *over, and the records take the radix passes.
constexpr uint32_t kMean = 512, kOver = 4, kSplitBuckets = 2048;
constexpr uint64_t kSplitMost = (uint64_t)kMean * kSplitBuckets;
constexpr uint32_t kSampleMost = kOver * kSplitBuckets;

template <int R>
__device__ __forceinline__ void split_of(unsigned long long *sk, const unsigned long long *__restrict__ keys, uint64_t n,
                                         uint32_t count, uint32_t m, unsigned long long *__restrict__ splitters) {
    const uint64_t step = (n << 20) / count;  // n <= 2^20, the index below 2^13
    unsigned long long v[R];
    unsigned ix[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const uint32_t i = threadIdx.x * R + r;
        v[r] = i < count ? keys[(i * step) >> 20] : ~0ull;
        ix[r] = 0;
    }
    bitonic<R, false>(v, ix, sk, nullptr, m);
#pragma unroll
    for (int r = 0; r < R; ++r) {  // bucket b: from splitters[b] (0: from the start) to splitters[b + 1]
        const uint32_t e = threadIdx.x * R + r;
        if (e < count && e % kOver == 0) splitters[e / kOver] = v[r];
    }
}

__global__ void __launch_bounds__(1024) k_sort_split(const unsigned long long *__restrict__ keys, uint64_t n, uint32_t nb,
                                                     unsigned long long *__restrict__ splitters,
                                                     unsigned *__restrict__ cursor, unsigned *__restrict__ over) {
    extern __shared__ __align__(16) unsigned char dyn[];
    unsigned long long *sk = reinterpret_cast<unsigned long long *>(dyn);
    const uint32_t count = kOver * nb;
    uint32_t m = 32;
    while (m < count) m <<= 1;
    if (m <= 1024) split_of<1>(sk, keys, n, count, m, splitters);
    else if (m <= 2048) split_of<2>(sk, keys, n, count, m, splitters);
    else if (m <= 4096) split_of<4>(sk, keys, n, count, m, splitters);
    else split_of<8>(sk, keys, n, count, m, splitters);
    for (uint32_t b = threadIdx.x; b < nb; b += 1024) cursor[b] = 0;
    if (threadIdx.x == 0) *over = 0;
}

// Records to their buckets' regions of kRoom records each, in any order.
constexpr int kSplitItems = 8;
__global__ void __launch_bounds__(256) k_sort_scatter(const unsigned long long *__restrict__ keys,
                                                      const unsigned long long *__restrict__ mult, uint64_t n, uint32_t nb,
                                                      const unsigned long long *__restrict__ splitters,
                                                      unsigned *__restrict__ cursor, unsigned *__restrict__ over,
                                                      unsigned long long *__restrict__ bkeys,
                                                      unsigned long long *__restrict__ bmult) {
    __shared__ unsigned long long sp[kSplitBuckets];
    __shared__ unsigned hist[kSplitBuckets];
    for (uint32_t b = threadIdx.x; b < nb; b += 256) {
        sp[b] = splitters[b];
        hist[b] = 0;
    }
    __syncthreads();
    unsigned long long kv[kSplitItems];
    unsigned at[kSplitItems];  // bucket | rank << 16
    const uint64_t r0 = (uint64_t)blockIdx.x * (256 * kSplitItems) + threadIdx.x;
#pragma unroll
    for (int i = 0; i < kSplitItems; ++i) {
        const uint64_t r = r0 + 256 * i;
        kv[i] = 0;
        at[i] = 0;
        if (r < n) {
            kv[i] = keys[r];
            uint32_t lo = 0, hi = nb;
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (sp[mid] <= kv[i]) lo = mid;
                else hi = mid;
            }
            at[i] = lo | atomicAdd(&hist[lo], 1u) << 16;
        }
    }
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < nb; b += 256)
        if (hist[b]) hist[b] = atomicAdd(&cursor[b], hist[b]);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSplitItems; ++i) {
        const uint64_t r = r0 + 256 * i;
        if (r < n) {
            const uint32_t b = at[i] & 0xffffu, p = hist[b] + (at[i] >> 16);
            if (p < kRoom) {
                bkeys[(uint64_t)b * kRoom + p] = kv[i];
                bmult[(uint64_t)b * kRoom + p] = mult[r];
            } else {
                *over = 1;
            }
        }
    }
}

// Bucket blockIdx.x ordered to its place: after the buckets before it.
__global__ void __launch_bounds__(1024) k_sort_buckets(const unsigned *__restrict__ cursor,
                                                       const unsigned *__restrict__ over,
                                                       const unsigned long long *__restrict__ bkeys,
                                                       const unsigned long long *__restrict__ bmult,
                                                       unsigned long long *__restrict__ okeys,
                                                       unsigned long long *__restrict__ omult) {
    __shared__ unsigned long long sk[kRoom];
    __shared__ unsigned short si[kRoom];
    __shared__ uint64_t wb[32];
    if (*over) return;
    uint64_t before = 0, base = 0;
    for (uint32_t b = threadIdx.x; b < blockIdx.x; b += 1024) before += cursor[b];
    block_exclusive_scan<1024>(before, wb, &base);
    const uint64_t r0 = (uint64_t)blockIdx.x * kRoom;
    sort_block(sk, si, bkeys + r0, bmult + r0, cursor[blockIdx.x], okeys + base, omult + base);
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
    const uint64_t nb = (n + kMean - 1) / kMean;
    const uint64_t split = n <= kSplitMost ? 16 * n + 16 * nb * kRoom + 16 * nb + 16 : 0;
    const uint64_t nc = (n + kTile - 1) / kTile * kDigits;
    return std::max(split, 32 * n + 8 * (nc + gscan_scratch(nc) + 1));
}

uint64_t sort_device_most() { return kSplitMost; }

void sort_records_device(const unsigned long long *d_keys, const unsigned long long *d_mult, uint64_t n, cudaStream_t s,
                         void *ws, unsigned long long **keys, unsigned long long **mult, unsigned **over) {
    unsigned long long *k = static_cast<unsigned long long *>(ws), *m = k + n;
    *keys = k;
    *mult = m;
    *over = nullptr;
    if (n <= kOne) {
        k_sort_one<<<1, 1024, 0, s>>>(d_keys, d_mult, (uint32_t)n, k, m);
        return;
    }
    const uint32_t nb = (uint32_t)((n + kMean - 1) / kMean);
    unsigned long long *bk = m + n, *bm = bk + (uint64_t)nb * kRoom, *sp = bm + (uint64_t)nb * kRoom;
    unsigned *cursor = reinterpret_cast<unsigned *>(sp + nb);
    *over = cursor + nb;
    allow_smem(k_sort_split, kSampleMost * sizeof(unsigned long long));
    k_sort_split<<<1, 1024, kSampleMost * sizeof(unsigned long long), s>>>(d_keys, n, nb, sp, cursor, *over);
    k_sort_scatter<<<(unsigned)((n + 256 * kSplitItems - 1) / (256 * kSplitItems)), 256, 0, s>>>(d_keys, d_mult, n, nb, sp,
                                                                                                cursor, *over, bk, bm);
    k_sort_buckets<<<nb, 1024, 0, s>>>(cursor, *over, bk, bm, k, m);
}

// ws: sort_scratch_bytes(n) of device scratch, 8-byte aligned. The inputs are
// not touched. radix: the radix passes whatever the size.
swg_status copy_records_sorted(const unsigned long long *d_keys, const unsigned long long *d_mult, uint64_t n, int bits,
                               cudaStream_t s, void *ws, uint64_t *keys, uint8_t *mult, bool radix) {
    if (!n) return SWG_OK;
    unsigned too_large = 0;
    unsigned long long *k[2], *m[2];
    k[0] = static_cast<unsigned long long *>(ws);
    m[0] = k[0] + n;
    int at = 0;
    if (n <= kOne || (n <= kSplitMost && !radix)) {
        unsigned *over = nullptr;
        sort_records_device(d_keys, d_mult, n, s, ws, &k[0], &m[0], &over);
        EMIT_CUDA(cudaGetLastError(), "sort kernels");
        if (over)
            EMIT_CUDA(cudaMemcpyAsync(&too_large, over, sizeof(unsigned), cudaMemcpyDeviceToHost, s), "sort status");
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
    return too_large ? copy_records_sorted(d_keys, d_mult, n, bits, s, ws, keys, mult, true) : SWG_OK;
}

}  // namespace swg
