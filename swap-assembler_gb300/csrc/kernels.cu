// sm_103a kernels of the k-mer graph build.
//
//   k_scan_*      exclusive prefix of k-mer occurrences per read
//   k_tiles       first read of every tile of kTileOcc occurrences
//   k_hll         HyperLogLog sketch of the distinct canonical k-molecules
//                 (sizes the table before the count)
//   k_count       K1: fused extraction + counting. Every thread takes one
//                 k-mer occurrence of the tile, builds its canonical
//                 k-molecule and arc slots (kmerGraph.cpp:240-296), equal
//                 keys inside a warp are merged (match.any), and one lane per
//                 key inserts or updates the open-addressing table in HBM with
//                 a 128-bit CAS on {key, 8 x uint8 counts} (saturating adds,
//                 graph.cpp:1058-1080)
//   k_compact     K2: the -c cutoff (graph.cpp:1092-1114) as one streaming
//                 pass over the table with block-level stream compaction
//   k_p1_*, k_sub_*, k_bucket_*
//                 bucketed build over single occurrences: two hash-partition
//                 scatters group their records by bucket, then one CTA per
//                 bucket counts it in a shared-memory table (super.cu has the
//                 one over super-k-mers, for odd k from 19)
//   k_probe       random-access roofline probe
//
// Every device-side retry loop is bounded; on exhaustion the kernel sets a
// status bit that the host reads after the build.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "dev_util.cuh"
#include "kmer_dev.cuh"
#include "swg_internal.h"

namespace swg {
namespace {

constexpr int kSmemReads = 512;
constexpr int kScanBlock = 256;
constexpr int kScanItems = 8;
constexpr uint64_t kScanChunk = (uint64_t)kScanBlock * kScanItems;
constexpr int kCBlock = 256;
constexpr int kCItems = 8;

// ---------------------------------------------------------------------
// Occurrence prefix: occ_prefix[r] = sum_{q<r} max(0, len[q]-k+1).
__global__ void __launch_bounds__(kScanBlock) k_scan_reduce(BuildArgs a) {
    __shared__ uint64_t wb[kScanBlock / 32];
    const uint64_t base = (uint64_t)blockIdx.x * kScanChunk;
    uint64_t s = 0;
    uint32_t longest = 0;
    for (int it = 0; it < kScanItems; ++it) {
        const uint64_t r = base + (uint64_t)it * kScanBlock + threadIdx.x;
        if (r < a.n_reads) {
            const uint32_t L = a.read_len[r];
            s += occ_of(L, k_of(a, seg_of(a, r)));
            longest = max(longest, L);
        }
    }
    uint64_t total;
    block_exclusive_scan<kScanBlock>(s, wb, &total);
    if (threadIdx.x == 0) a.scan_blocks[blockIdx.x] = total;
    if (a.max_len) {  // the longest read, for the choice of algorithm
        longest = __reduce_max_sync(kFull, longest);
        if ((threadIdx.x & 31) == 0 && longest) atomicMax(a.max_len, longest);
    }
}

// The occurrences of all reads (added to *total) and the longest read, for the
// builds that need no per-read prefix: one launch of resident blocks.
__global__ void __launch_bounds__(kScanBlock) k_occ_total(const uint32_t *__restrict__ len, uint64_t n_reads, int k,
                                                          unsigned long long *total, unsigned *longest) {
    unsigned long long s = 0;
    uint32_t most = 0;
    for (uint64_t r = (uint64_t)blockIdx.x * kScanBlock + threadIdx.x; r < n_reads; r += (uint64_t)gridDim.x * kScanBlock) {
        const uint32_t L = len[r];
        s += occ_of(L, k);
        most = max(most, L);
    }
#pragma unroll
    for (int d = 16; d; d >>= 1) s += __shfl_down_sync(kFull, s, d);
    most = __reduce_max_sync(kFull, most);
    if ((threadIdx.x & 31) == 0 && most) {
        atomicAdd(total, s);
        atomicMax(longest, most);
    }
}

__global__ void __launch_bounds__(1024) k_scan_blocks(uint64_t *block_sums, uint64_t nb,
                                                      uint64_t *occ_total) {
    __shared__ uint64_t wb[32];
    __shared__ uint64_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint64_t base = 0; base < nb; base += 1024) {
        const uint64_t i = base + threadIdx.x;
        const uint64_t v = i < nb ? block_sums[i] : 0;
        uint64_t total;
        const uint64_t ex = block_exclusive_scan<1024>(v, wb, &total);
        const uint64_t c = carry;
        if (i < nb) block_sums[i] = c + ex;
        __syncthreads();
        if (threadIdx.x == 0) carry = c + total;
        __syncthreads();
    }
    if (threadIdx.x == 0) *occ_total = carry;
}

__global__ void __launch_bounds__(kScanBlock) k_scan_write(BuildArgs a) {
    __shared__ uint64_t wb[kScanBlock / 32];
    const uint64_t base = (uint64_t)blockIdx.x * kScanChunk + (uint64_t)threadIdx.x * kScanItems;
    uint64_t v[kScanItems];
    uint64_t s = 0;
#pragma unroll
    for (int it = 0; it < kScanItems; ++it) {
        const uint64_t r = base + it;
        v[it] = r < a.n_reads ? occ_of(a.read_len[r], k_of(a, seg_of(a, r))) : 0;
        s += v[it];
    }
    uint64_t run = a.scan_blocks[blockIdx.x] + block_exclusive_scan<kScanBlock>(s, wb, nullptr);
#pragma unroll
    for (int it = 0; it < kScanItems; ++it) {
        const uint64_t r = base + it;
        if (r < a.n_reads) a.occ_prefix[r] = run;
        run += v[it];
    }
}

// First read of every tile: the read holding occurrence t*kTileOcc.
__global__ void k_tiles(const uint64_t *__restrict__ prefix, uint64_t n_reads, uint64_t n_tiles,
                        uint32_t *__restrict__ first) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_tiles) return;
    const uint64_t target = t * kTileOcc;
    uint64_t lo = 0, hi = n_reads + 1;  // upper_bound over prefix[0..n_reads]
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (prefix[mid] <= target) lo = mid + 1;
        else hi = mid;
    }
    first[t] = (uint32_t)(lo - 1);
}

// ---------------------------------------------------------------------
// Tile mapping shared by the HLL and count kernels.
struct TileSmem {
    uint64_t pre[kSmemReads + 1];
    uint64_t off[kSmemReads];
    uint32_t len[kSmemReads];
    uint32_t seg[kSmemReads];
};

struct TileView {
    uint64_t r0, nr;  // first read, reads overlapping the tile
    bool in_smem;
};

__device__ __forceinline__ TileView load_tile(const BuildArgs &a, uint64_t t, TileSmem &s) {
    TileView v;
    v.r0 = a.tile_first_read[t];
    const uint64_t r1 = (t + 1 < a.n_tiles) ? a.tile_first_read[t + 1] : a.n_reads - 1;
    v.nr = r1 - v.r0 + 1;
    v.in_smem = v.nr <= (uint64_t)kSmemReads;
    if (v.in_smem) {
        for (uint64_t j = threadIdx.x; j <= v.nr; j += blockDim.x) {
            s.pre[j] = a.occ_prefix[v.r0 + j];
            if (j < v.nr) {
                s.off[j] = a.read_off[v.r0 + j];
                s.len[j] = a.read_len[v.r0 + j];
                s.seg[j] = seg_of(a, v.r0 + j);
            }
        }
    }
    return v;
}

// Read holding occurrence i, with its prefix, offset and length.
__device__ __forceinline__ void find_read(const BuildArgs &a, const TileView &v,
                                          const TileSmem &s, uint64_t i, uint64_t &pre,
                                          uint64_t &off, uint32_t &len, uint64_t &ridx,
                                          uint32_t &seg) {
    if (v.in_smem) {
        uint64_t lo = 0, hi = v.nr;  // last j with pre[j] <= i
        while (hi - lo > 1) {
            const uint64_t mid = (lo + hi) >> 1;
            if (s.pre[mid] <= i) lo = mid;
            else hi = mid;
        }
        pre = s.pre[lo];
        off = s.off[lo];
        len = s.len[lo];
        ridx = v.r0 + lo;
        seg = s.seg[lo];
    } else {
        uint64_t lo = v.r0, hi = v.r0 + v.nr;
        while (hi - lo > 1) {
            const uint64_t mid = (lo + hi) >> 1;
            if (a.occ_prefix[mid] <= i) lo = mid;
            else hi = mid;
        }
        pre = a.occ_prefix[lo];
        off = a.read_off[lo];
        len = a.read_len[lo];
        ridx = lo;
        seg = seg_of(a, lo);
    }
}

// Canonical k-molecule of occurrence i and its arc increments (one byte per
// slot). kmerGraph.cpp:240-296 restated per occurrence j of a read:
// K = max(C, rc(C)), f = (C == K); right arc (j+k < L) -> slot
// (f ? 0 : 4) + base[j+k]; left arc (j >= 1) -> slot (f ? 4 : 0) + 3 - base[j-1].
__device__ __forceinline__ void make_occ(const BuildArgs &a, const TileView &v, const TileSmem &s,
                                         uint64_t i, uint64_t &key, uint64_t &inc, uint32_t &seg) {
    uint64_t pre, off, ridx;
    uint32_t len;
    find_read(a, v, s, i, pre, off, len, ridx, seg);
    const int k = k_of(a, seg);
    const uint64_t p = i - pre, g = off + p;
    const uint64_t win = window32(a.packed, a.n_words, g);
    const uint64_t fwd = win >> (64 - 2 * k);
    const uint64_t rc = revcomp_dev(fwd, k);
    const bool f = fwd >= rc;
    key = f ? fwd : rc;
    inc = 0;
    if (p + (uint64_t)k < len) {
        const uint32_t rb = (uint32_t)(win >> (62 - 2 * k)) & 3u;
        inc += 1ull << (8 * ((f ? 0u : 4u) + rb));
    }
    if (p >= 1) {
        const uint32_t lb = base_at(a.packed, a.n_words, g - 1);
        inc += 1ull << (8 * ((f ? 4u : 0u) + 3u - lb));
    }
}

// Rolling walk over the occurrences [i0, i1) of a tile: one read lookup and
// one window extraction where a read starts, then one base rolled in per
// occurrence. Calls fn(key, code) with the canonical k-molecule and its arc
// code: bits 0-2 right slot, bit 3 right arc present, bits 4-6 left slot,
// bit 7 left arc present (slots as in make_occ), and the read's index.
template <typename F>
__device__ __forceinline__ void walk_run(const BuildArgs &a, const TileView &v, const TileSmem &s,
                                         uint64_t i0, uint64_t i1, F &&fn) {
    int k = a.k;
    uint64_t kmask = 0;
    int top = 0;
    uint64_t fwd = 0, rc = 0, last = 0, g = 0, p = 0, ridx = 0;
    uint32_t len = 0, rb = 0, seg = 0;
    for (uint64_t i = i0; i < i1; ++i) {
        uint32_t lb;
        bool has_l;
        if (i == i0 || i > last) {
            uint64_t pre, off;
            find_read(a, v, s, i, pre, off, len, ridx, seg);
            k = k_of(a, seg);
            kmask = (1ull << (2 * k)) - 1;
            top = 2 * (k - 1);
            p = i - pre;
            g = off + p;
            last = pre + (len - (uint32_t)k);
            const uint64_t win = window32(a.packed, a.n_words, g);
            fwd = win >> (64 - 2 * k);
            rc = revcomp_dev(fwd, k);
            rb = (uint32_t)(win >> (62 - 2 * k)) & 3u;  // base g+k (used only if inside the read)
            has_l = p >= 1;
            lb = has_l ? base_at(a.packed, a.n_words, g - 1) : 0u;
        } else {
            lb = (uint32_t)(fwd >> top) & 3u;  // first base of the previous k-mer
            has_l = true;
            ++g;
            ++p;
            fwd = ((fwd << 2) | rb) & kmask;
            rc = (rc >> 2) | ((uint64_t)(3u - rb) << top);
            rb = (p + (uint64_t)k < len) ? base_at(a.packed, a.n_words, g + (uint64_t)k) : 0u;
        }
        const bool has_r = p + (uint64_t)k < len;
        const bool f = fwd >= rc;
        unsigned code = 0;
        if (has_r) code |= 0x08u | ((f ? 0u : 4u) + rb);
        if (has_l) code |= 0x80u | (((f ? 4u : 0u) + 3u - lb) << 4);
        fn(f ? fwd : rc, code, ridx, seg);
    }
}

// ---------------------------------------------------------------------
// HyperLogLog over the canonical keys (persistent over tiles). Each thread
// takes a run of kK1Items consecutive occurrences of the tile: one read lookup
// and one window extraction at the start of the run (and at every read
// boundary inside it), then the k-mer and its reverse complement are rolled
// one base at a time.
// HyperLogLog, one thread per read: the k-mer and its reverse complement
// are rolled base by base (one packed word loaded every 16 bases), so the
// lanes of a warp advance in lockstep over reads of equal length. Blocks take
// contiguous read ranges; the current sample's registers live in smem.
__global__ void __launch_bounds__(256) k_hll_reads(BuildArgs a) {
    __shared__ unsigned regs[1 << kHllBits];
    __shared__ uint32_t s_cur;
    for (int j = threadIdx.x; j < (1 << kHllBits); j += blockDim.x) regs[j] = 0;
    if (threadIdx.x == 0) s_cur = 0xffffffffu;
    const uint64_t r0 = a.n_reads * blockIdx.x / gridDim.x;
    const uint64_t r1 = a.n_reads * (blockIdx.x + 1) / gridDim.x;
    for (uint64_t base = r0; base < r1; base += blockDim.x) {
        __syncthreads();
        const uint32_t first = seg_of(a, base);
        if (first != s_cur) {
            if (s_cur != 0xffffffffu)
                for (int j = threadIdx.x; j < (1 << kHllBits); j += blockDim.x)
                    if (regs[j]) {
                        atomicMax(&a.hll[((uint64_t)s_cur << kHllBits) + j], regs[j]);
                        regs[j] = 0;
                    }
            __syncthreads();
            if (threadIdx.x == 0) s_cur = first;
            __syncthreads();
        }
        const uint32_t cur = s_cur;
        const uint64_t r = base + threadIdx.x;
        if (r >= r1) continue;
        const uint32_t seg = seg_of(a, r);
        const int k = k_of(a, seg);
        const uint32_t L = a.read_len[r];
        if (L < (uint32_t)k) continue;
        const uint64_t kmask = (1ull << (2 * k)) - 1;
        const int top = 2 * (k - 1);
        uint64_t g = a.read_off[r], fwd = 0, rc = 0;
        uint32_t w = ldw(a.packed, g >> 4, a.n_words);
        for (uint32_t p = 0; p < L; ++p, ++g) {
            if (p && (g & 15) == 0) w = ldw(a.packed, g >> 4, a.n_words);
            const uint32_t b = (w >> (30 - 2 * (int)(g & 15))) & 3u;
            fwd = ((fwd << 2) | b) & kmask;
            rc = (rc >> 2) | ((uint64_t)(3u - b) << top);
            if (p + 1 < (uint32_t)k) continue;
            const uint64_t key = fwd >= rc ? fwd : rc;
            const uint64_t h = mix64(key ^ 0x9e3779b97f4a7c15ull);
            const unsigned idx = (unsigned)(h >> (64 - kHllBits));
            const uint64_t rest = (h << kHllBits) | (1ull << (kHllBits - 1));
            const unsigned rank = (unsigned)__clzll(rest) + 1;
            if (seg == cur) {
                if (rank > regs[idx]) atomicMax(&regs[idx], rank);
            } else {
                atomicMax(&a.hll[((uint64_t)seg << kHllBits) + idx], rank);
            }
        }
    }
    __syncthreads();
    if (s_cur != 0xffffffffu)
        for (int j = threadIdx.x; j < (1 << kHllBits); j += blockDim.x)
            if (regs[j]) atomicMax(&a.hll[((uint64_t)s_cur << kHllBits) + j], regs[j]);
}

// HyperLogLog estimate per sample (the same formula as hll_estimate).
__global__ void __launch_bounds__(256) k_hll_est(const unsigned *regs, double *est) {
    __shared__ double ssum[256];
    __shared__ int szero[256];
    const unsigned *r = regs + ((uint64_t)blockIdx.x << kHllBits);
    double sum = 0;
    int zeros = 0;
    for (int j = threadIdx.x; j < (1 << kHllBits); j += blockDim.x) {
        sum += ldexp(1.0, -(int)r[j]);
        zeros += r[j] == 0;
    }
    ssum[threadIdx.x] = sum;
    szero[threadIdx.x] = zeros;
    __syncthreads();
    for (int d = 128; d > 0; d >>= 1) {
        if (threadIdx.x < d) {
            ssum[threadIdx.x] += ssum[threadIdx.x + d];
            szero[threadIdx.x] += szero[threadIdx.x + d];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const double m = (double)(1 << kHllBits);
        const double alpha = 0.7213 / (1.0 + 1.079 / m);
        double e = alpha * m * m / ssum[0];
        if (e <= 2.5 * m && szero[0] > 0) e = m * log(m / (double)szero[0]);
        est[blockIdx.x] = e;
    }
}

// Batched builds: the sample of every read and the shift of its offset into
// the concatenated packed stream.
__global__ void k_seg_setup(uint32_t n_segs, const uint64_t *__restrict__ seg_read_start,
                            const uint64_t *__restrict__ seg_base_shift,
                            uint32_t *__restrict__ read_seg, uint64_t *__restrict__ read_off) {
    const uint32_t sg = blockIdx.x % n_segs;
    const uint32_t part = blockIdx.x / n_segs, parts = gridDim.x / n_segs;
    const uint64_t rs = seg_read_start[sg], re = seg_read_start[sg + 1];
    const uint64_t shift = seg_base_shift[sg];
    for (uint64_t r = rs + (uint64_t)part * blockDim.x + threadIdx.x; r < re;
         r += (uint64_t)parts * blockDim.x) {
        read_seg[r] = sg;
        read_off[r] += shift;
    }
}

__global__ void k_gather_prefix(const uint64_t *__restrict__ prefix,
                                const uint64_t *__restrict__ idx, uint32_t n,
                                uint64_t *__restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = prefix[idx[i]];
}

// HyperLogLog of the canonical keys fused with each read's minimizer: the
// smallest 32-bit hash over the read's canonical k-molecules. Reads that share
// a minimizer overlap in the genome, so counting them one after another keeps
// their common k-molecules' table entries in L2.
__global__ void __launch_bounds__(kK1Block) k_sketch(BuildArgs a, unsigned *minhash) {
    __shared__ TileSmem s;
    __shared__ unsigned regs[1 << kHllBits];
    for (int j = threadIdx.x; j < (1 << kHllBits); j += blockDim.x) regs[j] = 0;
    for (uint64_t t = blockIdx.x; t < a.n_tiles; t += gridDim.x) {
        __syncthreads();
        const TileView v = load_tile(a, t, s);
        __syncthreads();
        const uint64_t A = t * kTileOcc;
        const uint64_t B = umin64(A + kTileOcc, a.total_occ);
        const uint64_t i0 = A + (uint64_t)threadIdx.x * kK1Items;
        uint64_t cur = ~0ull;
        unsigned best = 0xffffffffu;
        walk_run(a, v, s, i0, umin64(i0 + kK1Items, B), [&](uint64_t key, unsigned, uint64_t r, uint32_t) {
            const uint64_t h = mix64(key ^ 0x9e3779b97f4a7c15ull);
            const unsigned idx = (unsigned)(h >> (64 - kHllBits));
            const uint64_t rest = (h << kHllBits) | (1ull << (kHllBits - 1));
            const unsigned rank = (unsigned)__clzll(rest) + 1;
            if (rank > regs[idx]) atomicMax(&regs[idx], rank);
            if (r != cur) {
                if (cur != ~0ull) atomicMin(&minhash[cur], best);
                cur = r;
                best = 0xffffffffu;
            }
            const unsigned mh = (unsigned)(mix64(key) >> 32);
            best = mh < best ? mh : best;
        });
        if (cur != ~0ull) atomicMin(&minhash[cur], best);
    }
    __syncthreads();
    for (int j = threadIdx.x; j < (1 << kHllBits); j += blockDim.x)
        if (regs[j]) atomicMax(&a.hll[j], regs[j]);
}

// Counting sort of the reads into 2^16 buckets by the top bits of their
// minimizer (reads with equal minimizers end up next to each other).
constexpr int kBucketBits = 16;

__global__ void k_bucket_hist(const unsigned *__restrict__ minhash, uint64_t n,
                              unsigned *__restrict__ hist) {
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n;
         r += (uint64_t)gridDim.x * blockDim.x)
        atomicAdd(&hist[minhash[r] >> (32 - kBucketBits)], 1u);
}

__global__ void __launch_bounds__(1024) k_bucket_scan(unsigned *hist) {
    __shared__ uint64_t wb[32];
    constexpr int per = (1 << kBucketBits) / 1024;
    unsigned v[per];
    uint64_t sum = 0;
#pragma unroll
    for (int x = 0; x < per; ++x) {
        v[x] = hist[threadIdx.x * per + x];
        sum += v[x];
    }
    uint64_t run = block_exclusive_scan<1024>(sum, wb, nullptr);
#pragma unroll
    for (int x = 0; x < per; ++x) {
        hist[threadIdx.x * per + x] = (unsigned)run;
        run += v[x];
    }
}

__global__ void k_bucket_scatter(const unsigned *__restrict__ minhash, uint64_t n,
                                 unsigned *__restrict__ cursor, const uint64_t *__restrict__ off,
                                 const uint32_t *__restrict__ len, uint64_t *__restrict__ out_off,
                                 uint32_t *__restrict__ out_len) {
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n;
         r += (uint64_t)gridDim.x * blockDim.x) {
        const unsigned pos = atomicAdd(&cursor[minhash[r] >> (32 - kBucketBits)], 1u);
        out_off[pos] = off[r];
        out_len[pos] = len[r];
    }
}

// ---------------------------------------------------------------------
// K1: fused extraction + counting, one tile per block.
// kSeg: batched build (per-sample tables, status and counters).
template <bool kSeg>
__global__ void __launch_bounds__(kK1Block) k_count(BuildArgs a) {
    __shared__ TileSmem s;
    __shared__ unsigned s_stop;
    __shared__ uint32_t s_seg0;
    __shared__ unsigned long long s_ins;
    const uint64_t t = blockIdx.x;
    if (threadIdx.x == 0) s_ins = 0;
    const TileView v = load_tile(a, t, s);
    __syncthreads();
    if (threadIdx.x == 0) {
        s_seg0 = v.in_smem ? s.seg[0] : seg_of(a, v.r0);
        const unsigned *st0 = kSeg ? a.seg_status + s_seg0 : a.status;
        s_stop = (*(volatile const unsigned *)st0) & kStatusTableFull;
    }
    __syncthreads();
    const uint32_t seg0 = s_seg0;
    const bool stop0 = s_stop != 0;
    if (stop0 && !kSeg) return;  // the table is being rebuilt larger
    const int lane = threadIdx.x & 31;
    unsigned my_ins = 0;
    const uint64_t A = t * kTileOcc;
    const uint64_t B = umin64(A + kTileOcc, a.total_occ);
    for (uint64_t base = A; base < B; base += kK1Block) {
        const uint64_t i = base + threadIdx.x;
        const bool valid = i < B;
        const unsigned vmask = __ballot_sync(kFull, valid);
        if (!valid) continue;
        uint64_t key, inc;
        uint32_t seg;
        make_occ(a, v, s, i, key, inc, seg);
        // merge equal keys of this warp (tandem repeats, duplicated reads)
        unsigned peers = __match_any_sync(vmask, key);
        if (kSeg) peers &= __match_any_sync(vmask, seg);
        if (__any_sync(vmask, peers != (1u << lane))) {
            uint64_t tot = 0;
#pragma unroll
            for (int sl = 0; sl < 8; ++sl) {
                const unsigned b = __ballot_sync(vmask, (unsigned)(inc >> (8 * sl)) & 1u);
                tot |= (uint64_t)__popc(b & peers) << (8 * sl);
            }
            inc = tot;
        }
        if (lane != __ffs(peers) - 1) continue;
        if (!kSeg) {
            my_ins += insert_or_update(a.table, a.cap, key, inc, a.status);
            continue;
        }
        const SegParams &p = a.segs[seg];
        unsigned *st = a.seg_status + seg;
        if (seg == seg0) {
            if (!stop0) my_ins += insert_or_update(a.table + p.tbase, p.tcap, key, inc, st);
        } else if (!((*(volatile const unsigned *)st) & kStatusTableFull)) {
            if (insert_or_update(a.table + p.tbase, p.tcap, key, inc, st)) {
                const unsigned long long before = atomicAdd(&a.seg_counts[2 * seg], 1ull);
                if ((before + 1) * 20 > p.tcap * 19) atomicOr(st, kStatusTableFull);
            }
        }
    }
    if (my_ins) atomicAdd(&s_ins, (unsigned long long)my_ins);
    __syncthreads();
    if (threadIdx.x == 0 && s_ins) {
        unsigned long long *ctr = kSeg ? a.seg_counts + 2 * seg0 : a.counters;
        unsigned *st = kSeg ? a.seg_status + seg0 : a.status;
        const unsigned long long cap = kSeg ? a.segs[seg0].tcap : a.cap;
        const unsigned long long before = atomicAdd(ctr, s_ins);
        // stop early once the table is nearly full; the host retries larger
        if ((before + s_ins) * 20 > cap * 19) atomicOr(st, kStatusTableFull);
    }
}

// ---------------------------------------------------------------------
// K2: cutoff + compaction. multiplicity < c -> 0 (graph.cpp:1105); a key
// survives iff one of its 8 slots is nonzero (graph.cpp:1106-1108).
__global__ void __launch_bounds__(kCBlock) k_compact(BuildArgs a) {
    __shared__ uint64_t wb[kCBlock / 32];
    __shared__ unsigned long long s_base;
    const uint64_t chunk = (uint64_t)blockIdx.x * kCBlock * kCItems;
    int c = a.cutoff;
    unsigned long long *ctr = a.counters;
    uint64_t obase = 0, ocap = a.out_cap;
    if (a.segs) {  // sample regions start at multiples of the chunk
        uint32_t lo = 0, hi = a.n_segs;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (a.segs[mid].tbase <= chunk) lo = mid;
            else hi = mid;
        }
        c = a.segs[lo].cutoff;
        ctr = a.seg_counts + 2 * lo;
        obase = a.segs[lo].tbase;
        ocap = a.segs[lo].tcap;
    }
    const uint32_t thr = c <= 0 ? 0u : (c >= 256 ? 0u : (uint32_t)c * 0x01010101u);
    const bool all_cut = c >= 256;
    uint64_t keys[kCItems], cnts[kCItems];
    unsigned keep = 0;
    int nkeep = 0;
#pragma unroll
    for (int it = 0; it < kCItems; ++it) {
        const uint64_t idx = chunk + (uint64_t)it * kCBlock + threadIdx.x;
        keys[it] = 0;
        cnts[it] = 0;
        if (idx < a.cap) {
            const ulonglong2 e = *reinterpret_cast<const ulonglong2 *>(a.table + idx);
            uint64_t v = e.y;
            if (thr) {
                const uint32_t lo = (uint32_t)v & __vcmpgeu4((uint32_t)v, thr);
                const uint32_t hi = (uint32_t)(v >> 32) & __vcmpgeu4((uint32_t)(v >> 32), thr);
                v = ((uint64_t)hi << 32) | lo;
            }
            if (all_cut) v = 0;
            keys[it] = e.x;
            cnts[it] = v;
            if (e.x != 0 && v != 0) {
                keep |= 1u << it;
                nkeep++;
            }
        }
    }
    uint64_t total;
    const uint64_t ex = block_exclusive_scan<kCBlock>((uint64_t)nkeep, wb, &total);
    if (threadIdx.x == 0) s_base = total ? atomicAdd(&ctr[1], (unsigned long long)total) : 0;
    __syncthreads();
    uint64_t pos = s_base + ex;
#pragma unroll
    for (int it = 0; it < kCItems; ++it) {
        if (keep & (1u << it)) {
            if (pos < ocap) {
                a.out_keys[obase + pos] = keys[it];
                a.out_mult[obase + pos] = cnts[it];
            }
            pos++;
        }
    }
}

// ---------------------------------------------------------------------
// Partitioned build. A record is {the low 64-bits bits of h = rmix64(key),
// shifted left by 8 | arc code}; the partition is the top `bits` bits of h,
// so h (a bijection of the key) is whole again in the partition's pass.
constexpr int kMaxSlots = 64;
constexpr int kPartChunk = kCBlock * kCItems;  // slot capacities are multiples of this

__device__ __forceinline__ uint64_t slice_cap_of(const PartArgs &pa, unsigned long long count) {
    const uint64_t c = count * (uint64_t)pa.load_den / (uint64_t)pa.load_num + 16;
    return c < pa.slot_cap ? c : pa.slot_cap;
}

// Where a bin's records go: record j of the block's sorted round (j in the
// bin's run) is written to dst + j while j < lim (the run's part that fits
// the bin's region; the rest is dropped and the overflow flagged later).
struct __align__(16) BinDest {
    unsigned long long dst;  // global index of the run's first record, minus its start in the round
    unsigned lim;            // round index past the last record that fits
    unsigned pad;
};

// Shared memory of k_p1_scatter: a round's records, their partitions and
// order, and per partition its count, local offset and global run base.
size_t p1_scatter_smem(uint32_t n_parts, int round) {
    return (size_t)round * (sizeof(unsigned long long) + sizeof(unsigned short)) +
           (size_t)n_parts * (16 + 2 * sizeof(unsigned));
}

// One read per thread, rolled base by base: the state of one read's walk.
// Bases stream in from the packed words (one load per 16 bases, issued 16
// bases before they are needed); the left
// neighbour of a k-mer is the base its predecessor shifted out.
struct ReadWalk {
    uint64_t fwd, rc, kmask;
    uint64_t wnext;    // index of the next packed word
    uint32_t w;        // bases not yet consumed of the current word, MSB first
    uint32_t wn;       // the next word, loaded ahead
    uint32_t wrem;     // how many
    uint32_t L, p;     // read length, position of the current k-mer
    uint32_t nb;       // base p+k (valid when p+k < L)
    uint32_t lb;       // base p-1 (valid when p >= 1)
    int k, top;
    uint32_t left;     // occurrences still to emit
    uint64_t tag;      // sample index in the key's top bits (tagged batch), else 0
};

__device__ __forceinline__ uint32_t walk_next(const BuildArgs &a, ReadWalk &st) {
    if (st.wrem == 0) {
        st.w = st.wn;
        st.wn = ldw(a.packed, ++st.wnext, a.n_words);  // 16 bases ahead of its use
        st.wrem = 16;
    }
    const uint32_t b = st.w >> 30;
    st.w <<= 2;
    st.wrem--;
    return b;
}

// KC: k fixed at compile time (a single-sample build with that k), so the
// shifts and masks of the rolling update are constants; 0: k read at run time.
template <int KC = 0>
__device__ __forceinline__ void walk_init(const BuildArgs &a, ReadWalk &st, uint64_t r) {
    const uint32_t seg = seg_of(a, r);
    st.k = KC ? KC : k_of(a, seg);
    st.tag = a.tag_bits ? (uint64_t)seg << (64 - a.tag_bits) : 0ull;
    st.L = a.read_len[r];
    st.left = st.L >= (uint32_t)st.k ? st.L - (uint32_t)st.k + 1 : 0;
    if (!st.left) return;
    st.kmask = (1ull << (2 * st.k)) - 1;
    st.top = 2 * (st.k - 1);
    const int top = KC ? 2 * (KC - 1) : st.top;
    const uint64_t g0 = a.read_off[r];
    st.wnext = (g0 >> 4) + 1;
    st.w = ldw(a.packed, g0 >> 4, a.n_words) << (2 * (uint32_t)(g0 & 15));
    st.wn = ldw(a.packed, st.wnext, a.n_words);
    st.wrem = 16 - (uint32_t)(g0 & 15);
    st.fwd = st.rc = 0;
    for (int i = 0; i < (KC ? KC : st.k); ++i) {
        const uint32_t b = walk_next(a, st);
        st.fwd = (st.fwd << 2) | b;
        st.rc = (st.rc >> 2) | ((uint64_t)(3u - b) << top);
    }
    st.p = 0;
    st.lb = 0;
    st.nb = (uint32_t)st.k < st.L ? walk_next(a, st) : 0u;
}

// Emit the current occurrence (key, arc code) and advance to the next one.
// Arc slots as make_occ (kmerGraph.cpp:240-296): right (f ? 0 : 4) +
// base[p+k], left (f ? 4 : 0) + 3 - base[p-1], f = (forward k-mer is the
// canonical one).
template <int KC = 0>
__device__ __forceinline__ void walk_emit(const BuildArgs &a, ReadWalk &st, uint64_t &key,
                                          unsigned &code) {
    const int top = KC ? 2 * (KC - 1) : st.top;
    const uint64_t kmask = KC ? (1ull << (2 * KC)) - 1 : st.kmask;
    const bool f = st.fwd >= st.rc;
    key = (f ? st.fwd : st.rc);
    if (!KC) key |= st.tag;  // KC is used for single-sample builds only
    code = 0;
    if (st.left > 1) code = 0x08u | ((f ? 0u : 4u) + st.nb);  // p + k < L
    if (st.p) code |= 0x80u | (((f ? 4u : 0u) + 3u - st.lb) << 4);
    if (--st.left) {
        const uint32_t b = st.nb;
        st.lb = (uint32_t)(st.fwd >> top);
        st.fwd = ((st.fwd << 2) | b) & kmask;
        st.rc = (st.rc >> 2) | ((uint64_t)(3u - b) << top);
        ++st.p;
        if (st.left > 1) st.nb = walk_next(a, st);
    }
}

// Level-1 records per partition, one thread per read (blocks take batches of
// reads as they finish the previous one: reads of uneven length stay balanced).
__global__ void __launch_bounds__(256) k_p1_count(BuildArgs a, PartArgs pa) {
    __shared__ unsigned hist[1 << kPartBitsMax];
    for (uint32_t j = threadIdx.x; j < pa.n_parts; j += blockDim.x) hist[j] = 0;
    __syncthreads();
    __shared__ unsigned long long s_base;
    const int shift = 64 - pa.bits;
    for (;;) {  // batches of blockDim.x reads, handed out as blocks finish them
        if (threadIdx.x == 0) s_base = atomicAdd(&pa.work[0], (unsigned long long)blockDim.x);
        __syncthreads();
        const uint64_t r = s_base + threadIdx.x;
        if (s_base >= a.n_reads) break;
        __syncthreads();  // s_base read by all
        if (r < a.n_reads) {
            ReadWalk st;
            walk_init(a, st, r);
            while (st.left) {
                uint64_t key;
                unsigned code;
                walk_emit(a, st, key, code);
                atomicAdd(&hist[rmix64(key) >> shift], 1u);
            }
        }
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < pa.n_parts; j += blockDim.x)
        if (hist[j]) atomicAdd(&pa.part_count[j], (unsigned long long)hist[j]);
}

// Sampled sizes: every stride-th batch of reads, each record counted in its
// level-1 partition (shared histogram, flushed to part_count) and its bucket
// (cursor2, as a histogram). Reads are sampled whole, so a hot key weighs in
// with all its occurrences in the sampled reads.
__global__ void __launch_bounds__(256) k_p1_sample(BuildArgs a, PartArgs pa, BucketArgs b, uint32_t stride) {
    __shared__ unsigned hist[1 << kPartBitsMax];
    __shared__ unsigned long long s_base;
    for (uint32_t j = threadIdx.x; j < pa.n_parts; j += blockDim.x) hist[j] = 0;
    const int shift = 64 - pa.bits, bshift = 64 - b.b1 - b.b2;
    for (;;) {
        if (threadIdx.x == 0)
            s_base = atomicAdd(&pa.work[0], 1ull) * (unsigned long long)blockDim.x * stride;
        __syncthreads();
        const uint64_t base = s_base;
        if (base >= a.n_reads) break;
        __syncthreads();  // s_base read by all
        const uint64_t r = base + threadIdx.x;
        if (r < a.n_reads) {
            ReadWalk st;
            walk_init(a, st, r);
            while (st.left) {
                uint64_t key;
                unsigned code;
                walk_emit(a, st, key, code);
                const uint64_t h = rmix64(key);
                atomicAdd(&hist[h >> shift], 1u);
                atomicAdd(&b.cursor2[h >> bshift], 1ull);
            }
        }
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < pa.n_parts; j += blockDim.x)
        if (hist[j]) atomicAdd(&pa.part_count[j], (unsigned long long)hist[j]);
}

// Partition regions from the sampled counts: 1.25 x the partition's share of
// the n_rec records + 4096, laid out by exclusive prefix (one block); the
// sampled total goes to *sampled. Sum of regions <= 1.25 n_rec + 4097 P.
__global__ void __launch_bounds__(1024) k_part_caps(PartArgs pa, uint64_t n_rec, unsigned long long *sampled) {
    __shared__ uint64_t wb[32];
    const uint32_t j = threadIdx.x;
    const uint64_t c = j < pa.n_parts ? pa.part_count[j] : 0;
    uint64_t total;
    block_exclusive_scan<1024>(c, wb, &total);
    uint64_t cap = 0;
    if (j < pa.n_parts) {
        const double share = total ? (double)c / (double)total : 1.0 / (double)pa.n_parts;
        cap = (uint64_t)(share * (double)n_rec * 1.25) + 4096;
    }
    uint64_t all;
    const uint64_t ex = block_exclusive_scan<1024>(cap, wb, &all);
    if (j < pa.n_parts) {
        pa.part_start[j] = ex;
        pa.part_cursor[j] = ex;
    }
    if (j == 0) {
        pa.part_start[pa.n_parts] = all;
        *sampled = total;
    }
}

// Bucket regions from the sampled counts (counts): 1.5 x the bucket's share
// of the records + 256, into caps (scanned afterwards). Sum <= 1.5 n_rec + 257 nb.
__global__ void k_bucket_caps(const unsigned long long *counts, const unsigned long long *sampled,
                              uint64_t n_rec, uint64_t nb, unsigned long long *caps) {
    const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nb) return;
    const uint64_t t = *sampled;
    const double share = t ? (double)counts[j] / (double)t : 1.0 / (double)nb;
    caps[j] = (uint64_t)(share * (double)n_rec * 1.5) + 256;
}
// Level-1 scatter, one thread per read: every round each thread emits up to
// kK1Items records of its read into registers, taking its rank within the
// partition from the shared histogram; the block orders the round's records
// by partition in shared memory and writes one run per partition.
template <int NT, int IT, int MINB, int KC = 0, int B1C = 0>
__global__ void __launch_bounds__(NT, MINB) k_p1_scatter(BuildArgs a, PartArgs pa) {
    extern __shared__ __align__(16) unsigned char dyn[];
    unsigned long long *sorted = reinterpret_cast<unsigned long long *>(dyn);
    BinDest *dest = reinterpret_cast<BinDest *>(sorted + NT * IT);  // per partition: where its run goes
    unsigned *hist = reinterpret_cast<unsigned *>(dest + pa.n_parts);
    unsigned *loff = hist + pa.n_parts;
    unsigned short *spart = reinterpret_cast<unsigned short *>(loff + pa.n_parts);
    __shared__ uint64_t wb[NT / 32];
    const int bits = B1C ? B1C : pa.bits;
    const int shift = 64 - bits;
    const uint32_t n_parts = B1C ? (1u << B1C) : pa.n_parts;
    const uint32_t per = (n_parts + blockDim.x - 1) / blockDim.x;
    // the reads: [0, n_reads), or read_range (kept in shared memory, read
    // once per batch: no registers held through the rounds)
    __shared__ unsigned long long s_base, s_first, s_end;
    if (threadIdx.x == 0) {
        s_first = a.read_range ? a.read_range[0] : 0;
        s_end = a.read_range ? a.read_range[1] : a.n_reads;
    }
    for (;;) {  // batches of NT reads, handed out as blocks finish them
        if (threadIdx.x == 0) s_base = atomicAdd(&pa.work[1], (unsigned long long)NT);
        __syncthreads();
        const uint64_t r = s_first + s_base + threadIdx.x;
        if (s_first + s_base >= s_end) break;
        ReadWalk st;
        st.left = 0;
        if (r < s_end) walk_init<KC>(a, st, r);
        while (__syncthreads_or(st.left != 0)) {
            for (uint32_t j = threadIdx.x; j < n_parts; j += blockDim.x) hist[j] = 0;
            __syncthreads();
            unsigned long long rec[IT];
            unsigned pr[IT];  // partition | rank << 16; ~0 for no record
#pragma unroll
            for (int j = 0; j < IT; ++j) {
                pr[j] = ~0u;
                rec[j] = 0;
                if (st.left) {
                    uint64_t key;
                    unsigned code;
                    walk_emit<KC>(a, st, key, code);
                    const uint64_t h = rmix64(key);
                    const unsigned part = (unsigned)(h >> shift);
                    rec[j] = ((h << bits) >> (bits - 8)) | code;  // low 64-b1 bits << 8
                    pr[j] = part | (atomicAdd(&hist[part], 1u) << 16);
                }
            }
            __syncthreads();
            uint64_t mine = 0;
            for (uint32_t x = 0; x < per; ++x) {
                const uint32_t j = threadIdx.x * per + x;
                if (j < n_parts) mine += hist[j];
            }
            uint64_t total;
            uint64_t run = block_exclusive_scan<NT>(mine, wb, &total);
            for (uint32_t x = 0; x < per; ++x) {
                const uint32_t j = threadIdx.x * per + x;
                if (j < n_parts) {
                    const unsigned c = hist[j];
                    loff[j] = (unsigned)run;
                    BinDest d;
                    d.dst = 0;
                    d.lim = (unsigned)run;
                    d.pad = 0;
                    if (c) {
                        const unsigned long long g0 = atomicAdd(&pa.part_cursor[j], (unsigned long long)c);
                        const unsigned long long lim = pa.part_start[j + 1];  // region end
                        const unsigned f = g0 + c <= lim ? c : (g0 < lim ? (unsigned)(lim - g0) : 0u);
                        d.dst = g0 - run;
                        d.lim = (unsigned)run + f;
                    }
                    dest[j] = d;
                    run += c;
                }
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < IT; ++j) {
                if (pr[j] != ~0u) {
                    const unsigned part = pr[j] & 0xffffu;
                    const unsigned pos = loff[part] + (pr[j] >> 16);
                    sorted[pos] = rec[j];
                    spart[pos] = (unsigned short)part;
                }
            }
            __syncthreads();
            for (uint32_t j = threadIdx.x; j < (uint32_t)total; j += blockDim.x) {
                const BinDest d = dest[spart[j]];
                // records past the partition's region are dropped (the overflow
                // is flagged after the scatter and the build recounts)
                if (j < d.lim) pa.records[d.dst + j] = sorted[j];
            }
        }
    }
}


// Level-1 scatter with warp-cooperative extraction: blocks take tiles of
// NT * IT consecutive k-mer occurrences (the tiles of the occurrence prefix),
// and in round j the lanes of a warp take 32 consecutive occurrences —
// mostly of one read. Each lane cuts its k-mer from a 64-bit window of the
// packed words (loads its neighbours share through L1), its reverse
// complement by bit reversal, and its neighbour bases from the window and
// the word before; no state is carried from one occurrence to the next. The
// read of an occurrence: lane 0 searches the tile's reads in shared memory,
// the others step on from it. Records, ranks and the partition sort as in
// k_p1_scatter. Single-sample builds only (one k).
template <int NT, int IT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_p1_scatter_wc(BuildArgs a, PartArgs pa) {
    extern __shared__ __align__(16) unsigned char dyn[];
    unsigned long long *sorted = reinterpret_cast<unsigned long long *>(dyn);
    BinDest *dest = reinterpret_cast<BinDest *>(sorted + NT * IT);
    unsigned *hist = reinterpret_cast<unsigned *>(dest + pa.n_parts);
    unsigned *loff = hist + pa.n_parts;
    unsigned short *spart = reinterpret_cast<unsigned short *>(loff + pa.n_parts);
    __shared__ uint64_t wb[NT / 32];
    __shared__ TileSmem ts;
    const int shift = 64 - pa.bits;
    const uint32_t per = (pa.n_parts + NT - 1) / NT;
    const int k = a.k;
    const int lane = threadIdx.x & 31;
    for (uint64_t t = blockIdx.x; t < a.n_tiles; t += gridDim.x) {
        __syncthreads();  // the previous tile's rounds are written out
        const TileView v = load_tile(a, t, ts);
        for (uint32_t j = threadIdx.x; j < pa.n_parts; j += NT) hist[j] = 0;
        __syncthreads();
        unsigned long long rec[IT];
        unsigned pr[IT];  // partition | rank << 16; ~0 for no record
        uint64_t hint = 0;  // the read (index in the tile) of this lane's last occurrence
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            pr[it] = ~0u;
            rec[it] = 0;
            const uint64_t i = t * kTileOcc + (uint64_t)it * NT + threadIdx.x;
            const bool valid = i < a.total_occ;
            uint64_t pre = 0, off = 0;
            uint32_t len = 0;
            if (v.in_smem) {
                // lane 0 searches; the warp's 32 occurrences span few reads
                uint64_t r = hint;
                if (lane == 0 && valid) {
                    uint64_t lo = hint, hi = v.nr;
                    while (hi - lo > 1) {
                        const uint64_t mid = (lo + hi) >> 1;
                        if (ts.pre[mid] <= i) lo = mid;
                        else hi = mid;
                    }
                    r = lo;
                }
                r = __shfl_sync(kFull, r, 0);
                if (valid) {
                    while (r + 1 < v.nr && ts.pre[r + 1] <= i) ++r;
                    pre = ts.pre[r];
                    off = ts.off[r];
                    len = ts.len[r];
                }
                hint = r;
            } else if (valid) {
                uint64_t ridx;
                uint32_t seg;
                find_read(a, v, ts, i, pre, off, len, ridx, seg);
            }
            if (valid) {
                const uint64_t p = i - pre, g = off + p;
                const uint64_t win = window32(a.packed, a.n_words, g);
                const uint64_t fwd = win >> (64 - 2 * k);
                const uint64_t rc = revcomp_dev(fwd, k);
                const bool f = fwd >= rc;
                unsigned code = 0;
                if (p + (uint64_t)k < len) code = 0x08u | ((f ? 0u : 4u) + ((uint32_t)(win >> (62 - 2 * k)) & 3u));
                if (p >= 1) code |= 0x80u | (((f ? 4u : 0u) + 3u - base_at(a.packed, a.n_words, g - 1)) << 4);
                const uint64_t h = rmix64(f ? fwd : rc);
                const unsigned part = (unsigned)(h >> shift);
                rec[it] = ((h << pa.bits) >> (pa.bits - 8)) | code;
                pr[it] = part | (atomicAdd(&hist[part], 1u) << 16);
            }
        }
        __syncthreads();
        uint64_t mine = 0;
        for (uint32_t x = 0; x < per; ++x) {
            const uint32_t j = threadIdx.x * per + x;
            if (j < pa.n_parts) mine += hist[j];
        }
        uint64_t total;
        uint64_t run = block_exclusive_scan<NT>(mine, wb, &total);
        for (uint32_t x = 0; x < per; ++x) {
            const uint32_t j = threadIdx.x * per + x;
            if (j < pa.n_parts) {
                const unsigned c = hist[j];
                loff[j] = (unsigned)run;
                BinDest d;
                d.dst = 0;
                d.lim = (unsigned)run;
                d.pad = 0;
                if (c) {
                    const unsigned long long g0 = atomicAdd(&pa.part_cursor[j], (unsigned long long)c);
                    const unsigned long long lim = pa.part_start[j + 1];  // region end
                    const unsigned f = g0 + c <= lim ? c : (g0 < lim ? (unsigned)(lim - g0) : 0u);
                    d.dst = g0 - run;
                    d.lim = (unsigned)run + f;
                }
                dest[j] = d;
                run += c;
            }
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            if (pr[it] != ~0u) {
                const unsigned part = pr[it] & 0xffffu;
                const unsigned pos = loff[part] + (pr[it] >> 16);
                sorted[pos] = rec[it];
                spart[pos] = (unsigned short)part;
            }
        }
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < (uint32_t)total; j += NT) {
            const BinDest d = dest[spart[j]];
            if (j < d.lim) pa.records[d.dst + j] = sorted[j];  // past the region: flagged later, recounted
        }
    }
}

// Exclusive prefix over the partitions (n_parts <= 1024, one block).
__global__ void __launch_bounds__(1024) k_part_prefix(PartArgs pa) {
    __shared__ uint64_t wb[32];
    const uint32_t j = threadIdx.x;
    const uint64_t c = j < pa.n_parts ? pa.part_count[j] : 0;
    uint64_t total;
    const uint64_t ex = block_exclusive_scan<1024>(c, wb, &total);
    if (j < pa.n_parts) {
        pa.part_start[j] = ex;
        pa.part_cursor[j] = ex;
    }
    if (j == 0) pa.part_start[pa.n_parts] = total;
}

// Phase C: count the records of partitions [p0, p0+n) into their slices.
__global__ void __launch_bounds__(kK1Block) k_part_insert(BuildArgs a, PartArgs pa, uint32_t p0,
                                                          uint32_t n, uint64_t rb, uint64_t re) {
    __shared__ unsigned long long st[kMaxSlots + 1];
    for (uint32_t j = threadIdx.x; j <= n; j += blockDim.x) st[j] = pa.part_start[p0 + j];
    __syncthreads();
    const int shift = 64 - pa.bits;
    const int lane = threadIdx.x & 31;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t base = rb + (uint64_t)blockIdx.x * blockDim.x; base < re; base += stride) {
        const uint64_t r = base + threadIdx.x;
        const bool valid = r < re;
        const unsigned vmask = __ballot_sync(kFull, valid);
        if (!valid) continue;
        uint32_t lo = 0, hi = n;  // last slot j with st[j] <= r
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (st[mid] <= r) lo = mid;
            else hi = mid;
        }
        const unsigned long long rec = pa.records[r];
        const uint64_t h = ((uint64_t)(p0 + lo) << shift) | (rec >> 8);
        uint64_t inc = code_inc((unsigned)rec & 0xffu);
        const unsigned peers = __match_any_sync(vmask, h);
        if (__any_sync(vmask, peers != (1u << lane))) {
            uint64_t tot = 0;
#pragma unroll
            for (int sl = 0; sl < 8; ++sl) {
                const unsigned b = __ballot_sync(vmask, (unsigned)(inc >> (8 * sl)) & 1u);
                tot |= (uint64_t)__popc(b & peers) << (8 * sl);
            }
            inc = tot;
        }
        if (lane == __ffs(peers) - 1)
            insert_or_update(pa.slices + (uint64_t)lo * pa.slot_cap,
                             slice_cap_of(pa, st[lo + 1] - st[lo]), h, inc, a.status);
    }
}

// Phase D: cutoff + compaction of the slices of partitions [p0, p0+n); every
// used entry is zeroed for the next wave. One block per chunk of a slot.
__global__ void __launch_bounds__(kCBlock) k_part_compact(BuildArgs a, PartArgs pa, uint32_t p0) {
    __shared__ uint64_t wb[kCBlock / 32];
    __shared__ unsigned long long s_base;
    const uint64_t chunks_per_slot = pa.slot_cap / kPartChunk;
    const uint32_t j = (uint32_t)(blockIdx.x / chunks_per_slot);
    const uint64_t chunk = (blockIdx.x % chunks_per_slot) * (uint64_t)kPartChunk;
    const uint64_t cap = slice_cap_of(pa, pa.part_count[p0 + j]);
    Entry *slice = pa.slices + (uint64_t)j * pa.slot_cap;
    const int c = a.cutoff;
    const uint32_t thr = c <= 0 ? 0u : (c >= 256 ? 0u : (uint32_t)c * 0x01010101u);
    const bool all_cut = c >= 256;
    uint64_t keys[kCItems], cnts[kCItems];
    unsigned keep = 0;
    int nkeep = 0, nused = 0;
#pragma unroll
    for (int it = 0; it < kCItems; ++it) {
        const uint64_t idx = chunk + (uint64_t)it * kCBlock + threadIdx.x;
        keys[it] = 0;
        cnts[it] = 0;
        if (idx < cap) {
            Entry *e = slice + idx;
            const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(e);
            if (v.x != 0) {
                uint64_t w = v.y;
                if (thr) {
                    const uint32_t lo = (uint32_t)w & __vcmpgeu4((uint32_t)w, thr);
                    const uint32_t hi = (uint32_t)(w >> 32) & __vcmpgeu4((uint32_t)(w >> 32), thr);
                    w = ((uint64_t)hi << 32) | lo;
                }
                if (all_cut) w = 0;
                *reinterpret_cast<ulonglong2 *>(e) = make_ulonglong2(0ull, 0ull);
                nused++;
                if (w != 0) {
                    keys[it] = runmix64(v.x);
                    cnts[it] = w;
                    keep |= 1u << it;
                    nkeep++;
                }
            }
        }
    }
    uint64_t total;
    const uint64_t ex = block_exclusive_scan<kCBlock>((uint64_t)nkeep, wb, &total);
    uint64_t used;
    block_exclusive_scan<kCBlock>((uint64_t)nused, wb, &used);
    if (threadIdx.x == 0) {
        s_base = total ? atomicAdd(&a.counters[1], (unsigned long long)total) : 0;
        if (used) atomicAdd(&a.counters[0], (unsigned long long)used);
    }
    __syncthreads();
    uint64_t pos = s_base + ex;
#pragma unroll
    for (int it = 0; it < kCItems; ++it) {
        if (keep & (1u << it)) {
            if (pos < a.out_cap) {
                a.out_keys[pos] = keys[it];
                a.out_mult[pos] = cnts[it];
            }
            pos++;
        }
    }
}

// ---------------------------------------------------------------------
// Bucketed build. Level-1 records come from k_p1_scatter (2^b1 partitions,
// record = low 64-b1 bits of h shifted left by 8 | arc code); the next b2
// bits of h name the sub-bucket. The level-2 passes walk each partition in
// chunks of kBkChunk records (a chunk never spans two partitions). Each
// bucket is then counted by one CTA in a shared-memory hash table sized to
// the bucket, and compacted from there.
constexpr int kBkItems = 16;                     // records per thread in a chunk
constexpr int kBkChunk = 256 * kBkItems;         // records per chunk
constexpr int kBkBinsMax = 1 << 10;              // sub-buckets per partition (b2 <= 10)
constexpr int kBkTable = 4096;                   // largest shared-memory table (entries)
constexpr uint64_t kBkRecMax = 65535;            // 16-bit slot counters cannot carry past this
constexpr int kBkThreads = 512;                  // threads of a bucket CTA
constexpr int kBkBatch = 8;                      // records loaded ahead per thread
constexpr int kBkTable2 = 8192;                  // tier-2 table (entries), one CTA per SM
constexpr int kBkThreads2 = 1024;

__device__ __forceinline__ uint32_t sub_of(const BucketArgs &b, unsigned long long rec) {
    return b.b2 ? (uint32_t)((rec >> 8) >> (64 - b.b1 - b.b2)) : 0u;
}

// Record range [rb, re) of bucket bk: its region starts at off2[bk]; the
// records end at its cursor, clamped to the region (off2[bk+1]).
__device__ __forceinline__ void bucket_range(const BucketArgs &b, uint64_t bk, uint64_t &rb, uint64_t &re) {
    rb = b.off2[bk];
    re = umin64(b.cursor2[bk], b.off2[bk + 1]);
}

// End of every partition's records (its cursor, clamped to the partition's
// region, flagging an overflow) and the chunks per partition as an exclusive
// prefix (one block).
__global__ void __launch_bounds__(1024) k_chunk_prefix(BucketArgs b) {
    __shared__ uint64_t wb[32];
    const uint32_t j = threadIdx.x;
    uint64_t c = 0;
    if (j < b.n_parts) {
        uint64_t end = b.part_cursor[j];
        if (end > b.part_start[j + 1]) {  // the partition outgrew its region
            atomicOr(b.status, kStatusPartOverflow);
            end = b.part_start[j + 1];
        }
        b.part_end[j] = end;
        c = (end - b.part_start[j] + kBkChunk - 1) / kBkChunk;
    }
    uint64_t total;
    const uint64_t ex = block_exclusive_scan<1024>(c, wb, &total);
    if (j < b.n_parts) b.chunk_start[j] = ex;
    if (j == 0) b.chunk_start[b.n_parts] = total;
}

// Partition p and record range [r0, r1) of level-2 chunk q.
__device__ __forceinline__ uint32_t chunk_range(const BucketArgs &b, uint64_t q, uint64_t &r0,
                                                uint64_t &r1) {
    uint32_t lo = 0, hi = b.n_parts;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (b.chunk_start[mid] <= q) lo = mid;
        else hi = mid;
    }
    r0 = b.part_start[lo] + (q - b.chunk_start[lo]) * kBkChunk;
    r1 = umin64(r0 + kBkChunk, b.part_end[lo]);
    return lo;
}

// Records per bucket (into cursor2).
__global__ void __launch_bounds__(256) k_sub_hist(BucketArgs b) {
    __shared__ unsigned hist[kBkBinsMax];
    const uint32_t P2 = 1u << b.b2;
    const uint64_t nq = b.chunk_start[b.n_parts];
    for (uint64_t q = blockIdx.x; q < nq; q += gridDim.x) {
        uint64_t r0, r1;
        const uint32_t p = chunk_range(b, q, r0, r1);
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < P2; j += blockDim.x) hist[j] = 0;
        __syncthreads();
#pragma unroll 4
        for (int it = 0; it < kBkItems; ++it) {
            const uint64_t r = r0 + (uint64_t)it * 256 + threadIdx.x;
            if (r < r1) atomicAdd(&hist[sub_of(b, b.rec1[r])], 1u);
        }
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < P2; j += blockDim.x)
            if (hist[j]) atomicAdd(&b.cursor2[(uint64_t)p * P2 + j], (unsigned long long)hist[j]);
    }
}

// Level-2 scatter: a chunk is held in registers, ordered by sub-bucket in
// shared memory and written as one run per sub-bucket.
constexpr size_t kSubScatterDyn = kBkChunk * sizeof(unsigned long long) +
                                  kBkBinsMax * (3 * sizeof(unsigned) + sizeof(unsigned long long));

template <int NT, int IT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_sub_scatter(BucketArgs b) {
    extern __shared__ __align__(16) unsigned char dyn[];
    unsigned long long *sorted = reinterpret_cast<unsigned long long *>(dyn);
    unsigned long long *gbase = sorted + kBkChunk;
    unsigned *hist = reinterpret_cast<unsigned *>(gbase + kBkBinsMax);
    unsigned *loff = hist + kBkBinsMax;
    unsigned *fit = loff + kBkBinsMax;  // records of the run that fit the bucket's region
    __shared__ uint64_t wb[NT / 32];
    const uint32_t P2 = 1u << b.b2;
    const uint32_t per = (P2 + NT - 1) / NT;  // bins per thread in the scan
    const uint64_t nq = *b.status & kStatusPartOverflow ? 0 : b.chunk_start[b.n_parts];  // recount ahead
    for (uint64_t q = blockIdx.x; q < nq; q += gridDim.x) {
        uint64_t r0, r1;
        const uint32_t p = chunk_range(b, q, r0, r1);
        unsigned long long v[IT];
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const uint64_t r = r0 + (uint64_t)it * NT + threadIdx.x;
            v[it] = r < r1 ? b.rec1[r] : 0ull;
        }
        __syncthreads();  // the previous chunk is written out
        for (uint32_t j = threadIdx.x; j < P2; j += blockDim.x) hist[j] = 0;
        __syncthreads();
#pragma unroll
        for (int it = 0; it < IT; ++it)
            if (r0 + (uint64_t)it * NT + threadIdx.x < r1) atomicAdd(&hist[sub_of(b, v[it])], 1u);
        __syncthreads();
        uint64_t mine = 0;
        for (uint32_t x = 0; x < per; ++x) {
            const uint32_t j = threadIdx.x * per + x;
            if (j < P2) mine += hist[j];
        }
        uint64_t run = block_exclusive_scan<NT>(mine, wb, nullptr);
        for (uint32_t x = 0; x < per; ++x) {
            const uint32_t j = threadIdx.x * per + x;
            if (j < P2) {
                const unsigned c = hist[j];
                loff[j] = (unsigned)run;
                run += c;
                unsigned long long g0 = 0;
                unsigned f = 0;
                if (c) {
                    const uint64_t bkj = (uint64_t)p * P2 + j;
                    g0 = atomicAdd(&b.cursor2[bkj], (unsigned long long)c);
                    const unsigned long long lim = b.off2[bkj + 1];  // region end
                    f = g0 + c <= lim ? c : (g0 < lim ? (unsigned)(lim - g0) : 0u);
                }
                gbase[j] = g0;
                fit[j] = f;
                hist[j] = 0;
            }
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            if (r0 + (uint64_t)it * NT + threadIdx.x < r1) {
                const uint32_t bn = sub_of(b, v[it]);
                sorted[loff[bn] + atomicAdd(&hist[bn], 1u)] = v[it];
            }
        }
        __syncthreads();
        const uint32_t n = (uint32_t)(r1 - r0);
        for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) {
            const unsigned long long w = sorted[j];
            const uint32_t bn = sub_of(b, w);
            // records past the bucket's region are dropped (the overflow is
            // flagged by the bucket count and the build recounts)
            if (j - loff[bn] < fit[bn]) b.rec2[gbase[bn] + (j - loff[bn])] = w;
        }
    }
}

// Level-2 scatter, one shared atomic per record: the histogram's atomicAdd
// returns the record's rank within its bin, kept (16 bits each, two per
// register) until the records are ordered by bin in shared memory.
// Its shared memory: the chunk, then per bin (2^b2 of them) its destination,
// count and local offset.
size_t sub_scatter2_smem(int b2) {
    return kBkChunk * sizeof(unsigned long long) + ((size_t)1 << b2) * (sizeof(BinDest) + 2 * sizeof(unsigned));
}

template <int NT, int IT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_sub_scatter2(BucketArgs b) {
    static_assert(IT % 2 == 0, "ranks are packed two per register");
    extern __shared__ __align__(16) unsigned char dyn[];
    const uint32_t P2 = 1u << b.b2;
    unsigned long long *sorted = reinterpret_cast<unsigned long long *>(dyn);
    BinDest *dest = reinterpret_cast<BinDest *>(sorted + NT * IT);
    unsigned *hist = reinterpret_cast<unsigned *>(dest + P2);
    unsigned *loff = hist + P2;
    __shared__ uint64_t wb[NT / 32];
    const uint32_t per = (P2 + NT - 1) / NT;  // bins per thread in the scan
    const int sh = 64 - b.b1 - b.b2 + 8;      // record >> sh = its bin (b2 > 0)
    const uint64_t nq = *b.status & kStatusPartOverflow ? 0 : b.chunk_start[b.n_parts];  // recount ahead
    for (uint32_t j = threadIdx.x; j < P2; j += NT) hist[j] = 0;
    for (uint64_t q = blockIdx.x; q < nq; q += gridDim.x) {
        uint64_t r0, r1;
        const uint32_t p = chunk_range(b, q, r0, r1);
        const uint32_t n = (uint32_t)(r1 - r0);
        unsigned long long v[IT];
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const uint32_t r = (uint32_t)it * NT + threadIdx.x;
            v[it] = r < n ? b.rec1[r0 + r] : 0ull;
        }
        __syncthreads();  // hist cleared, the previous chunk written out
        unsigned rk[IT / 2];
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            unsigned x = 0;
            if ((uint32_t)it * NT + threadIdx.x < n) x = atomicAdd(&hist[b.b2 ? (uint32_t)(v[it] >> sh) : 0u], 1u);
            if (it & 1) rk[it / 2] |= x << 16;
            else rk[it / 2] = x;
        }
        __syncthreads();
        uint64_t mine = 0;
        for (uint32_t x = 0; x < per; ++x) {
            const uint32_t j = threadIdx.x * per + x;
            if (j < P2) mine += hist[j];
        }
        uint64_t run = block_exclusive_scan<NT>(mine, wb, nullptr);
        for (uint32_t x = 0; x < per; ++x) {
            const uint32_t j = threadIdx.x * per + x;
            if (j < P2) {
                const unsigned c = hist[j];
                loff[j] = (unsigned)run;
                BinDest d;
                d.dst = 0;
                d.lim = (unsigned)run;
                d.pad = 0;
                if (c) {
                    const uint64_t bkj = (uint64_t)p * P2 + j;
                    const unsigned long long g0 = atomicAdd(&b.cursor2[bkj], (unsigned long long)c);
                    const unsigned long long lim = b.off2[bkj + 1];  // region end
                    const unsigned f = g0 + c <= lim ? c : (g0 < lim ? (unsigned)(lim - g0) : 0u);
                    d.dst = g0 - run;
                    d.lim = (unsigned)run + f;
                }
                dest[j] = d;
                hist[j] = 0;  // cleared for the next chunk
                run += c;
            }
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            if ((uint32_t)it * NT + threadIdx.x < n) {
                const uint32_t bn = b.b2 ? (uint32_t)(v[it] >> sh) : 0u;
                const unsigned rank = (rk[it / 2] >> (16 * (it & 1))) & 0xffffu;
                sorted[loff[bn] + rank] = v[it];
            }
        }
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < n; j += NT) {
            const unsigned long long w = sorted[j];
            const BinDest d = dest[b.b2 ? (uint32_t)(w >> sh) : 0u];
            // records past the bucket's region are dropped (the overflow is
            // flagged by the bucket count and the build recounts)
            if (j < d.lim) b.rec2[d.dst + j] = w;
        }
    }
}

// ---- bulk (TMA) copies into shared memory, tracked by an mbarrier ----
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Orders this CTA's earlier generic-proxy shared-memory accesses before later
// bulk copies into the same memory.
__device__ __forceinline__ void fence_proxy_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// dst, src and bytes are multiples of 16.
__device__ __forceinline__ void bulk_load(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
constexpr int kMaxWait = 1 << 20;  // try_wait rounds before a copy is given up on
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
    for (int i = 0; i < kMaxWait; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// Level-2 scatter with the chunks brought in by bulk copies: while a chunk is
// ordered by sub-bucket and written out, the block's next chunk is already
// in flight into the other staging buffer. A chunk's staging buffer also
// holds it once ordered. Copies start at an even record (16-byte aligned)
// and end after an even record; the record buffer has two records of slack.
constexpr int kSubBuf = kBkChunk + 2;  // records per staging buffer
constexpr size_t kSubScatterTmaDyn = 2 * (size_t)kSubBuf * sizeof(unsigned long long) +
                                     kBkBinsMax * (2 * sizeof(unsigned) + sizeof(unsigned long long));

__global__ void __launch_bounds__(256, 2) k_sub_scatter_tma(BucketArgs b) {
    constexpr int NT = 256, IT = kBkChunk / 256;
    extern __shared__ __align__(16) unsigned char dyn[];
    unsigned long long *const buf0 = reinterpret_cast<unsigned long long *>(dyn);  // two staging buffers
    unsigned long long *gbase = buf0 + 2 * kSubBuf;
    unsigned *hist = reinterpret_cast<unsigned *>(gbase + kBkBinsMax);
    unsigned *loff = hist + kBkBinsMax;
    __shared__ __align__(8) uint64_t bar[2];
    __shared__ uint64_t wb[NT / 32];
    const uint32_t P2 = 1u << b.b2;
    const uint32_t per = (P2 + NT - 1) / NT;  // bins per thread in the scan
    const uint64_t nq = *b.status & kStatusPartOverflow ? 0 : b.chunk_start[b.n_parts];  // recount ahead
    const uint64_t stride = gridDim.x;
    auto issue = [&](uint64_t q, int k) {
        uint64_t r0, r1;
        chunk_range(b, q, r0, r1);
        const uint64_t a0 = r0 & ~1ull, a1 = (r1 + 1) & ~1ull;
        bulk_load(buf0 + k * kSubBuf, b.rec1 + a0, (uint32_t)((a1 - a0) * sizeof(unsigned long long)), &bar[k]);
    };
    if (threadIdx.x == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
        if (blockIdx.x < nq) issue(blockIdx.x, 0);
        if (blockIdx.x + stride < nq) issue(blockIdx.x + stride, 1);
    }
    __syncthreads();
    uint32_t parity = 0;  // bit k: phase parity of bar[k]
    int k = 0;
    for (uint64_t q = blockIdx.x; q < nq; q += stride, k ^= 1) {
        const bool ok = mbar_wait(&bar[k], (parity >> k) & 1u);
        if (__syncthreads_or(!ok)) {  // a copy never completed: flag it, let the others land, leave
            if (threadIdx.x == 0) {
                atomicOr(b.status, kStatusCasLimit);
                mbar_wait(&bar[k ^ 1], (parity >> (k ^ 1)) & 1u);
            }
            return;
        }
        parity ^= 1u << k;
        unsigned long long *cur = buf0 + k * kSubBuf;
        uint64_t r0, r1;
        const uint32_t p = chunk_range(b, q, r0, r1);
        const uint32_t off = (uint32_t)(r0 & 1);
        const uint32_t n = (uint32_t)(r1 - r0);
        unsigned long long v[IT];
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const uint32_t i = (uint32_t)it * NT + threadIdx.x;
            v[it] = i < n ? cur[off + i] : 0ull;
        }
        for (uint32_t j = threadIdx.x; j < P2; j += NT) hist[j] = 0;
        __syncthreads();  // v read from the staging buffer; the histogram cleared
#pragma unroll
        for (int it = 0; it < IT; ++it)
            if ((uint32_t)it * NT + threadIdx.x < n) atomicAdd(&hist[sub_of(b, v[it])], 1u);
        __syncthreads();
        uint64_t mine = 0;
        for (uint32_t x = 0; x < per; ++x) {
            const uint32_t j = threadIdx.x * per + x;
            if (j < P2) mine += hist[j];
        }
        uint64_t run = block_exclusive_scan<NT>(mine, wb, nullptr);
        for (uint32_t x = 0; x < per; ++x) {
            const uint32_t j = threadIdx.x * per + x;
            if (j < P2) {
                const unsigned c = hist[j];
                loff[j] = (unsigned)run;
                run += c;
                gbase[j] = c ? atomicAdd(&b.cursor2[(uint64_t)p * P2 + j], (unsigned long long)c) : 0;
                hist[j] = 0;
            }
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            if ((uint32_t)it * NT + threadIdx.x < n) {
                const uint32_t bn = sub_of(b, v[it]);
                cur[loff[bn] + atomicAdd(&hist[bn], 1u)] = v[it];
            }
        }
        __syncthreads();
        const uint64_t bk0 = (uint64_t)p * P2;
        for (uint32_t j = threadIdx.x; j < n; j += NT) {
            const unsigned long long w = cur[j];
            const uint32_t bn = sub_of(b, w);
            const uint64_t dst = gbase[bn] + (j - loff[bn]);
            // records past the bucket's region are dropped (the overflow is
            // flagged by the bucket count and the build recounts)
            if (dst < b.off2[bk0 + bn + 1]) b.rec2[dst] = w;
        }
        __syncthreads();  // the buffer is read out
        if (threadIdx.x == 0 && q + 2 * stride < nq) {
            fence_proxy_async_smem();
            issue(q + 2 * stride, k);
        }
    }
}

// Tagged batch: moves every survivor into its sample's range (cursor[s]
// starts at the sample's survivor prefix) and strips the tag from the key.
// A round of 2048 survivors takes its rank within each sample from a shared
// histogram and one range per sample from the global cursor.
__global__ void __launch_bounds__(256) k_group_by_sample(const unsigned long long *__restrict__ in_keys,
                                                         const unsigned long long *__restrict__ in_mult,
                                                         uint64_t n, int tag_bits, uint32_t n_samples,
                                                         unsigned long long *cursor,
                                                         unsigned long long *__restrict__ out_keys,
                                                         unsigned long long *__restrict__ out_mult) {
    constexpr int IT = 8;
    __shared__ unsigned hist[kMaxTagSamples];
    __shared__ unsigned long long base[kMaxTagSamples];
    const int shift = 64 - tag_bits;
    const uint64_t mask = (1ull << shift) - 1;
    for (uint64_t c0 = (uint64_t)blockIdx.x * 256 * IT; c0 < n; c0 += (uint64_t)gridDim.x * 256 * IT) {
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < n_samples; j += 256) hist[j] = 0;
        __syncthreads();
        unsigned long long kv[IT], mv[IT];
        unsigned pr[IT];  // sample | rank << 10
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const uint64_t i = c0 + (uint64_t)it * 256 + threadIdx.x;
            pr[it] = ~0u;
            kv[it] = mv[it] = 0;
            if (i < n) {
                kv[it] = in_keys[i];
                mv[it] = in_mult[i];
                const unsigned smp = (unsigned)(kv[it] >> shift);
                pr[it] = smp | (atomicAdd(&hist[smp], 1u) << 10);
            }
        }
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < n_samples; j += 256)
            base[j] = hist[j] ? atomicAdd(&cursor[j], (unsigned long long)hist[j]) : 0;
        __syncthreads();
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            if (pr[it] != ~0u) {
                const uint64_t pos = base[pr[it] & 1023u] + (pr[it] >> 10);
                out_keys[pos] = kv[it] & mask;
                out_mult[pos] = mv[it];
            }
        }
    }
}

// A warp's survivors (kept: their lanes) also go to the caller's host arrays
// at a global cursor: one atomic per warp, the lanes' slots in lane order;
// slots past host_cap are counted but not written.
__device__ __forceinline__ void host_append(const BuildArgs &a, unsigned kept, int lane, uint64_t m,
                                            uint64_t key) {
    unsigned long long at = 0;
    if (lane == __ffs(kept) - 1) at = atomicAdd(a.host_written, (unsigned long long)__popc(kept));
    at = __shfl_sync(kFull, at, __ffs(kept) - 1);
    if (m) {
        const uint64_t q = at + __popc(kept & ((1u << lane) - 1));
        if (q < a.host_cap) {
            a.host_keys[q] = key;
            a.host_mult[q] = m;
        }
    }
}

// Shared memory of a bucket CTA: T keys, T x 8 uint16 counters, and the list
// of used slots (uint16).
template <int T>
constexpr size_t bucket_smem() {
    return (size_t)T * (sizeof(unsigned long long) + 4 * sizeof(unsigned) + sizeof(unsigned short));
}
// ... plus, for a tagged batch, per-sample distinct and survivor counters.
constexpr size_t kBucketTagSmem = 2 * kMaxTagSamples * sizeof(unsigned);

// Persistent bucket counting. The CTA clears its table once; a bucket's
// keys are inserted into the first tsize entries (2x the bucket's records,
// at most kT), every newly used slot is appended to a shared list, and the
// compaction walks that list only, staging the survivors in the bucket's own
// record range (keys in stage_keys, multiplicities over the bucket's
// records, all read by then) and clearing the slots for the next bucket.
// The next bucket's first records are loaded during the compaction. A bucket
// whose keys do not fit, or with more records than the 16-bit slot counters
// hold, is appended to the overflow list instead. Buckets are
// list[0..n_items) if list is given, else 0..n_items.
template <int kT, int kNT, int kB = kBkBatch>
__device__ void bucket_pass(const BuildArgs &a, const BucketArgs &b, uint64_t n_items,
                            const unsigned long long *list, unsigned long long *ovf,
                            unsigned *ovf_count, uint32_t ovf_cap) {
    extern __shared__ __align__(16) unsigned char dyn[];
    unsigned long long *keys = reinterpret_cast<unsigned long long *>(dyn);
    unsigned *cnt = reinterpret_cast<unsigned *>(keys + kT);  // 8 x uint16 per entry
    unsigned short *used_list = reinterpret_cast<unsigned short *>(cnt + 4 * kT);
    unsigned *s_dist = reinterpret_cast<unsigned *>(used_list + kT);  // tagged batch only
    unsigned *s_surv = s_dist + kMaxTagSamples;
    __shared__ unsigned s_over, s_nused, s_kept;
    const int lane = threadIdx.x & 31;
    const int tb = a.tag_bits;
    for (uint32_t j = threadIdx.x; j < (uint32_t)kT; j += kNT) {
        keys[j] = 0;
        reinterpret_cast<uint4 *>(cnt)[j] = make_uint4(0, 0, 0, 0);
    }
    if (tb)
        for (uint32_t j = threadIdx.x; j < a.n_segs; j += kNT) s_dist[j] = s_surv[j] = 0;
    const int c = a.cutoff;
    const bool cut_all = c >= 256;
    const unsigned cbias = (c > 0 && c < 256) ? (0x8000u - (unsigned)c) * 0x00010001u : 0u;
    unsigned long long v[kB];
    uint64_t v_for = ~0ull;  // bucket whose first batch the registers v hold
    for (uint64_t it = blockIdx.x; it < n_items; it += gridDim.x) {
        const uint64_t bk = list ? list[it] : it;
        uint64_t rb, re;
        bucket_range(b, bk, rb, re);
        const uint64_t nrec = re - rb;
        if (threadIdx.x == 0 && b.cursor2[bk] > re) atomicOr(b.status, kStatusPartOverflow);
        if (threadIdx.x == 0 && it + gridDim.x < n_items) {  // the next bucket, into L2
            uint64_t nrb, nre;
            bucket_range(b, list ? list[it + gridDim.x] : it + gridDim.x, nrb, nre);
            prefetch_records_l2(b.rec2, nrb, nre);
        }
        __syncthreads();  // the previous bucket's compaction (and the clear) is done
        if (threadIdx.x == 0) {
            s_over = 0;
            s_nused = 0;
            s_kept = 0;
        }
        if (nrec == 0) {
            if (threadIdx.x == 0) b.surv[bk] = 0;
            continue;
        }
        uint32_t tsize = 256;
        while (tsize < (uint32_t)kT && (uint64_t)tsize < 2 * nrec) tsize <<= 1;
        const uint32_t tmask = tsize - 1;
        if (nrec > kBkRecMax) {
            if (threadIdx.x == 0) {
                b.surv[bk] = 0;
                const unsigned i = atomicAdd(ovf_count, 1u);
                if (i < ovf_cap) ovf[i] = bk;
            }
            continue;
        }
        if (v_for != bk) {
#pragma unroll
            for (int i = 0; i < kB; ++i) {
                const uint64_t r = rb + (uint64_t)i * kNT + threadIdx.x;
                v[i] = r < re ? b.rec2[r] : 0ull;
            }
        }
        __syncthreads();  // counters reset
        const uint64_t hp = (uint64_t)(bk >> b.b2) << (64 - b.b1);
        bool full = false;
        for (uint64_t base = rb; base < re; base += (uint64_t)kNT * kB) {
            if (base != rb) {
#pragma unroll
                for (int i = 0; i < kB; ++i) {  // the batch's loads are in flight together
                    const uint64_t r = base + (uint64_t)i * kNT + threadIdx.x;
                    v[i] = r < re ? b.rec2[r] : 0ull;
                }
            }
#pragma unroll
            for (int i = 0; i < kB; ++i) {
                if (base + (uint64_t)i * kNT >= re) break;  // no thread of the block has a record left
                const bool valid = !full && base + (uint64_t)i * kNT + threadIdx.x < re;
                bool fresh = false;
                uint32_t slot = 0;
                if (valid) {
                    const unsigned long long h = hp | (v[i] >> 8);
                    slot = (uint32_t)h & tmask;
                    uint32_t step = 0;
                    unsigned long long old = 0;
                    for (; step < tsize; ++step) {
                        old = atomicCAS(&keys[slot], 0ull, h);
                        if (old == 0 || old == h) break;
                        slot = (slot + 1) & tmask;
                    }
                    if (step == tsize) {  // table full
                        s_over = 1;
                        full = true;
                    } else {
                        fresh = old == 0;
                        const unsigned code = (unsigned)v[i] & 0xffu;
                        if (code & 0x08u) {
                            const unsigned t = code & 7u;
                            atomicAdd(&cnt[4 * slot + (t >> 1)], 1u << (16 * (t & 1)));
                        }
                        if (code & 0x80u) {
                            const unsigned t = (code >> 4) & 7u;
                            atomicAdd(&cnt[4 * slot + (t >> 1)], 1u << (16 * (t & 1)));
                        }
                    }
                }
                const unsigned fm = __ballot_sync(kFull, fresh);
                if (fm) {  // append the warp's new slots to the used list
                    unsigned at = 0;
                    if (lane == __ffs(fm) - 1) at = atomicAdd(&s_nused, (unsigned)__popc(fm));
                    at = __shfl_sync(kFull, at, __ffs(fm) - 1);
                    if (fresh) used_list[at + __popc(fm & ((1u << lane) - 1))] = (unsigned short)slot;
                }
            }
        }
        __syncthreads();
        const bool over = s_over != 0;
        const uint32_t nused = s_nused;
        // the next bucket's first batch loads while this one is compacted
        const uint64_t nit = it + gridDim.x;
        v_for = ~0ull;
        if (nit < n_items) {
            const uint64_t nbk = list ? list[nit] : nit;
            uint64_t nrb, nre;
            bucket_range(b, nbk, nrb, nre);
#pragma unroll
            for (int i = 0; i < kB; ++i) {
                const uint64_t r = nrb + (uint64_t)i * kNT + threadIdx.x;
                v[i] = r < nre ? b.rec2[r] : 0ull;
            }
            v_for = nbk;
        }
        for (uint32_t base = 0; base < nused; base += kNT) {
            const uint32_t j = base + threadIdx.x;
            unsigned long long h = 0;
            uint64_t m = 0;
            if (j < nused) {
                const uint32_t sl = used_list[j];
                h = keys[sl];
                if (!over) {
                    if (tb) {  // the sample's own cutoff, per-sample counts
                        const uint32_t smp = (uint32_t)(runmix64(h) >> (64 - tb));
                        const int cs = a.segs[smp].cutoff;
                        m = bucket_mult(cnt, sl, (cs > 0 && cs < 256) ? (0x8000u - (unsigned)cs) * 0x00010001u : 0u,
                                        cs >= 256);
                        atomicAdd(&s_dist[smp], 1u);
                        if (m) atomicAdd(&s_surv[smp], 1u);
                    } else {
                        m = bucket_mult(cnt, sl, cbias, cut_all);
                    }
                }
                keys[sl] = 0;
                reinterpret_cast<uint4 *>(cnt)[sl] = make_uint4(0, 0, 0, 0);
            }
            const unsigned kept = __ballot_sync(kFull, m != 0);
            if (kept) {
                unsigned at = 0;
                if (lane == __ffs(kept) - 1) at = atomicAdd(&s_kept, (unsigned)__popc(kept));
                at = __shfl_sync(kFull, at, __ffs(kept) - 1);
                if (m) {
                    const uint64_t pos = rb + at + __popc(kept & ((1u << lane) - 1));
                    b.stage_keys[pos] = runmix64(h);
                    b.rec2[pos] = m;
                }
                if (a.host_keys) host_append(a, kept, lane, m, runmix64(h));
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            if (over) {
                b.surv[bk] = 0;
                const unsigned i = atomicAdd(ovf_count, 1u);
                if (i < ovf_cap) ovf[i] = bk;
            } else {
                b.surv[bk] = s_kept;
                if (nused) atomicAdd(&a.counters[0], (unsigned long long)nused);
            }
        }
    }
    if (tb) {
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < a.n_segs; j += kNT) {
            if (s_dist[j]) atomicAdd(&a.seg_counts[2 * j], (unsigned long long)s_dist[j]);
            if (s_surv[j]) atomicAdd(&a.seg_counts[2 * j + 1], (unsigned long long)s_surv[j]);
        }
    }
}

// Tier 1: tables of up to kBkTable entries, two persistent CTAs per SM over
// all buckets; overflow to the big list.
__global__ void __launch_bounds__(kBkThreads, 2) k_bucket_count(BuildArgs a, BucketArgs b, uint64_t n_buckets) {
    if (block_reads_overflow(b.status)) return;  // a partition overflowed: the build recounts
    bucket_pass<kBkTable, kBkThreads>(a, b, n_buckets, nullptr, b.big, b.big_count, b.big_cap);
}

// Tier 1 for small buckets (a plan of at most kBkSmallRecords records per
// bucket on average): four CTAs of 256 threads per SM with 2048-entry tables
// and 4 records loaded ahead per thread — as many warps per SM, half as many
// threads behind each barrier. A bucket whose keys do not fit goes to tier 2.
constexpr int kBkTableS = 2048, kBkThreadsS = 256;
constexpr uint64_t kBkSmallRecords = 3072;
__global__ void __launch_bounds__(kBkThreadsS, 4) k_bucket_count_small(BuildArgs a, BucketArgs b, uint64_t n_buckets) {
    if (block_reads_overflow(b.status)) return;
    bucket_pass<kBkTableS, kBkThreadsS, 4>(a, b, n_buckets, nullptr, b.big, b.big_count, b.big_cap);
}

// Tier 2: the buckets tier 1 could not hold, one persistent CTA per SM with
// tables of up to kBkTable2 entries; overflow to the second list (counted in
// a global-memory table by the host-driven path).
__global__ void __launch_bounds__(kBkThreads2, 1) k_bucket_count_large(BuildArgs a, BucketArgs b) {
    if (block_reads_overflow(b.status)) return;
    const unsigned n = umin64(*b.big_count, b.big_cap);
    bucket_pass<kBkTable2, kBkThreads2>(a, b, n, b.big, b.big2, b.big2_count, b.big_cap);
}

// Packs the staged survivors of every bucket (warp per bucket) at the
// bucket's survivor prefix; the total goes to counters[1], after which the
// big-bucket path appends.
__global__ void __launch_bounds__(256) k_bucket_gather(BuildArgs a, BucketArgs b, uint64_t n_buckets) {
    const uint64_t bk = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (bk == 0 && lane == 0) a.counters[1] = b.surv_off[n_buckets];
    if (bk >= n_buckets) return;
    uint64_t rb, re;
    bucket_range(b, bk, rb, re);
    const uint64_t S = b.surv_off[bk], n = b.surv_off[bk + 1] - S;
    for (uint64_t i = lane; i < n; i += 32) {
        if (S + i < a.out_cap) {
            a.out_keys[S + i] = b.stage_keys[rb + i];
            a.out_mult[S + i] = b.rec2[rb + i];
        }
    }
}


// All buckets no shared-memory table held, in one global-memory table (their
// keys are disjoint): meta = rb [n] | hash prefix [n] | record prefix [n+1].
__global__ void __launch_bounds__(kK1Block) k_big_insert_multi(BuildArgs a, const unsigned long long *rec2,
                                                               const unsigned long long *meta, uint32_t n,
                                                               Entry *table, uint64_t cap) {
    const int lane = threadIdx.x & 31;
    const unsigned long long *rbs = meta, *hps = meta + n, *pre = meta + 2 * n;
    const uint64_t total = pre[n];
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < total; base += stride) {
        const uint64_t i = base + threadIdx.x;
        const bool valid = i < total;
        const unsigned vmask = __ballot_sync(kFull, valid);
        if (!valid) continue;
        uint32_t lo = 0, hi = n;  // last bucket j with pre[j] <= i
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (pre[mid] <= i) lo = mid;
            else hi = mid;
        }
        const unsigned long long rec = rec2[rbs[lo] + (i - pre[lo])];
        const uint64_t h = hps[lo] | (rec >> 8);
        uint64_t inc = code_inc((unsigned)rec & 0xffu);
        const unsigned peers = __match_any_sync(vmask, h);
        if (__any_sync(vmask, peers != (1u << lane))) {
            uint64_t tot = 0;
#pragma unroll
            for (int sl = 0; sl < 8; ++sl) {
                const unsigned bb = __ballot_sync(vmask, (unsigned)(inc >> (8 * sl)) & 1u);
                tot |= (uint64_t)__popc(bb & peers) << (8 * sl);
            }
            inc = tot;
        }
        if (lane == __ffs(peers) - 1) insert_or_update(table, cap, h, inc, a.status);
    }
}

__global__ void __launch_bounds__(kCBlock) k_big_compact(BuildArgs a, const Entry *table, uint64_t cap) {
    __shared__ uint64_t wb[kCBlock / 32];
    __shared__ unsigned long long s_base;
    const uint64_t chunk = (uint64_t)blockIdx.x * kCBlock * kCItems;
    const int c = a.cutoff;
    const uint32_t thr = c <= 0 ? 0u : (c >= 256 ? 0u : (uint32_t)c * 0x01010101u);
    uint64_t keys[kCItems], cnts[kCItems];
    unsigned keep = 0;
    int nkeep = 0, nused = 0;
#pragma unroll
    for (int it = 0; it < kCItems; ++it) {
        const uint64_t idx = chunk + (uint64_t)it * kCBlock + threadIdx.x;
        keys[it] = cnts[it] = 0;
        if (idx >= cap) continue;
        const ulonglong2 e = *reinterpret_cast<const ulonglong2 *>(table + idx);
        if (!e.x) continue;
        nused++;
        uint64_t v = e.y;
        uint32_t th = thr;
        int cc = c;
        uint32_t smp = 0;
        if (a.tag_bits) {  // tagged batch: the sample's own cutoff, per-sample counts
            smp = (uint32_t)(runmix64(e.x) >> (64 - a.tag_bits));
            cc = a.segs[smp].cutoff;
            th = cc <= 0 ? 0u : (cc >= 256 ? 0u : (uint32_t)cc * 0x01010101u);
        }
        if (th) {
            const uint32_t lo = (uint32_t)v & __vcmpgeu4((uint32_t)v, th);
            const uint32_t hi = (uint32_t)(v >> 32) & __vcmpgeu4((uint32_t)(v >> 32), th);
            v = ((uint64_t)hi << 32) | lo;
        }
        if (cc >= 256) v = 0;
        if (a.tag_bits) {
            atomicAdd(&a.seg_counts[2 * smp], 1ull);
            if (v) atomicAdd(&a.seg_counts[2 * smp + 1], 1ull);
        }
        if (v) {
            keys[it] = runmix64(e.x);
            cnts[it] = v;
            keep |= 1u << it;
            nkeep++;
        }
    }
    uint64_t total, used;
    const uint64_t ex = block_exclusive_scan<kCBlock>((uint64_t)nkeep, wb, &total);
    block_exclusive_scan<kCBlock>((uint64_t)nused, wb, &used);
    if (threadIdx.x == 0) {
        s_base = total ? atomicAdd(&a.counters[1], (unsigned long long)total) : 0;
        if (used) atomicAdd(&a.counters[0], (unsigned long long)used);
    }
    __syncthreads();
    uint64_t pos = s_base + ex;
#pragma unroll
    for (int it = 0; it < kCItems; ++it) {
        if (keep & (1u << it)) {
            if (pos < a.out_cap) {
                a.out_keys[pos] = keys[it];
                a.out_mult[pos] = cnts[it];
            }
            pos++;
        }
    }
    if (a.host_keys) {  // and to the caller's host arrays (see host_append)
        __shared__ unsigned long long s_hbase;
        if (threadIdx.x == 0) s_hbase = total ? atomicAdd(a.host_written, (unsigned long long)total) : 0;
        __syncthreads();
        uint64_t q = s_hbase + ex;
#pragma unroll
        for (int it = 0; it < kCItems; ++it) {
            if (keep & (1u << it)) {
                if (q < a.host_cap) {
                    a.host_keys[q] = keys[it];
                    a.host_mult[q] = cnts[it];
                }
                q++;
            }
        }
    }
}

// ---------------------------------------------------------------------
// Random-access probe (roofline denominator).
__global__ void __launch_bounds__(256) k_probe(int kind, Entry *table, uint64_t n16,
                                               uint64_t ops_per_thread, uint64_t seed,
                                               unsigned long long *sink) {
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    uint64_t x = mix64(seed ^ (tid * 0x9e3779b97f4a7c15ull)) | 1ull;
    unsigned long long acc = 0;
    for (uint64_t op = 0; op < ops_per_thread; ++op) {
        x ^= x >> 12;
        x ^= x << 25;
        x ^= x >> 27;
        const uint64_t r = x * 0x2545f4914f6cdd1dull;
        Entry *e = table + __umul64hi(r, n16);
        switch (kind) {
            case 0: atomicAdd(reinterpret_cast<unsigned *>(e), 1u); break;
            case 1: acc += atomicAdd(reinterpret_cast<unsigned long long *>(e), 1ull); break;
            case 2: acc += cas128(e, 0, 0, 0, 0).y; break;
            case 3: {
                const ulonglong2 v = ld_relaxed16(e);
                acc += v.x ^ v.y;
                break;
            }
            case 4: {
                const ulonglong2 v = ld_relaxed16(e);
                acc += cas128(e, v.x, v.y, v.x, v.y + 1).y;
                break;
            }
            case 5: {  // four independent 16-byte loads in flight
                const uint64_t r2 = r * 0x9e3779b97f4a7c15ull, r3 = r2 * 0x9e3779b97f4a7c15ull,
                               r4 = r3 * 0x9e3779b97f4a7c15ull;
                const ulonglong2 a0 = ld_relaxed16(e);
                const ulonglong2 a1 = ld_relaxed16(table + __umul64hi(r2, n16));
                const ulonglong2 a2 = ld_relaxed16(table + __umul64hi(r3, n16));
                const ulonglong2 a3 = ld_relaxed16(table + __umul64hi(r4, n16));
                acc += a0.x ^ a1.y ^ a2.x ^ a3.y;
                break;
            }
            default: {  // two independent load + CAS chains in flight
                Entry *e2 = table + __umul64hi(r * 0x9e3779b97f4a7c15ull, n16);
                const ulonglong2 v = ld_relaxed16(e);
                const ulonglong2 w = ld_relaxed16(e2);
                acc += cas128(e, v.x, v.y, v.x, v.y + 1).y;
                acc += cas128(e2, w.x, w.y, w.x, w.y + 1).y;
                break;
            }
        }
    }
    if (acc == 0x123456789ull) *sink = acc;  // keeps the loads live
}

}  // namespace

// ---------------------------------------------------------------------
// Host launchers.

int device_sm_count() {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    return n > 0 ? n : 1;
}

uint64_t scan_block_count(uint64_t n_reads) { return (n_reads + kScanChunk - 1) / kScanChunk; }

int launch_occ_scan(const BuildArgs &a, cudaStream_t s) {
    const uint64_t nb = scan_block_count(a.n_reads);
    if (nb == 0) return 0;
    k_scan_reduce<<<(unsigned)nb, kScanBlock, 0, s>>>(a);
    k_scan_blocks<<<1, 1024, 0, s>>>(a.scan_blocks, nb, a.occ_prefix + a.n_reads);
    k_scan_write<<<(unsigned)nb, kScanBlock, 0, s>>>(a);
    return 3;
}

int launch_occ_total(const BuildArgs &a, unsigned long long *total, cudaStream_t s) {
    if (!a.n_reads) return 0;
    const uint64_t blocks = (a.n_reads + 4 * kScanBlock - 1) / (4 * kScanBlock);
    k_occ_total<<<(unsigned)std::min<uint64_t>(blocks, (uint64_t)device_sm_count() * 8), kScanBlock, 0, s>>>(
        a.read_len, a.n_reads, a.k, total, a.max_len);
    return 1;
}


int launch_tiles(const BuildArgs &a, cudaStream_t s) {
    if (a.n_tiles == 0) return 0;
    const unsigned grid = (unsigned)((a.n_tiles + 255) / 256);
    k_tiles<<<grid, 256, 0, s>>>(a.occ_prefix, a.n_reads, a.n_tiles, a.tile_first_read);
    return 1;
}

int launch_hll(const BuildArgs &a, cudaStream_t s) {
    if (a.total_occ == 0 || a.n_reads == 0) return 0;
    const uint64_t grid = std::min<uint64_t>((a.n_reads + 255) / 256, (uint64_t)device_sm_count() * 8);
    k_hll_reads<<<(unsigned)grid, 256, 0, s>>>(a);
    return 1;
}

// Standard HyperLogLog estimate with the small-range (linear counting) correction.
double hll_estimate(const unsigned *regs) {
    const int m = 1 << kHllBits;
    double sum = 0;
    int zeros = 0;
    for (int j = 0; j < m; j++) {
        sum += ldexp(1.0, -(int)regs[j]);
        zeros += regs[j] == 0;
    }
    const double alpha = 0.7213 / (1.0 + 1.079 / m);
    double e = alpha * (double)m * (double)m / sum;
    if (e <= 2.5 * m && zeros > 0) e = m * log((double)m / zeros);
    return e;
}

int launch_sketch(const BuildArgs &a, unsigned *minhash, cudaStream_t s) {
    if (a.n_tiles == 0) return 0;
    const uint64_t grid = std::min<uint64_t>(a.n_tiles, (uint64_t)device_sm_count() * 8);
    k_sketch<<<(unsigned)grid, kK1Block, 0, s>>>(a, minhash);
    return 1;
}

uint64_t bucket_count() { return 1ull << kBucketBits; }

int launch_read_order(const BuildArgs &a, const unsigned *minhash, unsigned *hist,
                      uint64_t *out_off, uint32_t *out_len, cudaStream_t s) {
    if (a.n_reads == 0) return 0;
    const uint64_t grid = std::min<uint64_t>((a.n_reads + 255) / 256, (uint64_t)device_sm_count() * 8);
    cudaMemsetAsync(hist, 0, sizeof(unsigned) << kBucketBits, s);
    k_bucket_hist<<<(unsigned)grid, 256, 0, s>>>(minhash, a.n_reads, hist);
    k_bucket_scan<<<1, 1024, 0, s>>>(hist);
    k_bucket_scatter<<<(unsigned)grid, 256, 0, s>>>(minhash, a.n_reads, hist, a.read_off,
                                                    a.read_len, out_off, out_len);
    return 3;
}

int launch_seg_setup(const BuildArgs &a, const uint64_t *seg_read_start,
                     const uint64_t *seg_base_shift, uint32_t *read_seg, uint64_t *read_off,
                     cudaStream_t s) {
    if (a.n_segs == 0) return 0;
    const uint32_t parts = (uint32_t)std::max<uint64_t>(1, (uint64_t)device_sm_count() * 8 / a.n_segs);
    k_seg_setup<<<a.n_segs * parts, 256, 0, s>>>(a.n_segs, seg_read_start, seg_base_shift,
                                                 read_seg, read_off);
    return 1;
}

int launch_hll_estimates(const unsigned *regs, uint32_t n_segs, double *est, cudaStream_t s) {
    if (n_segs == 0) return 0;
    k_hll_est<<<n_segs, 256, 0, s>>>(regs, est);
    return 1;
}

int launch_gather_prefix(const uint64_t *prefix, const uint64_t *idx, uint32_t n, uint64_t *out,
                         cudaStream_t s) {
    if (n == 0) return 0;
    k_gather_prefix<<<(n + 255) / 256, 256, 0, s>>>(prefix, idx, n, out);
    return 1;
}

int launch_count(const BuildArgs &a, cudaStream_t s) {
    if (a.n_tiles == 0) return 0;
    if (a.segs) k_count<true><<<(unsigned)a.n_tiles, kK1Block, 0, s>>>(a);
    else k_count<false><<<(unsigned)a.n_tiles, kK1Block, 0, s>>>(a);
    return 1;
}

int launch_compact(const BuildArgs &a, cudaStream_t s) {
    const uint64_t per = (uint64_t)kCBlock * kCItems;
    const uint64_t grid = (a.cap + per - 1) / per;
    if (grid == 0) return 0;
    k_compact<<<(unsigned)grid, kCBlock, 0, s>>>(a);
    return 1;
}

int launch_part_count(const BuildArgs &a, const PartArgs &p, cudaStream_t s) {
    if (a.total_occ == 0 || a.n_reads == 0) return 0;
    const uint64_t grid = std::min<uint64_t>((a.n_reads + 255) / 256, resident_grid(k_p1_count, 256, 0));
    k_p1_count<<<(unsigned)grid, 256, 0, s>>>(a, p);
    return 1;
}


int launch_part_prefix(const PartArgs &p, cudaStream_t s) {
    k_part_prefix<<<1, 1024, 0, s>>>(p);
    return 1;
}

// Block shape of the two scatter passes: threads, records per thread per
// round, resident blocks per SM (SWG_SCATTER_SHAPE = 0..3 selects one; 3 is
// the level-2 scatter with bulk-copy staging).
int scatter_shape();
int level1_shape(int opt_shape) { return opt_shape ? opt_shape : scatter_shape(); }

int scatter_shape() {
    static int shape = [] {
        const char *e = std::getenv("SWG_SCATTER_SHAPE");
        const int v = e ? std::atoi(e) : 0;
        return v >= 0 && v <= 4 ? v : 0;
    }();
    return shape;
}

template <int NT, int IT, int MINB, int KC = 0, int B1C = 0>
int launch_p1_scatter_shape(const BuildArgs &a, const PartArgs &p, cudaStream_t s, int grid_mode) {
    auto kern = k_p1_scatter<NT, IT, MINB, KC, B1C>;
    const size_t smem = p1_scatter_smem(p.n_parts, NT * IT);
    allow_smem(kern, p1_scatter_smem(1u << kPartBitsMax, NT * IT));
    const uint64_t batches = (a.n_reads + NT - 1) / NT;
    const uint64_t resident = resident_grid(kern, NT, smem), sms = device_sm_count();
    uint64_t grid = batches;  // kScatterPerBatch
    if (grid_mode == kScatterResident) grid = std::min(batches, resident);
    if (grid_mode == kScatterShared) grid = std::min(batches, resident > sms ? resident - sms : resident);
    kern<<<(unsigned)grid, NT, smem, s>>>(a, p);
    return 1;
}

int launch_part_scatter(const BuildArgs &a, const PartArgs &p, cudaStream_t s, int grid_mode) {
    if (a.total_occ == 0 || a.n_reads == 0) return 0;
    const int shape = p.shape ? p.shape : scatter_shape();
    if (shape == 4 && a.tile_first_read && a.n_tiles && !a.segs && !a.tag_bits) {
        // warp-cooperative extraction (needs the occurrence prefix and tiles)
        auto kern = k_p1_scatter_wc<256, 16, 3>;
        const size_t smem = p1_scatter_smem(p.n_parts, 256 * 16);
        allow_smem(kern, p1_scatter_smem(1u << kPartBitsMax, 256 * 16));
        const uint64_t grid = std::min<uint64_t>(a.n_tiles, resident_grid(kern, 256, smem));
        kern<<<(unsigned)grid, 256, smem, s>>>(a, p);
        return 1;
    }
    const bool single = !a.segs && !a.read_seg && !a.tag_bits;
    // (Odd k from 19 to 31 come here for shapes 1 to 4, and to be counted again
    // exactly; otherwise they go by super-k-mers.)
    // Single-sample builds with 256 partitions and a common k: the walk's
    // shifts and masks and the record layout are compile-time constants, and
    // rounds of 12 records a thread fit 64 registers, so four blocks share an
    // SM (three in the shared grid, leaving a fourth block's room). Shapes 1
    // and 2 replace it in a resident or per-batch grid.
    if (single && p.bits == 8 && (grid_mode == kScatterShared || shape == 0 || shape == 3 || shape == 4))
        switch (a.k) {
            case 31: return launch_p1_scatter_shape<256, 12, 4, 31, 8>(a, p, s, grid_mode);
            case 27: return launch_p1_scatter_shape<256, 12, 4, 27, 8>(a, p, s, grid_mode);
            case 25: return launch_p1_scatter_shape<256, 12, 4, 25, 8>(a, p, s, grid_mode);
            case 21: return launch_p1_scatter_shape<256, 12, 4, 21, 8>(a, p, s, grid_mode);
            default: break;
        }
    // beside a concurrent stream otherwise: a 64-register shape of four blocks
    // an SM, so that three work while a fourth block's room stays free (for
    // 512 partitions with rounds of 16 records, which spill some registers:
    // a round of 2048 would write runs of 4)
    if (grid_mode == kScatterShared && p.bits == 8) return launch_p1_scatter_shape<256, 8, 4>(a, p, s, grid_mode);
    if (grid_mode == kScatterShared && single && p.bits == 9 && a.k == 31)
        return launch_p1_scatter_shape<256, 16, 4, 31, 9>(a, p, s, grid_mode);
    switch (shape) {  // shape 3 changes only the level-2 scatter, shape 4 only level 1
        case 1: return launch_p1_scatter_shape<512, 8, 2>(a, p, s, grid_mode);
        case 2: return launch_p1_scatter_shape<256, 8, 4>(a, p, s, grid_mode);
        default:
            if (single && p.bits == 9 && a.k == 31)  // past 400M occurrences: 512 partitions
                return launch_p1_scatter_shape<256, 16, 3, 31, 9>(a, p, s, grid_mode);
            return launch_p1_scatter_shape<256, 16, 3>(a, p, s, grid_mode);
    }
}

int launch_part_wave(const BuildArgs &a, const PartArgs &p, uint32_t p0, uint32_t n, uint64_t rb,
                     uint64_t re, cudaStream_t s) {
    int launches = 0;
    if (re > rb) {
        const uint64_t blocks = (re - rb + kK1Block - 1) / kK1Block;
        const uint64_t grid = std::min<uint64_t>(blocks, (uint64_t)device_sm_count() * 8);
        k_part_insert<<<(unsigned)grid, kK1Block, 0, s>>>(a, p, p0, n, rb, re);
        launches++;
    }
    const uint64_t grid = (uint64_t)n * (p.slot_cap / kPartChunk);
    if (grid) {
        k_part_compact<<<(unsigned)grid, kCBlock, 0, s>>>(a, p, p0);
        launches++;
    }
    return launches;
}

int launch_chunk_prefix(const BucketArgs &b, cudaStream_t s) {
    k_chunk_prefix<<<1, 1024, 0, s>>>(b);
    return 1;
}

int launch_sub_hist(const BucketArgs &b, cudaStream_t s) {
    if (!b.n_rec) return 0;
    const uint64_t chunks = b.n_rec / kBkChunk + b.n_parts;  // bound on the partition-aligned chunks
    const uint64_t grid = std::min<uint64_t>(chunks, resident_grid(k_sub_hist, 256, 0));
    k_sub_hist<<<(unsigned)grid, 256, 0, s>>>(b);
    return 1;
}

template <int NT, int IT, int MINB>
int launch_sub_scatter_shape(const BucketArgs &b, cudaStream_t s) {
    static_assert(NT * IT == kBkChunk, "a level-2 chunk is one block's round");
    auto kern = k_sub_scatter<NT, IT, MINB>;
    const uint64_t chunks = b.n_rec / kBkChunk + b.n_parts;  // bound on the partition-aligned chunks
    allow_smem(kern, kSubScatterDyn);
    const uint64_t grid = std::min<uint64_t>(chunks, resident_grid(kern, NT, kSubScatterDyn));
    kern<<<(unsigned)grid, NT, kSubScatterDyn, s>>>(b);
    return 1;
}

// One shared atomic per record (the histogram's returns the rank).
template <int NT, int IT, int MINB>
int launch_sub_scatter2_shape(const BucketArgs &b, cudaStream_t s) {
    static_assert(NT * IT == kBkChunk, "a level-2 chunk is one block's round");
    auto kern = k_sub_scatter2<NT, IT, MINB>;
    const uint64_t chunks = b.n_rec / kBkChunk + b.n_parts;
    const size_t smem = sub_scatter2_smem(b.b2);
    allow_smem(kern, sub_scatter2_smem(10));
    const uint64_t grid = std::min<uint64_t>(chunks, resident_grid(kern, NT, smem));
    kern<<<(unsigned)grid, NT, smem, s>>>(b);
    return 1;
}

int launch_sub_scatter(const BucketArgs &b, cudaStream_t s) {
    if (!b.n_rec) return 0;
    switch (b.shape ? b.shape : scatter_shape()) {
        case 1: return launch_sub_scatter_shape<512, 8, 2>(b, s);
        case 2: return launch_sub_scatter_shape<512, 8, 3>(b, s);
        default: return launch_sub_scatter2_shape<256, 16, 3>(b, s);
        case 3: {  // bulk-copy staging (measured slower on GB300: 2 blocks/SM instead of 3)
            const uint64_t chunks = b.n_rec / kBkChunk + b.n_parts;
            allow_smem(k_sub_scatter_tma, kSubScatterTmaDyn);
            const uint64_t grid =
                std::min<uint64_t>(chunks, resident_grid(k_sub_scatter_tma, 256, kSubScatterTmaDyn));
            k_sub_scatter_tma<<<(unsigned)grid, 256, kSubScatterTmaDyn, s>>>(b);
            return 1;
        }
    }
}

int bucket_count_table(bool tagged, uint64_t n_rec, uint64_t nb) {
    // SWG_BUCKET_SMALL: 0 keeps the 4096-entry tables, 2 takes the small ones
    // for every untagged build, unset or 1 picks by the mean bucket size
    const char *e = std::getenv("SWG_BUCKET_SMALL");
    const int small_mode = e ? std::atoi(e) : 1;
    return small_mode && !tagged && (small_mode == 2 || n_rec <= kBkSmallRecords * nb) ? kBkTableS : kBkTable;
}

int launch_bucket_count(const BuildArgs &a, const BucketArgs &b, cudaStream_t s) {
    const uint64_t nb = (uint64_t)b.n_parts << b.b2;
    const size_t tag = a.tag_bits ? kBucketTagSmem : 0;
    const size_t smem1 = bucket_smem<kBkTable>() + tag, smem2 = bucket_smem<kBkTable2>() + tag;
    if (bucket_count_table(a.tag_bits != 0, b.n_rec, nb) == kBkTableS) {  // small buckets on average
        const size_t smemS = bucket_smem<kBkTableS>();
        allow_smem(k_bucket_count_small, smemS);
        const uint64_t grid = std::min<uint64_t>(nb, resident_grid(k_bucket_count_small, kBkThreadsS, smemS));
        k_bucket_count_small<<<(unsigned)grid, kBkThreadsS, smemS, s>>>(a, b, nb);
    } else {
        allow_smem(k_bucket_count, bucket_smem<kBkTable>() + kBucketTagSmem);
        const uint64_t grid = std::min<uint64_t>(nb, resident_grid(k_bucket_count, kBkThreads, smem1));
        k_bucket_count<<<(unsigned)grid, kBkThreads, smem1, s>>>(a, b, nb);
    }
    allow_smem(k_bucket_count_large, bucket_smem<kBkTable2>() + kBucketTagSmem);
    k_bucket_count_large<<<(unsigned)device_sm_count(), kBkThreads2, smem2, s>>>(a, b);
    return 2;
}


int launch_group_by_sample(const unsigned long long *in_keys, const unsigned long long *in_mult,
                           uint64_t n, int tag_bits, uint32_t n_samples, unsigned long long *cursor,
                           unsigned long long *out_keys, unsigned long long *out_mult, cudaStream_t s) {
    if (!n) return 0;
    const uint64_t grid = std::min<uint64_t>((n + 2047) / 2048, (uint64_t)device_sm_count() * 8);
    k_group_by_sample<<<(unsigned)grid, 256, 0, s>>>(in_keys, in_mult, n, tag_bits, n_samples, cursor,
                                                     out_keys, out_mult);
    return 1;
}

int launch_bucket_gather(const BuildArgs &a, const BucketArgs &b, uint64_t n_buckets, cudaStream_t s) {
    const uint64_t threads = std::max<uint64_t>(n_buckets, 1) * 32;
    k_bucket_gather<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(a, b, n_buckets);
    return 1;
}

int launch_p1_sample(const BuildArgs &a, const PartArgs &p, const BucketArgs &b, uint32_t stride,
                     cudaStream_t s) {
    if (a.total_occ == 0 || a.n_reads == 0) return 0;
    const uint64_t batches = (a.n_reads + 255) / 256;
    const uint64_t grid = std::min<uint64_t>((batches + stride - 1) / stride, resident_grid(k_p1_sample, 256, 0));
    k_p1_sample<<<(unsigned)std::max<uint64_t>(grid, 1), 256, 0, s>>>(a, p, b, stride);
    return 1;
}

int launch_part_caps(const PartArgs &p, uint64_t n_rec, unsigned long long *sampled, cudaStream_t s) {
    k_part_caps<<<1, 1024, 0, s>>>(p, n_rec, sampled);
    return 1;
}

int launch_bucket_caps(const unsigned long long *counts, const unsigned long long *sampled, uint64_t n_rec,
                       uint64_t nb, unsigned long long *caps, cudaStream_t s) {
    k_bucket_caps<<<(unsigned)((nb + 255) / 256), 256, 0, s>>>(counts, sampled, n_rec, nb, caps);
    return 1;
}

int launch_big_multi(const BuildArgs &a, const BucketArgs &b, const unsigned long long *meta, uint32_t n,
                     uint64_t records, Entry *table, uint64_t cap, cudaStream_t s) {
    if (!n) return 0;
    const uint64_t blocks =
        std::min<uint64_t>((records + kK1Block - 1) / kK1Block, (uint64_t)device_sm_count() * 8);
    k_big_insert_multi<<<(unsigned)std::max<uint64_t>(blocks, 1), kK1Block, 0, s>>>(a, b.rec2, meta, n, table,
                                                                                     cap);
    return 1 + launch_big_compact(a, table, cap, s);
}

int launch_big_compact(const BuildArgs &a, const Entry *table, uint64_t cap, cudaStream_t s) {
    const uint64_t per = (uint64_t)kCBlock * kCItems;
    k_big_compact<<<(unsigned)((cap + per - 1) / per), kCBlock, 0, s>>>(a, table, cap);
    return 1;
}


// Shared-memory atomic probe (the on-chip roofline of the bucket count):
// two CTAs of 512 threads per SM, each with a zeroed table of kBkTable 64-bit
// slots and 4 x kBkTable 32-bit words (the bucket table's key and counter
// arrays), every thread issuing `iters` rounds of four independent operations
// at random slots. kind 0: 32-bit atomicAdd; kind 1: 64-bit atomicCAS (empty
// slot -> key; most find the slot taken, as most of a bucket's records do).
__global__ void __launch_bounds__(kBkThreads, 2) k_smem_probe(int kind, int iters, unsigned long long *sink) {
    extern __shared__ __align__(16) unsigned char dyn[];
    unsigned long long *keys = reinterpret_cast<unsigned long long *>(dyn);
    unsigned *cnt = reinterpret_cast<unsigned *>(keys + kBkTable);
    for (uint32_t j = threadIdx.x; j < (uint32_t)kBkTable; j += kBkThreads) {
        keys[j] = 0;
        reinterpret_cast<uint4 *>(cnt)[j] = make_uint4(0, 0, 0, 0);
    }
    __syncthreads();
    uint32_t x[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) x[q] = (blockIdx.x * kBkThreads + threadIdx.x) * 4u + q + 1u;
    unsigned long long acc = 0;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            x[q] = x[q] * 0x9e3779b1u + 0x7f4a7c15u;
            if (kind == 0) atomicAdd(&cnt[x[q] >> 18], 1u);  // 14 bits: 4 x kBkTable words
            else acc += atomicCAS(&keys[x[q] >> 20], 0ull, (unsigned long long)x[q] | 1ull);
        }
    }
    if (acc == 0x5a5a5a5a5a5a5a5aull) *sink = acc;  // keeps the CAS results live
}

cudaError_t run_smem_probe(int kind, uint64_t n_ops, cudaStream_t s, float *ms) {
    unsigned long long *sink = nullptr;
    cudaError_t err = cudaMalloc(&sink, sizeof(unsigned long long));
    if (err != cudaSuccess) return err;
    const size_t smem = (size_t)kBkTable * (sizeof(unsigned long long) + 4 * sizeof(unsigned));
    cudaFuncSetAttribute(k_smem_probe, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const unsigned grid = (unsigned)device_sm_count() * 2;
    const uint64_t per_round = (uint64_t)grid * kBkThreads * 4;
    const int iters = (int)std::max<uint64_t>(1, std::min<uint64_t>(n_ops / per_round, 1u << 20));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    k_smem_probe<<<grid, kBkThreads, smem, s>>>(kind, std::max(1, iters / 8), sink);  // warm-up
    cudaEventRecord(e0, s);
    k_smem_probe<<<grid, kBkThreads, smem, s>>>(kind, iters, sink);
    cudaEventRecord(e1, s);
    err = cudaEventSynchronize(e1);
    float t = 0;
    cudaEventElapsedTime(&t, e0, e1);
    *ms = t * (float)((double)n_ops / (double)(per_round * (uint64_t)iters));  // scale to n_ops
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    if (err == cudaSuccess) err = cudaGetLastError();
    return err;
}

cudaError_t run_probe(int kind, uint64_t table_bytes, uint64_t n_ops, cudaStream_t s, float *ms) {
    Entry *table = nullptr;
    unsigned long long *sink = nullptr;
    const uint64_t n16 = table_bytes / sizeof(Entry);
    if (n16 == 0) return cudaErrorInvalidValue;
    cudaError_t err = cudaMalloc(&table, n16 * sizeof(Entry));
    if (err != cudaSuccess) return err;
    err = cudaMalloc(&sink, sizeof(unsigned long long));
    if (err != cudaSuccess) {
        cudaFree(table);
        return err;
    }
    cudaMemsetAsync(table, 0, n16 * sizeof(Entry), s);
    const unsigned grid = (unsigned)device_sm_count() * 8;
    const uint64_t threads = (uint64_t)grid * 256;
    const uint64_t per = (n_ops + threads - 1) / threads;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    // warm-up launch, then the timed one
    k_probe<<<grid, 256, 0, s>>>(kind, table, n16, per / 4 + 1, 7, sink);
    cudaEventRecord(e0, s);
    k_probe<<<grid, 256, 0, s>>>(kind, table, n16, per, 11, sink);
    cudaEventRecord(e1, s);
    err = cudaEventSynchronize(e1);
    float t = 0;
    cudaEventElapsedTime(&t, e0, e1);
    *ms = t * (float)((double)n_ops / (double)(per * threads));  // scale to exactly n_ops
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    cudaFree(table);
    if (err == cudaSuccess) err = cudaGetLastError();
    return err;
}

}  // namespace swg
