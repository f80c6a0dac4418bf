// The bucketed build over super-k-mers (single k, odd, 19..31).
//
// The occurrences of a read are not written one by one. Every k-mer has a
// minimizer: the smallest hash among the canonical m-mers it contains, the
// same for both strands. Consecutive k-mers of a read mostly share it, so a
// read falls into runs (super-k-mers) of up to kSkRun k-mers with one
// minimizer, and all occurrences of a k-molecule fall into the bucket that
// their minimizer names. A run is one 16-byte record: its bases with the
// neighbour on each side, its k-mer count and flags. About one record per
// (w + 1) / 2 occurrences (w = k - m + 1) goes through the two scatters,
// 2 bytes an occurrence instead of 8, and the k-mers are cut out of the
// records only in the bucket's shared-memory count.
//
//   k_sk_pieces_*  long reads cut into pieces of kSkPiece k-mers
//   k_sk_scan      minimizers, runs; level-1 scatter of the records (or, on a
//                  sample of the reads, sizes per partition and bucket)
//   k_sk_regions (or k_sk_caps, k_sk_bucket_caps)   regions
//   k_sk_sub       level-2 scatter into buckets
//   k_sk_count*    per-bucket counting, cutoff, survivors
//   k_sk_big       buckets no shared-memory table holds
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "dev_util.cuh"
#include "kmer_dev.cuh"
#include "swg_internal.h"

namespace swg {
namespace {

// Record: bits 127..30 the run's bases, first base on top: left neighbour,
// n + k - 1 bases, right neighbour (at most 1 + 47 + 1); bits 0-4 n, bit 5 /
// 6 a left / right neighbour exists, bits 7-16 sub-bucket, 17-26 sample.
constexpr uint32_t kSkRun = 17;        // k-mers per record
constexpr int kSkThreads = 256;
constexpr unsigned kSkQueue = 320;     // runs found and not yet written, per warp
constexpr uint32_t kSkMaxStart = (1u << 14) - 1;  // k-mers of a read or piece
constexpr uint32_t kSkPiece = 256;     // k-mers of a piece of a long read
constexpr int kSubItems = 8;
constexpr uint32_t kSkChunk = 256 * kSubItems;  // records per level-2 chunk
// a bucket's records are counted this many at a time (16-bit counters: 3840 x
// 17 + 255 occurrences cannot carry), the counters clamped to 255 in between
constexpr uint32_t kSkClamp = 3840;
// larger buckets go to the global table: one CTA alone counts a bucket, others
// wait for it at the end (2.4G occurrences with 2% tandem repeats: count 17.5 ms
// with 16384, 16.0 with 8192, 14.6 with 4096, the build 27.6, 26.1 and 26.7)
constexpr uint64_t kSkBigRecords = 8192;

// Bucket of a minimizer (lowbias32 of Wellons's hash-prospector).
__device__ __forceinline__ uint32_t sk_mix(uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    return x ^ (x >> 16);
}

// ---- pieces of long reads: a piece's length word has bit 30 / 31 set when a
// base precedes / follows it in its read. A thread per read left 80 blocks for
// 20,000 reads of 3 to 15 kbp; level 1 over pieces takes 0.40 ms there (setup
// included 0.53), the single-occurrence scatter took 5.5 (7.3).
__global__ void __launch_bounds__(256) k_sk_pieces_count(BuildArgs a, uint64_t *__restrict__ n) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.n_reads) return;
    n[r] = (occ_of(a.read_len[r], a.k) + kSkPiece - 1) / kSkPiece;
}

// A warp per read.
__global__ void __launch_bounds__(256) k_sk_pieces_fill(BuildArgs a, const uint64_t *__restrict__ first,
                                                        uint64_t *__restrict__ off, uint32_t *__restrict__ len,
                                                        uint32_t *__restrict__ seg) {
    const uint64_t r = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (r >= a.n_reads) return;
    const uint64_t occ = occ_of(a.read_len[r], a.k), at = first[r], o = a.read_off[r];
    const uint64_t np = (occ + kSkPiece - 1) / kSkPiece;
    for (uint64_t j = threadIdx.x & 31; j < np; j += 32) {
        const uint64_t p = j * kSkPiece;
        const uint32_t nk = (uint32_t)umin64(kSkPiece, occ - p);
        off[at + j] = o + p;
        len[at + j] = (nk + (uint32_t)a.k - 1) | (j ? 1u << 30 : 0u) | (j + 1 < np ? 1u << 31 : 0u);
        if (seg) seg[at + j] = seg_of(a, r);
    }
}

// Minimizers and runs of every read, one thread per read (or piece). A block
// of W m-mers spans exactly K bases, one 64-bit window, so nothing but the
// window minima is carried along a read: m-mers and their reverse complements
// are cut from the top of the window at constant shifts. Window minima by the
// two-scan scheme of van Herk and of Gil and Werman: arr holds the suffix minima of the previous block's hashes;
// with the running minimum of this block they give one minimum per k-mer at
// three min operations each. A block leaves a bit mask of the positions where
// the minimum changes; the runs that end there are queued after it, a warp's
// lanes together (few lanes have one at any one position). Each warp fills
// its own part of the queue, without barriers, until it is full or its reads
// are done. Then the block writes the queue: every run's partition and its
// rank there (one shared atomic), one global atomic per partition for the
// run of records, and each thread cuts queued runs' 49-base windows out of
// the packed words (L1 hits) and stores them. Records of a partition are
// neighbours in memory, so L2 merges the 16-byte stores; ordering them in
// shared memory first is not needed. Queue entry: low word start (14 bits),
// k-mers (5), thread (8); high word the minimizer, then partition (10 bits),
// sub-bucket (10), rank (12).
// kSample: only counts, per partition and per bucket.
// Bound by the ALU pipe (80% busy: shifts, minima and selects at half rate).
// 2.5M reads of 100 bp, 175M occurrences, k = 31: 0.38 ms, where the scatter of
// single occurrences took 0.81 and wrote four times the bytes. With runs pushed
// from inside the block 0.61 (a warp's few lanes at a time); with every load
// checked against the read's end 0.40.
template <int M, int W, bool kSample>
__global__ void __launch_bounds__(kSkThreads, 4) k_sk_scan(BuildArgs a, SkArgs s, uint32_t stride) {
    constexpr int K = M + W - 1, NT = kSkThreads, NW = NT / 32;
    constexpr uint32_t kTop = ~0u << (32 - 2 * M);
    constexpr unsigned kEnd = 1u << 31;  // mask bit of the read's end
    static_assert(M <= 15 && K <= 31 && W <= (int)kSkRun, "one 64-bit window per block of m-mers");
    extern __shared__ __align__(16) unsigned char dyn[];
    uint2 *queue = reinterpret_cast<uint2 *>(dyn);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(queue + (kSample ? 0 : NW * kSkQueue));
    uint64_t *s_off = reinterpret_cast<uint64_t *>(dst + (kSample ? 0 : s.n_parts));
    unsigned *hist = reinterpret_cast<unsigned *>(s_off + (kSample ? 0 : NT));
    uint32_t *s_mv = hist + s.n_parts;  // [W][NT] window minima of a block
    unsigned *fit = s_mv + W * NT;
    unsigned *s_nk = fit + s.n_parts;
    unsigned *s_tag = s_nk + NT;
    __shared__ unsigned long long s_base, s_first, s_end;
    const uint32_t tid = threadIdx.x, lane = tid & 31, lt = (1u << lane) - 1;
    uint2 *const wqueue = queue + (tid >> 5) * kSkQueue;
    const int sh1 = 32 - s.b1, sh2 = 32 - s.b1 - s.b2;
    const uint32_t submask = (1u << s.b2) - 1;
    for (uint32_t j = tid; j < s.n_parts; j += NT) hist[j] = 0;
    if (tid == 0) {
        s_first = a.read_range ? a.read_range[0] : 0;
        s_end = a.read_range ? a.read_range[1] : s.n_pieces;
    }
    unsigned long long my_kmers = 0;
    const uint64_t inner = a.n_words > 4 ? a.n_words - 4 : 0;  // five words from any of these are in the reads
    for (;;) {
        if (tid == 0) s_base = atomicAdd(&s.work[kSample ? 0 : 1], kSample ? 1ull : (unsigned long long)NT) *
                               (kSample ? (unsigned long long)NT * stride : 1ull);
        __syncthreads();
        const uint64_t base = s_first + s_base;
        if (base >= s_end) break;
        __syncthreads();  // s_base read by all
        const uint64_t r = base + tid;
        uint32_t nk = 0, tag = 0;
        uint64_t off = 0;
        if (r < s_end) {
            const uint32_t lw = s.len[r], L = s.pieces ? lw & 0x3fffffffu : lw;
            nk = L >= (uint32_t)K ? L - (uint32_t)K + 1 : 0;
            if (nk > kSkMaxStart) nk = kSkMaxStart;  // the host does not use a result with such reads
            off = s.off[r];
            if (a.tag_bits) tag = s.seg[r];
            my_kmers += nk;
            if (!kSample) {
                s_off[tid] = off;
                s_nk[tid] = nk | (s.pieces ? lw & 0xc0000000u : 0u);
                if (a.tag_bits) s_tag[tid] = tag;
            }
        }
        __syncwarp();
        const uint32_t tmix = tag * 0x9e3779b1u;
        uint32_t arr[W];
        // cur, start: the open run's minimizer and first k-mer; ends: run ends
        // not yet queued, bit j at k-mer at + j; p: k-mers with a known minimum
        uint32_t cur = 0, start = 0, ends = 0, at = 0, p = 0, pos = 0;
        bool open = nk > 0;
        for (;;) {  // rounds: scan until the queue is full, write it out
            unsigned queued = 0;
            bool held = false;  // run ends left for the next round
            for (;;) {
                if (open && !ends) {
                    const uint64_t word = (off + pos) >> 4;
                    uint64_t win;
                    if (word < inner) {
                        const uint32_t *pk = a.packed + word;
                        const uint32_t sh = (uint32_t)((off + pos) & 15) * 2;
                        const uint32_t b0 = __ldg(pk), b1 = __ldg(pk + 1), b2 = __ldg(pk + 2);
                        win = (uint64_t)__funnelshift_l(b1, b0, sh) << 32 | __funnelshift_l(b2, b1, sh);
                    } else {
                        win = window32(a.packed, a.n_words, off + pos);
                    }
                    const uint64_t rct = revcomp_dev(win >> (64 - 2 * K), K) << (64 - 2 * K);
                    const uint32_t w1 = (uint32_t)(win >> 32), w0 = (uint32_t)win, r1 = (uint32_t)(rct >> 32),
                                   r0 = (uint32_t)rct;
                    uint32_t pre = ~0u, last = cur;
                    at = p;
#pragma unroll
                    for (int j = 0; j < W; ++j) {
                        if (j && j % 4 == 0 && pos && p + j >= nk) break;  // past the read's last k-mer
                        // (bits below the m-mer only break ties)
                        const uint32_t f = j < 16 ? __funnelshift_l(w0, w1, 2 * j) : w0;
                        const uint32_t v = W - 1 - j < 16 ? __funnelshift_l(r0, r1, 2 * (W - 1 - j)) : r0;
                        const uint32_t h = (min(f, v) & kTop) * 0x9e3779b1u + 0x7f4a7c15u;
                        pre = min(pre, h);
                        const uint32_t mv = j + 1 < W ? min(arr[j + 1 < W ? j + 1 : j], pre) : pre;
                        arr[j] = h;
                        if (pos) {
                            if (mv != last) ends |= 1u << j;
                            last = mv;
                            s_mv[j * NT + tid] = mv;
                        }
                    }
#pragma unroll
                    for (int j = W - 2; j >= 0; --j) arr[j] = min(arr[j], arr[j + 1]);
                    if (pos == 0) {  // the first K bases: one k-mer
                        cur = arr[0];
                        p = 1;
                    } else {
                        if (nk - p < (uint32_t)W) ends &= (1u << (nk - p)) - 1;
                        p += W;
                    }
                    pos += W;
                    if (p >= nk) {
                        ends |= kEnd;
                        open = false;
                    }
                }
                unsigned m;
                while ((m = __ballot_sync(kFull, ends != 0)) != 0) {
                    if (!kSample && queued + __popc(m) > kSkQueue) {
                        held = true;
                        break;
                    }
                    if (ends) {
                        const int j = __ffs(ends) - 1;
                        const uint32_t end = j == 31 ? nk : at + j;
                        const uint32_t n = min(end - start, kSkRun);
                        if (kSample) {
                            const uint32_t x = sk_mix(cur ^ tmix);
                            const uint32_t part = x >> sh1, sub = (x >> sh2) & submask;
                            atomicAdd(&hist[part], 1u);
                            atomicAdd(&s.cursor2[((uint64_t)part << s.b2) | sub], 1ull);
                        } else {
                            wqueue[queued + __popc(m & lt)] = make_uint2(start | n << 14 | tid << 19, cur ^ tmix);
                        }
                        start += n;
                        if (start == end) {
                            ends &= ends - 1;
                            if (j < 31) cur = s_mv[j * NT + tid];
                        }
                    }
                    queued += __popc(m);
                }
                if (held || !__any_sync(kFull, open)) break;
            }
            if (kSample) break;
            __syncwarp();  // the warp's queue is written
            for (uint32_t i = lane; i < queued; i += 32) {
                const uint32_t x = sk_mix(wqueue[i].y);
                const uint32_t part = x >> sh1, sub = (x >> sh2) & submask;
                wqueue[i].y = part | sub << 10 | atomicAdd(&hist[part], 1u) << 20;
            }
            const bool more = __syncthreads_or(held);  // every run is ranked
            for (uint32_t j = tid; j < s.n_parts; j += NT) {
                const unsigned c = hist[j];
                if (c) {
                    const unsigned long long g0 = atomicAdd(&s.part_cursor[j], (unsigned long long)c);
                    const unsigned long long lim = s.part_start[j + 1];
                    dst[j] = g0;
                    fit[j] = g0 + c <= lim ? c : (g0 < lim ? (unsigned)(lim - g0) : 0u);
                    hist[j] = 0;
                }
            }
            __syncthreads();
            for (uint32_t i = lane; i < queued; i += 32) {
                const uint2 e = wqueue[i];
                const uint32_t st = e.x & 0x3fffu, n = (e.x >> 14) & 31u, th = e.x >> 19;
                const uint32_t part = e.y & 1023u, sub = (e.y >> 10) & 1023u, rank = e.y >> 20;
                const uint32_t info = s_nk[th];
                const bool hl = st > 0 || (info & (1u << 30)), hr = st + n < (info & 0x3fffffffu) || (info >> 31);
                const uint64_t g = s_off[th] + st - 1;  // the left neighbour
                const uint64_t w = (uint64_t)((int64_t)g >> 4);
                const uint32_t sh = (uint32_t)(g & 15) * 2;
                uint32_t q0, q1, q2, q3, q4;
                if (w < inner) {
                    const uint32_t *pk = a.packed + w;
                    q0 = __ldg(pk), q1 = __ldg(pk + 1), q2 = __ldg(pk + 2), q3 = __ldg(pk + 3), q4 = __ldg(pk + 4);
                } else {
                    q0 = ldw(a.packed, w, a.n_words), q1 = ldw(a.packed, w + 1, a.n_words);
                    q2 = ldw(a.packed, w + 2, a.n_words), q3 = ldw(a.packed, w + 3, a.n_words);
                    q4 = ldw(a.packed, w + 4, a.n_words);
                }
                // bases past the run (and a neighbour that is none) are cleared:
                // equal runs are equal records
                const int bits = 2 * (int)(n + K) + (hr ? 2 : 0);
                uint4 rec;
                rec.x = __funnelshift_l(q1, q0, sh) & (hl ? ~0u : 0x3fffffffu);
                rec.y = __funnelshift_l(q2, q1, sh) & ~__funnelshift_rc(~0u, 0u, bits - 32);
                rec.z = __funnelshift_l(q3, q2, sh) & ~__funnelshift_rc(~0u, 0u, max(bits - 64, 0));
                rec.w = __funnelshift_l(q4, q3, sh) & ~__funnelshift_rc(~0u, 0u, max(bits - 96, 0));
                rec.w |= n | (hl ? 32u : 0u) | (hr ? 64u : 0u) | sub << 7;
                if (a.tag_bits) rec.w |= s_tag[th] << 17;
                if (rank < fit[part]) s.rec1[dst[part] + rank] = rec;  // past the region: flagged later
            }
            if (!more) break;
            __syncwarp();  // the queue is read
        }
    }
    if (kSample) {
        __syncthreads();
        for (uint32_t j = tid; j < s.n_parts; j += NT)
            if (hist[j]) atomicAdd(&s.part_count[j], (unsigned long long)hist[j]);
#pragma unroll
        for (int d = 16; d; d >>= 1) my_kmers += __shfl_down_sync(kFull, my_kmers, d);
        if (lane == 0 && my_kmers) atomicAdd(&s.sampled[1], my_kmers);
    }
}

size_t scan_smem(uint32_t n_parts, int w, bool sample) {
    const size_t both = (size_t)n_parts * sizeof(unsigned) + (size_t)w * kSkThreads * sizeof(uint32_t);
    if (sample) return both;
    return both + kSkThreads / 32 * kSkQueue * sizeof(uint2) +
           (size_t)n_parts * (sizeof(unsigned long long) + sizeof(unsigned)) +
           kSkThreads * (sizeof(uint64_t) + 2 * sizeof(unsigned));
}

// Records expected in the whole input, from the sample's records per k-mer,
// and at most rec_cap (which the buffers are sized for).
__device__ __forceinline__ double sk_records(const SkArgs &s, uint64_t sampled) {
    const unsigned long long km = s.sampled[1];
    double r = km ? (double)sampled / (double)km * (double)s.n_kmers * 1.02 : (double)s.rec_cap;
    return r < (double)s.rec_cap ? r : (double)s.rec_cap;
}

// What the regions follow from: the records expected and those per sampled
// record (worked out once a block: 64-bit arithmetic is slow here, and regions
// of single-precision sizes are as good).
struct SkScale {
    float r, f;
    bool sampled;
};
__device__ __forceinline__ SkScale sk_scale(const SkArgs &s, uint64_t sampled, SkScale *shared) {
    if (threadIdx.x == 0) {
        const double r = sk_records(s, sampled);
        shared->r = (float)r;
        shared->f = sampled ? (float)fmin(r / (double)sampled, s.scale_max) : 0.0f;
        shared->sampled = sampled != 0;
    }
    __syncthreads();
    return *shared;
}

// A partition's region: 1.25 x its share of the expected records + 1024.
__device__ __forceinline__ uint64_t part_cap(const SkArgs &s, uint64_t count, const SkScale &x) {
    return (uint64_t)(1.25f * (x.sampled ? (float)count * x.f : x.r / (float)s.n_parts)) + 1024;
}

// A bucket's region. Its sample is a few dozen records, so the region covers
// the mean that is six standard deviations of a Poisson count above what was
// seen, and a quarter more for tandem repeats, whose reads bring several
// records each to one bucket: 1.25 c + 18 + 6 sqrt(c + 9) sampled records,
// times the input's records per sampled one (at most scale_max, which the
// buffers are sized for).
__device__ __forceinline__ uint64_t bucket_cap(uint64_t count, const SkScale &x, uint64_t nb) {
    const float c = (float)count;
    return (uint64_t)(x.sampled ? x.f * (1.25f * c + 18.0f + 6.0f * sqrtf(c + 9.0f)) : x.r / (float)nb);
}

// Partition regions, laid out by exclusive prefix (one block). The sampled
// total goes to sampled[0].
__global__ void __launch_bounds__(1024) k_sk_caps(SkArgs s) {
    __shared__ uint64_t wb[32];
    const uint32_t j = threadIdx.x;
    const uint64_t c = j < s.n_parts ? s.part_count[j] : 0;
    uint64_t total;
    block_exclusive_scan<1024>(c, wb, &total);
    uint64_t cap = 0;
    __shared__ SkScale sc;
    const SkScale x = sk_scale(s, total, &sc);
    if (j < s.n_parts) cap = part_cap(s, c, x);
    uint64_t all;
    const uint64_t ex = block_exclusive_scan<1024>(cap, wb, &all);
    if (j < s.n_parts) {
        s.part_start[j] = ex;
        s.part_cursor[j] = ex;
    }
    if (j == 0) {
        s.part_start[s.n_parts] = all;
        s.sampled[0] = total;
    }
}

// Bucket regions (counts and caps may be the same array).
__global__ void __launch_bounds__(256) k_sk_bucket_caps(SkArgs s, const unsigned long long *counts, uint64_t nb,
                                                        unsigned long long *caps) {
    __shared__ SkScale sc;
    const SkScale x = sk_scale(s, s.sampled[0], &sc);
    const uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < nb) caps[j] = bucket_cap(counts[j], x, nb);
}

// Regions of one size, of the partitions and of the buckets of a second level.
__global__ void __launch_bounds__(1024) k_sk_uniform(SkArgs s, uint64_t part, uint32_t nb, uint64_t bucket) {
    const uint32_t j = blockIdx.x * 1024 + threadIdx.x;
    if (j < s.n_parts) s.part_start[j] = s.part_cursor[j] = j * part;
    if (j == 0) s.part_start[s.n_parts] = s.n_parts * part;
    if (j < nb) s.off2[j] = s.cursor2[j] = j * bucket;
    if (j == 0 && nb) s.off2[nb] = nb * bucket;
}

// Both kinds of regions of a plan of at most 1024 kRegionItems buckets, and
// the cursors at their starts, by one block (six launches otherwise, most of a
// small build's preparation). Single precision: 9 us for 2048 buckets, 25 in
// double.
constexpr int kRegionItems = 16;
__global__ void __launch_bounds__(1024) k_sk_regions(SkArgs s, uint32_t nb) {
    __shared__ uint64_t wb[32];
    const uint32_t j = threadIdx.x;
    const uint64_t pc = j < s.n_parts ? s.part_count[j] : 0;
    uint64_t sampled;
    block_exclusive_scan<1024>(pc, wb, &sampled);
    __shared__ SkScale sc;
    const SkScale x = sk_scale(s, sampled, &sc);
    uint64_t cap = 0, all;
    if (j < s.n_parts) cap = part_cap(s, pc, x);
    const uint64_t ex = block_exclusive_scan<1024>(cap, wb, &all);
    if (j < s.n_parts) {
        s.part_start[j] = ex;
        s.part_cursor[j] = ex;
    }
    if (j == 0) s.part_start[s.n_parts] = all;
    const uint32_t per = (nb + 1023) / 1024;
    uint64_t c[kRegionItems], sum = 0;
#pragma unroll
    for (int i = 0; i < kRegionItems; ++i) {
        const uint32_t b = j * per + i;
        c[i] = i < (int)per && b < nb ? bucket_cap(s.cursor2[b], x, nb) : 0;
        sum += c[i];
    }
    uint64_t at = block_exclusive_scan<1024>(sum, wb, &all);
#pragma unroll
    for (int i = 0; i < kRegionItems; ++i) {
        const uint32_t b = j * per + i;
        if (i < (int)per && b < nb) {
            s.off2[b] = at;
            s.cursor2[b] = at;
        }
        at += c[i];
    }
    if (j == 0) s.off2[nb] = all;
}

// Level-2 scatter: a chunk of one partition's records is held in registers,
// ordered by sub-bucket in shared memory and written as one run per bucket.
// Every block works out the partitions' chunks for itself (and flags a
// partition that outgrew its region). Bound by memory latency and bandwidth:
// 175M occurrences 0.145 ms, 0.68 for the records of single ones (8 B each,
// where these take 2 an occurrence).
size_t sub_smem(int b2, uint32_t n_parts) {
    return kSkChunk * sizeof(uint4) + ((size_t)1 << b2) * (sizeof(unsigned long long) + 3 * sizeof(unsigned)) +
           (n_parts + 1) * sizeof(unsigned);
}

__global__ void __launch_bounds__(256, 4) k_sk_sub(SkArgs s) {
    constexpr int NT = 256, IT = kSubItems;
    extern __shared__ __align__(16) unsigned char dyn[];
    const uint32_t P2 = 1u << s.b2;
    uint4 *sorted = reinterpret_cast<uint4 *>(dyn);
    unsigned long long *dst = reinterpret_cast<unsigned long long *>(sorted + kSkChunk);
    unsigned *hist = reinterpret_cast<unsigned *>(dst + P2);
    unsigned *loff = hist + P2, *lim = loff + P2;
    unsigned *chunk_start = lim + P2;
    __shared__ uint64_t wb[NT / 32];
    const uint32_t per = (P2 + NT - 1) / NT, submask = P2 - 1;
    for (uint32_t j = threadIdx.x; j < P2; j += NT) hist[j] = 0;
    const uint32_t pp = (s.n_parts + NT - 1) / NT;
    unsigned chunks = 0;
    bool outgrown = false;
    for (uint32_t x = 0; x < pp; ++x) {
        const uint32_t j = threadIdx.x * pp + x;
        if (j < s.n_parts) {
            const uint64_t end = s.part_cursor[j], lim2 = s.part_start[j + 1];
            outgrown |= end > lim2;
            const unsigned c = (unsigned)((umin64(end, lim2) - s.part_start[j] + kSkChunk - 1) / kSkChunk);
            chunk_start[j] = c;
            chunks += c;
        }
    }
    uint64_t nq;
    unsigned run0 = (unsigned)block_exclusive_scan<NT>(chunks, wb, &nq);
    for (uint32_t x = 0; x < pp; ++x) {
        const uint32_t j = threadIdx.x * pp + x;
        if (j < s.n_parts) {
            const unsigned c = chunk_start[j];
            chunk_start[j] = run0;
            run0 += c;
        }
    }
    if (__syncthreads_or(outgrown || (*s.status & kStatusPartOverflow))) {  // the build recounts
        if (threadIdx.x == 0) atomicOr(s.status, kStatusPartOverflow);
        return;
    }
    for (uint64_t q = blockIdx.x; q < nq; q += gridDim.x) {
        uint32_t lo = 0, hi = s.n_parts;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (chunk_start[mid] <= q) lo = mid;
            else hi = mid;
        }
        const uint64_t r0 = s.part_start[lo] + (q - chunk_start[lo]) * kSkChunk;
        const uint32_t n = (uint32_t)umin64(kSkChunk, umin64(s.part_cursor[lo], s.part_start[lo + 1]) - r0);
        uint4 v[IT];
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            const uint32_t r = (uint32_t)it * NT + threadIdx.x;
            v[it] = r < n ? s.rec1[r0 + r] : make_uint4(0, 0, 0, 0);
        }
        __syncthreads();  // hist cleared, the previous chunk written out
        unsigned rk[IT];
#pragma unroll
        for (int it = 0; it < IT; ++it) {
            rk[it] = 0;
            if ((uint32_t)it * NT + threadIdx.x < n) rk[it] = atomicAdd(&hist[(v[it].w >> 7) & submask], 1u);
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
                lim[j] = (unsigned)run;
                if (c) {
                    const uint64_t bkj = ((uint64_t)lo << s.b2) | j;
                    const unsigned long long g0 = atomicAdd(&s.cursor2[bkj], (unsigned long long)c);
                    const unsigned long long end = s.off2[bkj + 1];
                    lim[j] += g0 + c <= end ? c : (g0 < end ? (unsigned)(end - g0) : 0u);
                    dst[j] = g0 - run;
                }
                hist[j] = 0;
                run += c;
            }
        }
        __syncthreads();
#pragma unroll
        for (int it = 0; it < IT; ++it)
            if ((uint32_t)it * NT + threadIdx.x < n) sorted[loff[(v[it].w >> 7) & submask] + rk[it]] = v[it];
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < n; j += NT) {
            const uint4 x = sorted[j];
            const uint32_t b = (x.w >> 7) & submask;
            if (j < lim[b]) s.rec2[dst[b] + j] = x;  // past the region: flagged by the count
        }
    }
}

// The k-mer at position pos (0..16) of a record: canonical key, and its arc
// slots (kmerGraph.cpp:240-296) with an increment of inc, or 0 where the
// record has no neighbour: right slot rs, left slot ls. kK: k (0: k_run).
struct SkOcc {
    uint64_t key;
    uint32_t rs, ls, radd, ladd;
};
template <int kK>
__device__ __forceinline__ SkOcc sk_kmer(uint4 x, uint32_t pos, uint32_t inc, int k_run) {
    const int k = kK ? kK : k_run;
    const uint32_t sh = 2 * pos;
    const uint32_t y0 = __funnelshift_lc(x.y, x.x, sh), y1 = __funnelshift_lc(x.z, x.y, sh),
                   y2 = __funnelshift_lc(x.w, x.z, sh);
    const uint64_t z = ((uint64_t)__funnelshift_l(y1, y0, 2) << 32) | __funnelshift_l(y2, y1, 2);
    const uint64_t kr = z >> (62 - 2 * k);  // the k-mer and its right neighbour
    const uint64_t fwd = kr >> 2, rc = revcomp_dev(fwd, k);
    const bool f = fwd >= rc;
    SkOcc o;
    o.key = f ? fwd : rc;
    o.rs = (f ? 0u : 4u) + ((uint32_t)kr & 3u);
    o.ls = (f ? 7u : 3u) - (y0 >> 30);
    o.radd = pos + 1 < (x.w & 31u) || (x.w & 64u) ? inc : 0u;
    o.ladd = pos || (x.w & 32u) ? inc : 0u;
    return o;
}

// A warp's records expanded: fn(valid, occurrence, record) with 32
// consecutive k-mers at a time. Each lane gives one record (rec.w = 0 for
// none, records in the lowest lanes) and its weight. Lane i of a step finds
// its record from the bit mask of the record starts among the step's 32
// k-mers.
template <int kK, typename F>
__device__ __forceinline__ void sk_expand(uint4 rec, uint32_t weight, int k, F &&fn) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t n = rec.w & 31u;
    uint32_t inc = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, inc, d);
        if (lane >= d) inc += y;
    }
    const uint32_t first = inc - n, total = __shfl_sync(kFull, inc, 31);
    const uint32_t wf = first | weight << 16;  // at most 32 * 17 k-mers; weight < 2^16
    const uint32_t le = kFull >> (31 - lane);
    uint32_t before = ~0u;  // records that start before this step, less one
    for (uint32_t t = 0; t < total; t += 32) {
        const uint32_t at = first - t;
        const uint32_t starts = __reduce_or_sync(kFull, n && at < 32 ? 1u << (at & 31) : 0u);
        const int owner = (int)(before + __popc(starts & le));
        before += __popc(starts);
        uint4 x;
        x.x = __shfl_sync(kFull, rec.x, owner);
        x.y = __shfl_sync(kFull, rec.y, owner);
        x.z = __shfl_sync(kFull, rec.z, owner);
        x.w = __shfl_sync(kFull, rec.w, owner);
        const uint32_t o = __shfl_sync(kFull, wf, owner);
        fn(t + lane < total, sk_kmer<kK>(x, (t + lane - o) & 31u, o >> 16, k), x);
    }
}

// Shared memory of a counting CTA: T keys, T x 8 uint16 counters, the warps'
// lists of used slots (half as many again as an even split of the table).
template <int T, int NT>
constexpr size_t count_smem() {
    return (size_t)T * (sizeof(unsigned long long) + 4 * sizeof(unsigned)) + (size_t)T * 3 / 2 * sizeof(unsigned short);
}

// Whether one of a slot's 8 counters reaches c (bias = 0x8000 - c in both
// halves, 1 <= c <= 255).
__device__ __forceinline__ bool bucket_keep(const unsigned *cnt, uint32_t s, unsigned bias) {
    const uint4 v = reinterpret_cast<const uint4 *>(cnt)[s];
    const unsigned x = (__vminu2(v.x, 0x00ff00ffu) + bias) | (__vminu2(v.y, 0x00ff00ffu) + bias),
                   y = (__vminu2(v.z, 0x00ff00ffu) + bias) | (__vminu2(v.w, 0x00ff00ffu) + bias);
    return ((x | y) & 0x80008000u) != 0;
}

// Persistent bucket counting over super-k-mer records, in a shared-memory
// table of T keys with 8 x 16-bit counters.
//  1. Equal records are merged: at a coverage of 30 to 50 reads most runs of a
//     bucket repeat others base for base, so counting each distinct one once,
//     with a weight, spares most of the expansion and of the table's atomics.
//     Up to CH records (nearly every bucket's all) go to the counter array,
//     which is all zero between buckets; a small table there maps a record's
//     hash to the first record with these bases, and counts the others.
//  2. The distinct records are listed, with the k-mers before them, and each
//     warp takes an even share of the k-mers (the warps wait for each other at
//     the bucket's end) into registers; the counter array is zero again.
//  3. The warps expand their records, 32 k-mers at a time, into the table:
//     64-bit CAS on the key, two 32-bit adds on 16-bit halves, every new slot
//     in the warp's own list.
//  4. The listed slots give the survivors: counted first (one global atomic
//     per warp takes their place in the output, so that no warp waits for
//     another here), then written; the slots are cleared on the way.
// Buckets whose keys do not fit go to the overflow list uncounted; their
// records stay as they are.
// Bound on chip, by the table's shared-memory atomics and what feeds them.
// 2.5M reads of 100 bp at 1% errors (175M occurrences, 50M of them distinct):
// 1.49 ms, of which inserting 0.86 (the probes past a slot that is taken 0.38,
// the adds 0.14), cutting the k-mers out of the records 0.34, the rest 0.30.
// Without merging equal records 2.05. The count of single occurrences took
// 1.27, after scatters that took 1.0 ms more than the records' do. A load
// before the CAS, or 32-bit CAS on the halves of a key, took longer (1.68,
// 1.75 to 1.89 against 1.62 with 131072 buckets).
template <int T, int NT, int kK>
__device__ void count_pass(const BuildArgs &a, const SkArgs &s, uint64_t n_items, uint32_t set,
                           const unsigned long long *list, unsigned long long *ovf, unsigned *ovf_count) {
    constexpr int kBits = T == 2048 ? 11 : (T == 4096 ? 12 : 13);
    constexpr int NW = NT / 32, SEG = T * 3 / 2 / NW, R = NT == 1024 ? 3 : 4;
    constexpr uint32_t CH = R * NT;
    static_assert((1 << kBits) == T, "table sizes");
    constexpr uint32_t kEven = 16 * R * NW;  // distinct records shared out by their k-mers
    static_assert(CH <= kSkClamp && CH * 24 <= T * 16, "merged records fit the counters' 16 bits and their array");
    static_assert(CH * 4 + kEven * 2 <= NW * SEG * 2, "the distinct records' list fits the slots' lists");
    extern __shared__ __align__(16) unsigned char dyn[];
    unsigned long long *keys = reinterpret_cast<unsigned long long *>(dyn);
    unsigned *cnt = reinterpret_cast<unsigned *>(keys + T);
    unsigned short *lists = reinterpret_cast<unsigned short *>(cnt + 4 * T);
    unsigned *s_dist = reinterpret_cast<unsigned *>(lists + NW * SEG);  // tagged batch only
    unsigned *s_surv = s_dist + a.n_segs;
    uint4 *srec = reinterpret_cast<uint4 *>(cnt);                // merging: records,
    unsigned *stab = cnt + 4 * CH;                               // table: first record (index + 1) | others << 16;
    unsigned *sdis = reinterpret_cast<unsigned *>(lists);        // distinct records: index | weight << 16,
    unsigned short *sbefore = reinterpret_cast<unsigned short *>(sdis + CH);  // k-mers before each
    __shared__ unsigned s_over, s_total, s_added;
    __shared__ uint64_t s_start[2][4];
    __shared__ unsigned s_n[2][4];
    const uint32_t lane = threadIdx.x & 31, wp = threadIdx.x >> 5, lt = (1u << lane) - 1;
    unsigned short *const used = lists + wp * SEG;
    const int tb = a.tag_bits, k = s.k;
    for (uint32_t j = threadIdx.x; j < (uint32_t)T; j += NT) {
        keys[j] = 0;
        reinterpret_cast<uint4 *>(cnt)[j] = make_uint4(0, 0, 0, 0);
    }
    if (tb)
        for (uint32_t j = threadIdx.x; j < a.n_segs; j += NT) s_dist[j] = s_surv[j] = 0;
    const int c = a.cutoff;
    // (a cutoff of 0 keeps what 1 keeps: a multiplicity of 0 is no arc)
    const unsigned cbias = (0x8000u - (unsigned)min(max(c, 1), 255)) * 0x00010001u;
    const uint4 none = make_uint4(0, 0, 0, 0);
    // The CTA's buckets come in sets of `set` neighbours; it counts as many of a
    // set at once as it expects to fit its table (by the distinct keys a record
    // that it has seen) and the merging's CH records: what is done once per
    // pass, half the time of a pass over a bucket of few distinct k-molecules,
    // is then shared. Two sets' bounds are kept, the later one read ahead.
    const uint32_t n_sets = (uint32_t)((n_items + set - 1) / set);  // (at most 2^20 buckets)
    bool outgrown = false;
    auto fetch = [&](uint32_t q, int buf) {
        if (threadIdx.x < set) {
            const uint64_t it = (uint64_t)q * set + threadIdx.x;
            uint64_t start = 0, n = 0;
            if (it < n_items) {
                const uint64_t bk = list ? list[it] : it;
                start = s.off2[bk];
                const uint64_t end = s.cursor2[bk], lim = s.off2[bk + 1];
                outgrown |= end > lim;
                n = umin64(end, lim) - start;
            }
            s_start[buf][threadIdx.x] = start;
            s_n[buf][threadIdx.x] = (unsigned)umin64(n, 1u << 30);
        }
    };
    uint32_t per_record = 32 << 8;  // distinct keys a record so far, 8 fraction bits (before the first pass: one bucket)
    uint32_t cur = blockIdx.x;      // set, its buffer, the pass's first bucket in it, how many, their records
    int buf = 0;
    uint32_t i0 = 0, nb = 0, nrec = 0;
    auto pick = [&]() {
        nb = 1;
        nrec = s_n[buf][i0];
        while (i0 + nb < set) {
            const uint32_t n = nrec + s_n[buf][i0 + nb];
            if (n > CH || (n * per_record) >> 8 > (uint32_t)T * 15 / 32) break;  // (no overflow: n <= CH, a record's 17 k-mers)
            nrec = n;
            ++nb;
        }
    };
    uint4 rec[R];
    auto load = [&]() {  // record i * NT + threadIdx.x of the pass's first min(nrec, CH)
        if (nb == 1) {
            const uint4 *from = s.rec2 + s_start[buf][i0];
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const uint32_t r = i * NT + threadIdx.x;
                rec[i] = r < nrec ? from[r] : none;
            }
            return;
        }
#pragma unroll
        for (int i = 0; i < R; ++i) {
            uint32_t r = i * NT + threadIdx.x, j = i0;
            rec[i] = none;
            if (r < nrec) {
                while (j + 1 < i0 + nb && r >= s_n[buf][j]) r -= s_n[buf][j++];
                rec[i] = s.rec2[s_start[buf][j] + r];
            }
        }
    };
    auto overflow = [&]() {  // the pass's buckets to the overflow list (one thread)
        for (uint32_t j = i0; j < i0 + nb; ++j) {
            const uint64_t it = (uint64_t)cur * set + j;
            if (!s_n[buf][j]) continue;
            const unsigned i = atomicAdd(ovf_count, 1u);
            if (i < s.big_cap) ovf[i] = list ? list[it] : it;
        }
    };
    fetch(cur, 0);
    fetch(cur + gridDim.x, 1);
    __syncthreads();
    pick();
    load();
    unsigned long long distinct = 0;  // keys this warp added to tables
    // to the next pass's buckets; the set after the next one is fetched at the
    // top of the first pass over a set, which is past all reads of its buffer
    bool fresh_set = false;
    auto advance = [&]() {
        i0 += nb;
        if (i0 >= set) {
            i0 = 0;
            cur += gridDim.x;
            buf ^= 1;
            fresh_set = true;
        }
        pick();
    };
    while (cur < n_sets) {
        __syncthreads();  // the previous pass is done: the table is all zero
        if (fresh_set) fetch(cur + gridDim.x, buf ^ 1);
        fresh_set = false;
        if (nrec > kSkBigRecords) {
            if (threadIdx.x == 0) overflow();
            __syncthreads();  // (the bounds fetched above are read from here on)
            advance();
            load();
            continue;
        }
        if (threadIdx.x == 0) {
            s_over = 0;
            s_total = 0;
            s_added = 0;
        }
        // equal records among the first CH merged
        const uint32_t n0 = min(nrec, CH);
        const int tbits = min(31 - __clz(4 * n0 + 255), 31 - __clz(2 * CH));
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (i * NT + threadIdx.x < n0) srec[i * NT + threadIdx.x] = rec[i];
        __syncthreads();
        uint32_t first[R];   // slot of the table where record i is the first with its bases; ~0: it is not
        uint32_t own = 0;    // this thread's distinct records << 16 | their k-mers
#pragma unroll
        for (int i = 0; i < R; ++i) {
            first[i] = ~0u;
            const uint32_t r = i * NT + threadIdx.x;
            if (r < n0) {
                uint32_t h = (rec[i].x * 0x9e3779b1u ^ rec[i].y * 0x85ebca6bu) + (rec[i].z * 0xc2b2ae35u ^ rec[i].w * 0x27d4eb2fu);
                h = (h ^ h >> 15) * 0x2c1b3c6du >> (32 - tbits);
                for (;;) {  // ends: the table has free slots
                    const unsigned old = atomicCAS(&stab[h], 0u, r + 1);
                    if (old == 0) {
                        first[i] = h;
                        own += 1u << 16 | (rec[i].w & 31u);
                        break;
                    }
                    const uint4 x = srec[(old & 0xffffu) - 1];
                    if (x.x == rec[i].x && x.y == rec[i].y && x.z == rec[i].z && x.w == rec[i].w) {
                        atomicAdd(&stab[h], 1u << 16);
                        break;
                    }
                    h = (h + 1) & ((1u << tbits) - 1);
                }
            }
        }
        uint32_t at = own;  // where this thread's distinct records go in the list << 16 | k-mers before them
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, at, d);
            if ((int)lane >= d) at += y;
        }
        unsigned base = 0;
        if (lane == 31 && at) base = atomicAdd(&s_total, at);
        at += __shfl_sync(kFull, base, 31) - own;
        __syncthreads();
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const uint32_t r = i * NT + threadIdx.x;
            if (first[i] != ~0u) {
                sdis[at >> 16] = r | (1u + (stab[first[i]] >> 16)) << 16;
                if (at >> 16 < kEven) sbefore[at >> 16] = (unsigned short)at;
                stab[first[i]] = 0;
                at += 1u << 16 | (rec[i].w & 31u);
            } else if (r < n0) {
                srec[r] = none;
            }
        }
        __syncthreads();
        // the warp's share of the distinct records (at most R a lane): an even
        // number of them if they are many or short, else of their k-mers, by
        // where the records start
        const uint32_t nd = s_total >> 16, nk = s_total & 0xffffu;
        uint32_t p0, p1;
        if (nd > kEven || nk < 4 * nd) {
            p0 = nd * wp / NW;
            p1 = nd * (wp + 1) / NW;
        } else {
            const uint32_t want = nk * (wp + (lane & 1)) / NW;  // lane 0: the share's start, lane 1: its end
            uint32_t lo = 0, hi = nd;
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (sbefore[mid] < want) lo = mid + 1;
                else hi = mid;
            }
            p0 = __shfl_sync(kFull, lo, 0);
            p1 = wp + 1 == NW ? nd : __shfl_sync(kFull, lo, 1);
        }
        uint32_t weight[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const uint32_t p = p0 + 32 * i + lane;
            rec[i] = none;
            weight[i] = 0;
            if (p < p1) {
                const uint32_t x = sdis[p];
                rec[i] = srec[x & 0xffffu];
                weight[i] = x >> 16;
                srec[x & 0xffffu] = none;
            }
        }
        for (uint32_t p = p0 + 32 * R + lane; p < p1; p += 32) {  // (uneven beyond that room: the next tier's)
            srec[sdis[p] & 0xffffu] = none;
            s_over = 1;
        }
        __syncthreads();  // the counter array is zero again, the list is read
        bool full = false;
        uint32_t nu = 0;  // slots in the warp's list
        auto insert = [&](bool valid, const SkOcc &o, const uint4 &x) {
            bool fresh = false;
            const unsigned long long key = tb ? o.key | (unsigned long long)((x.w >> 17) & 1023u) << (64 - tb) : o.key;
            // (double hashing: a warp's step takes as long as its longest probe sequence, and linear probing's clusters
            // made those longer: 1.51 -> 1.47 ms at 175M occurrences)
            const uint32_t hash = (uint32_t)key * 0x9e3779b1u + (uint32_t)(key >> 32) * 0x85ebca6bu;
            const uint32_t stride = (hash >> 7) | 1u;
            uint32_t slot = hash >> (32 - kBits);
            if (valid && !full) {
                uint32_t step = 0;
                unsigned long long old = 0;
                for (; step < (uint32_t)T; ++step) {
                    old = atomicCAS(&keys[slot], 0ull, key);
                    if (old == 0 || old == key) break;
                    slot = (slot + stride) & (T - 1);
                }
                if (step == (uint32_t)T) {
                    s_over = 1;
                    full = true;
                } else {
                    fresh = old == 0;
                    atomicAdd(&cnt[4 * slot + (o.rs >> 1)], o.radd << (16 * (o.rs & 1)));
                    atomicAdd(&cnt[4 * slot + (o.ls >> 1)], o.ladd << (16 * (o.ls & 1)));
                }
            }
            const unsigned fm = __ballot_sync(kFull, fresh);
            if (fresh) {
                const uint32_t q = nu + __popc(fm & lt);
                if (q < SEG) used[q] = (unsigned short)slot;
                else s_over = 1;
            }
            nu += __popc(fm);
        };
#pragma unroll
        for (int i = 0; i < R; ++i) {
            if (p0 + 32 * i >= p1) break;
            sk_expand<kK>(rec[i], weight[i], k, insert);
        }
        // a larger bucket's other records, one by one; the counters (which
        // saturate at 255 in the end) are clamped before they can carry
        for (uint32_t c0 = CH; c0 < nrec; c0 += kSkClamp) {
            __syncthreads();
            for (uint32_t j = threadIdx.x; j < (uint32_t)T; j += NT) {
                uint4 *e = reinterpret_cast<uint4 *>(cnt) + j;
                uint4 v = *e;
                v.x = __vminu2(v.x, 0x00ff00ffu);
                v.y = __vminu2(v.y, 0x00ff00ffu);
                v.z = __vminu2(v.z, 0x00ff00ffu);
                v.w = __vminu2(v.w, 0x00ff00ffu);
                *e = v;
            }
            __syncthreads();
            const uint32_t cn = min(nrec - c0, kSkClamp);
            const uint64_t rb = s_start[buf][i0];  // (a pass with more than CH records has one bucket)
            const uint64_t g1 = rb + c0 + cn * (wp + 1) / NW;
            for (uint64_t g = rb + c0 + cn * wp / NW; g < g1; g += 32)
                sk_expand<kK>(g + lane < g1 ? s.rec2[g + lane] : none, 1, k, insert);
        }
        if (lane == 0) atomicAdd(&s_added, nu);
        __syncthreads();
        const bool over = s_over != 0;
        if (over && threadIdx.x == 0) overflow();
        if (nrec >= 32) {  // a pass weighs a quarter; an eighth more for the spread
            const uint32_t seen = (s_added * 288u) / nrec;
            per_record = over ? min(2 * per_record, 32u << 8) : (per_record == 32 << 8 ? seen : (3 * per_record + seen) / 4);
        }
        advance();
        load();  // the next pass's records load while this one is compacted
        if (over) {
            for (uint32_t j = threadIdx.x; j < (uint32_t)T; j += NT) {
                keys[j] = 0;
                reinterpret_cast<uint4 *>(cnt)[j] = none;
            }
            continue;
        }
        // slots of no count >= c are cleared, the others move to the list's front
        uint32_t ns = 0;
        for (uint32_t i = 0; i < nu; i += 32) {
            uint32_t sl = 0;
            bool keep = false;
            if (i + lane < nu) {
                sl = used[i + lane];
                unsigned bias = cbias;
                int cs = c;
                if (tb) {
                    const uint32_t smp = (uint32_t)(keys[sl] >> (64 - tb));
                    cs = a.segs[smp].cutoff;
                    bias = (0x8000u - (unsigned)max(cs, 1)) * 0x00010001u;
                    atomicAdd(&s_dist[smp], 1u);
                }
                keep = cs < 256 && bucket_keep(cnt, sl, bias);
                if (!keep) {
                    keys[sl] = 0;
                    reinterpret_cast<uint4 *>(cnt)[sl] = none;
                } else if (tb) {
                    atomicAdd(&s_surv[(uint32_t)(keys[sl] >> (64 - tb))], 1u);
                }
            }
            const unsigned m = __ballot_sync(kFull, keep);
            __syncwarp();  // (a vote orders no memory: the lanes' slots are read before they are overwritten)
            if (keep) used[ns + __popc(m & lt)] = (unsigned short)sl;
            ns += __popc(m);
        }
        __syncwarp();  // the list's front is written: other lanes read it below
        distinct += nu;
        unsigned long long out = 0;
        if (lane == 0 && ns) {
            out = atomicAdd(&a.counters[1], (unsigned long long)ns);
            if (a.host_keys) atomicAdd(a.host_written, (unsigned long long)ns);
        }
        out = __shfl_sync(kFull, out, 0);
        for (uint32_t i = lane; i < ns; i += 32) {
            const uint32_t sl = used[i];
            const uint64_t pos = out + i;
            const unsigned long long key = keys[sl];
            unsigned bias = cbias;
            if (tb) {
                const int cs = a.segs[key >> (64 - tb)].cutoff;
                bias = cs > 0 ? (0x8000u - (unsigned)cs) * 0x00010001u : 0u;
            }
            const uint64_t m = bucket_mult(cnt, sl, bias, false);
            if (pos < a.out_cap) {
                a.out_keys[pos] = key;
                a.out_mult[pos] = m;
            }
            if (a.host_keys && pos < a.host_cap) {
                a.host_keys[pos] = key;
                a.host_mult[pos] = m;
            }
            keys[sl] = 0;
            reinterpret_cast<uint4 *>(cnt)[sl] = none;
        }
    }
    if (lane == 0 && distinct) atomicAdd(&a.counters[0], distinct);
    if (outgrown) atomicOr(s.status, kStatusPartOverflow);
    if (tb) {
        __syncthreads();
        for (uint32_t j = threadIdx.x; j < a.n_segs; j += NT) {
            if (s_dist[j]) atomicAdd(&a.seg_counts[2 * j], (unsigned long long)s_dist[j]);
            if (s_surv[j]) atomicAdd(&a.seg_counts[2 * j + 1], (unsigned long long)s_surv[j]);
        }
    }
}

// Tier 1 for plans of small buckets: four CTAs of 256 threads an SM with
// 2048-entry tables; else two of 512 threads with 4096 entries. Tier 2: one
// CTA of 1024 threads an SM with 8192 entries, over tier 1's overflow list.
template <int T, int NT, int kK>
__global__ void __launch_bounds__(NT, 1024 / NT) k_sk_count(BuildArgs a, SkArgs s, uint64_t n) {
    if (block_reads_overflow(s.status) || (T == 8192 && blockIdx.x >= *s.big_count)) return;
    if (T == 8192) {
        count_pass<T, NT, kK>(a, s, umin64(*s.big_count, s.big_cap), 1, s.big, s.big2, s.big2_count);
    } else {  // sets of four buckets, fewer where the CTAs would not get a dozen sets each
        const uint32_t set = n >= 48ull * gridDim.x ? 4 : (n >= 12ull * gridDim.x ? 2 : 1);
        count_pass<T, NT, kK>(a, s, n, set, nullptr, s.big, s.big_count);
    }
}

// First record and records of the buckets no shared-memory table holds.
__global__ void k_sk_big_bounds(SkArgs s, uint32_t n, unsigned long long *meta) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned long long b = s.big2[i], start = s.off2[b];
    meta[i] = start;
    meta[n + i] = umin64(s.cursor2[b], s.off2[b + 1]) - start;
}

// Those buckets, in one global-memory table of record hashes (rmix64 of the
// key, as k_big_compact reads it): meta = first record [n] | record prefix
// [n+1]. They are tandem repeats, so their k-mers are few and hot, and updates
// of the same entry go one after the other: equal records of a chunk are merged
// first, as in the tables' count, then equal keys of a warp's step. 2.4G
// occurrences with 2% tandem repeats, 31 such buckets: 1.0 ms, 2.9 record by
// record.
constexpr uint32_t kSkBigChunk = 1024;
__global__ void __launch_bounds__(256) k_sk_big(BuildArgs a, SkArgs s, const unsigned long long *meta, uint32_t n,
                                                Entry *table, uint64_t cap) {
    constexpr int R = kSkBigChunk / 256, kSlotBits = 11;
    __shared__ uint4 srec[kSkBigChunk];
    __shared__ unsigned stab[1 << kSlotBits], sdis[kSkBigChunk];  // first record (index + 1) | others << 16; distinct ones
    __shared__ unsigned s_distinct;
    const uint32_t lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const unsigned long long *rbs = meta, *pre = meta + n;
    const uint64_t total = pre[n];
    for (uint64_t g0 = (uint64_t)blockIdx.x * kSkBigChunk; g0 < total; g0 += (uint64_t)gridDim.x * kSkBigChunk) {
        for (uint32_t j = threadIdx.x; j < 1u << kSlotBits; j += 256) stab[j] = 0;
        if (threadIdx.x == 0) s_distinct = 0;
        uint4 rec[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const uint64_t g = g0 + i * 256 + threadIdx.x;
            if (g < total) {
                uint32_t lo = 0, hi = n;
                while (hi - lo > 1) {
                    const uint32_t mid = (lo + hi) >> 1;
                    if (pre[mid] <= g) lo = mid;
                    else hi = mid;
                }
                srec[i * 256 + threadIdx.x] = rec[i] = s.rec2[rbs[lo] + (g - pre[lo])];
            }
        }
        __syncthreads();
        uint32_t first[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            first[i] = ~0u;
            if (g0 + i * 256 + threadIdx.x >= total) continue;
            uint32_t h = (rec[i].x * 0x9e3779b1u ^ rec[i].y * 0x85ebca6bu) + (rec[i].z * 0xc2b2ae35u ^ rec[i].w * 0x27d4eb2fu);
            h = (h ^ h >> 15) * 0x2c1b3c6du >> (32 - kSlotBits);
            for (;;) {  // ends: the table has twice the chunk's slots
                const unsigned old = atomicCAS(&stab[h], 0u, i * 256 + threadIdx.x + 1);
                if (old == 0) {
                    first[i] = h;
                    break;
                }
                const uint4 x = srec[(old & 0xffffu) - 1];
                if (x.x == rec[i].x && x.y == rec[i].y && x.z == rec[i].z && x.w == rec[i].w) {
                    atomicAdd(&stab[h], 1u << 16);
                    break;
                }
                h = (h + 1) & ((1u << kSlotBits) - 1);
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (first[i] != ~0u)
                sdis[atomicAdd(&s_distinct, 1u)] = i * 256 + threadIdx.x | (1u + (stab[first[i]] >> 16)) << 16;
        __syncthreads();
        const uint32_t nd = s_distinct;
        for (uint32_t p0 = wp * 32; p0 < nd; p0 += 256) {
            uint4 one = make_uint4(0, 0, 0, 0);
            uint32_t weight = 0;
            if (p0 + lane < nd) {
                one = srec[sdis[p0 + lane] & 0xffffu];
                weight = sdis[p0 + lane] >> 16;
            }
            sk_expand<0>(one, weight, s.k, [&](bool valid, const SkOcc &o, const uint4 &x) {
                const unsigned vmask = __ballot_sync(kFull, valid);
                if (!valid) return;
                uint64_t key = o.key;
                if (a.tag_bits) key |= (uint64_t)((x.w >> 17) & 1023u) << (64 - a.tag_bits);
                // (counts saturate at 255: so may the sums on the way)
                const uint64_t inc = (uint64_t)min(o.radd, 255u) << (8 * o.rs) | (uint64_t)min(o.ladd, 255u) << (8 * o.ls);
                const unsigned peers = __match_any_sync(vmask, key);
                unsigned low = 0, high = 0;
                for (unsigned left = peers; __any_sync(vmask, left); left &= left - 1) {  // a round per lane of the largest group
                    const int from = left ? __ffs(left) - 1 : (int)lane;
                    const unsigned l = __shfl_sync(vmask, (unsigned)inc, from), h = __shfl_sync(vmask, (unsigned)(inc >> 32), from);
                    if (left) {
                        low = __vaddus4(low, l);
                        high = __vaddus4(high, h);
                    }
                }
                if (lane == (uint32_t)__ffs(peers) - 1)
                    insert_or_update(table, cap, rmix64(key), (uint64_t)high << 32 | low, a.status);
            });
        }
        __syncthreads();
    }
}

template <int M, int W>
int scan_launch(const BuildArgs &a, const SkArgs &s, uint64_t bound, uint32_t stride, bool sample, int grid_mode,
                cudaStream_t st) {
    const size_t smem = scan_smem(s.n_parts, W, sample);
    const uint64_t batches = (bound + kSkThreads - 1) / kSkThreads;
    const uint64_t sms = device_sm_count();
    if (sample) {
        auto kern = k_sk_scan<M, W, true>;
        allow_smem(kern, scan_smem(1u << kPartBitsMax, W, true));
        const uint64_t want = (batches + stride - 1) / stride;
        kern<<<(unsigned)std::max<uint64_t>(1, std::min(want, resident_grid(kern, kSkThreads, smem))), kSkThreads, smem,
               st>>>(a, s, stride);
        return 1;
    }
    auto kern = k_sk_scan<M, W, false>;
    allow_smem(kern, scan_smem(1u << kPartBitsMax, W, false));
    const uint64_t resident = resident_grid(kern, kSkThreads, smem);
    uint64_t grid = batches;
    if (grid_mode == kScatterResident) grid = std::min(batches, resident);
    if (grid_mode == kScatterShared) grid = std::min(batches, resident > sms ? resident - sms : resident);
    kern<<<(unsigned)std::max<uint64_t>(1, grid), kSkThreads, smem, st>>>(a, s, 1);
    return 1;
}

}  // namespace

// Window w of m-mers per k-mer (0: no super-k-mer build for this k), m = k - w
// + 1. Short m-mers make long runs, fewer records and more k-mers per block of
// the scan (up to the record's 17): but 4^m / 2 minimizers have to be several
// per bucket, or single ones make buckets uneven and too full. Builds at k =
// 21: of 216M occurrences of a 5 Mbp genome 2.13 ms with m = 11, 2.24 with 12,
// 2.37 with 13; of 693M of 40 Mbp 10.0 (329 buckets recounted), 7.8 and 8.2.
int super_window(int k, uint64_t occurrences) {
    const int m = occurrences <= (256ull << 20) ? 11 : (occurrences <= (2048ull << 20) ? 12 : 13);
    switch (k) {
        case 31: return 17;
        case 29: return 17;
        case 27: return 15;
        case 25: return m == 13 ? 13 : 14;
        case 23: case 21: case 19: return k - m + 1;
        default: return 0;
    }
}

int launch_super_scan(const BuildArgs &a, const SkArgs &s, uint64_t bound, uint32_t stride, bool sample, int grid_mode,
                      cudaStream_t st) {
    if (!bound) return 0;
#define SWG_SCAN(M, W) \
    if (s.k == M + W - 1 && s.w == W) return scan_launch<M, W>(a, s, bound, stride, sample, grid_mode, st)
    SWG_SCAN(15, 17);
    SWG_SCAN(13, 17);
    SWG_SCAN(13, 15);
    SWG_SCAN(12, 14);
    SWG_SCAN(13, 13);
    SWG_SCAN(11, 13);
    SWG_SCAN(12, 12);
    SWG_SCAN(13, 11);
    SWG_SCAN(11, 11);
    SWG_SCAN(12, 10);
    SWG_SCAN(13, 9);
    SWG_SCAN(11, 9);
    SWG_SCAN(12, 8);
    SWG_SCAN(13, 7);
#undef SWG_SCAN
    return 0;  // (super_window names no other)
}

// sum over the buckets, by the square root's concavity
uint64_t super_bucket_room(uint64_t records, uint64_t nb, double scale_max) {
    const double mean = (double)records / (double)nb / scale_max;
    const double most = 1.25 * (double)records + (double)nb * scale_max * (18.0 + 6.0 * std::sqrt(mean + 9.0));
    return (uint64_t)(1.001 * most) + nb;  // (the regions are worked out in single precision)
}

uint64_t super_pieces_bound(uint64_t n_reads, uint64_t occurrences) { return n_reads + occurrences / kSkPiece + 1; }

int launch_super_pieces(const BuildArgs &a, uint64_t *count, uint64_t *first, uint64_t *scratch, uint64_t *total,
                        uint64_t *off, uint32_t *len, uint32_t *seg, cudaStream_t st) {
    k_sk_pieces_count<<<(unsigned)((a.n_reads + 255) / 256), 256, 0, st>>>(a, count);
    const int n = launch_gscan(count, first, a.n_reads, scratch, total, st);
    k_sk_pieces_fill<<<(unsigned)((a.n_reads * 32 + 255) / 256), 256, 0, st>>>(a, first, off, len, seg);
    return 2 + n;
}

int launch_super_uniform(const SkArgs &s, uint64_t part, uint64_t nb, uint64_t bucket, cudaStream_t st) {
    k_sk_uniform<<<(unsigned)std::max<uint64_t>(1, (nb + 1023) / 1024), 1024, 0, st>>>(s, part, (uint32_t)nb, bucket);
    return 1;
}

int launch_super_caps(const SkArgs &s, uint64_t nb, uint64_t *scratch, cudaStream_t st) {
    if (nb <= 1024 * kRegionItems) {
        k_sk_regions<<<1, 1024, 0, st>>>(s, (uint32_t)nb);
        return 1;
    }
    k_sk_caps<<<1, 1024, 0, st>>>(s);
    k_sk_bucket_caps<<<(unsigned)((nb + 255) / 256), 256, 0, st>>>(s, s.cursor2, nb, s.cursor2);
    const int n = launch_gscan(reinterpret_cast<const uint64_t *>(s.cursor2), reinterpret_cast<uint64_t *>(s.off2), nb,
                               scratch, reinterpret_cast<uint64_t *>(s.off2 + nb), st);
    cudaMemcpyAsync(s.cursor2, s.off2, nb * 8, cudaMemcpyDeviceToDevice, st);
    return 2 + n;
}

int launch_super_sub(const SkArgs &s, cudaStream_t st) {
    const size_t smem = sub_smem(s.b2, s.n_parts);
    allow_smem(k_sk_sub, sub_smem(10, 1u << kPartBitsMax));
    const uint64_t chunks = s.rec_cap * 5 / 4 / kSkChunk + s.n_parts;
    k_sk_sub<<<(unsigned)std::min<uint64_t>(chunks, resident_grid(k_sk_sub, 256, smem)), 256, smem, st>>>(s);
    return 1;
}

template <int kK>
int count_launch(const BuildArgs &a, const SkArgs &s, uint64_t nb, int table, cudaStream_t st) {
    const size_t tag = a.tag_bits ? 2 * a.n_segs * sizeof(unsigned) : 0;
    constexpr size_t tag_most = 2 * kMaxTagSamples * sizeof(unsigned);
    if (table == 2048) {
        auto kern = k_sk_count<2048, 256, kK>;
        const size_t smem = count_smem<2048, 256>() + tag;
        allow_smem(kern, count_smem<2048, 256>() + tag_most);
        kern<<<(unsigned)std::min<uint64_t>(nb, resident_grid(kern, 256, smem)), 256, smem, st>>>(a, s, nb);
    } else {
        auto kern = k_sk_count<4096, 512, kK>;
        const size_t smem = count_smem<4096, 512>() + tag;
        allow_smem(kern, count_smem<4096, 512>() + tag_most);
        kern<<<(unsigned)std::min<uint64_t>(nb, resident_grid(kern, 512, smem)), 512, smem, st>>>(a, s, nb);
    }
    auto large = k_sk_count<8192, 1024, kK>;
    const size_t smem = count_smem<8192, 1024>() + tag;
    allow_smem(large, count_smem<8192, 1024>() + tag_most);
    large<<<(unsigned)device_sm_count(), 1024, smem, st>>>(a, s, nb);
    return 2;
}

int launch_super_count(const BuildArgs &a, const SkArgs &s, uint64_t nb, int table, cudaStream_t st) {
    switch (s.k) {
        case 31: return count_launch<31>(a, s, nb, table, st);
        case 29: return count_launch<29>(a, s, nb, table, st);
        case 27: return count_launch<27>(a, s, nb, table, st);
        case 25: return count_launch<25>(a, s, nb, table, st);
        case 23: return count_launch<23>(a, s, nb, table, st);
        case 21: return count_launch<21>(a, s, nb, table, st);
        default: return count_launch<19>(a, s, nb, table, st);
    }
}

int launch_super_big_bounds(const SkArgs &s, uint32_t n, unsigned long long *meta, cudaStream_t st) {
    k_sk_big_bounds<<<(n + 255) / 256, 256, 0, st>>>(s, n, meta);
    return 1;
}

int launch_super_big(const BuildArgs &a, const SkArgs &s, const unsigned long long *meta, uint32_t n, uint64_t records,
                     Entry *table, uint64_t cap, cudaStream_t st) {
    const uint64_t blocks =
        std::min<uint64_t>((records + kSkBigChunk - 1) / kSkBigChunk, (uint64_t)device_sm_count() * 6);
    k_sk_big<<<(unsigned)std::max<uint64_t>(blocks, 1), 256, 0, st>>>(a, s, meta, n, table, cap);
    return 1;
}

}  // namespace swg
