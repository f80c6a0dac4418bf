// Device helpers shared by the build's kernels (kernels.cu, super.cu): packed
// reads, hashes, the open-addressing table in HBM, multiplicities.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <set>
#include <utility>

#include "swg_internal.h"

namespace swg {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kMaxProbe = 1 << 14;
constexpr int kMaxCas = 1 << 20;

__device__ __forceinline__ uint64_t mix64(uint64_t x) {
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ull;
    x ^= x >> 33;
    return x;
}

// Reverse complement of a k-mer held in the low 2k bits (k <= 31): complement
// every base (b -> 3-b, i.e. bitwise NOT), reverse the 2-bit groups. Same
// value as the reference's O(k) loop (kmerGraph.cpp:5-14).
__device__ __forceinline__ uint64_t revcomp_dev(uint64_t x, int k) {
    uint64_t y = __brevll(~x);
    y = ((y >> 1) & 0x5555555555555555ull) | ((y & 0x5555555555555555ull) << 1);
    return y >> (64 - 2 * k);
}

__device__ __forceinline__ uint32_t ldw(const uint32_t *__restrict__ p, uint64_t i, uint64_t n) {
    return i < n ? __ldg(p + i) : 0u;
}

// 32 bases starting at base g, first base in bits 63..62.
__device__ __forceinline__ uint64_t window32(const uint32_t *__restrict__ p, uint64_t n,
                                             uint64_t g) {
    const uint64_t w = g >> 4;
    const int sh = (int)(g & 15) * 2;
    const uint64_t hi = ((uint64_t)ldw(p, w, n) << 32) | ldw(p, w + 1, n);
    if (sh == 0) return hi;
    return (hi << sh) | (uint64_t)(ldw(p, w + 2, n) >> (32 - sh));
}

__device__ __forceinline__ uint32_t base_at(const uint32_t *__restrict__ p, uint64_t n,
                                            uint64_t g) {
    return (ldw(p, g >> 4, n) >> (30 - 2 * (int)(g & 15))) & 3u;
}

__device__ __forceinline__ uint64_t umin64(uint64_t a, uint64_t b) { return a < b ? a : b; }

// Asks L2 to fetch records [r0, r1) of a record array ahead of their loads
// (one bulk prefetch from the calling thread). The range is narrowed to
// whole 16-byte pairs of records inside it, as the bulk prefetch requires.
__device__ __forceinline__ void prefetch_records_l2(const unsigned long long *rec, uint64_t r0, uint64_t r1) {
    const uint64_t a = (r0 + 1) & ~1ull, e = r1 & ~1ull;
    if (e <= a) return;
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(rec + a), "r"((uint32_t)((e - a) * 8))
                 : "memory");
}

__device__ __forceinline__ uint64_t occ_of(uint32_t len, int k) {
    return len >= (uint32_t)k ? (uint64_t)(len - (uint32_t)k + 1) : 0ull;
}

// Sample (segment) of read r and its parameters; a single-sample build has no
// segment arrays and takes k, cutoff, table and counters from BuildArgs.
__device__ __forceinline__ uint32_t seg_of(const BuildArgs &a, uint64_t r) {
    return a.read_seg ? a.read_seg[r] : 0u;
}

__device__ __forceinline__ int k_of(const BuildArgs &a, uint32_t seg) {
    return a.segs ? a.segs[seg].k : a.k;
}

__device__ __forceinline__ ulonglong2 ld_relaxed16(const Entry *e) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];"
                 : "=l"(v.x), "=l"(v.y)
                 : "l"(e)
                 : "memory");
    return v;
}

// 128-bit compare-and-swap on {key, cnt}; returns the previous contents.
__device__ __forceinline__ ulonglong2 cas128(Entry *e, uint64_t cmp_key, uint64_t cmp_cnt,
                                             uint64_t new_key, uint64_t new_cnt) {
    ulonglong2 old;
    asm volatile(
        "{\n\t"
        ".reg .b128 cmpv, newv, oldv;\n\t"
        "mov.b128 cmpv, {%2, %3};\n\t"
        "mov.b128 newv, {%4, %5};\n\t"
        "atom.relaxed.gpu.global.cas.b128 oldv, [%6], cmpv, newv;\n\t"
        "mov.b128 {%0, %1}, oldv;\n\t"
        "}"
        : "=l"(old.x), "=l"(old.y)
        : "l"(cmp_key), "l"(cmp_cnt), "l"(new_key), "l"(new_cnt), "l"(e)
        : "memory");
    return old;
}

// Per-byte saturating add of 8 uint8 counts (min(a+b, 255) in each byte).
__device__ __forceinline__ uint64_t satadd8(uint64_t a, uint64_t b) {
    const uint32_t lo = __vaddus4((uint32_t)a, (uint32_t)b);
    const uint32_t hi = __vaddus4((uint32_t)(a >> 32), (uint32_t)(b >> 32));
    return ((uint64_t)hi << 32) | lo;
}

// Add `inc` to the counts of `key` (present at e, last seen counts `cur`).
__device__ __forceinline__ void update_counts(Entry *e, uint64_t key, uint64_t cur, uint64_t inc,
                                              unsigned *status) {
    for (int tries = 0; tries < kMaxCas; ++tries) {
        const uint64_t nxt = satadd8(cur, inc);
        if (nxt == cur) return;  // every touched slot already at 255
        const ulonglong2 old = cas128(e, key, cur, key, nxt);
        if (old.y == cur) return;
        cur = old.y;
    }
    atomicOr(status, kStatusCasLimit);
}

// Insert `key` with counts `inc`, or add `inc` to its counts. Returns 1 when
// this call inserted the key.
__device__ __forceinline__ unsigned insert_or_update(Entry *__restrict__ table, uint64_t cap,
                                                     uint64_t key, uint64_t inc,
                                                     unsigned *status) {
    uint64_t h = __umul64hi(mix64(key), cap);
    for (int step = 0; step < kMaxProbe; ++step) {
        Entry *e = table + h;
        const ulonglong2 v = ld_relaxed16(e);
        if (v.x == key) {
            update_counts(e, key, v.y, inc, status);
            return 0;
        }
        if (v.x == 0) {
            const ulonglong2 old = cas128(e, 0, 0, key, inc);
            if (old.x == 0) return 1;  // empty entries always hold zero counts
            if (old.x == key) {
                update_counts(e, key, old.y, inc, status);
                return 0;
            }
        }
        h = (h + 1 == cap) ? 0 : h + 1;
    }
    atomicOr(status, kStatusTableFull);
    return 0;
}

__device__ __forceinline__ uint64_t code_inc(unsigned code) {
    uint64_t inc = 0;
    if (code & 0x08u) inc += 1ull << (8 * (code & 7u));
    if (code & 0x80u) inc += 1ull << (8 * ((code >> 4) & 7u));
    return inc;
}

// Record hash of the level-1 scatter (bucketed and partitioned builds): a
// bijection on 64 bits, cheaper than mix64 on the per-occurrence path. An odd
// multiplier carries every key bit into the top bits (the partition and the
// bucket); folding the high half into the low half gives the low bits (the
// table slot) every key bit too. rmix64's inverse: undo the fold (the high
// half is unchanged), multiply by the multiplier's inverse modulo 2^64.
__device__ __forceinline__ uint64_t rmix64(uint64_t x) {
    x *= 0x9e3779b97f4a7c15ull;
    return x ^ (x >> 32);
}
__device__ __forceinline__ uint64_t runmix64(uint64_t x) {
    x ^= x >> 32;
    return x * 0xf1de83e19937733dull;
}

// Eight saturated uint8 multiplicities of table entry s (8 x uint16
// counters, slot t in half t&1 of word t>>1), after the -c cutoff
// (graph.cpp:1105: a multiplicity below c becomes 0). SWAR on the 16-bit
// halves: min(v, 255), then v + 0x8000 - c has bit 15 set iff v >= c (no
// carry leaves a half since v <= 255 and 1 <= c <= 255).
__device__ __forceinline__ uint64_t bucket_mult(const unsigned *cnt, uint32_t s, unsigned cbias,
                                                bool cut_all) {
    const uint4 cv = reinterpret_cast<const uint4 *>(cnt)[s];
    unsigned w[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        w[t] = __vminu2(w[t], 0x00ff00ffu);
        if (cbias) {
            const unsigned ge = ((w[t] + cbias) >> 15) & 0x00010001u;
            w[t] &= ge * 0xffffu;
        }
    }
    const uint64_t m = ((uint64_t)__byte_perm(w[2], w[3], 0x6420) << 32) | __byte_perm(w[0], w[1], 0x6420);
    return cut_all ? 0 : m;
}

// Whether a region has been outgrown, so that the build will count again: one
// answer for the whole block. The blocks of a counting kernel set the bit
// themselves when they find a bucket outgrown, so threads that each read it
// could disagree, and those that stayed would count with tables that the
// others never cleared, at barriers the others never reach.
__device__ __forceinline__ bool block_reads_overflow(const unsigned *status) {
    return __syncthreads_or(threadIdx.x == 0 && (*(const volatile unsigned *)status & kStatusPartOverflow));
}

}  // namespace

// Lets a kernel use up to `most` bytes of dynamic shared memory (its largest
// use, not the launch's own), once per device: builds run in several threads,
// and the attribute of a kernel that another thread is launching must not
// change under it.
template <typename K>
void allow_smem(K kernel, size_t most) {
    static std::mutex mu;
    static std::set<std::pair<int, K>> done;
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> lock(mu);
    if (!done.count({dev, kernel}) &&
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) == cudaSuccess)
        done.insert({dev, kernel});
}

// Blocks of a persistent kernel that are resident at once on the device.
template <typename K>
uint64_t resident_grid(K kernel, int threads, size_t dyn_smem) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, dyn_smem) != cudaSuccess ||
        per_sm < 1) {
        cudaGetLastError();
        per_sm = 1;
    }
    return (uint64_t)per_sm * device_sm_count();
}


}  // namespace swg
