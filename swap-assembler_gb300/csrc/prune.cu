// The reference's rank-0 passes over the merged graph that follow the merge,
// on the device: masterTipsRemoval (graph.cpp:2194-2265),
// masterLowCoverageEdgeRemoval (graph.cpp:2267-2300) and the re-merge the
// reference runs after each, masterSimplifyNodeGraph (graph.cpp:2089-2192,
// described with its kernels below). They work on the merged graph's lines (node key, per
// arc slot its length, multiplicity, string offset and the far end's arc
// back) and then rewrite its text (gathered node lines in key order, deleted
// and arc-less nodes left out as gatherDistNodeGraph does, graph.cpp:587-596).
//
// Tips: a node with exactly one arc, shorter than k, loses that arc, so does
// the far node's arc back, and the node is deleted. The reference visits the
// nodes in its node map's order, removing tips as it meets them; here every
// node that is a tip when the pass starts is judged on that state — the same
// as visiting all other nodes first and then the tips in key order. Of two
// tips whose arcs join them to each other, the one with the smaller key is
// deleted and the other keeps no arc. An arc that leads back to its own node
// is left alone (graph.cpp:2244).
//
// Low coverage: avg = sum(len * m) / sum(len) over the arcs of the nodes left
// (integer division); every arc shorter than 2k with m < avg / 4 is cut (both
// ends' arcs meet the test alike, having the same length and multiplicity).
// The reference divides by zero when no arc is left; here nothing is cut.
#include <cuda_runtime.h>

#include <cooperative_groups.h>
#include <cooperative_groups/reduce.h>

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "swg_internal.h"
#include "text_dev.cuh"

namespace swg {
namespace {

namespace cg = cooperative_groups;

constexpr unsigned char kNoTip = 8;

__device__ __forceinline__ void agg_add(unsigned long long *ctr, unsigned long long v) {
    cg::coalesced_group g = cg::coalesced_threads();
    const unsigned long long sum = cg::reduce(g, v, cg::plus<unsigned long long>());
    if (g.thread_rank() == 0) atomicAdd(ctr, sum);
}

// The slot of a node's one arc when the node is a tip, else kNoTip.
__global__ void k_pr_tipslot(MergedGraph m, unsigned char *__restrict__ tip) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= m.lines) return;
    unsigned char t = kNoTip;
    if (!m.del[q]) {
        int num = 0, slot = 0;
        for (int s = 0; s < 8; ++s)
            if (m.len[8 * q + s]) ++num, slot = s;
        if (num == 1 && m.len[8 * q + slot] < (unsigned)m.k) t = (unsigned char)slot;
    }
    tip[q] = t;
}

__global__ void k_pr_tips(MergedGraph m, const unsigned char *__restrict__ tip, unsigned long long *count) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= m.lines || tip[q] == kNoTip) return;
    const unsigned s = tip[q];
    const unsigned b = m.back[8 * q + s];
    const uint64_t far = b >> 3, fs = b & 7;
    if (far == q) return;  // the arc leads back to this node
    m.len[8 * q + s] = 0;
    m.mult[8 * q + s] = 0;
    // a tip at the far end joined only to this one: the smaller key goes first,
    // removes both arcs, and the other is left without arcs (lines are in key order)
    if (tip[far] != kNoTip && far < q) return;
    m.len[8 * far + fs] = 0;
    m.mult[8 * far + fs] = 0;
    m.del[q] = 1;
    agg_add(count, 1);
}

// sums[0] = sum(len * m), sums[1] = sum(len) over the arcs of nodes left.
__global__ void k_pr_cov(MergedGraph m, unsigned long long *sums) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= m.lines || m.del[q]) return;
    unsigned long long cov = 0, nuc = 0;
    for (int s = 0; s < 8; ++s) {
        const unsigned l = m.len[8 * q + s];
        nuc += l;
        cov += (unsigned long long)l * m.mult[8 * q + s];
    }
    agg_add(&sums[0], cov);
    agg_add(&sums[1], nuc);
}

__global__ void k_pr_low(MergedGraph m, const unsigned long long *sums, unsigned long long *count) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= m.lines || m.del[q]) return;
    const unsigned long long avg = sums[1] ? sums[0] / sums[1] : 0;
    unsigned cut = 0;
    for (int s = 0; s < 8; ++s) {
        const unsigned l = m.len[8 * q + s];
        // multiplicity < 0.25 * avgCoverage (graph.cpp:2294), exactly: 4 * m < avg
        if (l < 2u * (unsigned)m.k && 4ull * m.mult[8 * q + s] < avg) {
            cut += l != 0;
            m.len[8 * q + s] = 0;
            m.mult[8 * q + s] = 0;
        }
    }
    if (cut) agg_add(count, cut);
}

// ---- rewrite of the text
// (count: what the pass before counted, put beside what the host reads next)
__global__ void k_pr_len(MergedGraph m, uint64_t *__restrict__ out, unsigned long long *printed,
                         const unsigned long long *__restrict__ count) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q == 0 && count) printed[1] = *count;
    if (q >= m.lines) return;
    uint64_t sum = 0;
    if (!m.del[q])
        for (int s = 0; s < 8; ++s) sum += m.len[8 * q + s];
    out[q] = sum ? 69 + sum : 0;
    if (sum) agg_add(printed, 1);
}

// Eight lanes a line, one per arc slot (as the merge writes them).
__global__ void __launch_bounds__(256) k_pr_write(MergedGraph m, const uint64_t *__restrict__ off, char *__restrict__ text) {
    const uint64_t q = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const int s = threadIdx.x & 7;
    const bool in = q < m.lines && off[q + 1] != off[q];
    const unsigned l = in ? m.len[8 * q + s] : 0, mult = in ? m.mult[8 * q + s] : 0;
    const unsigned dig = 1 + ndig(mult);
    unsigned long long al = l + 2ull;
    unsigned dl = dig;
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) {
        const unsigned long long x = __shfl_up_sync(0xffffffffu, al, d, 8);
        const unsigned y = __shfl_up_sync(0xffffffffu, dl, d, 8);
        if (s >= d) {
            al += x;
            dl += y;
        }
    }
    const unsigned long long arcs = __shfl_sync(0xffffffffu, al, 7, 8);
    const unsigned digits = __shfl_sync(0xffffffffu, dl, 7, 8);
    if (!in) return;
    char *const start = text + off[q];
    const uint64_t key = m.key[q];
    const unsigned head = ndig(key);
    char *p = start + head + (al - l - 2);  // this lane's " arc#"
    *p = ' ';
    p[1 + l] = '#';
    m.src2[8 * q + s] = (unsigned long long)(p + 1 - text);
    char *d = start + head + arcs + (dl - dig);  // this lane's " m"
    *d = ' ';
    put_u64(d + 1, mult);
    const uint64_t vlen = off[q + 1] - off[q];
    for (uint64_t i = head + arcs + digits + s; i < vlen - 1; i += 8) start[i] = ' ';
    if (s == 0) {
        put_u64(start, key);
        start[vlen - 1] = '\n';
    }
}

// The arc strings move from the old text to the new one, a piece's first KiB
// by eight lanes; the rest of a long one is listed in parts of a KiB, a warp
// each, so that a few very long arcs (whole chains) spread over the GPU too.
// Bound by the loads' latency, so every lane has sixteen bytes under way. A
// piece is an arc's own string (its first `own` bytes, the whole arc unless a
// merge lengthened it) or, after a merge, a merged node's arc string placed
// inside an end's new arc. 50,000 pieces, 1 MB: first parts of 4 KiB by a warp,
// a byte a lane at a time, took 29 to 62 us, parts' counts scanned and searched
// 13 to 27; now 14 and 8.
constexpr unsigned kPart = 1024;   // bytes of a piece moved at a time
constexpr unsigned kChunk = 4096;  // of a contig
constexpr int kBytes = 16;         // a lane's under way

// `l` bytes by `lanes` neighbouring lanes, of which this one is `lane`.
__device__ __forceinline__ void move_bytes(char *b, const char *a, unsigned l, unsigned lane, unsigned lanes) {
    for (unsigned c = lane; c < l; c += kBytes * lanes) {
        char v[kBytes];
#pragma unroll
        for (int j = 0; j < kBytes; ++j)
            if (c + j * lanes < l) v[j] = a[c + j * lanes];
#pragma unroll
        for (int j = 0; j < kBytes; ++j)
            if (c + j * lanes < l) b[c + j * lanes] = v[j];
    }
}

struct Pieces {
    const unsigned *own;                    // per arc slot: bytes of its old string (nullptr: len)
    uint64_t n;                             // extra pieces
    const unsigned long long *src;          // old-text offset
    const unsigned *len;
    const unsigned *arc;                    // the arc slot whose new string receives it
    const unsigned long long *at;           // offset inside that string
};

__device__ __forceinline__ unsigned own_len(const MergedGraph &m, const Pieces &x, uint64_t a) {
    if (m.del[a >> 3]) return 0;
    return x.own ? x.own[a] : m.len[a];
}

// Where piece i's string lies and goes, and its length.
__device__ __forceinline__ unsigned piece(const MergedGraph &m, const Pieces &x, uint64_t i, uint64_t &src, uint64_t &dst) {
    const uint64_t arcs = 8 * m.lines;
    if (i < arcs) {
        const unsigned l = own_len(m, x, i);
        if (l) {
            src = m.src[i];
            dst = m.src2[i];
        }
        return l;
    }
    const uint64_t j = i - arcs;
    const unsigned l = x.len[j];
    if (l) {
        src = x.src[j];
        dst = m.src2[x.arc[j]] + x.at[j];
    }
    return l;
}

// Eight lanes a piece: they move its first part, and list the other parts of a
// long one (piece << 24 | part; a part's number is below 2^22), counted in
// *listed. (A warp that looked at 32 pieces and moved four at a time waited for
// eight rounds of loads: 17 to 26 us for 50,000 pieces, 14 now.)
__global__ void __launch_bounds__(256) k_pr_short(MergedGraph m, Pieces x, const char *__restrict__ from,
                                                  char *__restrict__ to, unsigned long long *__restrict__ parts,
                                                  unsigned long long *__restrict__ listed) {
    const uint64_t pieces = 8 * m.lines + x.n;
    const uint64_t i = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const unsigned lane = threadIdx.x & 7;
    uint64_t src = 0, dst = 0;
    const unsigned len = i < pieces ? piece(m, x, i, src, dst) : 0;
    const unsigned more = len ? (len - 1) / kPart : 0;
    unsigned long long at = 0;
    if (lane == 0 && more) at = atomicAdd(listed, (unsigned long long)more);
    at = __shfl_sync(0xffffffffu, at, 0, 8);
    for (unsigned c = lane; c < more; c += 8) parts[at + c] = i << 24 | (c + 1);
    if (len) move_bytes(to + dst, from + src, len < kPart ? len : kPart, lane, 8);
}

// The listed parts, a warp each; their number is read on the device.
__global__ void __launch_bounds__(256) k_pr_long(MergedGraph m, Pieces x, const unsigned long long *__restrict__ parts,
                                                 const unsigned long long *__restrict__ listed,
                                                 const char *__restrict__ from, char *__restrict__ to) {
    const uint64_t n = *listed, warps = (uint64_t)gridDim.x * (blockDim.x >> 5);
    for (uint64_t c = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < n; c += warps) {
        uint64_t src = 0, dst = 0;
        const unsigned len = piece(m, x, parts[c] >> 24, src, dst);
        const uint64_t at = (parts[c] & 0xffffffu) * kPart;
        const uint64_t rest = len - at;
        move_bytes(to + dst + at, from + src + at, rest < kPart ? (unsigned)rest : kPart, threadIdx.x & 31, 32);
    }
}

inline unsigned blocks(uint64_t n) { return (unsigned)std::max<uint64_t>((n + 255) / 256, 1); }

// Writes the lines into the spare text, then swaps it in.
swg_status rewrite(MergedGraph *m, cudaStream_t s, Scratch &scr, const Pieces &x = Pieces{},
                   const unsigned long long *d_count = nullptr, uint64_t *count = nullptr) {
    uint64_t *len = nullptr, *off = nullptr;
    unsigned long long *printed = nullptr;
    if (!scr.get(&len, m->lines) || !scr.get(&off, m->lines + 4))
        return cuda_err(cudaErrorMemoryAllocation, "rewrite workspace");
    // read together with the text's size: printed lines, the pass's count; the listed parts' comes after them
    printed = reinterpret_cast<unsigned long long *>(off + m->lines + 1);
    EMIT_CUDA(cudaMemsetAsync(printed, 0, 24, s), "rewrite");
    if (m->lines) k_pr_len<<<blocks(m->lines), 256, 0, s>>>(*m, len, printed, d_count);
    swg_status st = scan_lengths(len, off, m->lines, scr, s);
    if (st) return st;
    uint64_t h[3] = {0, 0, 0};
    EMIT_CUDA(cudaMemcpyAsync(h, off + m->lines, 24, cudaMemcpyDeviceToHost, s), "text size");
    EMIT_CUDA(cudaStreamSynchronize(s), "text size");
    if (count) *count = h[2];
    const uint64_t bytes = h[0] + 1;
    if (bytes > m->text2_cap) {
        cudaFree(m->text2);
        m->text2 = nullptr;
        m->text2_cap = 0;
        EMIT_CUDA(cudaMalloc((void **)&m->text2, bytes), "merged text");
        m->text2_cap = bytes;
    }
    if (m->lines) {
        const uint64_t pieces = 8 * m->lines + x.n;
        const uint64_t most = h[0] / kPart;  // a part per KiB of the new text
        unsigned long long *parts = nullptr;
        if (!scr.get(&parts, most)) return cuda_err(cudaErrorMemoryAllocation, "rewrite workspace");
        k_pr_write<<<blocks(8 * m->lines), 256, 0, s>>>(*m, off, m->text2);
        k_pr_short<<<blocks(8 * pieces), 256, 0, s>>>(*m, x, m->text, m->text2, parts, printed + 2);
        if (most)
            k_pr_long<<<(unsigned)std::min<uint64_t>((most + 7) / 8, 4096), 256, 0, s>>>(*m, x, parts, printed + 2,
                                                                                        m->text, m->text2);
    }
    EMIT_CUDA(cudaMemsetAsync(m->text2 + h[0], '\n', 1, s), "merged text");
    EMIT_CUDA(cudaGetLastError(), "rewrite kernels");
    EMIT_CUDA(cudaStreamSynchronize(s), "rewrite");
    std::swap(m->text, m->text2);
    std::swap(m->text_cap, m->text2_cap);
    std::swap(m->src, m->src2);
    m->text_bytes = bytes;
    m->nodes = h[1];
    return SWG_OK;
}


// ---- masterSimplifyNodeGraph (graph.cpp:2089-2192) over the lines: a node
// left with exactly one arc on each side (the last nonempty slot of each
// half) whose arcs do not lead back to itself is merged away; each chain of
// such nodes between two other nodes collapses into the two end arcs, whose
// strings are the concatenation of the chain's arcs. The multiplicity is the
// reference's weighted average in size_t arithmetic (graph.cpp:2157-2163),
// taken in the merge's visiting order — chain numbered from its smaller end
// arc (key, slot), node p at level ctz(p) — so a pairwise reduction of the
// chain's arcs weighted by their lengths. A cycle of such nodes is cut at its
// largest key. Chains are found by pointer jumping over two walk states per
// node (the line graph is small next to the k-molecule graph).
constexpr unsigned long long kTerm = 1ull << 63;
constexpr unsigned kNone = 0xffffffffu;

struct SimplifyArgs {
    MergedGraph m;
    unsigned char *fl;  // bit0 merged away, bits1-2 right slot, bits3-4 left slot - 4
    unsigned long long *nx[2], *ws[2], *mx[2];
    unsigned *cn[2];
    unsigned *chain_of;  // per arc slot of an end: chain id (at its start arc)
    unsigned long long *ch_eoff;
    unsigned *ch_m;
    unsigned char *ent_m;
    unsigned long long *ent_l;
    unsigned *ent_chain;
    unsigned long long *cls_count, *cls_cursor;
    unsigned long long *ctr;  // [0] mergeable nodes [1] cycles cut [2] chains [3] states left in cycles
    unsigned *own;
    unsigned long long *xsrc, *xat;
    unsigned *xlen, *xarc;
};

__device__ __forceinline__ bool sm_m(const SimplifyArgs &a, uint64_t q) { return a.fl[q] & 1u; }
__device__ __forceinline__ int sm_rs(unsigned char f) { return (f >> 1) & 3; }
__device__ __forceinline__ int sm_ls(unsigned char f) { return 4 + ((f >> 3) & 3); }

__device__ __forceinline__ unsigned long long agg_inc(unsigned long long *ctr) {
    cg::coalesced_group g = cg::coalesced_threads();
    unsigned long long base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(ctr, (unsigned long long)g.size());
    return g.shfl(base, 0) + g.thread_rank();
}

__device__ __forceinline__ unsigned long long agg_add_labeled(unsigned long long *ctr, int label,
                                                              unsigned long long step) {
    cg::coalesced_group g = cg::labeled_partition(cg::coalesced_threads(), label);
    unsigned long long base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(ctr + label, step * g.size());
    return g.shfl(base, 0) + step * g.thread_rank();
}

__device__ __forceinline__ bool sm_arc_less(const SimplifyArgs &a, uint64_t x, uint64_t y) {
    const unsigned long long kx = a.m.key[x >> 3], ky = a.m.key[y >> 3];
    return kx < ky || (kx == ky && (x & 7) < (y & 7));
}

struct SmPos {
    unsigned m, pos;
    uint64_t alpha, beta;  // end arcs reached going back / forward
    bool fwd;              // the chain runs through the node leaving by its right arc
};

__device__ __forceinline__ SmPos sm_pos(const SimplifyArgs &a, int in, uint64_t q) {
    SmPos c;
    const unsigned la = __ldcg(a.cn[in] + 2 * q), lb = __ldcg(a.cn[in] + 2 * q + 1);
    c.beta = __ldcg(a.nx[in] + 2 * q) & ~kTerm;
    c.alpha = __ldcg(a.nx[in] + 2 * q + 1) & ~kTerm;
    c.m = la + lb - 1;
    c.fwd = sm_arc_less(a, c.alpha, c.beta);
    c.pos = c.fwd ? lb : la;
    return c;
}

__device__ __forceinline__ int sm_class(unsigned m) { return m == 0 ? 0 : 64 - __clzll((unsigned long long)m); }

// Lines merged away, their walk states ranked by pointer jumping, cycles and
// chains counted: all in one cooperative launch, since each step is a few
// microseconds over a few thousand lines and a grid barrier costs less than a
// launch (one block of 1024 an SM at most: a barrier's time grows with them).
//  - A line with one arc on each side that does not lead back to it is merged.
//  - Walk state 2q+d leaves line q by its right (d = 0) or left (d = 1) arc; the
//    next line is entered by the slot the back link names: entered from the
//    left (slot >= 4), it is traversed leaving by its right arc.
//  - Jumping rounds go in pairs, so that the result is in the first buffers
//    again, until every state has reached an end (those of a cycle never do).
//  - Lines still in a cycle then (ctr[3]): the cycle's largest key ends it, and
//    the host launches this again (first = 0); the chains are counted anew.
// 6,300 lines: the five kernels 37 and 55 us (after tips, after low coverage),
// this 26 and 42.
__global__ void __launch_bounds__(1024) k_sm_rank(SimplifyArgs a, int pairs, unsigned *moved, int first) {
    const uint64_t lines = a.m.lines, states = 2 * lines, stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (first) {
        for (uint64_t q = t; q < lines; q += stride) {
            int rc = 0, lc = 0, rs = 0, ls = 4;
            if (!a.m.del[q])
                for (int s = 0; s < 8; ++s)
                    if (a.m.len[8 * q + s]) {
                        if (s < 4) ++rc, rs = s;
                        else ++lc, ls = s;
                    }
            const bool merged =
                rc == 1 && lc == 1 && (a.m.back[8 * q + rs] >> 3) != q && (a.m.back[8 * q + ls] >> 3) != q;
            a.fl[q] = (unsigned char)((merged ? 1 : 0) | (rs << 1) | ((ls - 4) << 3));
            if (merged) agg_inc(&a.ctr[0]);
        }
        cg::this_grid().sync();
    }
    for (uint64_t q = t; q < lines; q += stride) {
        if (!sm_m(a, q)) continue;
        const unsigned char f = a.fl[q];
        for (int d = 0; d < 2; ++d) {
            const int slot = d ? sm_ls(f) : sm_rs(f);
            const unsigned b = a.m.back[8 * q + slot];
            const uint64_t far = b >> 3;
            const uint64_t st = 2 * q + d;
            a.nx[0][st] = sm_m(a, far) ? 2 * far + ((b & 7) >= 4 ? 0 : 1) : (kTerm | b);
            a.cn[0][st] = 1;
            a.ws[0][st] = a.m.len[8 * q + slot];
            a.mx[0][st] = a.m.key[q];
        }
    }
    cg::this_grid().sync();
    for (int r = 0; r < pairs; ++r) {
        for (int in = 0; in < 2; ++in) {
            const int out = in ^ 1;
            bool left = false;
            for (uint64_t st = t; st < states; st += stride) {
                if (!sm_m(a, st >> 1)) continue;
                unsigned long long nx = __ldcg(a.nx[in] + st), ws = __ldcg(a.ws[in] + st), mx = __ldcg(a.mx[in] + st);
                unsigned cn = __ldcg(a.cn[in] + st);
                if (!(nx & kTerm)) {
                    const unsigned long long to = nx;
                    nx = __ldcg(a.nx[in] + to);
                    cn += __ldcg(a.cn[in] + to);
                    ws += __ldcg(a.ws[in] + to);
                    const unsigned long long y = __ldcg(a.mx[in] + to);
                    mx = y > mx ? y : mx;
                    left |= !(nx & kTerm);
                }
                a.nx[out][st] = nx;
                a.cn[out][st] = cn;
                a.ws[out][st] = ws;
                a.mx[out][st] = mx;
            }
            if (in && left) moved[r] = 1;
            cg::this_grid().sync();
        }
        if (!*(volatile unsigned *)(moved + r)) break;
    }
    for (uint64_t q = t; q < lines; q += stride) {
        if (!sm_m(a, q)) continue;
        if (!(__ldcg(a.nx[0] + 2 * q) & kTerm)) {
            if (!first) continue;
            agg_inc(&a.ctr[3]);
            if (a.m.key[q] == __ldcg(a.mx[0] + 2 * q)) {
                a.fl[q] &= (unsigned char)~1u;
                agg_inc(&a.ctr[1]);
            }
            continue;
        }
        const SmPos c = sm_pos(a, 0, q);
        if (c.pos == 1) agg_add_labeled(a.cls_count, sm_class(c.m), 1);
    }
}

__global__ void k_sm_chain_alloc(SimplifyArgs a, int in) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= a.m.lines || !sm_m(a, q)) return;
    const SmPos c = sm_pos(a, in, q);
    if (c.pos != 1) return;
    const int cl = sm_class(c.m);
    const unsigned id = (unsigned)agg_inc(&a.ctr[2]);
    a.ch_eoff[id] = agg_add_labeled(a.cls_cursor, cl, 1ull << cl);
    a.ch_m[id] = c.m;
    a.chain_of[c.fwd ? c.alpha : c.beta] = id;
}

// Unit arc p of a chain (multiplicity, length): node p's arc towards the far
// end; node 1 also stores the arc back to the start.
__global__ void k_sm_entries(SimplifyArgs a, int in) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= a.m.lines || !sm_m(a, q)) return;
    const SmPos c = sm_pos(a, in, q);
    const unsigned id = a.chain_of[c.fwd ? c.alpha : c.beta];
    const uint64_t e = a.ch_eoff[id];
    const unsigned char f = a.fl[q];
    const int out = c.fwd ? sm_rs(f) : sm_ls(f), back = c.fwd ? sm_ls(f) : sm_rs(f);
    a.ent_m[e + c.pos] = a.m.mult[8 * q + out];
    a.ent_l[e + c.pos] = a.m.len[8 * q + out];
    a.ent_chain[e + c.pos] = id;
    if (c.pos == 1) {
        a.ent_m[e] = a.m.mult[8 * q + back];
        a.ent_l[e] = a.m.len[8 * q + back];
        a.ent_chain[e] = id;
    }
}

// Levels t0 .. t0 + kLevels - 1 (below top) of the weighted pairwise reduction
// (graph.cpp:2157-2163), a block's entries in shared memory (as the merge's).
constexpr int kLevels = 10;
__global__ void __launch_bounds__(256) k_sm_levels(SimplifyArgs a, uint64_t total, int t0, int top) {
    constexpr unsigned N = 1u << kLevels;
    __shared__ unsigned char v[N];
    __shared__ unsigned long long w[N];
    __shared__ unsigned cm[N / 2], rel[N / 2];  // of every even entry: its chain's m (kNone: no chain), its position >> t0
    const uint64_t q0 = (uint64_t)blockIdx.x << kLevels;
    for (unsigned i = threadIdx.x; i < N; i += 256) {
        const uint64_t e = (q0 + i) << t0;
        v[i] = e < total ? a.ent_m[e] : 0;
        w[i] = e < total ? a.ent_l[e] : 0;
        if (!(i & 1)) {
            const unsigned id = e < total ? a.ent_chain[e] : kNone;
            cm[i / 2] = id == kNone ? kNone : a.ch_m[id];
            rel[i / 2] = id == kNone ? 0 : (unsigned)((e - a.ch_eoff[id]) >> t0);
        }
    }
    for (int l = 0; l < kLevels && t0 + l < top; ++l) {
        __syncthreads();
        for (unsigned q = threadIdx.x; q < (N >> (l + 1)); q += 256) {
            const unsigned i = q << (l + 1), r = i + (1u << l);
            if (cm[i / 2] == kNone || (((uint64_t)(rel[i / 2] >> l) + 1) << (t0 + l)) > cm[i / 2]) continue;
            const uint64_t ll = w[i], lr = w[r];
            v[i] = (unsigned char)(((uint64_t)v[i] * ll + (uint64_t)v[r] * lr) / (ll + lr));
            w[i] = ll + lr;
        }
    }
    __syncthreads();
    for (unsigned i = threadIdx.x; i < N; i += 256) {
        const uint64_t e = (q0 + i) << t0;
        if (e < total && !(i & 1)) {
            a.ent_m[e] = v[i];
            a.ent_l[e] = w[i];
        }
    }
}

// The two end arcs of every chain take the chain: its total length and
// multiplicity, each other as the arc back; every merged node hands its two
// arc strings to them as pieces at the offsets its walk states summed (the
// arcs between it and the far start, which mirror the arcs before it). own[]
// keeps the ends' old string lengths for the rewrite.
__global__ void k_sm_apply(SimplifyArgs a, int in) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= a.m.lines || !sm_m(a, q)) return;
    a.m.del[q] = 1;
    const SmPos c = sm_pos(a, in, q);
    const uint64_t start = c.fwd ? c.alpha : c.beta, end = c.fwd ? c.beta : c.alpha;
    const unsigned id = a.chain_of[start];
    const uint64_t e = a.ch_eoff[id];
    const unsigned char f = a.fl[q];
    const int out = c.fwd ? sm_rs(f) : sm_ls(f), back = c.fwd ? sm_ls(f) : sm_rs(f);
    const int d_out = c.fwd ? 0 : 1;
    a.xsrc[2 * q] = a.m.src[8 * q + out];
    a.xlen[2 * q] = a.m.len[8 * q + out];
    a.xarc[2 * q] = (unsigned)start;
    a.xat[2 * q] = a.ws[in][2 * q + (d_out ^ 1)];
    a.xsrc[2 * q + 1] = a.m.src[8 * q + back];
    a.xlen[2 * q + 1] = a.m.len[8 * q + back];
    a.xarc[2 * q + 1] = (unsigned)end;
    a.xat[2 * q + 1] = a.ws[in][2 * q + d_out];
    if (c.pos == 1 || c.pos == c.m) {
        const unsigned char mm = a.ent_m[e];
        const unsigned long long tl = a.ent_l[e];
        if (c.pos == 1) {
            a.m.len[start] = (unsigned)tl;
            a.m.mult[start] = mm;
            a.m.back[start] = (unsigned)end;
        }
        if (c.pos == c.m) {
            a.m.len[end] = (unsigned)tl;
            a.m.mult[end] = mm;
            a.m.back[end] = (unsigned)start;
        }
    }
}

int sm_ceil_log2(uint64_t v) {
    int r = 0;
    while ((1ull << r) < v) ++r;
    return r;
}


// ---- printContigs (graph.cpp:1139-1202): every arc of at least
// Contig_Length - k bases (Contig_Length = 100, sequence.h:15) is printed
// once, from the end whose key is not smaller than the far end's, as
// ">proc0: " + the node's k-mer oriented for the arc's side + the arc string.
constexpr int kContigLength = 100;

__device__ __forceinline__ bool ct_prints(const MergedGraph &m, uint64_t a) {
    const uint64_t q = a >> 3;
    const unsigned l = m.len[a];
    if (m.del[q] || l == 0 || (int)l < kContigLength - m.k) return false;
    return m.key[q] >= m.key[m.back[a] >> 3];
}

__global__ void k_ct_len(MergedGraph m, uint64_t *__restrict__ out, unsigned long long *count) {
    const uint64_t a = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= 8 * m.lines) return;
    const bool p = ct_prints(m, a);
    out[a] = p ? 8 + (uint64_t)m.k + m.len[a] + 1 : 0;
    if (p) agg_add(count, 1);
}

__global__ void k_ct_write(MergedGraph m, const uint64_t *__restrict__ off, char *__restrict__ text) {
    const uint64_t a = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (a >= 8 * m.lines || off[a + 1] == off[a]) return;
    char *p = text + off[a];
    const char head[8] = {'>', 'p', 'r', 'o', 'c', '0', ':', ' '};
    for (int i = 0; i < 8; ++i) *p++ = head[i];
    const uint64_t key = m.key[a >> 3];
    const uint64_t o = (a & 7) < 4 ? key : rc_dev(key, m.k);
    for (int i = m.k - 1; i >= 0; --i) *p++ = "ACGT"[(o >> (2 * i)) & 3];
    p[m.len[a]] = '\n';  // the arc string itself is copied in chunks
}

__global__ void k_ct_chunks(MergedGraph m, const uint64_t *__restrict__ off, uint64_t *__restrict__ chunks) {
    const uint64_t a = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (a < 8 * m.lines) chunks[a] = off[a + 1] == off[a] ? 0 : (m.len[a] + kChunk - 1) / kChunk;
}

__global__ void k_ct_copy(MergedGraph m, const uint64_t *__restrict__ off, const uint64_t *__restrict__ first,
                          uint64_t n_chunks, char *__restrict__ out) {
    const uint64_t arcs = 8 * m.lines;
    for (uint64_t c = blockIdx.x; c < n_chunks; c += gridDim.x) {
        uint64_t lo = 0, hi = arcs;
        while (hi - lo > 1) {
            const uint64_t mid = (lo + hi) / 2;
            if (first[mid] <= c) lo = mid;
            else hi = mid;
        }
        const uint64_t at = (c - first[lo]) * kChunk;
        const uint64_t rest = m.len[lo] - at;
        const unsigned l = rest < kChunk ? (unsigned)rest : kChunk;
        const char *a = m.text + m.src[lo] + at;
        char *b = out + off[lo] + 8 + m.k + at;
        for (unsigned i = threadIdx.x; i < l; i += blockDim.x) b[i] = a[i];
    }
}
}  // namespace

swg_status prune_tips(MergedGraph *m, cudaStream_t s, uint64_t *count) {
    Scratch scr(s, m->pool);
    unsigned char *tip = nullptr;
    unsigned long long *ctr = nullptr;
    if (!scr.get(&tip, m->lines) || !scr.get(&ctr, 1)) return cuda_err(cudaErrorMemoryAllocation, "tips workspace");
    EMIT_CUDA(cudaMemsetAsync(ctr, 0, 8, s), "tips");
    if (m->lines) {
        k_pr_tipslot<<<blocks(m->lines), 256, 0, s>>>(*m, tip);
        k_pr_tips<<<blocks(m->lines), 256, 0, s>>>(*m, tip, ctr);
    }
    return rewrite(m, s, scr, Pieces{}, ctr, count);
}

swg_status simplify_lines(MergedGraph *m, cudaStream_t s, uint64_t *count) {
    *count = 0;
    Scratch scr(s, m->pool);
    const uint64_t L = m->lines;
    SimplifyArgs a{};
    a.m = *m;
    constexpr int kCls = 40;
    if (!scr.get(&a.fl, L) || !scr.get(&a.nx[0], 2 * L) || !scr.get(&a.nx[1], 2 * L) ||
        !scr.get(&a.ws[0], 2 * L) || !scr.get(&a.ws[1], 2 * L) || !scr.get(&a.mx[0], 2 * L) ||
        !scr.get(&a.mx[1], 2 * L) || !scr.get(&a.cn[0], 2 * L) || !scr.get(&a.cn[1], 2 * L) ||
        !scr.get(&a.chain_of, 8 * L) || !scr.get(&a.ctr, 8 + 2 * kCls) || !scr.get(&a.own, 8 * L) ||
        !scr.get(&a.xsrc, 2 * L) || !scr.get(&a.xat, 2 * L) || !scr.get(&a.xlen, 2 * L) ||
        !scr.get(&a.xarc, 2 * L))
        return cuda_err(cudaErrorMemoryAllocation, "simplify workspace");
    a.cls_count = a.ctr + 8;
    a.cls_cursor = a.ctr + 8 + kCls;
    EMIT_CUDA(cudaMemsetAsync(a.ctr, 0, (8 + 2 * kCls) * 8, s), "simplify");
    EMIT_CUDA(cudaMemsetAsync(a.xlen, 0, std::max<uint64_t>(2 * L, 1) * 4, s), "simplify");
    if (L == 0) return rewrite(m, s, scr);
    int pairs = (sm_ceil_log2(2 * L) + 2) / 2;
    unsigned *moved = nullptr;
    if (!scr.get(&moved, 64)) return cuda_err(cudaErrorMemoryAllocation, "simplify workspace");
    int sms = 0, dev = 0;
    EMIT_CUDA(cudaGetDevice(&dev), "device");
    EMIT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "device attribute");
    const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)std::max(1, sms), (2 * L + 1023) / 1024);
    unsigned long long h[8 + kCls] = {0};
    const int in = 0;  // the jumps leave their result in the first buffers
    for (int first = 1; first >= 0; --first) {  // again after cutting cycles
        EMIT_CUDA(cudaMemsetAsync(moved, 0, 64 * sizeof(unsigned), s), "simplify");
        if (!first) EMIT_CUDA(cudaMemsetAsync(a.cls_count, 0, kCls * 8, s), "simplify");
        void *args[] = {&a, &pairs, &moved, &first};
        EMIT_CUDA(cudaLaunchCooperativeKernel((const void *)k_sm_rank, dim3(grid), dim3(1024), args, 0, s), "simplify");
        EMIT_CUDA(cudaMemcpyAsync(h, a.ctr, sizeof(h), cudaMemcpyDeviceToHost, s), "simplify");
        EMIT_CUDA(cudaStreamSynchronize(s), "simplify");
        if (!h[3]) break;
    }
    const unsigned long long *cls = h + 8;
    unsigned long long cursor[kCls];
    uint64_t total = 0, n_chains = 0;
    int top = 0;
    for (int c = kCls - 1; c >= 0; --c) {
        cursor[c] = total;
        total += cls[c] << c;
        n_chains += cls[c];
        if (cls[c] && !top) top = c;
    }
    EMIT_CUDA(cudaMemcpyAsync(a.cls_cursor, cursor, sizeof(cursor), cudaMemcpyHostToDevice, s), "simplify");
    if (!scr.get(&a.ch_eoff, n_chains) || !scr.get(&a.ch_m, n_chains) || !scr.get(&a.ent_m, total) ||
        !scr.get(&a.ent_l, total) || !scr.get(&a.ent_chain, total))
        return cuda_err(cudaErrorMemoryAllocation, "simplify chains");
    EMIT_CUDA(cudaMemsetAsync(a.ent_chain, 0xff, std::max<uint64_t>(total, 1) * 4, s), "simplify");
    EMIT_CUDA(cudaMemcpyAsync(a.own, m->len, 8 * L * 4, cudaMemcpyDeviceToDevice, s), "simplify");
    k_sm_chain_alloc<<<blocks(L), 256, 0, s>>>(a, in);
    k_sm_entries<<<blocks(L), 256, 0, s>>>(a, in);
    for (int t = 0; t < top; t += kLevels) {
        const uint64_t per = 1ull << (t + kLevels);
        k_sm_levels<<<(unsigned)((total + per - 1) / per), 256, 0, s>>>(a, total, t, top);
    }
    k_sm_apply<<<blocks(L), 256, 0, s>>>(a, in);
    EMIT_CUDA(cudaGetLastError(), "simplify kernels");
    *count = h[0] - h[1];
    Pieces x;
    x.own = a.own;
    x.n = 2 * L;
    x.src = a.xsrc;
    x.len = a.xlen;
    x.arc = a.xarc;
    x.at = a.xat;
    return rewrite(m, s, scr, x);
}

swg_status write_contigs(MergedGraph *m, const char *path, cudaStream_t s, uint64_t *count) {
    *count = 0;
    Scratch scr(s, m->pool);
    const uint64_t arcs = 8 * m->lines;
    uint64_t *len = nullptr, *off = nullptr, *chunks = nullptr, *first = nullptr;
    unsigned long long *ctr = nullptr;
    if (!scr.get(&len, arcs) || !scr.get(&off, arcs + 1) || !scr.get(&chunks, arcs) ||
        !scr.get(&first, arcs + 1) || !scr.get(&ctr, 1))
        return cuda_err(cudaErrorMemoryAllocation, "contig workspace");
    EMIT_CUDA(cudaMemsetAsync(ctr, 0, 8, s), "contigs");
    if (arcs) k_ct_len<<<blocks(arcs), 256, 0, s>>>(*m, len, ctr);
    swg_status st = scan_lengths(len, off, arcs, scr, s);
    if (st) return st;
    uint64_t h[2] = {0, 0};
    EMIT_CUDA(cudaMemcpyAsync(&h[0], off + arcs, 8, cudaMemcpyDeviceToHost, s), "contigs");
    EMIT_CUDA(cudaMemcpyAsync(&h[1], ctr, 8, cudaMemcpyDeviceToHost, s), "contigs");
    EMIT_CUDA(cudaStreamSynchronize(s), "contigs");
    char *text = nullptr;
    if (!scr.get(&text, h[0])) return cuda_err(cudaErrorMemoryAllocation, "contig text");
    if (arcs) {
        k_ct_write<<<blocks(arcs), 256, 0, s>>>(*m, off, text);
        k_ct_chunks<<<blocks(arcs), 256, 0, s>>>(*m, off, chunks);
        st = scan_lengths(chunks, first, arcs, scr, s);
        if (st) return st;
        uint64_t n_chunks = 0;
        EMIT_CUDA(cudaMemcpyAsync(&n_chunks, first + arcs, 8, cudaMemcpyDeviceToHost, s), "contigs");
        EMIT_CUDA(cudaStreamSynchronize(s), "contigs");
        if (n_chunks)
            k_ct_copy<<<(unsigned)std::min<uint64_t>(n_chunks, 1u << 20), 256, 0, s>>>(*m, off, first, n_chunks,
                                                                                      text);
    }
    EMIT_CUDA(cudaGetLastError(), "contig kernels");
    *count = h[1];
    return stream_to_file(text, h[0], path, s);
}

swg_status prune_low_coverage(MergedGraph *m, cudaStream_t s, uint64_t *count) {
    Scratch scr(s, m->pool);
    unsigned long long *ctr = nullptr;
    if (!scr.get(&ctr, 3)) return cuda_err(cudaErrorMemoryAllocation, "low-coverage workspace");
    EMIT_CUDA(cudaMemsetAsync(ctr, 0, 24, s), "low coverage");
    if (m->lines) {
        k_pr_cov<<<blocks(m->lines), 256, 0, s>>>(*m, ctr);
        k_pr_low<<<blocks(m->lines), 256, 0, s>>>(*m, ctr, ctr + 2);
    }
    return rewrite(m, s, scr, Pieces{}, ctr + 2, count);
}

}  // namespace swg
