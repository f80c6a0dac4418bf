// Merging of semi-extended k-molecules on the device: the result of the
// reference's SWAP merge loop (simplifyDistNodeGraph, graph.cpp:1392-1566,
// with the edge messages of recvProc, graph.cpp:1204-1389) over the filtered
// k-mer graph, written as the gathered node lines of its -d file
// contigGraph.txt (gatherDistNodeGraph, graph.cpp:576-696).
//
// A node with exactly one arc on each side whose arcs do not lead back to
// itself is merged away; all other nodes end the chains of merged nodes, and
// each end arc finally spells the whole chain up to the next end node (the
// arc strings do not depend on the order the merge visits nodes in). The
// multiplicity of a merged arc is the reference's running weighted average
// (graph.cpp:1322-1324: 64-bit sum kept in an int, divided by the new length,
// truncated to 8 bits), which does depend on that order. The device follows
// one fixed order: a chain of m merged nodes is numbered 1..m from its
// smaller end arc (node key, then slot) and node p is visited at level
// ctz(p), so each level merges disjoint pairs of neighbouring segments — a
// pairwise tree reduction of the chain's unit arcs. A cycle made only of
// mergeable nodes is cut at its largest key, which is visited last and keeps
// the whole cycle on its two arcs.
//
// Steps (one stream): open-addressing index key -> node (4-byte entries);
// per node the neighbour of each arc; for every mergeable node two
// directed walk states; list ranking of the walks in three steps (within
// tiles of neighbouring nodes, in shared memory; over the states where walks
// enter tiles, each eighth walking to the next; over those by pointer
// jumping); cycles (states that are not reached so, or whose list never
// ends) are found, cut and ranked by pointer jumping; chains are laid out in
// power-of-two aligned segments so the tree reduction runs level by level in
// place; finally the surviving nodes are ordered by key, each formats its
// line and every merged node writes its two bases straight into the arc
// strings of the two ends. Node indices follow the build's output order,
// which the result does not depend on: chains are numbered by the keys of
// their end nodes.
#include <cuda_runtime.h>

#include <cooperative_groups.h>
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cstdint>
#include <cstring>

#include "swg_internal.h"
#include "text_dev.cuh"

namespace swg {
namespace {

constexpr unsigned long long kTerm = 1ull << 63;  // walk successor: end arc code (node * 8 + slot)
constexpr unsigned kEnd = 1u << 31;               // 32-bit successor or list entry: an end arc is reached
constexpr unsigned kHead = 1u << 30;              // ruler list entry: the walk's first
constexpr unsigned kNone = 0xffffffffu;
constexpr unsigned kNodeMask = (1u << 29) - 1;
constexpr int kClasses = 40;  // chain segment size classes 2^0 .. 2^39

// error bits
constexpr unsigned kErrIndex = 1u, kErrNeighbour = 2u, kErrWalk = 4u, kErrCycle = 8u, kErrOrder = 16u;

// Per chain position of a merge in a given visiting order: the visit time of
// the node at the position, and the two segments that meet there (the first
// arc of the left one, the last arc of the right one, their multiplicities)
// once both are merged; `arrive` counts the sides that have arrived.
struct CartSlot {
    unsigned t;
    unsigned lb, rb;
    unsigned arrive;
    unsigned char lv, rv;
};

__device__ __forceinline__ uint64_t fmix64(uint64_t x) {  // MurmurHash3 finaliser
    x ^= x >> 33;
    x *= 0xff51afd7ed558ccdull;
    x ^= x >> 33;
    x *= 0xc4ceb9fe1a85ec53ull;
    x ^= x >> 33;
    return x;
}

namespace cg = cooperative_groups;

// Counter increments aggregated over the threads of a warp that make them
// together (one atomic per counter per warp); returns this thread's slot.
__device__ __forceinline__ unsigned long long agg_inc(unsigned long long *ctr) {
    cg::coalesced_group g = cg::coalesced_threads();
    unsigned long long base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(ctr, (unsigned long long)g.size());
    return g.shfl(base, 0) + g.thread_rank();
}

// The same for threads that target different counters ctr[label], each
// adding step(label).
__device__ __forceinline__ unsigned long long agg_add_labeled(unsigned long long *ctr, int label,
                                                              unsigned long long step) {
    cg::coalesced_group g = cg::labeled_partition(cg::coalesced_threads(), label);
    unsigned long long base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(ctr + label, step * g.size());
    return g.shfl(base, 0) + step * g.thread_rank();
}

struct MergeArgs {
    int k;
    uint64_t n;
    const unsigned long long *keys;
    const unsigned long long *mult;  // byte s = multiplicity of slot s
    unsigned *ht;                    // index: the key's hash's top 3 bits << 29 | node (kNone when free)
    uint64_t hmask;
    unsigned *nb;              // n*8: (neighbour << 1) | arrival side, kNone for an empty slot
    unsigned char *fl;         // bit0 mergeable, bits1-2 right slot, bits3-4 left slot - 4
    unsigned long long *oo;    // per state: its ruler << 32 | distance from it (~0: none)
    unsigned *rpos;            // ruler list position of a ruler state
    uint2 *rp0;                // ruler list: next ruler or end arc, states to it | kEnd at an end arc, kHead
    uint2 *ro;                 // per ruler: its pole, distance from it (kNone: none)
    uint2 *pp0, *pp1;          // pole list: next pole or end arc, states to it | kEnd at an end arc
    unsigned *heads;           // poles that are walks' first rulers (then: chains' first nodes)
    unsigned *moved;           // per pair of rounds of the pole list's jumping: a pole had not arrived
    uint2 *lt;                 // per state: states from it to the end of its walk, end arc reached
    unsigned *clist;
    unsigned long long *cx0, *cx1, *cy0, *cy1;  // cycle pointer jumping
    unsigned *chain_of;        // per arc code: chain id (set at the chain's start arc)
    unsigned long long *ch_eoff;
    unsigned *ch_m;
    unsigned long long *ch_dfwd, *ch_drev;
    unsigned char *ent;        // chain unit-arc multiplicities, reduced in place
    unsigned *ent_chain;
    unsigned long long *cls_count, *cls_cursor;
    unsigned long long *ctr;   // [0] rulers [1] cycle states [2] chains' first nodes [3] cycles cut [4] merged nodes
                               // [5] surviving nodes [6] poles listed
    unsigned long long *skey;  // surviving nodes: keys, then (sorted) node indices
    unsigned long long *sidx;
    unsigned *err;             // (the word after the counters [0] to [6])
    // merge in a given visiting order (null: the fixed tree order)
    unsigned long long *vt;    // per node: its visit time
    CartSlot *cart;            // per chain position (the ent layout)
};

// The index holds nodes, not keys: 4 bytes a slot keep it, and the keys, in L2
// for ten times the nodes that 16-byte slots did (5M nodes: 67 MB where it was
// 268, and 67 MB to clear). A key is read where the slot's 3 bits of its hash
// agree, so probes past other keys seldom read one. (n < 2^29: an entry is
// never kNone.)
__device__ __forceinline__ unsigned lookup(const MergeArgs &a, uint64_t key) {
    const uint64_t f = fmix64(key);
    const unsigned tag = (unsigned)(f >> 61);
    uint64_t h = f & a.hmask;
    for (uint64_t probe = 0; probe <= a.hmask; ++probe) {
        const unsigned e = a.ht[h];
        if (e == kNone) return kNone;
        if (e >> 29 == tag && a.keys[e & kNodeMask] == key) return e & kNodeMask;
        h = (h + 1) & a.hmask;
    }
    return kNone;
}

__device__ __forceinline__ unsigned mbyte(uint64_t m, int s) { return (unsigned)(m >> (8 * s)) & 0xffu; }
__device__ __forceinline__ bool is_m(const MergeArgs &a, uint64_t i) { return a.fl[i] & 1u; }
__device__ __forceinline__ int rslot(unsigned char f) { return (f >> 1) & 3; }
__device__ __forceinline__ int lslot(unsigned char f) { return 4 + ((f >> 3) & 3); }

__global__ void k_mg_index(MergeArgs a) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const unsigned long long key = a.keys[i];
    const uint64_t f = fmix64(key);
    const unsigned tag = (unsigned)(f >> 61);
    uint64_t h = f & a.hmask;
    for (uint64_t probe = 0; probe <= a.hmask; ++probe) {
        const unsigned prev = atomicCAS(&a.ht[h], kNone, tag << 29 | (unsigned)i);
        if (prev == kNone || (prev >> 29 == tag && a.keys[prev & kNodeMask] == key)) return;
        h = (h + 1) & a.hmask;
    }
    atomicOr(a.err, kErrIndex);
}

// Neighbour of every arc (node::getNodeID, graph.cpp:164-196: oriented k-mer
// plus the arc base, last k bases, canonical id and the side reached) and
// whether the node is merged away. A thread goes through its node's arcs, not
// through the eight slots: the lanes of a warp have theirs in different slots,
// and a warp then waits for two lookups where it waited for eight. One counter
// update a block: one a warp, all of them to the same word, took longer than
// the lookups. 5M nodes: 325 us with 16-byte index slots, eight
// rounds and a counter update a warp, 141 now (4.2 TB/s of DRAM traffic).
__global__ void __launch_bounds__(256) k_mg_classify(MergeArgs a) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    bool merged = false;
    if (i < a.n) {
        const int k = a.k;
        const uint64_t kmask = (1ull << (2 * k)) - 1;
        const uint64_t key = a.keys[i], m = a.mult[i], rk = rc_dev(key, k);
        const uint64_t full = (((m & 0x7f7f7f7f7f7f7f7full) + 0x7f7f7f7f7f7f7f7full) | m) & 0x8080808080808080ull;
        uint4 *nb = reinterpret_cast<uint4 *>(a.nb + i * 8);
        nb[0] = nb[1] = make_uint4(kNone, kNone, kNone, kNone);
        bool ok = true;  // every neighbour is there and none is the node itself
        for (uint64_t left = full; left; left &= left - 1) {
            const int s = (__ffsll((long long)left) - 1) >> 3;
            const uint64_t e = (((s < 4 ? key : rk) << 2) | (uint64_t)(s & 3)) & kmask;
            const uint64_t r = rc_dev(e, k);
            const unsigned side = e >= r;
            const unsigned j = lookup(a, side ? e : r);
            if (j == kNone) {
                atomicOr(a.err, kErrNeighbour);
                ok = false;
            } else {
                a.nb[i * 8 + s] = (j << 1) | side;
                ok &= (uint64_t)j != i;
            }
        }
        const unsigned right = (unsigned)full, l = (unsigned)(full >> 32);
        merged = ok && __popc(right) == 1 && __popc(l) == 1;
        const int rs = right ? (31 - __clz(right)) >> 3 : 0, ls = l ? (31 - __clz(l)) >> 3 : 0;
        a.fl[i] = (unsigned char)((merged ? 1 : 0) | (rs << 1) | (ls << 3));
    }
    const int c = __syncthreads_count(merged);
    if (threadIdx.x == 0 && c) atomicAdd(&a.ctr[4], (unsigned long long)c);
}

// Walk state 2i+d of a merged node: d = 0 traverses it as its key (leaves by
// the right arc), d = 1 as the reverse complement (leaves by the left arc).
// The successor is the next merged node's state, or the end arc that points
// back from the end node reached: its side of arrival picks the half, the
// first base of the k-mer just left gives the slot.
__device__ __forceinline__ unsigned long long walk_next(const MergeArgs &a, uint64_t i, int d) {
    const unsigned char f = a.fl[i];
    const unsigned v = a.nb[i * 8 + (d ? lslot(f) : rslot(f))];
    const uint64_t j = v >> 1;
    const unsigned side = v & 1u;
    if (is_m(a, j)) return v ^ 1u;  // state 2 * j + (side ? 0 : 1)
    const uint64_t o = d ? rc_dev(a.keys[i], a.k) : a.keys[i];
    const unsigned first = (unsigned)(o >> (2 * (a.k - 1))) & 3u;
    return kTerm | (j * 8 + (side ? 4 : 0) + 3 - first);
}

// The same, with kEnd for any end arc.
__device__ __forceinline__ unsigned walk_state(const MergeArgs &a, unsigned char f, uint64_t i, int d) {
    const unsigned v = a.nb[i * 8 + (d ? lslot(f) : rslot(f))];
    return is_m(a, v >> 1) ? v ^ 1u : kEnd;  // state 2 * j + (side ? 0 : 1)
}

// Both walk states of a merged node, ranked within the block's 512 nodes. The
// build leaves the k-molecules of a bucket side by side, and a walk stays in a
// bucket for six to nine nodes, so most of it is a matter of shared memory
// here, with coalesced reads and writes around it, where walking node by node
// through memory took as long as all else together. A state whose predecessor
// (its twin's successor's twin) lies in another tile, or which has none, is a
// ruler; the others are ranked from theirs by pointer jumping, as many rounds
// as the tile's longest stretch needs (states of a cycle within the tile never
// get there). Per state in shared memory: predecessor | distance << 11 | rooted.
// 5M nodes: 103 us (116 with tiles of 1024 nodes, fewer of them an SM); with
// the ruler list's kernel 236 where states, walks and list took 347.
constexpr int kTile = 512;
__global__ void __launch_bounds__(kTile, 4) k_mg_states(MergeArgs a) {
    constexpr unsigned kRooted = 1u << 31, kDist = 0xffffu << 11;
    __shared__ unsigned v[2 * kTile], pos[2 * kTile];
    __shared__ unsigned rulers;
    __shared__ unsigned long long base;
    const unsigned t = threadIdx.x;
    const uint64_t first = (uint64_t)blockIdx.x * kTile, i = first + t;
    if (t == 0) rulers = 0;
    const unsigned char f = i < a.n ? a.fl[i] : 0;
    const bool in = f & 1u;
    unsigned nx[2] = {kEnd, kEnd}, w[2];
    if (in) {
        nx[0] = walk_state(a, f, i, 0);
        nx[1] = walk_state(a, f, i, 1);
    }
    __syncthreads();
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        const unsigned pred = nx[d ^ 1] ^ 1u;  // (if the twin has a successor)
        const bool here = in && !(nx[d ^ 1] & kEnd) && (pred >> 1) - first < (uint64_t)kTile;
        w[d] = here ? (pred - (unsigned)(2 * first)) | 1u << 11 : (2 * t + d) | kRooted;
        v[2 * t + d] = w[d];
        if (in && !here) pos[2 * t + d] = atomicAdd(&rulers, 1u);
    }
    __syncthreads();
    if (t == 0 && rulers) base = atomicAdd(&a.ctr[0], (unsigned long long)rulers);
    for (int r = 0; r < 12; ++r) {  // stretches are at most 2 * kTile - 1 states
        bool open = false;
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            if (w[d] & kRooted) continue;
            const unsigned u = v[w[d] & (2 * kTile - 1)];
            w[d] = (u & (kRooted | (2 * kTile - 1))) | (((w[d] & kDist) + (u & kDist)) & kDist);
            open |= !(w[d] & kRooted);
        }
        const bool more = __syncthreads_or(open);
        v[2 * t] = w[0];
        v[2 * t + 1] = w[1];
        __syncthreads();
        if (!more) break;
    }
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        if (!in || w[d] != ((2 * t + d) | kRooted)) continue;
        const unsigned at = (unsigned)base + pos[2 * t + d];
        a.rpos[2 * i + d] = at;
        a.rp0[at] = make_uint2(0, kEnd);  // (stays if arcs do not lead back)
    }
    __syncthreads();
    if (!in) return;
    unsigned long long o[2];
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        const unsigned root = w[d] & (2 * kTile - 1), dist = (w[d] & kDist) >> 11;
        const unsigned at = (unsigned)base + pos[root];
        o[d] = w[d] & kRooted ? (unsigned long long)at << 32 | dist : ~0ull;
        if (!(w[d] & kRooted)) continue;
        // the stretch's last state knows where it leads, and whether it is a walk's first stretch
        const bool end = nx[d] & kEnd;
        if (end || (nx[d] >> 1) - first >= (uint64_t)kTile) {
            const uint64_t r = first + (root >> 1);
            const bool head = root == 2 * t + d ? nx[d ^ 1] & kEnd : walk_state(a, a.fl[r], r, (root & 1) ^ 1) & kEnd;
            a.rp0[at] = make_uint2(end ? (unsigned)walk_next(a, i, d) : nx[d], (dist + 1) | (end ? kEnd : 0) | (head ? kHead : 0));
        }
    }
    *reinterpret_cast<ulonglong2 *>(a.oo + 2 * i) = make_ulonglong2(o[0], o[1]);
}

// The ruler list ranked, in one cooperative launch (a grid barrier costs less
// than a launch, and one block of 1024 an SM less than more): every eighth
// ruler and every walk's first is a pole; the poles walk to the next pole,
// noting the rulers on the way; the poles' list is ranked by pointer jumping;
// the rulers take over their pole's result. Bound by the latency of random
// loads, all of L2: so as few rounds over as short a list as walks of some
// twenty steps leave. Jumping rounds go in pairs, so that the result is in pp0
// again, and end once every pole has reached an end (the poles of a cycle never
// do). 5M nodes: 133 us. (A longest walk has twelve times the mean: every fourth
// ruler a pole shortens it, but doubles the list, 25 us more in all; blocks for
// n / 8192, up to one an SM, because a barrier's time grows with them.)
constexpr unsigned kPole = 8;
__global__ void __launch_bounds__(1024) k_mg_rank(MergeArgs a, int pairs) {
    const uint64_t n_rul = a.ctr[0], stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t p0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, every = (n_rul + kPole - 1) / kPole;
    for (uint64_t q = p0; q < n_rul; q += stride) {  // next rulers from states to list positions
        const uint2 v = __ldcg(a.rp0 + q);
        if (!(v.y & kEnd)) {
            const unsigned next = a.rpos[v.x];
            if (next >= n_rul) atomicOr(a.err, kErrWalk);  // (arcs that do not lead back)
            a.rp0[q].x = next < n_rul ? next : 0;
        }
        uint2 o = make_uint2(kNone, 0);
        if (q % kPole == 0) {
            o.x = (unsigned)(q / kPole);
        } else if (v.y & kHead) {
            const uint64_t h = agg_inc(&a.ctr[6]);
            a.heads[h] = (unsigned)q;
            o.x = (unsigned)(every + h);
        }
        a.ro[q] = o;
    }
    cg::this_grid().sync();
    const uint64_t n_pole = every + __ldcg(&a.ctr[6]);
    for (uint64_t p = p0; p < n_pole; p += stride) {
        uint64_t cur = p < every ? p * kPole : __ldcg(a.heads + (p - every));
        uint2 out = make_uint2(0, kEnd);
        bool done = false;
        unsigned o = 0;
        for (uint64_t step = 0; step <= n_rul && !done; ++step) {
            const uint2 v = __ldcg(a.rp0 + cur);
            o += v.y & (kHead - 1);
            done = (v.y & kEnd) || v.x % kPole == 0;
            if (done) {
                out = v.y & kEnd ? make_uint2(v.x, o | kEnd) : make_uint2(v.x / kPole, o);
            } else {
                a.ro[v.x] = make_uint2((unsigned)p, o);
                cur = v.x;
            }
        }
        if (!done) atomicOr(a.err, kErrWalk);
        a.pp0[p] = out;
    }
    cg::this_grid().sync();
    for (int r = 0; r < pairs; ++r) {
        bool moved = false;
        for (int half = 0; half < 2; ++half) {
            const uint2 *in = half ? a.pp1 : a.pp0;
            uint2 *out = half ? a.pp0 : a.pp1;
            for (uint64_t p = p0; p < n_pole; p += stride) {
                uint2 v = __ldcg(in + p);
                if (!(v.y & kEnd)) {  // (a cycle's sums mean nothing, and stay below kEnd)
                    const uint2 w = __ldcg(in + v.x);
                    v = make_uint2(w.x, ((v.y + (w.y & ~kEnd)) & ~kEnd) | (w.y & kEnd));
                    moved |= !(v.y & kEnd);
                }
                out[p] = v;
            }
            if (half && moved) a.moved[r] = 1;
            cg::this_grid().sync();
            moved = false;
        }
        if (!*(volatile unsigned *)(a.moved + r)) break;
    }
    for (uint64_t q = p0; q < n_rul; q += stride) {
        const uint2 o = __ldcg(a.ro + q);
        uint2 v = make_uint2(0, 0);
        if (o.x != kNone) {
            const uint2 w = __ldcg(a.pp0 + o.x);
            if (w.y & kEnd) v = make_uint2(w.x, w.y - o.y);
        }
        a.rp0[q] = v;
    }
}

// ---- chains
// End arcs compare by (key of the end node, slot). Only end nodes' keys are
// read here: a small, cache-resident set.
__device__ __forceinline__ bool arc_less(const MergeArgs &a, uint64_t x, uint64_t y) {
    const unsigned long long kx = a.keys[x >> 3], ky = a.keys[y >> 3];
    return kx < ky || (kx == ky && (x & 7) < (y & 7));
}

struct ChainPos {
    unsigned m, pos;
    uint64_t start;  // the smaller end arc code: the chain's start
    bool fwd;        // the chain runs through this node as its key (state 2i)
};

__device__ __forceinline__ ChainPos chain_pos_of(const MergeArgs &a, uint4 lt) {
    ChainPos c;
    const unsigned la = lt.x, lb = lt.z;
    const uint64_t beta = lt.y, alpha = lt.w;
    c.m = la + lb - 1;
    c.fwd = arc_less(a, alpha, beta);
    c.pos = c.fwd ? lb : la;
    c.start = c.fwd ? alpha : beta;
    return c;
}

__device__ __forceinline__ ChainPos chain_pos(const MergeArgs &a, uint64_t i) {
    return chain_pos_of(a, *reinterpret_cast<const uint4 *>(a.lt + 2 * i));
}

__device__ __forceinline__ int size_class(unsigned m) {  // ceil(log2(m + 1))
    return m == 0 ? 0 : 64 - __clzll((unsigned long long)m);
}

// A chain's first node counts it by size and lists itself.
__device__ __forceinline__ void count_chain(const MergeArgs &a, uint64_t i, const ChainPos &c) {
    if (c.pos != 1) return;
    agg_add_labeled(a.cls_count, size_class(c.m), 1);
    a.heads[agg_inc(&a.ctr[2])] = (unsigned)i;  // (the poles' list is done with)
}

// Per state the distance to its walk's end and the end arc, and the chains
// counted while both are at hand (again by k_mg_chain_count once cycles are
// cut; their states, at 0, are no chain's). 5M nodes: 40 us, two kernels took 62.
__global__ void k_mg_finish(MergeArgs a) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n || !is_m(a, i)) return;
    const ulonglong2 oo = *reinterpret_cast<const ulonglong2 *>(a.oo + 2 * i);
    uint2 lt[2];
#pragma unroll
    for (int d = 0; d < 2; ++d) {
        const unsigned long long o = d ? oo.y : oo.x;
        uint2 v = make_uint2(0, 0);
        if (o != ~0ull) v = a.rp0[o >> 32];
        const bool ends = v.y & kEnd;
        lt[d] = ends ? make_uint2((v.y & ~kEnd) - (unsigned)o, v.x) : make_uint2(0, 0);
        if (!ends) a.clist[agg_inc(&a.ctr[1])] = (unsigned)(2 * i + d);
    }
    const uint4 both = make_uint4(lt[0].x, lt[0].y, lt[1].x, lt[1].y);
    *reinterpret_cast<uint4 *>(a.lt + 2 * i) = both;
    count_chain(a, i, chain_pos_of(a, both));
}

// ---- cycles of merged nodes: largest key by pointer jumping, cut there
// A cycle keeps the node the merge visits last: the largest key in the fixed
// order, the latest visit time in a given one.
__device__ __forceinline__ unsigned long long cut_rank(const MergeArgs &a, uint64_t node) {
    return a.vt ? a.vt[node] : a.keys[node];
}

__global__ void k_mg_cyc_init(MergeArgs a, uint64_t c) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= c) return;
    const unsigned st = a.clist[t];
    a.cx0[st] = cut_rank(a, st >> 1);
    a.cy0[st] = walk_next(a, st >> 1, (int)(st & 1));  // (no end arc in a cycle)
}

__global__ void k_mg_cyc_max(MergeArgs a, uint64_t c, const unsigned long long *__restrict__ mx_in,
                             const unsigned long long *__restrict__ nx_in, unsigned long long *__restrict__ mx_out,
                             unsigned long long *__restrict__ nx_out) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= c) return;
    const unsigned st = a.clist[t];
    const unsigned long long nx = nx_in[st];
    mx_out[st] = max(mx_in[st], mx_in[nx]);
    nx_out[st] = nx_in[nx];
}

__global__ void k_mg_cyc_cut(MergeArgs a, uint64_t c, const unsigned long long *__restrict__ mx) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= c) return;
    const unsigned st = a.clist[t];
    if (cut_rank(a, st >> 1) == mx[st]) {
        a.fl[st >> 1] &= (unsigned char)~1u;  // both states of the node store the same
        if (!(st & 1)) atomicAdd(&a.ctr[3], 1ull);
    }
}

__global__ void k_mg_cyc_succ(MergeArgs a, uint64_t c) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= c) return;
    const unsigned st = a.clist[t];
    if (!is_m(a, st >> 1)) return;
    a.cy0[st] = walk_next(a, st >> 1, (int)(st & 1));
    a.cx0[st] = 1;
}

__global__ void k_mg_cyc_rank(MergeArgs a, uint64_t c, const unsigned long long *__restrict__ ln_in,
                              const unsigned long long *__restrict__ nx_in, unsigned long long *__restrict__ ln_out,
                              unsigned long long *__restrict__ nx_out) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= c) return;
    const unsigned st = a.clist[t];
    if (!is_m(a, st >> 1)) return;
    const unsigned long long nx = nx_in[st];
    if (nx & kTerm) {
        ln_out[st] = ln_in[st];
        nx_out[st] = nx;
    } else {
        ln_out[st] = ln_in[st] + ln_in[nx];
        nx_out[st] = nx_in[nx];
    }
}

__global__ void k_mg_cyc_done(MergeArgs a, uint64_t c, const unsigned long long *__restrict__ ln,
                              const unsigned long long *__restrict__ nx) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= c) return;
    const unsigned st = a.clist[t];
    if (!is_m(a, st >> 1)) return;
    if (!(nx[st] & kTerm)) atomicOr(a.err, kErrCycle);
    a.lt[st] = make_uint2((unsigned)ln[st], (unsigned)nx[st]);
}

__global__ void k_mg_chain_count(MergeArgs a) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n || !is_m(a, i)) return;
    count_chain(a, i, chain_pos(a, i));
}

__global__ void k_mg_chain_alloc(MergeArgs a, uint64_t n_chains) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_chains) return;
    const ChainPos c = chain_pos(a, a.heads[q]);
    const int cl = size_class(c.m);
    const unsigned id = (unsigned)q;
    a.ch_eoff[id] = agg_add_labeled(a.cls_cursor, cl, 1ull << cl);
    a.ch_m[id] = c.m;
    a.chain_of[c.start] = id;
}

// Unit arc p (0..m) of a chain: between its nodes at positions p and p+1
// (0 and m+1 are the end nodes); node p stores the arc it leaves by, node 1
// also the arc it enters by.
__global__ void k_mg_entries(MergeArgs a) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    if (!is_m(a, i)) {  // a node left: listed for the key-order sort
        const unsigned long long q = agg_inc(&a.ctr[5]);
        a.skey[q] = a.keys[i];
        a.sidx[q] = i;
        return;
    }
    const ChainPos c = chain_pos(a, i);
    const unsigned id = a.chain_of[c.start];
    const uint64_t e = a.ch_eoff[id];
    const unsigned char f = a.fl[i];
    const uint64_t m = a.mult[i];
    a.ent[e + c.pos] = (unsigned char)mbyte(m, c.fwd ? rslot(f) : lslot(f));
    a.ent_chain[e + c.pos] = id;
    if (a.cart) {
        CartSlot z;
        z.t = (unsigned)a.vt[i];
        z.lb = z.rb = z.arrive = 0;
        z.lv = z.rv = 0;
        a.cart[e + c.pos] = z;
    }
    if (c.pos == 1) {
        a.ent[e] = (unsigned char)mbyte(m, c.fwd ? lslot(f) : rslot(f));
        a.ent_chain[e] = id;
    }
}

// Levels t0 .. t0 + kLevels - 1 (below top) of the pairwise reduction: at
// level t the node at position (2b+1)*2^t merges segment b (left) with segment
// b+1 (right), graph.cpp:1322-1324. Segments are aligned to their size, so a
// block that holds 2^kLevels entries at stride 2^t0 in shared memory takes all
// of these levels alone (a launch per level, 21 for a chain of millions, took
// 4 us each for almost no work past the first few).
constexpr int kLevels = 12;
__global__ void __launch_bounds__(512) k_mg_levels(MergeArgs a, uint64_t total, int t0, int top) {
    constexpr unsigned N = 1u << kLevels;
    __shared__ unsigned char v[N];
    __shared__ unsigned cm[N / 2], rel[N / 2];  // of every even entry: its chain's m (kNone: no chain), its position >> t0
    const uint64_t q0 = (uint64_t)blockIdx.x << kLevels;
    for (unsigned i = threadIdx.x; i < N; i += 512) {
        const uint64_t e = (q0 + i) << t0;
        v[i] = e < total ? a.ent[e] : 0;
        if (!(i & 1)) {
            const unsigned id = e < total ? a.ent_chain[e] : kNone;
            cm[i / 2] = id == kNone ? kNone : a.ch_m[id];
            rel[i / 2] = id == kNone ? 0 : (unsigned)((e - a.ch_eoff[id]) >> t0);
        }
    }
    for (int l = 0; l < kLevels && t0 + l < top; ++l) {
        __syncthreads();
        const int t = t0 + l;
        for (unsigned q = threadIdx.x; q < (N >> (l + 1)); q += 512) {
            const unsigned i = q << (l + 1);
            if (cm[i / 2] == kNone) continue;
            const uint64_t m = cm[i / 2], b = rel[i / 2] >> l;
            if (((b + 1) << t) > m) continue;  // no node in the middle: the segment carries over
            const uint64_t ll = 1ull << t;
            const uint64_t lr = min((b + 2) << t, m + 1) - ((b + 1) << t);
            const uint64_t sum = (uint64_t)v[i] * ll + (uint64_t)v[i + (1u << l)] * lr;
            const int pre = (int)(unsigned)sum;
            v[i] = (unsigned char)((uint64_t)(int64_t)pre / (ll + lr));
        }
    }
    __syncthreads();
    for (unsigned i = threadIdx.x; i < N; i += 512) {
        const uint64_t e = (q0 + i) << t0;
        if (e < total && !(i & 1)) a.ent[e] = v[i];
    }
}

// Merge in a given visiting order. Visiting the node at position p merges the
// segment of unit arcs to its left with the one to its right, each spanning
// up to the nearest node on that side still unvisited (or the chain's end):
// the chain's merge tree is the Cartesian tree of the visit times. One thread
// starts at every unit arc; a segment belongs to whichever of its two
// bounding nodes is visited first; a thread publishes its segment there, and
// the second of the two sides to arrive combines them (the weighted average
// of graph.cpp:1322-1324) and carries the merged segment on. The root (no
// unvisited bound left) writes the chain's multiplicity to its first entry.
__global__ void k_mg_cart(MergeArgs a, uint64_t total) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= total) return;
    const unsigned id = a.ent_chain[e];
    if (id == kNone) return;
    const uint64_t e0 = a.ch_eoff[id], m = a.ch_m[id];
    uint64_t l = e - e0, r = l;  // the segment: unit arcs l..r
    unsigned v = a.ent[e];
    for (uint64_t step = 0; step <= m; ++step) {
        const unsigned tl = l == 0 ? kNone : a.cart[e0 + l].t;      // node l bounds it on the left
        const unsigned tr = r == m ? kNone : a.cart[e0 + r + 1].t;  // node r+1 on the right
        if (tl == kNone && tr == kNone) {
            a.ent[e0] = (unsigned char)v;
            return;
        }
        const bool as_right = tl < tr;  // node l is visited first: this is its right side
        const uint64_t p = as_right ? l : r + 1;
        CartSlot *cs = a.cart + e0 + p;
        if (as_right) {
            cs->rv = (unsigned char)v;
            cs->rb = (unsigned)r;
        } else {
            cs->lv = (unsigned char)v;
            cs->lb = (unsigned)l;
        }
        __threadfence();
        if (atomicAdd(&cs->arrive, 1u) == 0) return;  // the other side carries on
        __threadfence();
        volatile CartSlot *vs = cs;
        const uint64_t L = as_right ? vs->lb : l, R = as_right ? r : vs->rb;
        const unsigned vl = as_right ? vs->lv : v, vr = as_right ? v : vs->rv;
        const uint64_t ll = p - L, lr = R - p + 1;
        const uint64_t sum = (uint64_t)vl * ll + (uint64_t)vr * lr;
        const int pre = (int)(unsigned)sum;
        v = (unsigned)(unsigned char)((uint64_t)(int64_t)pre / (ll + lr));
        l = L;
        r = R;
    }
    atomicOr(a.err, kErrWalk);
}

// Visit times from a list of keys in visiting order: every node exactly once.
__global__ void k_mg_vtime(MergeArgs a, const unsigned long long *__restrict__ order, uint64_t n_order) {
    const uint64_t q = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n_order) return;
    const unsigned i = lookup(a, order[q]);
    if (i == kNone || atomicCAS(&a.vt[i], ~0ull, (unsigned long long)q) != ~0ull) atomicOr(a.err, kErrOrder);
}

// ---- the gathered node lines (graph.cpp:615-645): id, per slot " " + arc + "#",
// 8 multiplicities, blanks up to sum(len+1)+61 bytes, '\n' as the last byte.
__device__ __forceinline__ uint64_t first_state(unsigned v) {
    return 2 * (uint64_t)(v >> 1) + ((v & 1u) ? 0 : 1);
}

// (eight lanes a line, one per arc slot: a line's arcs are chains of dependent
// loads, and few lines are left of a graph; unordered: nothing to read yet)
__global__ void k_mg_line_len(MergeArgs a, const unsigned long long *__restrict__ order, uint64_t n_lines,
                              uint64_t *__restrict__ out, const unsigned *__restrict__ unordered,
                              unsigned *__restrict__ pos_of) {
    if (unordered && *unordered) return;
    const uint64_t q = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const int s = threadIdx.x & 7;
    unsigned long long l = 0;
    if (q < n_lines) {
        const uint64_t j = order[q];
        if (mbyte(a.mult[j], s)) {
            const unsigned v = a.nb[j * 8 + s];
            l = 1 + (is_m(a, v >> 1) ? a.lt[first_state(v)].x : 0);
        }
    }
#pragma unroll
    for (int d = 4; d; d >>= 1) l += __shfl_xor_sync(0xffffffffu, l, d);
    if (q < n_lines && s == 0) {
        out[q] = 69 + l;
        pos_of[order[q]] = (unsigned)q;  // the line's position, for the arcs back
    }
}

// Eight lanes a line: lane s writes arc s's place, its multiplicity and an
// eighth of the blanks.
__global__ void __launch_bounds__(256) k_mg_line_write(MergeArgs a, const unsigned long long *__restrict__ order, uint64_t n_lines,
                                const uint64_t *__restrict__ off, char *__restrict__ text,
                                const unsigned *__restrict__ pos_of, MergedGraph mg) {
    const uint64_t q = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
    const int s = threadIdx.x & 7;
    const bool in = q < n_lines;
    const uint64_t j = in ? order[q] : 0, key = in ? a.keys[j] : 0;
    unsigned mm = in ? mbyte(a.mult[j], s) : 0;
    unsigned long long l = 0;  // the arc's length
    unsigned back = kNone, id = 0;
    bool chain = false, first = false;
    if (mm) {
        const unsigned v = a.nb[j * 8 + s];
        l = 1;
        if (is_m(a, v >> 1)) {
            const uint64_t st = first_state(v);
            const uint64_t mine = j * 8 + s, other = a.lt[st].y;
            chain = true;
            first = arc_less(a, mine, other);  // this end starts the chain
            id = a.chain_of[first ? mine : other];
            mm = a.ent[a.ch_eoff[id]];
            l += a.lt[st].x;
            back = pos_of[other >> 3] * 8u + (unsigned)(other & 7);
        } else {  // one base to the next node left: its arc back, as walk_next finds it
            const uint64_t o = s < 4 ? key : rc_dev(key, a.k);
            const unsigned base = (unsigned)(o >> (2 * (a.k - 1))) & 3u;
            back = pos_of[v >> 1] * 8u + ((v & 1u) ? 4u : 0u) + 3u - base;
        }
    }
    const unsigned dig = 1 + ndig(mm);  // " m"
    unsigned long long al = l + 2;      // " arc#"
    unsigned dl = dig;
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) {  // the line's arcs and multiplicities up to and with this lane's
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
    const unsigned head = ndig(key);
    char *p = start + head + (al - l - 2);  // this lane's " arc#"
    *p = ' ';
    p[1 + l] = '#';
    const unsigned long long dest = (unsigned long long)(p + 1 - text);
    if (l) p[1] = "ACGT"[s & 3];
    if (chain) {
        if (first) a.ch_dfwd[id] = dest;
        else a.ch_drev[id] = dest;
    }
    char *d = start + head + arcs + (dl - dig);  // this lane's " m"
    *d = ' ';
    put_u64(d + 1, mm);
    const uint64_t vlen = off[q + 1] - off[q];
    for (uint64_t i = head + arcs + digits + s; i < vlen - 1; i += 8) start[i] = ' ';
    mg.src[8 * q + s] = l ? dest : 0;
    mg.len[8 * q + s] = (unsigned)l;
    mg.mult[8 * q + s] = (unsigned char)mm;
    mg.back[8 * q + s] = back;
    if (s == 0) {
        put_u64(start, key);
        start[vlen - 1] = '\n';
        mg.key[q] = key;
        mg.del[q] = 0;
    }
}

__global__ void k_mg_chars(MergeArgs a, char *__restrict__ text) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n || !is_m(a, i)) return;
    const ChainPos c = chain_pos(a, i);
    const unsigned id = a.chain_of[c.start];
    const unsigned char f = a.fl[i];
    const int out_fwd = c.fwd ? rslot(f) : lslot(f);  // leaving towards the chain's far end
    const int out_rev = c.fwd ? lslot(f) : rslot(f);
    text[a.ch_dfwd[id] + c.pos] = "ACGT"[out_fwd & 3];
    text[a.ch_drev[id] + (c.m + 1 - c.pos)] = "ACGT"[out_rev & 3];
}

inline unsigned blocks(uint64_t n) { return (unsigned)std::max<uint64_t>((n + 255) / 256, 1); }

int ceil_log2(uint64_t v) {
    int r = 0;
    while ((1ull << r) < v) ++r;
    return r;
}

}  // namespace

// Grows the merged graph's buffers (the text, the spare text for rewrites,
// the per-line arrays) to hold `bytes` of text and `lines` lines.
swg_status merged_reserve(MergedGraph *m, uint64_t bytes, uint64_t lines) {
    if (bytes > m->text_cap) {
        cudaFree(m->text);
        cudaFree(m->text2);
        m->text = m->text2 = nullptr;
        m->text_cap = m->text2_cap = 0;
        EMIT_CUDA(cudaMalloc((void **)&m->text, bytes), "merged text");
        m->text_cap = bytes;
    }
    if (lines > m->line_cap || !m->key) {
        const uint64_t c = std::max<uint64_t>(lines, 1);
        cudaFree(m->key);
        cudaFree(m->len);
        cudaFree(m->mult);
        cudaFree(m->src);
        cudaFree(m->src2);
        cudaFree(m->back);
        cudaFree(m->del);
        m->key = nullptr;
        m->len = nullptr;
        m->mult = nullptr;
        m->src = m->src2 = nullptr;
        m->back = nullptr;
        m->del = nullptr;
        m->line_cap = 0;
        EMIT_CUDA(cudaMalloc((void **)&m->key, c * 8), "merged lines");
        EMIT_CUDA(cudaMalloc((void **)&m->len, c * 32), "merged lines");
        EMIT_CUDA(cudaMalloc((void **)&m->mult, c * 8), "merged lines");
        EMIT_CUDA(cudaMalloc((void **)&m->src, c * 64), "merged lines");
        EMIT_CUDA(cudaMalloc((void **)&m->src2, c * 64), "merged lines");
        EMIT_CUDA(cudaMalloc((void **)&m->back, c * 32), "merged lines");
        EMIT_CUDA(cudaMalloc((void **)&m->del, c), "merged lines");
        m->line_cap = c;
    }
    return SWG_OK;
}

void merged_free(MergedGraph *m) {
    cudaFree(m->text);
    cudaFree(m->text2);
    cudaFree(m->key);
    cudaFree(m->len);
    cudaFree(m->mult);
    cudaFree(m->src);
    cudaFree(m->src2);
    cudaFree(m->back);
    cudaFree(m->del);
    if (m->pool) cudaMemPoolDestroy(m->pool);
    *m = MergedGraph();
}

swg_status merge_graph(const unsigned long long *d_keys, const unsigned long long *d_mult, uint64_t n, int k,
                       cudaStream_t s, MergedGraph *mg, MergeResult *res, const unsigned long long *h_order,
                       uint64_t n_order) {
    *res = MergeResult();
    if (n >= (1ull << 29)) {
        set_error("merge: more than 2^29 k-molecules");
        return SWG_ERR_BAD_INPUT;
    }
    if (k % 2 == 0) {  // the reference's k is odd (sequence.cpp:44): no k-mer is its own reverse complement
        set_error("merge: k must be odd (an even k-mer can be its own reverse complement)");
        return SWG_ERR_BAD_INPUT;
    }
    Scratch scr(s, mg->pool);
    MergeArgs a;
    std::memset(&a, 0, sizeof(a));
    a.k = k;
    a.n = n;
    unsigned long long *ctr = nullptr;
    uint64_t hcap = 1024;
    while (hcap < 2 * n) hcap *= 2;
    a.hmask = hcap - 1;
    if (!scr.get(&a.ht, hcap) || !scr.get(&a.nb, 8 * n) || !scr.get(&a.fl, n) ||
        !scr.get(&a.oo, 2 * n) || !scr.get(&a.rpos, 2 * n) || !scr.get(&a.heads, 2 * n) ||
        !scr.get(&a.lt, 2 * n) || !scr.get(&a.clist, 2 * n) ||
        !scr.get(&a.chain_of, 8 * n) || !scr.get(&ctr, 8 + 2 * kClasses))
        return cuda_err(cudaErrorMemoryAllocation, "merge workspace");
    a.ctr = ctr;
    a.err = reinterpret_cast<unsigned *>(ctr + 7);
    a.cls_count = ctr + 8;
    a.cls_cursor = ctr + 8 + kClasses;
    a.keys = d_keys;
    a.mult = d_mult;
    EMIT_CUDA(cudaMemsetAsync(ctr, 0, (8 + 2 * kClasses) * sizeof(unsigned long long), s), "merge clear");
    EMIT_CUDA(cudaMemsetAsync(a.ht, 0xff, hcap * sizeof(unsigned), s), "merge clear");
    int launches = 0;
    k_mg_index<<<blocks(n), 256, 0, s>>>(a);
    if (h_order) {  // visit times from the caller's order
        if (n_order != n) {
            set_error("merge: the visiting order must list every k-molecule once");
            return SWG_ERR_BAD_INPUT;
        }
        unsigned long long *d_order = nullptr;
        if (!scr.get(&a.vt, n) || !scr.get(&d_order, n))
            return cuda_err(cudaErrorMemoryAllocation, "visiting order");
        EMIT_CUDA(cudaMemsetAsync(a.vt, 0xff, std::max<uint64_t>(n, 1) * sizeof(unsigned long long), s), "merge clear");
        if (n)
            EMIT_CUDA(cudaMemcpyAsync(d_order, h_order, n * sizeof(unsigned long long), cudaMemcpyHostToDevice, s),
                      "visiting order");
        k_mg_vtime<<<blocks(n), 256, 0, s>>>(a, d_order, n);
        unsigned herr = 0;
        EMIT_CUDA(cudaMemcpyAsync(&herr, a.err, sizeof(unsigned), cudaMemcpyDeviceToHost, s), "merge status");
        EMIT_CUDA(cudaStreamSynchronize(s), "visiting order");
        if (herr & kErrOrder) {
            set_error("merge: the visiting order names a key twice or a key the graph does not hold");
            return SWG_ERR_BAD_INPUT;
        }
        ++launches;
    }
    k_mg_classify<<<blocks(n), 256, 0, s>>>(a);
    // rulers: at most one per state; counts stay on the device
    if (!scr.get(&a.rp0, 2 * n) || !scr.get(&a.ro, 2 * n) || !scr.get(&a.pp0, 2 * n) || !scr.get(&a.pp1, 2 * n) ||
        !scr.get(&a.moved, 64))
        return cuda_err(cudaErrorMemoryAllocation, "ruler list");
    EMIT_CUDA(cudaMemsetAsync(a.moved, 0, 64 * sizeof(unsigned), s), "merge clear");
    k_mg_states<<<(unsigned)std::max<uint64_t>((n + kTile - 1) / kTile, 1), kTile, 0, s>>>(a);
    launches += 3;
    int sms = 0, dev = 0;
    EMIT_CUDA(cudaGetDevice(&dev), "device");
    EMIT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "device attribute");
    {
        int pairs = (ceil_log2(std::max<uint64_t>(2 * n, 1)) + 2) / 2;
        void *args[] = {&a, &pairs};
        const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)std::max(1, sms), n / 8192 + 1);
        EMIT_CUDA(cudaLaunchCooperativeKernel((const void *)k_mg_rank, dim3(grid), dim3(1024), args, 0, s), "ruler list");
    }
    k_mg_finish<<<blocks(n), 256, 0, s>>>(a);
    launches += 2;
    unsigned long long h[8 + kClasses];
    EMIT_CUDA(cudaMemcpyAsync(h, ctr, sizeof(h), cudaMemcpyDeviceToHost, s), "merge counts");
    EMIT_CUDA(cudaStreamSynchronize(s), "merge counts");
    unsigned herr = (unsigned)h[7];
    if (herr & (kErrIndex | kErrNeighbour)) {
        set_error("merge: node index or neighbour lookup failed (arc without its neighbour k-molecule)");
        return SWG_ERR_BAD_INPUT;
    }
    if (herr) {
        set_error("merge: a walk did not end (internal error)");
        return SWG_ERR_TIMEOUT;
    }
    const uint64_t n_cyc_states = h[1];
    if (n_cyc_states) {
        if (!scr.get(&a.cx0, 2 * n) || !scr.get(&a.cx1, 2 * n) || !scr.get(&a.cy0, 2 * n) ||
            !scr.get(&a.cy1, 2 * n))
            return cuda_err(cudaErrorMemoryAllocation, "cycle workspace");
        const uint64_t c = n_cyc_states;
        const int rounds = ceil_log2(c) + 1;
        unsigned long long *bx[2] = {a.cx0, a.cx1}, *by[2] = {a.cy0, a.cy1};
        k_mg_cyc_init<<<blocks(c), 256, 0, s>>>(a, c);
        for (int r = 0; r < rounds; ++r)
            k_mg_cyc_max<<<blocks(c), 256, 0, s>>>(a, c, bx[r & 1], by[r & 1], bx[(r + 1) & 1], by[(r + 1) & 1]);
        k_mg_cyc_cut<<<blocks(c), 256, 0, s>>>(a, c, bx[rounds & 1]);
        k_mg_cyc_succ<<<blocks(c), 256, 0, s>>>(a, c);
        for (int r = 0; r < rounds; ++r)
            k_mg_cyc_rank<<<blocks(c), 256, 0, s>>>(a, c, bx[r & 1], by[r & 1], bx[(r + 1) & 1], by[(r + 1) & 1]);
        k_mg_cyc_done<<<blocks(c), 256, 0, s>>>(a, c, bx[rounds & 1], by[rounds & 1]);
        EMIT_CUDA(cudaMemsetAsync(a.cls_count, 0, kClasses * sizeof(unsigned long long), s), "cycle chains");
        EMIT_CUDA(cudaMemsetAsync(&a.ctr[2], 0, sizeof(unsigned long long), s), "cycle chains");
        k_mg_chain_count<<<blocks(n), 256, 0, s>>>(a);
        launches += 5 + 2 * rounds;
        EMIT_CUDA(cudaMemcpyAsync(h, ctr, sizeof(h), cudaMemcpyDeviceToHost, s), "cycle chains");
        EMIT_CUDA(cudaStreamSynchronize(s), "cycle chains");
        if (h[7]) {
            set_error("merge: a walk did not end (internal error)");
            return SWG_ERR_TIMEOUT;
        }
    }
    const unsigned long long *cls = h + 8;
    // segments of 2^c entries, largest class first: every offset is aligned
    unsigned long long cursor[kClasses];
    uint64_t total = 0, n_chains = 0;
    int top = 0;
    for (int c = kClasses - 1; c >= 0; --c) {
        cursor[c] = total;
        total += cls[c] << c;
        n_chains += cls[c];
        if (cls[c] && !top) top = c;
    }
    const uint64_t n_lines = n - h[4] + h[3];  // nodes left
    EMIT_CUDA(cudaMemcpyAsync(a.cls_cursor, cursor, sizeof(cursor), cudaMemcpyHostToDevice, s), "chain layout");
    if (!scr.get(&a.ch_eoff, n_chains) || !scr.get(&a.ch_m, n_chains) || !scr.get(&a.ch_dfwd, n_chains) ||
        !scr.get(&a.ch_drev, n_chains) || !scr.get(&a.ent, total) || !scr.get(&a.ent_chain, total) ||
        !scr.get(&a.skey, n_lines) || !scr.get(&a.sidx, n_lines))
        return cuda_err(cudaErrorMemoryAllocation, "chain workspace");
    EMIT_CUDA(cudaMemsetAsync(a.ent_chain, 0xff, std::max<uint64_t>(total, 1) * sizeof(unsigned), s), "chain clear");
    if (a.vt && !scr.get(&a.cart, total)) return cuda_err(cudaErrorMemoryAllocation, "merge tree");
    k_mg_chain_alloc<<<blocks(n_chains), 256, 0, s>>>(a, n_chains);
    k_mg_entries<<<blocks(n), 256, 0, s>>>(a);
    launches += 2;
    if (a.vt) {
        if (total) k_mg_cart<<<blocks(total), 256, 0, s>>>(a, total);
        ++launches;
    } else {
        for (int t = 0; t < top; t += kLevels) {
            const uint64_t per = 1ull << (t + kLevels);
            k_mg_levels<<<(unsigned)((total + per - 1) / per), 512, 0, s>>>(a, total, t, top);
            ++launches;
        }
    }
    // the nodes left, in key order
    unsigned long long *skey2 = nullptr, *sidx2 = nullptr;
    uint64_t *lens = nullptr, *loff = nullptr;
    unsigned *pos_of = nullptr;
    if (!scr.get(&lens, n_lines) || !scr.get(&loff, n_lines + 1) || !scr.get(&pos_of, n))
        return cuda_err(cudaErrorMemoryAllocation, "line workspace");
    uint64_t bytes = 0;
    // by splitters (three launches, 37 us for 6,000 lines; the library's passes
    // took eight and 61), or by the library's passes if there are more lines
    // than those take, one of their buckets runs full or there is no room
    for (bool library = n_lines > sort_device_most();; library = true) {
        unsigned *over = nullptr;
        unsigned unordered = 0;
        unsigned char *ws = nullptr;
        if (n_lines && !library && scr.get(&ws, sort_scratch_bytes(n_lines))) {
            sort_records_device(a.skey, a.sidx, n_lines, s, ws, &skey2, &sidx2, &over);
        } else if (n_lines) {
            if (!scr.get(&skey2, n_lines) || !scr.get(&sidx2, n_lines))
                return cuda_err(cudaErrorMemoryAllocation, "line workspace");
            size_t tb = 0;
            EMIT_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, a.skey, skey2, a.sidx, sidx2, (int64_t)n_lines, 0,
                                                      2 * k, s),
                      "sort size");
            unsigned char *tmp = nullptr;
            if (!scr.get(&tmp, tb)) return cuda_err(cudaErrorMemoryAllocation, "sort scratch");
            EMIT_CUDA(cub::DeviceRadixSort::SortPairs(tmp, tb, a.skey, skey2, a.sidx, sidx2, (int64_t)n_lines, 0,
                                                      2 * k, s),
                      "sort");
        }
        if (over) EMIT_CUDA(cudaMemcpyAsync(&unordered, over, sizeof(unsigned), cudaMemcpyDeviceToHost, s), "sort status");
        if (n_lines) {
            k_mg_line_len<<<blocks(8 * n_lines), 256, 0, s>>>(a, sidx2, n_lines, lens, over, pos_of);
            ++launches;
        }
        swg_status st = scan_lengths(lens, loff, n_lines, scr, s);
        if (st) return st;
        EMIT_CUDA(cudaMemcpyAsync(&bytes, loff + n_lines, 8, cudaMemcpyDeviceToHost, s), "text size");
        EMIT_CUDA(cudaStreamSynchronize(s), "text size");
        if (!unordered) break;
    }
    swg_status gst = merged_reserve(mg, bytes + 1, n_lines);
    if (gst) return gst;
    mg->k = k;
    mg->lines = n_lines;
    if (n_lines) {
        k_mg_line_write<<<blocks(8 * n_lines), 256, 0, s>>>(a, sidx2, n_lines, loff, mg->text, pos_of, *mg);
    }
    k_mg_chars<<<blocks(n), 256, 0, s>>>(a, mg->text);
    launches += 2;
    EMIT_CUDA(cudaMemsetAsync(mg->text + bytes, '\n', 1, s), "merged text");
    EMIT_CUDA(cudaGetLastError(), "merge kernels");
    EMIT_CUDA(cudaMemcpyAsync(&herr, a.err, sizeof(unsigned), cudaMemcpyDeviceToHost, s), "merge status");
    EMIT_CUDA(cudaStreamSynchronize(s), "merge");
    if (herr) {
        set_error("merge: a merge tree did not end (internal error)");
        return SWG_ERR_TIMEOUT;
    }
    res->text_bytes = bytes + 1;
    mg->text_bytes = bytes + 1;
    mg->nodes = n_lines;
    res->nodes = n_lines;
    res->chains = n_chains;
    res->cycles = h[3];
    res->rulers = h[0];
    res->launches = launches + 3;  // + the scan
    return SWG_OK;
}

}  // namespace swg
