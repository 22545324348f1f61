// The per-root shortest-path tree kernel shared by the tree handle (mcbgpu_trees.cu)
// and the device candidate generation (mcbgpu_gen.cu).
//
// Shortest-path trees of many roots of one graph (the host's per-root tree searches,
// include/Dijkstra.h:78-124, as one persistent launch): for each root, the distances
// to every vertex and every vertex's parent slot, chosen by the rule that makes any
// exact search agree with the reference's heap search, plus a flag for the roots
// where that rule cannot decide.
//
// Graph: the reduced multigraph's CSR (row offsets, columns, weights, reverse slots),
// every weight at least 1 and every distance below 2^31 (checked at creation).
//
// One CTA per root, persistent over a root counter:
//   1. distances, label-correcting by buckets: each round takes lo = (a lower
//      bound of) the smallest distance among dirty vertices and relaxes (atomicMin)
//      the arcs of every dirty vertex nearer than lo + delta, marking improved heads
//      dirty.  The dirty vertex at lo is final once relaxed (weights >= 1).  The loop
//      stops after 2 (n + 1) rounds, far more than any tree has taken, and flags the root
//      if it has not converged (a vertex that finds the round's list full waits, so that
//      is a check and not a bound).  A round first lists the vertices to relax, then gives
//      each kTreeLanes lanes, one arc at a time each: one thread per dirty word with its
//      vertices and arcs one after the other left a few threads with all of a frontier
//      of neighbours (planar-chain graph of 65k points: 14.8 us per root, 5.2 with lists; random
//      graph of 20k vertices 3.2, 1.0 with them; 2 or 8 lanes are within 8%).  Distances and dirty bits live in shared
//      memory up to kTreeSharedMaxN vertices, in a per-CTA global slice beyond.  delta (the
//      bucket width) trades rounds (each a pass over the dirty bits and a barrier)
//      against relaxations repeated inside a bucket; the callers time a few widths
//      and CTA shapes on their first roots and keep the fastest.
//   2. parents: for each vertex c, among its neighbours x on a shortest path
//      (d[x] + w = d[c]) the nearest one, entered through its first slot to c (the
//      smallest slot index of x's row among those arcs); the reference keeps exactly
//      that parent (only a strictly shorter path replaces one, and parents at
//      different distances settle in distance order) unless two different
//      neighbours tie at that nearest distance, which sets the root's flag so that
//      the host searches that root itself.  The same pass checks that the distances
//      are exact: every vertex but the root has a parent with d[x] + w = d[c] (so
//      d[c] is a path length) and no slot offers a shorter one (so it is the
//      shortest); a root that fails is flagged too.  So every tree handed out with
//      its flag clear is the reference's, whatever the rounds before did.
// CTA barriers are cta_sync / cta_sync_and (the non-aligned barrier): the loops
// before them diverge within warps.
#pragma once

#include <algorithm>
#include <climits>
#include <type_traits>
#include <vector>

#include "mcbgpu_internal.cuh"

namespace mcbgpu {
namespace sssp {
// internal linkage: every file that includes this header gets its own copy of the
// kernel, registered with its own module
namespace {

constexpr int kTreeThreads = 1024;      // the shared-memory form's CTA
constexpr int kTreeSharedMaxN = 53248;  // 208 KB of distances + 6.5 KB of dirty bits + 8 KB of list (of 227 KB)
constexpr int kTreeLanes = 4;  // lanes that share a listed vertex's arcs
constexpr int kTreeSharedList = 4096;   // vertices listed per round: shared form (16 bits each)
constexpr int kTreeGlobalList = 1024;   // global form: at least (tree_list_cap)
constexpr int kTreeNearList = 1024;     // and the form with two bitmaps
constexpr int kTreeMaxCtasPerSm = 16;   // the global form's per-CTA slices are sized for this many

// A vertex's first kArcSlots arcs at a fixed place, (column, weight) together: relaxing
// is a chain of L2 reads (the vertex's distance and arcs, then its neighbours'), one
// shorter than with the row's offsets read first (planar-chain graph of 65k points: 4.8
// us per root with those, 3.8 with the table).  Unused entries have column
// kNoArc; the last entry's top bit says that the vertex has more arcs (in cols / w).
constexpr int kArcSlots = 8;
constexpr uint32_t kNoArc = 0x7fffffffu, kMoreArcs = 0x80000000u;

inline std::vector<uint2> arc_table(int32_t n, const uint32_t *ro, const uint32_t *cols, const int32_t *w) {
    std::vector<uint2> t((size_t)n * kArcSlots, make_uint2(kNoArc, 0u));
    for (int32_t v = 0; v < n; v++) {
        for (uint32_t o = ro[v]; o < ro[v + 1] && o < ro[v] + kArcSlots; o++)
            t[(size_t)v * kArcSlots + (o - ro[v])] = make_uint2(cols[o], (uint32_t)w[o]);
        if (ro[v + 1] - ro[v] > (uint32_t)kArcSlots) t[(size_t)v * kArcSlots + kArcSlots - 1].x |= kMoreArcs;
    }
    return t;
}

struct TreeArgs {
    const uint32_t *ro;
    const uint32_t *cols;
    const int32_t *w;
    const uint32_t *rev;
    const uint2 *arcs;   // n x kArcSlots: the first arcs of every vertex (arc_table)
    int32_t n;
    int32_t delta;
    int32_t list_cap;    // vertices listed per round (global form only)
    const uint32_t *roots;
    int32_t count;
    int32_t *dist_out;   // count x n
    int32_t *pedge_out;  // count x n
    uint8_t *tied_out;   // count
    int32_t *gdist;      // gridDim.x x n (global form only)
    uint32_t *gdirty;    // gridDim.x x words (global form only)
    uint32_t *gsumm;     // gridDim.x x summary words (global form only)
    int32_t *next_root;
    unsigned *status;
};

// Relaxes the arcs of v (distance dv) that fall to lane `sub` of kTreeLanes: lower(x, nd)
// is called for each, two of the fixed places at once.
template <typename Lower>
__device__ __forceinline__ void relax_arcs(const TreeArgs &a, uint32_t v, int dv, int sub, const Lower &lower) {
    static_assert(kArcSlots == 2 * kTreeLanes, "two entries per lane");
    const uint2 e0 = __ldg(a.arcs + (size_t)v * kArcSlots + sub), e1 = __ldg(a.arcs + (size_t)v * kArcSlots + kTreeLanes + sub);
    const uint32_t x1 = e1.x & ~kMoreArcs;
    lower(e0.x, dv + (int)e0.y, x1, dv + (int)e1.y);
    const unsigned group = ((1u << kTreeLanes) - 1) << (threadIdx.x & 31 & ~(kTreeLanes - 1));
    if (__shfl_sync(group, e1.x, kTreeLanes - 1, kTreeLanes) & kMoreArcs) {
        const uint32_t o1 = __ldg(a.ro + v + 1);
        for (uint32_t o = __ldg(a.ro + v) + kArcSlots + sub; o < o1; o += kTreeLanes)
            lower(__ldg(a.cols + o), dv + __ldg(a.w + o), kNoArc, 0);
    }
}

// 2. parents by the rule into the root's rows, with its distances; returns whether this
// thread saw a tie or an inexact distance (or the distances have not converged).
template <typename Get>
__device__ __forceinline__ int tree_parents(const TreeArgs &a, int r, uint32_t src, const Get &get, bool converged) {
    const int n = a.n, tid = threadIdx.x, nt = blockDim.x;
    int tie = converged ? 0 : 1;
    for (int c = tid; c < n; c += nt) {
        const int dc = get((uint32_t)c);
        int32_t slot = -1;
        if ((uint32_t)c != src && dc != INT_MAX) {
            int bestd = INT_MAX, rival = 0;  // rival: another neighbour as near as the best
            int shorter = 0;                 // some slot offers c a shorter path
            uint32_t bestx = 0xffffffffu, bests = 0xffffffffu;
            const uint32_t o1 = __ldg(a.ro + c + 1);
            for (uint32_t ob = __ldg(a.ro + c); ob < o1; ob += 4) {  // four arcs in flight
                uint32_t xs[4];
                int dxs[4], ws[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    xs[q] = ob + q < o1 ? __ldg(a.cols + ob + q) : 0u;
                    ws[q] = ob + q < o1 ? __ldg(a.w + ob + q) : 0;
                }
#pragma unroll
                for (int q = 0; q < 4; q++) dxs[q] = ob + q < o1 ? get(xs[q]) : INT_MAX;
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int dx = dxs[q];
                    if (dx == INT_MAX) continue;
                    // the certificate of exact distances: no slot gives c a shorter
                    // path (with every vertex's distance that of a real path through
                    // its parent, below, the distances are the shortest); a root
                    // that fails it is left to the host
                    const long long via = (long long)dx + ws[q];
                    if (via < (long long)dc) shorter = 1;
                    if (via != (long long)dc) continue;
                    if (dx < bestd) {
                        bestd = dx;
                        bestx = xs[q];
                        bests = __ldg(a.rev + ob + q);
                        rival = 0;
                    } else if (dx == bestd) {
                        if (xs[q] == bestx)
                            bests = min(bests, __ldg(a.rev + ob + q));
                        else
                            rival = 1;
                    }
                }
            }
            slot = bests == 0xffffffffu ? -1 : (int32_t)bests;
            if (rival || shorter || slot < 0) tie = 1;  // (no shortest-path neighbour cannot happen; left to the host)
        } else if ((uint32_t)c != src) {
            tie = 1;  // unreachable vertex (the graph is not connected): left to the host
        }
        a.dist_out[(size_t)r * n + c] = dc;
        a.pedge_out[(size_t)r * n + c] = slot;
    }
    return tie;
}

// Threads per CTA: the shared-memory form runs one 1024-thread CTA per SM (its
// distances fill the shared memory); the other forms run kThreads-thread CTAs, several
// per SM, so that the bucket rounds of different roots overlap: their distances are in
// the CTA's global slice (trees_near_kernel by tree_form()'s rule, else the dirty bits too,
// with a summary).  They wait on L2 half of their time, so a full SM of threads
// (32 registers, a few spills) is worth more than registers.
enum TreeForm { kTreeShared, kTreeNear, kTreeGlobal };
template <int kForm, int kThreads>
__global__ void __launch_bounds__(kThreads, kForm == kTreeShared ? 1 : 2048 / kThreads) trees_kernel(TreeArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_next[3];
    __shared__ int s_root;
    __shared__ int s_cnt[2], s_nv[2];
    const int n = a.n;
    const int words = (n + 31) >> 5;
    const int swords = (words + 31) >> 5;  // summary: one bit per dirty word
    int32_t *dist;
    uint32_t *dirty, *summ;
    constexpr bool kShared = kForm == kTreeShared, kSummary = kForm == kTreeGlobal;
    using VertT = typename std::conditional<kShared, uint16_t, uint32_t>::type;
    const int list_cap = kShared ? kTreeSharedList : a.list_cap;
    VertT *s_verts;  // the vertices of a round
    if (kShared) {
        dist = reinterpret_cast<int32_t *>(smem);
        dirty = reinterpret_cast<uint32_t *>(smem + (((size_t)n * 4 + 15) & ~(size_t)15));
        summ = nullptr;
        s_verts = reinterpret_cast<VertT *>(dirty + words);
    } else {
        dist = a.gdist + (size_t)blockIdx.x * n;
        dirty = a.gdirty + (size_t)blockIdx.x * words;
        summ = a.gsumm + (size_t)blockIdx.x * swords;
        s_verts = reinterpret_cast<VertT *>(smem);
    }
    // global form: the dirty words of a round (words < 65536 entries, 16-bit)
    uint16_t *s_list = reinterpret_cast<uint16_t *>(smem + 4 * (size_t)list_cap);
    volatile int32_t *vdist = dist;
    // a distance as the CTA's atomics left it; global ones from L2, loads free to overlap
    auto get = [&](uint32_t v) -> int { return kShared ? vdist[v] : __ldcg(dist + v); };
    volatile uint32_t *vdirty = dirty;
    volatile uint32_t *vsumm = summ;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
    for (;;) {
        if (tid == 0) s_root = atomicAdd(a.next_root, 1);
        cta_sync();
        const int r = s_root;
        cta_sync();  // every thread has read s_root before thread 0 writes it again
        if (r >= a.count) return;
        const uint32_t src = a.roots[r];  // < n, checked by the host
        for (int v = tid; v < n; v += nt) dist[v] = INT_MAX;
        for (int k = tid; k < words; k += nt) dirty[k] = 0;
        if (kSummary)
            for (int k = tid; k < swords; k += nt) summ[k] = 0;
        if (tid == 0) {
            s_next[0] = INT_MAX;
            s_next[1] = INT_MAX;
            s_cnt[0] = 0;
            s_cnt[1] = 0;
            s_nv[0] = 0;
            s_nv[1] = 0;
        }
        cta_sync();
        if (tid == 0) {
            dist[src] = 0;
            dirty[src >> 5] = 1u << (src & 31);
            if (kSummary) summ[src >> 10] = 1u << ((src >> 5) & 31);
        }
        cta_sync();
        // 1. distances.  One pass per round over the dirty bits: vertices nearer than
        // hi = lo + delta are listed and relaxed, the others skipped; the next round's lo is the
        // smallest distance of a skipped vertex or of an improvement made in this
        // round (at most the smallest distance left dirty, so no vertex is missed;
        // an underestimate only costs a round).  The dirty vertex at the true lo is
        // final once relaxed (weights >= 1); it may wait while a list is full, so the
        // number of rounds is checked: past 2 (n + 1), far more than any tree took, the
        // root is flagged as not converged.  The round's
        // minimum goes to s_next[round % 3]: the slot read after this round's
        // barrier, reset two rounds later, when every thread has read it.
        bool converged = false;
        int lo = 0;
        for (int round = 0; round <= 2 * n + 1; round++) {
            if (lo == INT_MAX) {
                converged = true;
                break;
            }
            const int hi = lo > INT_MAX - a.delta ? INT_MAX : lo + a.delta;
            const int slot = round % 3;
            if (tid == 0) s_next[(round + 1) % 3] = INT_MAX;
            int mynext = INT_MAX;
            int *nv = &s_nv[round & 1];
            if (tid == 0) s_nv[(round + 1) & 1] = 0;  // read last in round - 1, before its barrier
            // One dirty word: its vertices nearer than hi leave it for the round's list, the
            // others stay (and their smallest distance counts for the next round), as do
            // those that find the list full.  Returns whether some vertex was left dirty.
            auto list_word = [&](int k) {
                if (*(volatile int *)nv >= list_cap) {  // no room in this round: not looked at
                    mynext = lo < mynext ? lo : mynext;
                    return true;
                }
                const uint32_t bits = vdirty[k];
                uint32_t take = 0;
                for (uint32_t m = bits; m;) {  // four distances in flight
                    int b[4], d[4];
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        b[q] = __ffs(m) - 1;
                        m &= m - 1;
                        d[q] = b[q] >= 0 ? get((uint32_t)((k << 5) + b[q])) : INT_MAX;
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        if (d[q] < hi)
                            take |= 1u << b[q];
                        else
                            mynext = d[q] < mynext ? d[q] : mynext;
                    }
                }
                if (take) {
                    int at = atomicAdd(nv, __popc(take));
                    uint32_t listed = 0;
                    for (uint32_t m = take; m; m &= m - 1, at++) {
                        const int b = __ffs(m) - 1;
                        if (at < list_cap) {
                            s_verts[at] = (VertT)((k << 5) + b);
                            listed |= 1u << b;
                        } else {
                            mynext = lo < mynext ? lo : mynext;
                        }
                    }
                    // the bits go before the barrier, the distances are read after it: a
                    // distance lowered since sets its bit again
                    if (listed) atomicAnd(&dirty[k], ~listed);
                    take = listed;
                }
                return (bits & ~take) != 0;
            };
            if (!kSummary) {
                for (int k = tid; k < words; k += nt) list_word(k);
            } else {
                // the summary words: a set bit marks a dirty word as possibly non-zero.
                // A writer sets the dirty bit, then the summary bit (fence between).
                // Phase 1 clears the summary bits and lists their words; the barrier
                // orders the clears before phase 2's reads of the words, so a bit set
                // before a clear is seen in its word and one set after it leaves the
                // summary bit set for the next round; a word left with skipped
                // vertices gets its summary bit back.
                int *cnt = &s_cnt[round & 1];
                if (tid == 0) s_cnt[(round + 1) & 1] = 0;  // read last in round - 1, before its barrier
                for (int q = tid; q < swords; q += nt) {
                    uint32_t sb = vsumm[q];
                    if (!sb) continue;
                    atomicAnd(&summ[q], ~sb);
                    while (sb) {
                        const int kb = __ffs(sb) - 1;
                        sb &= sb - 1;
                        s_list[atomicAdd(cnt, 1)] = (uint16_t)((q << 5) + kb);
                    }
                }
                cta_sync();
                const int m = *(volatile int *)cnt;
                for (int i = tid; i < m; i += nt) {
                    const int k = s_list[i];
                    if (list_word(k)) atomicOr(&summ[k >> 5], 1u << (k & 31));
                }
            }
            __threadfence_block();
            cta_sync();
            // the listed vertices' arcs, kTreeLanes at a time
            const int listed = min(*(volatile int *)nv, list_cap);
            auto improve = [&](uint32_t x, int nd) {
                const int old = atomicMin(&dist[x], nd);
                if (nd < old) {
                    __threadfence_block();  // the new distance before the dirty bit
                    atomicOr(&dirty[x >> 5], 1u << (x & 31));
                    if (kSummary) {
                        __threadfence_block();  // the dirty bit before the summary bit
                        atomicOr(&summ[x >> 10], 1u << ((x >> 5) & 31));
                    }
                    mynext = nd < mynext ? nd : mynext;
                }
            };
            for (int i = tid / kTreeLanes; i < listed; i += nt / kTreeLanes) {
                const uint32_t v = s_verts[i];
                relax_arcs(a, v, get(v), tid % kTreeLanes, [&](uint32_t x0, int n0, uint32_t x1, int n1) {
                    const int d0 = x0 != kNoArc ? get(x0) : INT_MIN, d1 = x1 != kNoArc ? get(x1) : INT_MIN;
                    if (n0 < d0) improve(x0, n0);
                    if (n1 < d1) improve(x1, n1);
                });
            }
            mynext = __reduce_min_sync(0xffffffffu, mynext);
            if (lane == 0 && mynext != INT_MAX) atomicMin(&s_next[slot], mynext);
            cta_sync();
            lo = s_next[slot];
        }
        int tie = tree_parents(a, r, src, get, converged);
        tie = cta_sync_and(tie == 0) ? 0 : 1;
        if (tid == 0) a.tied_out[r] = tie ? 1 : 0;
        if (!converged && tid == 0) atomicOr(a.status, ST_DIVERGED);
    }
}

// The form for distances in global memory with everything else in shared memory: two
// bitmaps instead of one.  `near` holds the vertices to relax now (nearer than hi), `far`
// the improved ones beyond hi.  A round relaxes all of near, and only when that is empty
// does hi move on and far get looked at: a bucket's several rounds no longer read the
// distances of every vertex that waits for a later one.  Planar-chain graph of 65k points:
// 650 rounds of 125 vertices per root, 4.8 us per root (5.2 with one bitmap; 3.8 with
// arc_table).  Bound by the chain of L2 reads of each relaxation at eight CTAs per SM
// (512 or 128 threads per CTA: 4.6 and 5.4).
//
// The line: eight CTAs' bitmaps (19.4 KB), lists (4 KB) and the system's 1 KB each must fit the
// SM's last split but one of shared memory and L1 (196 of 228 KB): up to 79,360 vertices.
// Past it a random graph takes 24 us per root against 14 with the dirty bits in global
// memory, a planar-chain graph 7.4 against 6.9.  Up to it planar-chain and grid graphs gain
// 15-25% (60k vertices 4.0 / 5.2, 79k 5.4 / 6.7) and RGGs nothing (5.6); random ones of mean
// degree 4.4 gain 3% to 63k and lose 10% beyond (66k 11.4 / 10.0); of degree 6.3 and 8.1 they
// lose 10-25% from the start (57k 12.9 / 11.7, 60k 19.8 / 16.9): more waits than a list
// holds.  So the degree decides too.
constexpr int kTreeNearMaxN = 79360;
constexpr int kTreeNearMaxDegree = 6;

template <int kThreads>
__global__ void __launch_bounds__(kThreads, 2048 / kThreads) trees_near_kernel(TreeArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_root, s_lo, s_nv[3];
    const int n = a.n, words = (n + 31) >> 5;
    uint32_t *s_verts = reinterpret_cast<uint32_t *>(smem);
    uint32_t *near = s_verts + kTreeNearList, *far = near + words;
    int32_t *dist = a.gdist + (size_t)blockIdx.x * n;
    const int tid = threadIdx.x, lane = tid & 31;
    auto get = [&](uint32_t v) -> int { return __ldcg(dist + v); };
    for (;;) {
        if (tid == 0) s_root = atomicAdd(a.next_root, 1);
        cta_sync();
        const int r = s_root;
        cta_sync();  // every thread has read s_root before thread 0 writes it again
        if (r >= a.count) return;
        const uint32_t src = a.roots[r];  // < n, checked by the host
        for (int v = tid; v < n; v += kThreads) dist[v] = (uint32_t)v == src ? 0 : INT_MAX;
        for (int k = tid; k < 2 * words; k += kThreads) near[k] = 0;
        cta_sync();
        if (tid == 0) {
            near[src >> 5] = 1u << (src & 31);
            s_nv[0] = 0;
        }
        cta_sync();
        bool converged = false;
        int hi = a.delta, beyond = INT_MAX;  // beyond: this thread's smallest distance put or left in far
        for (int it = 0; it <= 4 * n + 16; it++) {
            int *nv = &s_nv[it % 3];
            if (tid == 0) s_nv[(it + 1) % 3] = 0;  // read last two barriers ago
            // the near vertices leave the bitmap for the list (those that find it full stay)
            for (int k = tid; k < words; k += kThreads) {
                uint32_t bits = near[k];
                if (!bits) continue;
                int at = atomicAdd(nv, __popc(bits));
                while (bits && at < kTreeNearList) {
                    const int b = __ffs(bits) - 1;
                    bits &= bits - 1;
                    s_verts[at++] = (uint32_t)((k << 5) + b);
                }
                near[k] = bits;
            }
            cta_sync();
            const int listed = min(*(volatile int *)nv, kTreeNearList);
            if (listed > 0) {
                // their arcs, kTreeLanes at a time; bits were cleared before the barrier and
                // distances are read after it, so a distance lowered since sets its bit again
                auto improved = [&](uint32_t x, int nd) {
                    __threadfence_block();  // the new distance before the bit
                    atomicOr((nd < hi ? near : far) + (x >> 5), 1u << (x & 31));
                    if (nd >= hi) beyond = min(beyond, nd);
                };
                for (int i = tid / kTreeLanes; i < listed; i += kThreads / kTreeLanes) {
                    const uint32_t v = s_verts[i];
                    relax_arcs(a, v, get(v), tid % kTreeLanes, [&](uint32_t x0, int n0, uint32_t x1, int n1) {
                        const int d0 = x0 != kNoArc ? get(x0) : INT_MIN, d1 = x1 != kNoArc ? get(x1) : INT_MIN;
                        const bool t0 = n0 < d0, t1 = n1 < d1;
                        const int o0 = t0 ? atomicMin(&dist[x0], n0) : INT_MIN, o1 = t1 ? atomicMin(&dist[x1], n1) : INT_MIN;
                        if (n0 < o0) improved(x0, n0);
                        if (n1 < o1) improved(x1, n1);
                    });
                }
                cta_sync();
                continue;
            }
            // near is empty: the next bucket starts at far's smallest distance (or below it,
            // where that vertex has been improved into near since: an empty bucket)
            if (tid == 0) s_lo = INT_MAX;
            cta_sync();
            beyond = __reduce_min_sync(0xffffffffu, beyond);
            if (lane == 0 && beyond != INT_MAX) atomicMin(&s_lo, beyond);
            cta_sync();
            const int lo = s_lo;
            if (lo == INT_MAX) {
                converged = true;
                break;
            }
            hi = lo > INT_MAX - a.delta ? INT_MAX : lo + a.delta;
            beyond = INT_MAX;
            auto sort_out = [&](uint32_t v, int d) {  // out of far: into near, or back
                if (d < hi)
                    atomicOr(near + (v >> 5), 1u << (v & 31));
                else {
                    atomicOr(far + (v >> 5), 1u << (v & 31));
                    beyond = min(beyond, d);
                }
            };
            it++;
            nv = &s_nv[it % 3];
            if (tid == 0) s_nv[(it + 1) % 3] = 0;
            for (int k = tid; k < words; k += kThreads) {
                uint32_t bits = far[k];
                if (!bits) continue;
                far[k] = 0;
                int at = atomicAdd(nv, __popc(bits));
                for (; bits; bits &= bits - 1, at++) {
                    const uint32_t v = (uint32_t)((k << 5) + __ffs(bits) - 1);
                    if (at < kTreeNearList)
                        s_verts[at] = v;
                    else
                        sort_out(v, get(v));  // its word is this thread's
                }
            }
            cta_sync();
            const int nfar = min(*(volatile int *)nv, kTreeNearList);
            for (int i = tid; i < nfar; i += kThreads) {
                const uint32_t v = s_verts[i];
                sort_out(v, get(v));
            }
            cta_sync();
        }
        int tie = tree_parents(a, r, src, get, converged);
        tie = cta_sync_and(tie == 0) ? 0 : 1;
        if (tid == 0) a.tied_out[r] = tie ? 1 : 0;
        if (!converged && tid == 0) atomicOr(a.status, ST_DIVERGED);
    }
}

// The form for a graph of n vertices and `slots` arcs.
inline TreeForm tree_form(int n, long long slots) {
    if (n <= kTreeSharedMaxN) return kTreeShared;
    return n <= kTreeNearMaxN && slots <= (long long)kTreeNearMaxDegree * n ? kTreeNear : kTreeGlobal;
}

// Dynamic shared memory for n vertices: the shared form's distances, dirty bits and a
// round's vertices; the other forms' vertices and bitmaps or dirty words of a round.
inline size_t trees_smem_bytes(int n) {
    const size_t words = ((size_t)n + 31) / 32;
    return (((size_t)n * 4 + 15) & ~(size_t)15) + words * 4 + 2 * kTreeSharedList;
}
inline size_t trees_global_smem_bytes(TreeForm form, int n, int list_cap) {
    const size_t words = ((size_t)n + 31) / 32;
    return form == kTreeNear ? 4 * kTreeNearList + 8 * words : 4 * (size_t)list_cap + 2 * ((words + 7) & ~(size_t)7);
}
constexpr int kTreeGlobalMaxN = 65536 * 32;  // the global form's 16-bit word list: at most 128 KB

// A launch shape of trees_kernel: CTA size, CTAs per SM (global form) and the
// bucket width as a multiple of the mean edge weight, in quarters.
struct TreeShape {
    int threads, ctas_per_sm, delta_quarters;
};

// The bucket width of a shape on a graph whose mean slot weight is mean_w.
inline int32_t shape_delta(const TreeShape &sh, int32_t mean_w) {
    const long long d = ((long long)mean_w * sh.delta_quarters + 3) / 4;
    return (int32_t)(d < 1 ? 1 : d > (1ll << 30) ? (1ll << 30) : d);
}

// The kernel for a CTA size of the forms with distances in global memory.
typedef void (*TreeKernel)(TreeArgs);
inline TreeKernel tree_kernel(TreeForm form, int threads) {
    const bool d = form == kTreeNear;
    switch (threads) {
    case 128: return d ? trees_near_kernel<128> : trees_kernel<kTreeGlobal, 128>;
    case 256: return d ? trees_near_kernel<256> : trees_kernel<kTreeGlobal, 256>;
    case 512: return d ? trees_near_kernel<512> : trees_kernel<kTreeGlobal, 512>;
    default: return d ? trees_near_kernel<1024> : trees_kernel<kTreeGlobal, 1024>;
    }
}

// The global form's list entries per CTA, and its shape where none is timed.  A frontier of
// tens of thousands of vertices (random graphs) takes a round per list, so larger lists are
// faster, until eight CTAs' lists and dirty words leave the SM a smaller L1: from 180k
// vertices on they get half, and four CTAs of twice the threads, which keep theirs, are the
// first choice.  Microseconds per root: no list and one thread per dirty word (as it was) /
// 1,024 entries in eight CTAs and every waiting vertex read in every round / the rule: random
// graphs of 104k, 166k, 249k and 332k vertices 28 / 28 / 20, 51 / 64 / 41, 73 / 121 / 54, 107 /
// 208 / 85; of degree eight, 159k and 238k 73 / 84 / 55, 126 / 171 / 96; planar-chain graphs of
// 166k, 242k and 368k 39 / 14 / 14, 55 / 25 / 22, 97 / 34 / 34 (with eight CTAs' lists twice as
// long beyond 180k 276k vertices take 53 instead of 28).
constexpr int kTreeWideN = 180000;
inline int tree_list_cap(int n, const TreeShape &sh) {
    const int ctas = std::max(sh.ctas_per_sm, 1);
    return std::max(kTreeGlobalList, (n > kTreeWideN && ctas >= 8 ? 8 : 16) * kTreeGlobalList / ctas);
}
inline TreeShape first_shape(TreeForm form, int n) {
    if (form == kTreeGlobal && n > kTreeWideN) return TreeShape{512, 4, 8};
    return TreeShape{256, 8, 8};
}

// Launches the form's kernel in `shape` over grid CTAs (the shared form: 1024 threads,
// smem bytes of dynamic shared memory).
inline cudaError_t launch_trees(TreeForm form, const TreeShape &shape, int grid, size_t smem, cudaStream_t st,
                                TreeArgs a) {
    a.list_cap = tree_list_cap(a.n, shape);
    if (form == kTreeShared)
        trees_kernel<kTreeShared, kTreeThreads><<<grid, kTreeThreads, smem, st>>>(a);
    else
        tree_kernel(form, shape.threads)<<<grid, shape.threads <= 512 ? shape.threads : 1024,
                                           trees_global_smem_bytes(form, a.n, a.list_cap), st>>>(a);
    return cudaGetLastError();
}

inline cudaError_t set_trees_smem_limit() {
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(trees_kernel<kTreeShared, kTreeThreads>, attr, (int)trees_smem_bytes(kTreeSharedMaxN));
    for (int threads : {128, 256, 512, 1024})
        for (TreeForm form : {kTreeNear, kTreeGlobal})
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(tree_kernel(form, threads), attr,
                                         (int)trees_global_smem_bytes(form, form == kTreeNear ? kTreeNearMaxN : kTreeGlobalMaxN,
                                                                      2 * 8 * kTreeGlobalList));
    return e;
}

}  // namespace
}  // namespace sssp
}  // namespace mcbgpu

