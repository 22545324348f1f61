// Candidate generation on the device: the per-root shortest-path trees, the
// candidate test and the cycle coordinate lists of the host preparation
// (include/Dijkstra.h:78-254, include/work_per_thread.h:92-147, include/cycles.h:144-195),
// for a problem whose host preparation stopped after the spanning tree
// (mcbh_options.structure_only).  The host keeps the two steps whose result only
// the standard library's own routines reproduce: the heap-ordered search of the
// roots whose tree has a tie (mcbh_search_trees) and the per-root group maps + the
// sort on weight (mcbh_rank_candidates).
//
// Per chunk of roots (FVS indices t0 .. t0+count):
//   1. trees_kernel (mcbgpu_sssp.cuh): distances into the chunk's distance rows,
//      parent slots into the resident parent array (F x n' int32, kept for the
//      lists), a tie flag per root; the host replaces the tied roots' trees.
//   2. per vertex, its branch: the child of the root its tree path runs through, or
//      "blocked" if that path holds an FVS vertex with a smaller id than the root, by
//      pointer jumping up the parent chains (O(n' log height)); and per non-tree pair of
//      slots the reference's test (both ends unblocked, paths meeting only at the root)
//      as a bitmap, and a count per root: branch_test_kernel, one CTA per root with the
//      branches in shared memory (up to kBranchMaxN vertices), else codes_kernel and
//      cand_count_kernel over global memory; then cand_write_kernel: the accepted pairs
//      in pair order with their weights d(a) + d(b) + w, one warp per root, at offsets
//      from a scan of the counts.
// After the host has ranked all candidates:
//   4. walk_kernel (twice): per rank, the coordinates on its two root paths and of
//      its own edge; first the lengths, then (after a scan) the lists;
//      sort_lists_kernel sorts each list ascending (one warp per list, bitonic in
//      shared memory; one CTA per list above 1024 entries).
// Every index read from a caller's array is range-checked; a bad one sets a status
// bit (MCBGPU_E_DEVICE) instead of being followed, and every walk is bounded by n'.
#include <algorithm>
#include <climits>
#include <cstring>
#include <new>
#include <type_traits>
#include <vector>

#include "mcbgpu_sssp.cuh"

using namespace mcbgpu;
using namespace mcbgpu::sssp;

// (a named namespace: an anonymous one here would clash, in the generated launch
// stubs, with the one of mcbgpu_sssp.cuh)
namespace mcbgpu {
namespace gen {

constexpr int kCodeThreads = 1024;
constexpr int kJumpRounds = 40;  // pointer jumping halves every chain per round: heights below 2^39
constexpr int kCandThreads = 512;
constexpr int kWalkThreads = 256;
constexpr int kSortWarpMax = 1024;   // lists up to this length: one warp, 4 KB of shared memory
constexpr int kSortLongMax = 32768;  // longer lists: one CTA, up to 128 KB of shared memory
constexpr int kScanThreads = 1024;

struct GenGraph {
    const uint32_t *ro, *rows, *cols, *rev, *pair_slot, *roots;
    const int32_t *w, *ec, *fvs;
    const uint4 *slot_info;      // per slot: row, column, pair index, coordinate or -1
    const uint32_t *pair_ends;   // per pair: its lower slot's row and column, 16 bits each (n <= kBranchMaxN)
    int32_t n, F;
    int64_t slots, npairs;
};

// A vertex's pointer starts as its parent, or as itself below the root (its branch), or
// as "blocked" where it blocks; jumping to its pointer's pointer until that points to
// itself (or is blocked) leaves its branch.  Pointers are updated in place: a vertex
// reads its ancestor's whole, which is at least as far along as in the synchronous
// scheme, so each round at least halves every remaining chain.
constexpr int32_t kCodeRoot = -1, kCodeBlocked = -2;

// What a vertex starts with: its pointer, with kCodeRoot / kCodeBlocked; bad: its parent
// slot is none of its own (it is left blocked, so it joins no candidate).
__device__ __forceinline__ int32_t first_pointer(const GenGraph &g, uint32_t v, uint32_t src, int32_t o, uint32_t &pair,
                                                 bool &bad) {
    pair = 0xffffffffu;
    if (v == src) return kCodeRoot;
    if (o < 0 || (int64_t)o >= g.slots) {
        bad = true;
        return kCodeBlocked;
    }
    const uint4 si = __ldg(g.slot_info + o);
    if (si.y != v) {
        bad = true;
        return kCodeBlocked;
    }
    pair = si.z;
    if (g.fvs[v] >= 0 && v < src) return kCodeBlocked;
    return (int32_t)(si.x == src ? v : si.x);
}

// Branches and candidate test of a root in one CTA: 16-bit pointers and the tree's pairs
// (a bit each) in shared memory, so that a pair costs its packed ends, two lookups and a
// ballot, and nothing of a root goes through global memory but its parent slots and the
// bitmap.  Planar-chain graph of 65k points (59.6k vertices, 130k pairs): the two kernels
// over global memory took 3.0 us per root, this 0.7 us.
constexpr int kBranchMaxN = 65534;
constexpr size_t kBranchSmemMax = 220 * 1024;
constexpr uint16_t kRoot16 = 0xfffeu, kBlocked16 = 0xffffu;
inline size_t branch_smem_bytes(int n, int64_t npairs) {
    return (((size_t)n * 2 + 15) & ~(size_t)15) + 4 * (size_t)((npairs + 31) / 32);
}

__global__ void __launch_bounds__(kCodeThreads) branch_test_kernel(GenGraph g, const int32_t *__restrict__ pedge, int t0,
                                                                   int count, uint32_t *bits, int64_t words_per_root,
                                                                   int64_t *counts, unsigned *status) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_cnt[kCodeThreads / 32];
    const int n = g.n, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    volatile uint16_t *J = reinterpret_cast<volatile uint16_t *>(smem);
    uint32_t *tree = reinterpret_cast<uint32_t *>(smem + (((size_t)n * 2 + 15) & ~(size_t)15));
    const int words = (int)words_per_root;
    for (int r = blockIdx.x; r < count; r += gridDim.x) {
        const int t = t0 + r;
        const uint32_t src = g.roots[t];
        const int32_t *pe = pedge + (size_t)t * n;
        for (int i = tid; i < words; i += kCodeThreads) tree[i] = 0;
        cta_sync();
        bool bad = false;
        for (int v0 = tid; v0 < n; v0 += 4 * kCodeThreads) {
            int32_t o[4];
#pragma unroll
            for (int q = 0; q < 4; q++) o[q] = v0 + q * kCodeThreads < n ? __ldg(pe + v0 + q * kCodeThreads) : -1;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int v = v0 + q * kCodeThreads;
                if (v >= n) break;
                uint32_t pair;
                const int32_t p = first_pointer(g, (uint32_t)v, src, o[q], pair, bad);
                J[v] = p == kCodeRoot ? kRoot16 : p == kCodeBlocked ? kBlocked16 : (uint16_t)p;
                if (pair != 0xffffffffu) atomicOr(&tree[pair >> 5], 1u << (pair & 31u));
            }
        }
        if (!cta_sync_and(!bad) && tid == 0) atomicOr(status, ST_BAD_INPUT);
        bool done = false;
        for (int round = 0; round < kJumpRounds && !done; round++) {
            bool open = false;
            for (int v = tid; v < n; v += kCodeThreads) {
                const uint16_t p = J[v];
                if (p >= kRoot16 || p == v) continue;
                const uint16_t y = J[p];
                if (y == p) continue;  // a branch
                J[v] = y;
                open |= y < kRoot16;
            }
            done = cta_sync_and(!open);
        }
        if (!done && tid == 0) atomicOr(status, ST_BAD_INPUT);  // deeper than any tree of checked parents
        int cnt = 0;
        uint32_t *bw = bits + (size_t)r * words_per_root;
        for (int wi = warp; wi < words; wi += kCodeThreads / 32) {
            const int64_t k = (int64_t)wi * 32 + lane;
            bool acc = false;
            if (k < g.npairs && !((tree[wi] >> lane) & 1u)) {
                const uint32_t ab = __ldg(g.pair_ends + k);
                const uint32_t a = ab & 0xffffu, b = ab >> 16;
                const uint16_t ca = J[a], cb = J[b];
                acc = ca != kBlocked16 && cb != kBlocked16 && (a == src || b == src || ca != cb);
            }
            const uint32_t m = __ballot_sync(0xffffffffu, acc);
            if (lane == 0) bw[wi] = m;
            cnt += __popc(m);
        }
        if (lane == 0) s_cnt[warp] = cnt;
        cta_sync();
        if (tid == 0) {
            long long sum = 0;
            for (int i = 0; i < kCodeThreads / 32; i++) sum += s_cnt[i];
            counts[r] = sum;
        }
        cta_sync();
    }
}

// Host-made parents (mcbgpu_gen_put_trees), one CTA per tree: each vertex's chain must reach
// the root.  The jumps above do not show that: a vertex of a parent cycle may come to point
// to itself, as a branch does, or to a blocking vertex of its cycle, and then stands.  Here
// only the root stands, so a cycle stays open.  The device's own parents lie nearer to the
// root than their children and are not checked.  Slots that are no parent's are left to
// first_pointer().
template <bool kShared>
__global__ void __launch_bounds__(kCodeThreads) put_check_kernel(GenGraph g, const int32_t *__restrict__ pedge,
                                                                 const int32_t *__restrict__ trees, int count, int t0,
                                                                 int32_t *code, unsigned *status) {
    extern __shared__ __align__(16) unsigned char smem[];
    using Ptr = typename std::conditional<kShared, uint16_t, int32_t>::type;
    const int n = g.n;
    for (int i = blockIdx.x; i < count; i += gridDim.x) {
        const int t = trees[i];
        const uint32_t src = g.roots[t];
        const int32_t *pe = pedge + (size_t)t * n;
        volatile Ptr *J = kShared ? reinterpret_cast<volatile Ptr *>(smem)
                                  : reinterpret_cast<volatile Ptr *>(code + (size_t)(t - t0) * n);
        for (int v = threadIdx.x; v < n; v += blockDim.x) {
            const int32_t o = (uint32_t)v == src ? -1 : pe[v];
            J[v] = (Ptr)(o >= 0 && (int64_t)o < g.slots ? __ldg(g.slot_info + o).x : src);
        }
        cta_sync();
        bool done = false;
        for (int round = 0; round < kJumpRounds && !done; round++) {
            bool open = false;
            for (int v = threadIdx.x; v < n; v += blockDim.x) {
                const Ptr p = J[v];
                if ((uint32_t)p == src) continue;
                const Ptr y = J[p];
                J[v] = y;
                open |= (uint32_t)y != src;
            }
            done = cta_sync_and(!open);
        }
        if (!done && threadIdx.x == 0) atomicOr(status, ST_BAD_INPUT);
        cta_sync();  // the pointers are the next tree's
    }
}

// Branch codes of the chunk's trees, one CTA per root, in global memory: the pointers are
// jumped in the code array itself.
__global__ void __launch_bounds__(kCodeThreads) codes_kernel(GenGraph g, const int32_t *__restrict__ pedge, int t0,
                                                             int count, int32_t *code, unsigned *status) {
    const int n = g.n;
    for (int r = blockIdx.x; r < count; r += gridDim.x) {
        const int t = t0 + r;
        const uint32_t src = g.roots[t];
        const int32_t *pe = pedge + (size_t)t * n;
        volatile int32_t *J = code + (size_t)r * n;
        bool bad = false;
        for (int v = threadIdx.x; v < n; v += blockDim.x) {
            uint32_t pair;
            J[v] = first_pointer(g, (uint32_t)v, src, pe[v], pair, bad);
        }
        if (!cta_sync_and(!bad) && threadIdx.x == 0) atomicOr(status, ST_BAD_INPUT);
        bool done = false;
        for (int round = 0; round < kJumpRounds && !done; round++) {
            bool open = false;
            for (int v = threadIdx.x; v < n; v += blockDim.x) {
                const int32_t p = J[v];
                if (p < 0 || p == v) continue;
                const int32_t y = J[p];
                if (y == p) continue;  // a branch
                J[v] = y;
                open |= y >= 0;
            }
            done = cta_sync_and(!open);
        }
        if (!done && threadIdx.x == 0) atomicOr(status, ST_BAD_INPUT);  // deeper than any tree of checked parents
        cta_sync();
    }
}

// The reference's candidate test per non-tree pair of slots, as one bit per pair
// (32 pairs per warp step), and the number of candidates per root.
__global__ void __launch_bounds__(kCandThreads) cand_count_kernel(GenGraph g, const int32_t *__restrict__ pedge,
                                                                  const int32_t *__restrict__ code, int t0, int count,
                                                                  uint32_t *bits, int64_t words_per_root,
                                                                  int64_t *counts) {
    __shared__ long long s_cnt[kCandThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int n = g.n;
    for (int r = blockIdx.x; r < count; r += gridDim.x) {
        const int t = t0 + r;
        const uint32_t src = g.roots[t];
        const int32_t *pe = pedge + (size_t)t * n;
        const int32_t *cd = code + (size_t)r * n;
        uint32_t *bw = bits + (size_t)r * words_per_root;
        long long cnt = 0;
        for (int64_t wi = warp; wi < words_per_root; wi += nwarps) {
            const int64_t k = wi * 32 + lane;
            int acc = 0;
            if (k < g.npairs) {
                const uint32_t o = g.pair_slot[k];
                const uint32_t a = g.rows[o], b = g.cols[o];
                if (pe[b] != (int32_t)o && pe[a] != (int32_t)g.rev[o]) {
                    const int32_t ca = cd[a], cb = cd[b];
                    acc = ca != kCodeBlocked && cb != kCodeBlocked && (a == src || b == src || ca != cb);
                }
            }
            const uint32_t m = __ballot_sync(0xffffffffu, acc);
            if (lane == 0) {
                bw[wi] = m;
                cnt += __popc(m);
            }
        }
        if (lane == 0) s_cnt[warp] = cnt;
        cta_sync();
        if (threadIdx.x == 0) {
            long long s = 0;
            for (int i = 0; i < nwarps; i++) s += s_cnt[i];
            counts[r] = s;
        }
        cta_sync();
    }
}

// Exclusive prefix sum of `count` int64 values in one CTA; out[count] = the total.
__global__ void __launch_bounds__(kScanThreads) scan_small_kernel(const int64_t *in, int count, int64_t *out) {
    __shared__ long long s_part[kScanThreads / 32];
    __shared__ long long s_carry;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_carry = 0;
    cta_sync();
    for (int base = 0; base < count; base += blockDim.x) {
        const int i = base + threadIdx.x;
        long long v = i < count ? in[i] : 0;
        long long x = v;
        for (int d = 1; d < 32; d <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, x, d);
            if (lane >= d) x += y;
        }
        if (lane == 31) s_part[warp] = x;
        cta_sync();
        if (warp == 0) {
            long long p = lane < (int)(blockDim.x >> 5) ? s_part[lane] : 0;
            for (int d = 1; d < 32; d <<= 1) {
                const long long y = __shfl_up_sync(0xffffffffu, p, d);
                if (lane >= d) p += y;
            }
            s_part[lane] = p;  // inclusive prefix of the warp sums
        }
        cta_sync();
        const long long before = s_carry + (warp > 0 ? s_part[warp - 1] : 0);
        if (i < count) out[i] = before + x - v;
        cta_sync();
        if (threadIdx.x == blockDim.x - 1) s_carry = before + x;
        cta_sync();
    }
    if (threadIdx.x == 0) out[count] = s_carry;
}

// The accepted pairs of each root in pair order with their weights, one warp per
// root, written at the root's offset.
__global__ void __launch_bounds__(kCandThreads) cand_write_kernel(GenGraph g, const int32_t *__restrict__ dist,
                                                                  const uint32_t *__restrict__ bits,
                                                                  int64_t words_per_root, int count,
                                                                  const int64_t *__restrict__ offsets, int64_t cap,
                                                                  uint32_t *out_pair, int32_t *out_weight,
                                                                  unsigned *status) {
    const int lane = threadIdx.x & 31;
    const int n = g.n;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, nw = (gridDim.x * blockDim.x) >> 5;
    for (int r = gw; r < count; r += nw) {
        const uint32_t *bw = bits + (size_t)r * words_per_root;
        const int32_t *d = dist + (size_t)r * n;
        int64_t pos = offsets[r];
        const int64_t end = offsets[r + 1];
        for (int64_t wb = 0; wb < words_per_root; wb += 32) {
            const int64_t wi = wb + lane;
            uint32_t m = wi < words_per_root ? bw[wi] : 0u;
            const int c = __popc(m);
            int x = c;
            for (int dd = 1; dd < 32; dd <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, dd);
                if (lane >= dd) x += y;
            }
            int64_t p = pos + x - c;
            while (m) {
                const int j = __ffs(m) - 1;
                m &= m - 1;
                const int64_t k = wi * 32 + j;
                const uint32_t o = g.pair_slot[k];
                if (p < end && p < cap) {
                    out_pair[p] = (uint32_t)k;
                    out_weight[p] = d[g.rows[o]] + d[g.cols[o]] + g.w[o];
                } else {
                    atomicOr(status, ST_BAD_INPUT);
                }
                p++;
            }
            pos += __shfl_sync(0xffffffffu, x, 31);
        }
    }
}

__device__ __forceinline__ uint16_t to_bf16(float f) {
    uint32_t u = __float_as_uint(f);
    u += 0x7fffu + ((u >> 16) & 1u);  // round to nearest even (finite inputs)
    return (uint16_t)(u >> 16);
}

// The learned proposal's 16 features of one candidate (bf16), from its walk: its
// weight against the list's median weight, the two root distances and the edge
// weight as shares of the weight, the path hop counts, the list length, its rank
// quantile, the degrees of its root and ends.
__device__ void candidate_features(uint16_t *f, float W, float wmed, float da, float db, float we, int ha, int hb,
                                   int len, float quantile, int deg_root, int deg_ends) {
    const float Wp = W > 0.0f ? W : 1.0f;
    const float v[16] = {W / wmed,
                         fminf(da, db) / Wp,
                         fmaxf(da, db) / Wp,
                         we / Wp,
                         log2f(1.0f + (float)(ha + hb)) * 0.125f,
                         log2f(1.0f + (float)len) * 0.125f,
                         quantile,
                         log2f(1.0f + (float)deg_root) * 0.25f,
                         log2f(1.0f + (float)deg_ends) * 0.25f,
                         fabsf((float)(ha - hb)) / (1.0f + (float)(ha + hb)),
                         1.0f,
                         0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < 16; i++) f[i] = to_bf16(v[i]);
}

// Per rank: the coordinates of its cycle (its own edge's, then the root paths of its
// two ends).  Without `out`, the count into len[r] (and with `feat`, the candidate's
// features); with it, the coordinates at out[off[r] ...] in walk order.  A hop is two
// dependent reads (parent slot, from HBM; its row and coordinate in one 16-byte entry,
// from L2), and the two paths are walked side by side so that theirs overlap: 1.1M
// candidates of a 65k-point planar-chain graph, 130 hops each, 5.4 -> 4.8 ms per pass, 1.3
// by tree (tree_order_kernel).
__global__ void __launch_bounds__(kWalkThreads) walk_kernel(GenGraph g, const int32_t *__restrict__ pedge, int64_t K,
                                                            const int32_t *__restrict__ tree,
                                                            const int32_t *__restrict__ eoff, int32_t *len,
                                                            const int64_t *__restrict__ off, int32_t *out,
                                                            unsigned *status, uint16_t *feat,
                                                            const int32_t *__restrict__ weight, float wmed,
                                                            const int32_t *__restrict__ order, int64_t count) {
    const int n = g.n;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
        const int64_t r = order ? order[i] : i;
        if (r >= K) continue;
        const int32_t t = tree[r], o = eoff[r];
        if (t < 0 || t >= g.F || o < 0 || (int64_t)o >= g.slots) {
            atomicOr(status, ST_BAD_INPUT);
            if (!out) len[r] = 0;
            if (feat) candidate_features(feat + r * 16, 0, 1, 0, 0, 0, 0, 0, 0, 0, 0, 0);
            continue;
        }
        const uint32_t src = g.roots[t];
        const int32_t *pe = pedge + (size_t)t * n;
        int64_t p = out ? off[r] : 0;
        const int64_t end = out ? off[r + 1] : 0;
        int c = 0;
        auto emit = [&](int32_t coord) {
            if (coord < 0) return;
            if (out) {
                if (p < end)
                    out[p++] = coord;
                else
                    atomicOr(status, ST_BAD_INPUT);
            }
            c++;
        };
        const uint4 own = __ldg(g.slot_info + o);
        emit((int32_t)own.w);
        float dist[2] = {0.0f, 0.0f};
        int hops[2] = {0, 0};
        uint32_t x[2] = {own.x, own.y};
        for (int steps = 0; x[0] != src || x[1] != src; steps++) {
            int32_t q[2];
#pragma unroll
            for (int side = 0; side < 2; side++) q[side] = x[side] != src ? pe[x[side]] : -1;
            uint4 si[2];
#pragma unroll
            for (int side = 0; side < 2; side++) {
                si[side] = make_uint4(src, 0, 0, 0xffffffffu);
                if (x[side] == src) continue;
                if (steps >= n || q[side] < 0 || (int64_t)q[side] >= g.slots)
                    atomicOr(status, ST_BAD_INPUT);  // the path ends here
                else
                    si[side] = __ldg(g.slot_info + q[side]);
            }
#pragma unroll
            for (int side = 0; side < 2; side++) {
                if (x[side] == src) continue;
                emit((int32_t)si[side].w);
                if (feat && q[side] >= 0 && (int64_t)q[side] < g.slots) {
                    dist[side] += (float)g.w[q[side]];
                    hops[side]++;
                }
                x[side] = si[side].x;
            }
        }
        if (!out) len[r] = c;
        if (feat) {
            const uint32_t a = g.rows[o], b = g.cols[o];
            const int deg_root = (int)(g.ro[src + 1] - g.ro[src]);
            const int deg_ends = (int)(g.ro[a + 1] - g.ro[a] + g.ro[b + 1] - g.ro[b]);
            candidate_features(feat + r * 16, (float)weight[r], wmed, dist[0], dist[1], (float)g.w[o], hops[0],
                               hops[1], c, (float)r / (float)K, deg_root, deg_ends);
        }
    }
}

// The walks go tree by tree where few of them share a tree larger than L2 holds: ranks are
// by weight, so neighbouring ones walk trees gigabytes apart, and every hop was a sector
// of its own from HBM.  A counting sort: place[r] in its tree's group (ranks with a bad
// tree: group F), then order[start[tree] + place[r]] = r.  The order inside a group is
// any; the lists do not depend on it.  Two walks, by rank / by tree with the sort:
// planar-chain graphs of 65k points (4.7 GB of parent slots, 1,060 per candidate) 9.6 /
// 2.7 ms, 12k points (159 MB, 390) 250 / 200 us, 8k (69 MB, 290) 197 / 157 us, 4k (17 MB)
// 117 / 97 us, which the sort's launches take back; random graphs of 20k vertices (313 MB,
// 15) 1.82 / 2.42 ms, 8k (50 MB, 12) 271 / 368 us: the sort costs by candidate, and
// their sectors are in L2 from other walks.
constexpr int64_t kOrderBytes = 64 << 20;
constexpr int64_t kOrderSlots = 64;  // parent slots per candidate from here on

__global__ void __launch_bounds__(kScanThreads) tree_place_kernel(const int32_t *__restrict__ tree, int64_t K, int F,
                                                                  int32_t *size, int32_t *place) {
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < K; r += (int64_t)gridDim.x * blockDim.x) {
        const int t = tree[r];
        place[r] = atomicAdd(size + (t >= 0 && t < F ? t : F), 1);
    }
}

__global__ void __launch_bounds__(kScanThreads) tree_order_kernel(const int32_t *__restrict__ tree, int64_t K, int F,
                                                                  const int64_t *__restrict__ start,
                                                                  const int32_t *__restrict__ place, int32_t *order) {
    for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < K; r += (int64_t)gridDim.x * blockDim.x) {
        const int t = tree[r];
        order[start[t >= 0 && t < F ? t : F] + place[r]] = (int32_t)r;
    }
}

// Block-level exclusive scan over int32 lengths -> int64 offsets (three passes:
// per-block sums, a scan of the sums in one block, the offsets).
constexpr int kScanItems = 8;  // items per thread in the per-block passes

__global__ void __launch_bounds__(kScanThreads) block_sums_kernel(const int32_t *len, int64_t K, int64_t *sums) {
    __shared__ long long s_part[kScanThreads / 32];
    const int64_t base = (int64_t)blockIdx.x * kScanThreads * kScanItems;
    long long s = 0;
    for (int i = 0; i < kScanItems; i++) {
        const int64_t r = base + (int64_t)i * kScanThreads + threadIdx.x;
        if (r < K) s += len[r];
    }
    for (int d = 16; d > 0; d >>= 1) s += __shfl_down_sync(0xffffffffu, s, d);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = s;
    cta_sync();
    if (threadIdx.x == 0) {
        long long tot = 0;
        for (int i = 0; i < (int)(blockDim.x >> 5); i++) tot += s_part[i];
        sums[blockIdx.x] = tot;
    }
}

__global__ void __launch_bounds__(kScanThreads) block_offsets_kernel(const int32_t *len, int64_t K,
                                                                     const int64_t *block_base, int64_t *off) {
    __shared__ long long s_part[kScanThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * kScanThreads * kScanItems;
    // each thread takes kScanItems consecutive items
    const int64_t r0 = base + (int64_t)threadIdx.x * kScanItems;
    long long v[kScanItems];
    long long s = 0;
    for (int i = 0; i < kScanItems; i++) {
        v[i] = r0 + i < K ? len[r0 + i] : 0;
        s += v[i];
    }
    long long x = s;
    for (int d = 1; d < 32; d <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, x, d);
        if (lane >= d) x += y;
    }
    if (lane == 31) s_part[warp] = x;
    cta_sync();
    if (warp == 0) {
        long long p = lane < (int)(blockDim.x >> 5) ? s_part[lane] : 0;
        for (int d = 1; d < 32; d <<= 1) {
            const long long y = __shfl_up_sync(0xffffffffu, p, d);
            if (lane >= d) p += y;
        }
        s_part[lane] = p;
    }
    cta_sync();
    long long run = block_base[blockIdx.x] + (warp > 0 ? s_part[warp - 1] : 0) + x - s;
    for (int i = 0; i < kScanItems; i++) {
        if (r0 + i < K) off[r0 + i] = run;
        run += v[i];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == blockDim.x - 1) off[K] = run;
}

// Bitonic sort of s[0, P) (P a power of two) by the calling threads: `lane` of
// `width` cooperating threads; sync() between the stages.
template <typename Sync>
__device__ __forceinline__ void bitonic(int32_t *s, int P, int lane, int width, Sync sync) {
    for (int k = 2; k <= P; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = lane; i < P; i += width) {
                const int l = i ^ j;
                if (l > i) {
                    const int32_t a = s[i], b = s[l];
                    if ((a > b) == ((i & k) == 0)) {
                        s[i] = b;
                        s[l] = a;
                    }
                }
            }
            sync();
        }
    }
}

constexpr int kSortWarps = 8;

// Sorts each list ascending: one warp per list of up to kSortWarpMax entries; longer
// lists are appended to `longs` for sort_long_kernel.
__global__ void __launch_bounds__(kSortWarps * 32) sort_lists_kernel(int64_t K, const int64_t *__restrict__ off,
                                                                     int32_t *coords, int64_t *longs,
                                                                     unsigned *nlong, unsigned long long cap_long) {
    __shared__ int32_t s_buf[kSortWarps][kSortWarpMax];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t *s = s_buf[warp];
    const int64_t gw = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r = gw; r < K; r += nw) {
        const int64_t b = off[r];
        const int L = (int)(off[r + 1] - b);
        if (L <= 1) continue;
        if (L > kSortWarpMax) {
            if (lane == 0) {
                const unsigned q = atomicAdd(nlong, 1u);
                if (q < cap_long) longs[q] = r;
            }
            continue;
        }
        int P = 2;
        while (P < L) P <<= 1;
        for (int i = lane; i < P; i += 32) s[i] = i < L ? coords[b + i] : INT_MAX;
        __syncwarp();
        bitonic(s, P, lane, 32, [] { __syncwarp(); });
        for (int i = lane; i < L; i += 32) coords[b + i] = s[i];
        __syncwarp();
    }
}

__global__ void __launch_bounds__(1024) sort_long_kernel(const int64_t *__restrict__ off, int32_t *coords,
                                                         const int64_t *longs, int count, unsigned *status) {
    extern __shared__ int32_t s_long[];
    for (int q = blockIdx.x; q < count; q += gridDim.x) {
        const int64_t r = longs[q];
        const int64_t b = off[r];
        const int64_t L = off[r + 1] - b;
        if (L > kSortLongMax) {
            if (threadIdx.x == 0) atomicOr(status, ST_BAD_INPUT);
            continue;
        }
        int P = 2;
        while (P < L) P <<= 1;
        for (int i = threadIdx.x; i < P; i += blockDim.x) s_long[i] = i < L ? coords[b + i] : INT_MAX;
        cta_sync();
        bitonic(s_long, P, threadIdx.x, blockDim.x, [] { cta_sync(); });
        for (int i = threadIdx.x; i < L; i += blockDim.x) coords[b + i] = s_long[i];
        cta_sync();
    }
}

}  // namespace gen
}  // namespace mcbgpu

using namespace mcbgpu::gen;

struct mcbgpu_gen {
    int32_t n = 0, F = 0, chunk = 0, N = 0;
    int64_t slots = 0, npairs = 0, words_per_root = 0;
    int sm_count = 0;
    TreeForm form = kTreeShared;
    size_t smem = 0;
    int delta = 1;  // the mean slot weight
    // launch shapes of the tree kernel: while tuning, call i of mcbgpu_gen_trees
    // runs shapes[i] and records its time per root; then the fastest is kept
    std::vector<TreeShape> shapes;
    std::vector<double> shape_us;  // microseconds per root, per shape tried
    int chosen = -1;
    // two tree slots, so that the trees of the next chunk run while the host searches
    // the current chunk's tied roots: distances, tie flags (device and pinned host),
    // the events around the launch, and what was submitted into each
    int32_t *d_dist_slot[2] = {nullptr, nullptr};
    uint8_t *d_tied_slot[2] = {nullptr, nullptr};
    uint8_t *h_tied[2] = {nullptr, nullptr};
    cudaEvent_t ev_begin[2] = {nullptr, nullptr}, ev_end[2] = {nullptr, nullptr};
    int32_t slot_t0[2] = {-1, -1}, slot_count[2] = {0, 0};
    int slot_shape[2] = {-1, -1};
    int submitted = 0;
    int cur_slot = 0;
    // graph
    uint32_t *d_ro = nullptr, *d_rows = nullptr, *d_cols = nullptr, *d_rev = nullptr, *d_pairs = nullptr,
             *d_roots = nullptr;
    uint2 *d_arcs = nullptr;
    int32_t *d_w = nullptr, *d_ec = nullptr, *d_fvs = nullptr;
    // trees
    int32_t *d_pedge = nullptr;  // F x n, resident
    int32_t *d_dist = nullptr;   // chunk x n
    int32_t *d_code = nullptr;   // chunk x n (without branch_shared)
    int32_t *d_put = nullptr;    // chunk: the trees a call of mcbgpu_gen_put_trees brings
    uint4 *d_slot_info = nullptr;
    uint32_t *d_pair_ends = nullptr;
    bool branch_shared = false;  // branch_test_kernel
    uint32_t *d_bits = nullptr;  // chunk x words_per_root
    int32_t *d_gdist = nullptr, *d_next = nullptr;
    uint32_t *d_gdirty = nullptr, *d_gsumm = nullptr;
    uint8_t *d_tied = nullptr;
    int64_t *d_counts = nullptr, *d_coff = nullptr;  // chunk, chunk + 1
    uint32_t *d_cpair = nullptr;
    int32_t *d_cweight = nullptr;
    int64_t cand_cap = 0;
    int32_t cur_t0 = -1, cur_count = 0;
    // lists
    int64_t K = 0, K_lists = 0, nnz = 0;
    // list buffers, kept from one ranking to the next; their sizes in bytes
    int64_t cap_tree = 0, cap_eoff = 0, cap_len = 0, cap_weight = 0, cap_off = 0, cap_bsum = 0, cap_coords = 0,
            cap_longs = 0;
    int64_t cap_order = 0;
    unsigned char *d_order = nullptr;  // ranks tree by tree (mcbgpu_gen_rank), and scratch
    bool ranked = false, ordered = false;
    int32_t *d_tree = nullptr, *d_eoff = nullptr, *d_len = nullptr, *d_coords = nullptr, *d_weight = nullptr;
    int64_t *d_off = nullptr, *d_bsum = nullptr, *d_longs = nullptr;
    unsigned *d_nlong = nullptr;
    unsigned *d_status = nullptr;
    long long bytes = 0;
    long long diverged_runs = 0;
};

template <typename T>
static void drop_room(T *&p, int64_t &cap) {
    cudaFree(p);
    p = nullptr;
    cap = 0;
}

// Room for `need` bytes in *p (contents are lost when it grows).
template <typename T>
static cudaError_t keep_room(T *&p, int64_t &cap, int64_t need) {
    if (need <= cap) return cudaSuccess;
    drop_room(p, cap);
    const cudaError_t e = cudaMalloc((void **)&p, (size_t)need);
    if (e == cudaSuccess) cap = need;
    return e;
}

// Room for what a ranking cannot do without.  Where the memory is short, the walks' order and
// (`all`, before a new ranking) the former lists are given back for it.
template <typename T>
static cudaError_t must_room(mcbgpu_gen *g, T *&p, int64_t &cap, int64_t need, bool all) {
    cudaError_t e = keep_room(p, cap, need);
    if (e != cudaErrorMemoryAllocation) return e;
    (void)cudaGetLastError();
    drop_room(g->d_order, g->cap_order);
    g->ordered = false;
    if (all) {
        drop_room(g->d_coords, g->cap_coords);
        drop_room(g->d_longs, g->cap_longs);
    }
    return keep_room(p, cap, need);
}

static void gen_free_lists(mcbgpu_gen *g) {
    cudaFree(g->d_order);
    cudaFree(g->d_tree);
    cudaFree(g->d_eoff);
    cudaFree(g->d_len);
    cudaFree(g->d_coords);
    cudaFree(g->d_off);
    cudaFree(g->d_bsum);
    cudaFree(g->d_longs);
    cudaFree(g->d_weight);
}

static void gen_free(mcbgpu_gen *g) {
    for (int k = 0; k < 2; k++) {
        if (g->ev_begin[k]) cudaEventDestroy(g->ev_begin[k]);
        if (g->ev_end[k]) cudaEventDestroy(g->ev_end[k]);
        if (g->h_tied[k]) cudaFreeHost(g->h_tied[k]);
        cudaFree(g->d_tied_slot[k]);
    }
    cudaFree(g->d_dist_slot[1]);  // slot 0's distances are d_dist
    void *ps[] = {g->d_arcs, g->d_ro,   g->d_rows,    g->d_cols,   g->d_rev,    g->d_pairs,  g->d_roots,  g->d_w,
                  g->d_ec,   g->d_fvs,     g->d_pedge,  g->d_dist_slot[0], g->d_code, g->d_slot_info, g->d_pair_ends, g->d_put, g->d_bits,
                  g->d_gdist, g->d_next,   g->d_gdirty, g->d_gsumm, g->d_tied,   g->d_counts, g->d_coff,   g->d_cpair,
                  g->d_cweight, g->d_nlong, g->d_status};
    for (void *p : ps) cudaFree(p);
    gen_free_lists(g);
    delete g;
}

static GenGraph graph_of(const mcbgpu_gen *g) {
    GenGraph a;
    a.ro = g->d_ro;
    a.rows = g->d_rows;
    a.cols = g->d_cols;
    a.rev = g->d_rev;
    a.pair_slot = g->d_pairs;
    a.roots = g->d_roots;
    a.w = g->d_w;
    a.ec = g->d_ec;
    a.fvs = g->d_fvs;
    a.slot_info = g->d_slot_info;
    a.pair_ends = g->d_pair_ends;
    a.n = g->n;
    a.F = g->F;
    a.slots = g->slots;
    a.npairs = g->npairs;
    return a;
}

static int check_status(mcbgpu_gen *g, cudaStream_t st, const char *what) {
    unsigned h = 0;
    MCB_CUDA(cudaMemcpyAsync(&h, g->d_status, sizeof h, cudaMemcpyDeviceToHost, st));
    MCB_CUDA(cudaStreamSynchronize(st));
    if (h & ST_DIVERGED) g->diverged_runs++;
    if (h & ~(unsigned)ST_DIVERGED) {
        MCB_CUDA(cudaMemsetAsync(g->d_status, 0, sizeof(unsigned), st));
        set_error("%s: device status 0x%x (an index out of range was skipped)", what, h);
        return MCBGPU_E_DEVICE;
    }
    MCB_CUDA(cudaMemsetAsync(g->d_status, 0, sizeof(unsigned), st));
    return MCBGPU_OK;
}

extern "C" {

int mcbgpu_gen_create(mcbgpu_gen **out, int32_t nodes, int64_t slots, const uint32_t *row_offsets,
                      const uint32_t *rows, const uint32_t *cols, const int32_t *weights, const uint32_t *rev,
                      const int32_t *edge_coord, int32_t num_coords, const int32_t *fvs_array,
                      const uint32_t *fvs_vertices, int32_t fvs_size, const uint32_t *pair_slot, int32_t chunk) {
    if (!out || nodes <= 0 || slots <= 0 || slots >= (1ll << 31) || (slots & 1) || fvs_size <= 0 || chunk <= 0 ||
        num_coords < 0 || !row_offsets || !rows || !cols || !weights || !rev || !edge_coord || !fvs_array ||
        !fvs_vertices || !pair_slot) {
        set_error("mcbgpu_gen_create: invalid arguments");
        return MCBGPU_E_ARG;
    }
    *out = nullptr;
    if (nodes > kTreeGlobalMaxN) {
        set_error("mcbgpu_gen_create: %d vertices after chain contraction (at most %d)", (int)nodes, kTreeGlobalMaxN);
        return MCBGPU_E_ARG;
    }
    // the graph is checked here once, so the kernels can index with it
    if (row_offsets[0] != 0 || (int64_t)row_offsets[nodes] != slots) {
        set_error("mcbgpu_gen_create: row offsets must run from 0 to the slot count");
        return MCBGPU_E_ARG;
    }
    for (int32_t v = 0; v < nodes; v++)
        if (row_offsets[v + 1] < row_offsets[v]) {
            set_error("mcbgpu_gen_create: row offsets decrease at vertex %d", (int)v);
            return MCBGPU_E_ARG;
        }
    long long wsum = 0, wmax = 0;
    for (int32_t v = 0; v < nodes; v++)
        for (uint32_t o = row_offsets[v]; o < row_offsets[v + 1]; o++)
            if (rows[o] != (uint32_t)v) {
                set_error("mcbgpu_gen_create: slot %u is in row %d but names row %u", o, (int)v, rows[o]);
                return MCBGPU_E_ARG;
            }
    for (int64_t o = 0; o < slots; o++) {
        if (cols[o] >= (uint32_t)nodes || rev[o] >= (uint64_t)slots || rev[rev[o]] != (uint32_t)o ||
            rows[rev[o]] != cols[o] || weights[o] < 1 || weights[rev[o]] != weights[o] || edge_coord[o] < -1 ||
            edge_coord[o] >= num_coords) {
            set_error("mcbgpu_gen_create: slot %lld is not a consistent reverse pair with weight >= 1 and a "
                      "coordinate in [-1, N)",
                      (long long)o);
            return MCBGPU_E_ARG;
        }
        wsum += weights[o];
        wmax = weights[o] > wmax ? weights[o] : wmax;
    }
    if (path_length_bound(nodes, slots, weights, rev) + wmax >= (long long)INT_MAX) {
        set_error("mcbgpu_gen_create: distances could reach 2^31 (the n' - 1 heaviest edges weigh too much)");
        return MCBGPU_E_ARG;
    }
    const int64_t npairs = slots / 2;
    for (int64_t k = 0; k < npairs; k++)
        if ((int64_t)pair_slot[k] >= slots || pair_slot[k] >= rev[pair_slot[k]] ||
            (k > 0 && pair_slot[k] <= pair_slot[k - 1])) {
            set_error("mcbgpu_gen_create: pair %lld is not the lower slot of an ascending pair list", (long long)k);
            return MCBGPU_E_ARG;
        }
    for (int32_t t = 0; t < fvs_size; t++)
        if (fvs_vertices[t] >= (uint32_t)nodes || fvs_array[fvs_vertices[t]] != t) {
            set_error("mcbgpu_gen_create: FVS vertex %d is not consistent with the FVS array", (int)t);
            return MCBGPU_E_ARG;
        }
    mcbgpu_gen *g = new mcbgpu_gen();
    g->n = nodes;
    g->F = fvs_size;
    g->N = num_coords;
    g->slots = slots;
    g->npairs = npairs;
    g->chunk = chunk < fvs_size ? chunk : fvs_size;
    g->words_per_root = (npairs + 31) / 32;
    g->delta = (int32_t)((wsum + slots - 1) / slots);
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&g->sm_count, cudaDevAttrMultiProcessorCount, dev);
    const int words = (nodes + 31) / 32;
    g->form = tree_form(nodes, slots);
    g->smem = g->form == kTreeShared ? trees_smem_bytes(nodes) : 0;
    const size_t n = (size_t)nodes, C = (size_t)g->chunk;
#define GALLOC(ptr, sz)                                            \
    do {                                                           \
        size_t _b = (size_t)(sz);                                  \
        if (_b < 16) _b = 16;                                      \
        if (e == cudaSuccess) e = cudaMalloc((void **)&(ptr), _b); \
        g->bytes += (long long)_b;                                 \
    } while (0)
    GALLOC(g->d_ro, 4 * (n + 1));
    GALLOC(g->d_rows, 4 * (size_t)slots);
    GALLOC(g->d_cols, 4 * (size_t)slots);
    GALLOC(g->d_rev, 4 * (size_t)slots);
    GALLOC(g->d_w, 4 * (size_t)slots);
    GALLOC(g->d_arcs, sizeof(uint2) * kArcSlots * n);
    GALLOC(g->d_ec, 4 * (size_t)slots);
    GALLOC(g->d_fvs, 4 * n);
    GALLOC(g->d_pairs, 4 * (size_t)npairs);
    GALLOC(g->d_roots, 4 * (size_t)fvs_size);
    GALLOC(g->d_pedge, 4 * n * (size_t)fvs_size);
    GALLOC(g->d_dist, 4 * n * C);
    g->d_dist_slot[0] = g->d_dist;
    GALLOC(g->d_slot_info, sizeof(uint4) * (size_t)slots);
    GALLOC(g->d_put, 4 * C);
    g->branch_shared = nodes <= kBranchMaxN && branch_smem_bytes(nodes, npairs) <= kBranchSmemMax;
    if (g->branch_shared)
        GALLOC(g->d_pair_ends, 4 * (size_t)npairs);
    else
        GALLOC(g->d_code, 4 * n * C);
    GALLOC(g->d_bits, 4 * (size_t)g->words_per_root * C);
    GALLOC(g->d_tied, C);
    GALLOC(g->d_counts, 8 * C);
    GALLOC(g->d_coff, 8 * (C + 1));
    GALLOC(g->d_next, 4);
    GALLOC(g->d_status, 4);
    GALLOC(g->d_nlong, 4);
    if (g->form != kTreeShared) {
        GALLOC(g->d_gdist, 4 * n * (size_t)g->sm_count * kTreeMaxCtasPerSm);
        GALLOC(g->d_gdirty, 4 * (size_t)words * (size_t)g->sm_count * kTreeMaxCtasPerSm);
        GALLOC(g->d_gsumm, 4 * (size_t)((words + 31) / 32) * (size_t)g->sm_count * kTreeMaxCtasPerSm);
    }
    // shapes the tuner tries (the shared form: one 1024-thread CTA per SM, bucket
    // widths only); with fewer chunks than twice the shapes, the first one is kept
    if (g->form == kTreeShared)
        g->shapes = {{kTreeThreads, 1, 8}, {kTreeThreads, 1, 4}, {kTreeThreads, 1, 16}, {kTreeThreads, 1, 2}};
    else {
        g->shapes = {first_shape(g->form, nodes)};
        for (const TreeShape sh : {TreeShape{256, 8, 8}, TreeShape{256, 8, 4}, TreeShape{256, 8, 12}, TreeShape{256, 8, 16},
                                   TreeShape{512, 4, 8}, TreeShape{128, 16, 8}})
            if (sh.threads != g->shapes[0].threads || sh.delta_quarters != g->shapes[0].delta_quarters) g->shapes.push_back(sh);
    }
    const int nchunks = (fvs_size + g->chunk - 1) / g->chunk;
    if (nchunks < 2 * (int)g->shapes.size()) g->chosen = 0;
    for (int k = 0; k < 2; k++) {
        if (e == cudaSuccess) e = cudaEventCreate(&g->ev_begin[k]);
        if (e == cudaSuccess) e = cudaEventCreate(&g->ev_end[k]);
        if (e == cudaSuccess) e = cudaMallocHost((void **)&g->h_tied[k], C);
        if (e == cudaSuccess) e = cudaMalloc((void **)&g->d_tied_slot[k], C);
    }
    if (e == cudaSuccess) e = cudaMalloc((void **)&g->d_dist_slot[1], 4 * n * C);
    g->bytes += 4ll * (long long)n * (long long)C + 2ll * (long long)C;
#undef GALLOC
    auto up = [&](void *dst, const void *src, size_t b) {
        if (e == cudaSuccess) e = cudaMemcpy(dst, src, b, cudaMemcpyHostToDevice);
    };
    up(g->d_ro, row_offsets, 4 * (n + 1));
    up(g->d_rows, rows, 4 * (size_t)slots);
    up(g->d_cols, cols, 4 * (size_t)slots);
    up(g->d_rev, rev, 4 * (size_t)slots);
    up(g->d_w, weights, 4 * (size_t)slots);
    try {
        const std::vector<uint2> arcs = arc_table(nodes, row_offsets, cols, weights);
        up(g->d_arcs, arcs.data(), sizeof(uint2) * arcs.size());
    } catch (const std::bad_alloc &) {  // host memory: reported as the device's
        e = cudaErrorMemoryAllocation;
    }
    up(g->d_ec, edge_coord, 4 * (size_t)slots);
    up(g->d_fvs, fvs_array, 4 * n);
    up(g->d_pairs, pair_slot, 4 * (size_t)npairs);
    up(g->d_roots, fvs_vertices, 4 * (size_t)fvs_size);
    try {
        std::vector<uint4> info((size_t)slots);
        std::vector<uint32_t> ends(g->branch_shared ? (size_t)npairs : 0);
        for (int64_t o = 0; o < slots; o++) info[(size_t)o] = make_uint4(rows[o], cols[o], 0, (uint32_t)edge_coord[o]);
        for (int64_t k = 0; k < npairs; k++) {
            const uint32_t o = pair_slot[k];
            info[o].z = info[rev[o]].z = (uint32_t)k;
            if (g->branch_shared) ends[(size_t)k] = rows[o] | (cols[o] << 16);
        }
        up(g->d_slot_info, info.data(), sizeof(uint4) * (size_t)slots);
        if (g->branch_shared) up(g->d_pair_ends, ends.data(), 4 * (size_t)npairs);
    } catch (const std::bad_alloc &) {
        e = cudaErrorMemoryAllocation;
    }
    if (e == cudaSuccess) e = cudaMemset(g->d_status, 0, 4);
    if (e == cudaSuccess) e = set_trees_smem_limit();
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(branch_test_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBranchSmemMax);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(put_check_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * kBranchMaxN);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(sort_long_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(sizeof(int32_t) * kSortLongMax));
    if (e != cudaSuccess) {
        const int rc = cuda_fail(e, "mcbgpu_gen_create");
        gen_free(g);
        return rc;
    }
    *out = g;
    return MCBGPU_OK;
}

int mcbgpu_gen_trees_submit(mcbgpu_gen *g, int32_t t0, int32_t count, void *stream) {
    if (!g || t0 < 0 || count <= 0 || count > g->chunk || t0 + (int64_t)count > g->F) {
        set_error("mcbgpu_gen_trees_submit: invalid arguments");
        return MCBGPU_E_ARG;
    }
    if (!g->d_pedge) {
        set_error("mcbgpu_gen_trees_submit: the trees were released");
        return MCBGPU_E_STATE;
    }
    const int k = g->submitted & 1;
    if (g->slot_t0[k] >= 0) {
        set_error("mcbgpu_gen_trees_submit: both tree slots are taken (collect a chunk first)");
        return MCBGPU_E_STATE;
    }
    cudaStream_t st = (cudaStream_t)stream;
    // the shape: the next untried one while tuning; once every shape has been
    // submitted, the fastest collected so far (the chosen one once all are timed)
    int si;
    if (g->chosen >= 0)
        si = g->chosen;
    else if (g->submitted < (int)g->shapes.size())
        si = g->submitted;
    else
        si = g->shape_us.empty() ? 0
                                 : (int)(std::min_element(g->shape_us.begin(), g->shape_us.end()) - g->shape_us.begin());
    const TreeShape shape = g->shapes[(size_t)si];
    MCB_CUDA(cudaMemsetAsync(g->d_next, 0, 4, st));
    TreeArgs a;
    a.ro = g->d_ro;
    a.cols = g->d_cols;
    a.w = g->d_w;
    a.rev = g->d_rev;
    a.arcs = g->d_arcs;
    a.n = g->n;
    a.delta = shape_delta(shape, g->delta);
    a.roots = g->d_roots + t0;
    a.count = count;
    a.dist_out = g->d_dist_slot[k];
    a.pedge_out = g->d_pedge + (size_t)t0 * g->n;
    a.tied_out = g->d_tied_slot[k];
    a.gdist = g->d_gdist;
    a.gdirty = g->d_gdirty;
    a.gsumm = g->d_gsumm;
    a.next_root = g->d_next;
    a.status = g->d_status;
    const int cap = g->sm_count * shape.ctas_per_sm;
    const int grid = count < cap ? count : cap;
    MCB_CUDA(cudaEventRecord(g->ev_begin[k], st));
    MCB_CUDA(launch_trees(g->form, shape, grid, g->smem, st, a));
    MCB_CUDA(cudaEventRecord(g->ev_end[k], st));
    MCB_CUDA(cudaMemcpyAsync(g->h_tied[k], g->d_tied_slot[k], (size_t)count, cudaMemcpyDeviceToHost, st));
    g->slot_t0[k] = t0;
    g->slot_count[k] = count;
    g->slot_shape[k] = si;
    g->submitted++;
    return MCBGPU_OK;
}

int mcbgpu_gen_trees_collect(mcbgpu_gen *g, int32_t t0, uint8_t *tied, void *stream) {
    if (!g || !tied) {
        set_error("mcbgpu_gen_trees_collect: invalid arguments");
        return MCBGPU_E_ARG;
    }
    const int k = g->slot_t0[0] == t0 ? 0 : g->slot_t0[1] == t0 ? 1 : -1;
    if (k < 0 || t0 < 0) {
        set_error("mcbgpu_gen_trees_collect: no chunk at tree %d was submitted", (int)t0);
        return MCBGPU_E_STATE;
    }
    cudaStream_t st = (cudaStream_t)stream;
    MCB_CUDA(cudaEventSynchronize(g->ev_end[k]));
    const int count = g->slot_count[k];
    // the tie flags' copy follows ev_end on the same stream
    MCB_CUDA(cudaStreamSynchronize(st));
    std::memcpy(tied, g->h_tied[k], (size_t)count);
    g->cur_t0 = t0;
    g->cur_count = count;
    g->cur_slot = k;
    g->d_dist = g->d_dist_slot[k];
    const int rc = check_status(g, st, "mcbgpu_gen_trees");
    if (rc) return rc;
    const int si = g->slot_shape[k];
    if (g->chosen < 0 && si == (int)g->shape_us.size() && si < (int)g->shapes.size()) {
        float ms = 0;
        MCB_CUDA(cudaEventElapsedTime(&ms, g->ev_begin[k], g->ev_end[k]));
        g->shape_us.push_back(1e3 * (double)ms / count);
        if (g->shape_us.size() == g->shapes.size())
            g->chosen = (int)(std::min_element(g->shape_us.begin(), g->shape_us.end()) - g->shape_us.begin());
    }
    g->slot_t0[k] = -1;  // free for the next submission (its distances stay until then)
    return MCBGPU_OK;
}

int mcbgpu_gen_trees(mcbgpu_gen *g, int32_t t0, int32_t count, uint8_t *tied, void *stream) {
    if (!tied) {
        set_error("mcbgpu_gen_trees: invalid arguments");
        return MCBGPU_E_ARG;
    }
    int rc = mcbgpu_gen_trees_submit(g, t0, count, stream);
    if (rc) return rc;
    return mcbgpu_gen_trees_collect(g, t0, tied, stream);
}

int mcbgpu_gen_tuning(const mcbgpu_gen *g) { return g && g->chosen < 0 ? 1 : 0; }

int mcbgpu_gen_put_trees(mcbgpu_gen *g, const int32_t *trees, int32_t count, const int32_t *dist,
                         const int32_t *parent_slot, void *stream) {
    if (!g || count < 0 || (count > 0 && (!trees || !dist || !parent_slot))) {
        set_error("mcbgpu_gen_put_trees: invalid arguments");
        return MCBGPU_E_ARG;
    }
    for (int32_t i = 0; i < count; i++)
        if (trees[i] < g->cur_t0 || trees[i] >= g->cur_t0 + g->cur_count) {
            set_error("mcbgpu_gen_put_trees: tree %d is not in the current chunk", (int)trees[i]);
            return MCBGPU_E_ARG;
        }
    cudaStream_t st = (cudaStream_t)stream;
    const size_t n = (size_t)g->n;
    for (int32_t i = 0; i < count; i++) {
        const int32_t t = trees[i];
        MCB_CUDA(cudaMemcpyAsync(g->d_dist + (size_t)(t - g->cur_t0) * n, dist + (size_t)i * n, 4 * n,
                                 cudaMemcpyHostToDevice, st));
        MCB_CUDA(cudaMemcpyAsync(g->d_pedge + (size_t)t * n, parent_slot + (size_t)i * n, 4 * n,
                                 cudaMemcpyHostToDevice, st));
    }
    // a bad tree is reported with the candidates (device status)
    const GenGraph gg = graph_of(g);
    for (int32_t at = 0; at < count; at += g->chunk) {
        const int32_t some = count - at < g->chunk ? count - at : g->chunk;
        const int grid = some < g->sm_count * 2 ? some : g->sm_count * 2;
        MCB_CUDA(cudaMemcpyAsync(g->d_put, trees + at, 4 * (size_t)some, cudaMemcpyHostToDevice, st));
        if (g->n <= kBranchMaxN)
            put_check_kernel<true><<<grid, kCodeThreads, 2 * n, st>>>(gg, g->d_pedge, g->d_put, some, g->cur_t0, nullptr,
                                                                      g->d_status);
        else
            put_check_kernel<false><<<grid, kCodeThreads, 0, st>>>(gg, g->d_pedge, g->d_put, some, g->cur_t0, g->d_code,
                                                                   g->d_status);
        MCB_CUDA(cudaGetLastError());
    }
    MCB_CUDA(cudaStreamSynchronize(st));
    return MCBGPU_OK;
}

int mcbgpu_gen_candidates(mcbgpu_gen *g, int64_t *counts, int64_t *total, void *stream) {
    if (!g || !counts || !total || g->cur_t0 < 0) {
        set_error("mcbgpu_gen_candidates: invalid arguments (mcbgpu_gen_trees first)");
        return MCBGPU_E_ARG;
    }
    cudaStream_t st = (cudaStream_t)stream;
    const GenGraph gg = graph_of(g);
    const int count = g->cur_count;
    const int grid = count < g->sm_count * 2 ? count : g->sm_count * 2;
    if (g->branch_shared) {
        branch_test_kernel<<<grid, kCodeThreads, branch_smem_bytes(g->n, g->npairs), st>>>(
            gg, g->d_pedge, g->cur_t0, count, g->d_bits, g->words_per_root, g->d_counts, g->d_status);
        MCB_CUDA(cudaGetLastError());
    } else {
        codes_kernel<<<grid, kCodeThreads, 0, st>>>(gg, g->d_pedge, g->cur_t0, count, g->d_code, g->d_status);
        MCB_CUDA(cudaGetLastError());
        cand_count_kernel<<<count < g->sm_count * 4 ? count : g->sm_count * 4, kCandThreads, 0, st>>>(
            gg, g->d_pedge, g->d_code, g->cur_t0, count, g->d_bits, g->words_per_root, g->d_counts);
        MCB_CUDA(cudaGetLastError());
    }
    scan_small_kernel<<<1, kScanThreads, 0, st>>>(g->d_counts, count, g->d_coff);
    MCB_CUDA(cudaGetLastError());
    MCB_CUDA(cudaMemcpyAsync(counts, g->d_counts, 8 * (size_t)count, cudaMemcpyDeviceToHost, st));
    MCB_CUDA(cudaMemcpyAsync(total, g->d_coff + count, 8, cudaMemcpyDeviceToHost, st));
    int rc = check_status(g, st, "mcbgpu_gen_candidates");
    if (rc) return rc;
    if (*total > g->cand_cap) {
        cudaFree(g->d_cpair);
        cudaFree(g->d_cweight);
        g->d_cpair = nullptr;
        g->d_cweight = nullptr;
        const int64_t cap = *total + *total / 4 + 1024;
        MCB_CUDA(cudaMalloc((void **)&g->d_cpair, 4 * (size_t)cap));
        MCB_CUDA(cudaMalloc((void **)&g->d_cweight, 4 * (size_t)cap));
        g->cand_cap = cap;
    }
    const int wgrid = (int)std::min<long long>((count + (kCandThreads / 32) - 1) / (kCandThreads / 32),
                                               (long long)g->sm_count * 8);
    cand_write_kernel<<<wgrid, kCandThreads, 0, st>>>(gg, g->d_dist, g->d_bits, g->words_per_root, count, g->d_coff,
                                                      g->cand_cap, g->d_cpair, g->d_cweight, g->d_status);
    MCB_CUDA(cudaGetLastError());
    return MCBGPU_OK;
}

int mcbgpu_gen_fetch(mcbgpu_gen *g, int64_t total, uint32_t *pair_index, int32_t *weight, void *stream) {
    if (!g || total < 0 || total > g->cand_cap || (total > 0 && (!pair_index || !weight))) {
        set_error("mcbgpu_gen_fetch: invalid arguments");
        return MCBGPU_E_ARG;
    }
    cudaStream_t st = (cudaStream_t)stream;
    if (total > 0) {
        MCB_CUDA(cudaMemcpyAsync(pair_index, g->d_cpair, 4 * (size_t)total, cudaMemcpyDeviceToHost, st));
        MCB_CUDA(cudaMemcpyAsync(weight, g->d_cweight, 4 * (size_t)total, cudaMemcpyDeviceToHost, st));
    }
    return check_status(g, st, "mcbgpu_gen_fetch");
}

int mcbgpu_gen_rank(mcbgpu_gen *g, int64_t K, const int32_t *tree, const int32_t *edge_offset,
                    const int32_t *weight, uint16_t *features, void *stream) {
    if (!g || K < 0 || (K > 0 && (!tree || !edge_offset || !weight))) {
        set_error("mcbgpu_gen_rank: invalid arguments");
        return MCBGPU_E_ARG;
    }
    if (!g->d_pedge) {
        set_error("mcbgpu_gen_rank: the trees were released");
        return MCBGPU_E_STATE;
    }
    cudaStream_t st = (cudaStream_t)stream;
    g->ranked = false;
    g->K = K;
    g->K_lists = 0;
    g->nnz = 0;
    const int64_t k1 = K > 0 ? K : 1;
    const int64_t nblk = (K + (int64_t)kScanThreads * kScanItems - 1) / ((int64_t)kScanThreads * kScanItems);
    MCB_CUDA(must_room(g, g->d_tree, g->cap_tree, 4 * k1, true));
    MCB_CUDA(must_room(g, g->d_eoff, g->cap_eoff, 4 * k1, true));
    MCB_CUDA(must_room(g, g->d_len, g->cap_len, 4 * k1, true));
    MCB_CUDA(must_room(g, g->d_weight, g->cap_weight, 4 * k1, true));
    MCB_CUDA(must_room(g, g->d_off, g->cap_off, 8 * (K + 1), true));
    MCB_CUDA(must_room(g, g->d_bsum, g->cap_bsum, 8 * (nblk + 1), true));
    g->ranked = true;
    if (K == 0) return MCBGPU_OK;
    MCB_CUDA(cudaMemcpyAsync(g->d_tree, tree, 4 * (size_t)K, cudaMemcpyHostToDevice, st));
    MCB_CUDA(cudaMemcpyAsync(g->d_eoff, edge_offset, 4 * (size_t)K, cudaMemcpyHostToDevice, st));
    MCB_CUDA(cudaMemcpyAsync(g->d_weight, weight, 4 * (size_t)K, cudaMemcpyHostToDevice, st));
    g->ordered = false;
    if (4 * (int64_t)g->F * g->n > kOrderBytes && (int64_t)g->F * g->n / K >= kOrderSlots && K < INT32_MAX) {
        // [order K | start F + 2 | sums | sizes F + 1]; without the room the walks go by rank
        const int64_t items = (int64_t)g->F + 1;
        const int64_t ob = (items + (int64_t)kScanThreads * kScanItems - 1) / ((int64_t)kScanThreads * kScanItems);
        const int64_t at_start = (4 * K + 15) & ~15ll, at_sums = at_start + 8 * (items + 1), at_size = at_sums + 8 * (ob + 1);
        if (keep_room(g->d_order, g->cap_order, at_size + 4 * items) == cudaSuccess) {
            int64_t *start = reinterpret_cast<int64_t *>(g->d_order + at_start), *sums = reinterpret_cast<int64_t *>(g->d_order + at_sums);
            int32_t *size = reinterpret_cast<int32_t *>(g->d_order + at_size), *order = reinterpret_cast<int32_t *>(g->d_order);
            const int ogrid = (int)std::min<long long>((K + kScanThreads - 1) / kScanThreads, (long long)g->sm_count * 8);
            MCB_CUDA(cudaMemsetAsync(size, 0, 4 * (size_t)items, st));
            tree_place_kernel<<<ogrid, kScanThreads, 0, st>>>(g->d_tree, K, g->F, size, g->d_len);
            block_sums_kernel<<<(unsigned)ob, kScanThreads, 0, st>>>(size, items, sums);
            scan_small_kernel<<<1, kScanThreads, 0, st>>>(sums, (int)ob, sums);
            block_offsets_kernel<<<(unsigned)ob, kScanThreads, 0, st>>>(size, items, sums, start);
            tree_order_kernel<<<ogrid, kScanThreads, 0, st>>>(g->d_tree, K, g->F, start, g->d_len, order);
            MCB_CUDA(cudaGetLastError());
            g->ordered = true;
        } else {
            (void)cudaGetLastError();
        }
    }
    const float wmed = (float)(weight[K / 2] > 0 ? weight[K / 2] : 1);  // the list is sorted by weight
    const GenGraph gg = graph_of(g);
    const int wgrid = (int)std::min<long long>((K + kWalkThreads - 1) / kWalkThreads, (long long)g->sm_count * 16);
    walk_kernel<<<wgrid, kWalkThreads, 0, st>>>(gg, g->d_pedge, K, g->d_tree, g->d_eoff, g->d_len, nullptr, nullptr,
                                                g->d_status, features, g->d_weight, wmed,
                                                g->ordered ? reinterpret_cast<const int32_t *>(g->d_order) : nullptr, K);
    MCB_CUDA(cudaGetLastError());
    return check_status(g, st, "mcbgpu_gen_rank");
}

int mcbgpu_gen_build_lists(mcbgpu_gen *g, int64_t K_keep, int64_t *nnz, void *stream) {
    if (!g || !nnz || K_keep < 0 || K_keep > g->K || !g->ranked) {
        set_error("mcbgpu_gen_build_lists: invalid arguments (mcbgpu_gen_rank first)");
        return MCBGPU_E_ARG;
    }
    if (!g->d_pedge) {
        set_error("mcbgpu_gen_build_lists: the trees were released");
        return MCBGPU_E_STATE;
    }
    cudaStream_t st = (cudaStream_t)stream;
    g->K_lists = K_keep;
    g->nnz = 0;
    if (K_keep == 0) {
        MCB_CUDA(cudaMemsetAsync(g->d_off, 0, 8, st));
        MCB_CUDA(cudaStreamSynchronize(st));
        *nnz = 0;
        return MCBGPU_OK;
    }
    const int64_t K = K_keep;
    const int64_t nblk = (K + (int64_t)kScanThreads * kScanItems - 1) / ((int64_t)kScanThreads * kScanItems);
    block_sums_kernel<<<(unsigned)nblk, kScanThreads, 0, st>>>(g->d_len, K, g->d_bsum);
    MCB_CUDA(cudaGetLastError());
    scan_small_kernel<<<1, kScanThreads, 0, st>>>(g->d_bsum, (int)nblk, g->d_bsum);
    MCB_CUDA(cudaGetLastError());
    block_offsets_kernel<<<(unsigned)nblk, kScanThreads, 0, st>>>(g->d_len, K, g->d_bsum, g->d_off);
    MCB_CUDA(cudaGetLastError());
    int64_t total = 0;
    MCB_CUDA(cudaMemcpyAsync(&total, g->d_off + K, 8, cudaMemcpyDeviceToHost, st));
    int rc = check_status(g, st, "mcbgpu_gen_build_lists (offsets)");
    if (rc) return rc;
    MCB_CUDA(must_room(g, g->d_coords, g->cap_coords, 4 * (total > 0 ? total : 1), false));
    const GenGraph gg = graph_of(g);
    const int32_t *order = g->ordered ? reinterpret_cast<const int32_t *>(g->d_order) : nullptr;
    const int64_t walks = order ? g->K : K;  // the order is over all ranks
    const int wgrid = (int)std::min<long long>((walks + kWalkThreads - 1) / kWalkThreads, (long long)g->sm_count * 16);
    walk_kernel<<<wgrid, kWalkThreads, 0, st>>>(gg, g->d_pedge, K, g->d_tree, g->d_eoff, g->d_len, g->d_off,
                                                g->d_coords, g->d_status, nullptr, nullptr, 1.0f, order, walks);
    MCB_CUDA(cudaGetLastError());
    const unsigned long long cap_long = (unsigned long long)(K < 65536 ? K : 65536);
    MCB_CUDA(must_room(g, g->d_longs, g->cap_longs, 8 * (int64_t)cap_long, false));
    MCB_CUDA(cudaMemsetAsync(g->d_nlong, 0, 4, st));
    const int sgrid = (int)std::min<long long>((K + kSortWarps - 1) / kSortWarps, (long long)g->sm_count * 8);
    sort_lists_kernel<<<sgrid, kSortWarps * 32, 0, st>>>(K, g->d_off, g->d_coords, g->d_longs, g->d_nlong, cap_long);
    MCB_CUDA(cudaGetLastError());
    unsigned nlong = 0;
    MCB_CUDA(cudaMemcpyAsync(&nlong, g->d_nlong, 4, cudaMemcpyDeviceToHost, st));
    MCB_CUDA(cudaStreamSynchronize(st));
    if (nlong > cap_long) {
        set_error("mcbgpu_gen_build_lists: %u lists longer than %d entries (at most %llu)", nlong, kSortWarpMax,
                  cap_long);
        return MCBGPU_E_ARG;
    }
    if (nlong > 0) {
        sort_long_kernel<<<std::min<unsigned>(nlong, (unsigned)g->sm_count), 1024, sizeof(int32_t) * kSortLongMax,
                           st>>>(g->d_off, g->d_coords, g->d_longs, (int)nlong, g->d_status);
        MCB_CUDA(cudaGetLastError());
    }
    rc = check_status(g, st, "mcbgpu_gen_build_lists");
    if (rc) return rc;
    g->nnz = total;
    *nnz = total;
    return MCBGPU_OK;
}

int mcbgpu_gen_lists(mcbgpu_gen *g, int64_t K, const int32_t *tree, const int32_t *edge_offset,
                     const int32_t *weight, int64_t *nnz, void *stream) {
    if (!nnz) {
        set_error("mcbgpu_gen_lists: NULL nnz");
        return MCBGPU_E_ARG;
    }
    int rc = mcbgpu_gen_rank(g, K, tree, edge_offset, weight, nullptr, stream);
    if (rc) return rc;
    return mcbgpu_gen_build_lists(g, K, nnz, stream);
}

int mcbgpu_gen_get_lists(const mcbgpu_gen *g, const int32_t **weight, const int64_t **offsets,
                         const int32_t **coords) {
    if (!g || !weight || !offsets || !coords || !g->d_off || (g->K_lists > 0 && !g->d_coords)) {
        set_error("mcbgpu_gen_get_lists: no lists (mcbgpu_gen_build_lists first)");
        return MCBGPU_E_STATE;
    }
    *weight = g->d_weight;
    *offsets = g->d_off;
    *coords = g->d_coords;
    return MCBGPU_OK;
}

int mcbgpu_gen_copy_lists(const mcbgpu_gen *g, int64_t *offsets, int32_t *coords, void *stream) {
    if (!g || !offsets || (g->nnz > 0 && !coords) || !g->d_off || (g->K_lists > 0 && !g->d_coords)) {
        set_error("mcbgpu_gen_copy_lists: invalid arguments or no lists");
        return MCBGPU_E_ARG;
    }
    cudaStream_t st = (cudaStream_t)stream;
    MCB_CUDA(cudaMemcpyAsync(offsets, g->d_off, 8 * (size_t)(g->K_lists + 1), cudaMemcpyDeviceToHost, st));
    if (g->nnz > 0)
        MCB_CUDA(cudaMemcpyAsync(coords, g->d_coords, 4 * (size_t)g->nnz, cudaMemcpyDeviceToHost, st));
    MCB_CUDA(cudaStreamSynchronize(st));
    return MCBGPU_OK;
}

int mcbgpu_gen_release_trees(mcbgpu_gen *g) {
    if (!g) return MCBGPU_OK;
    cudaFree(g->d_pedge);
    g->d_pedge = nullptr;
    g->bytes -= 4ll * g->n * g->F;
    return MCBGPU_OK;
}

int mcbgpu_gen_tree_shapes(const mcbgpu_gen *g, int32_t *shapes, double *us_per_root, int32_t cap, int32_t *count,
                           int32_t *chosen) {
    if (!g || !count || !chosen || (cap > 0 && (!shapes || !us_per_root))) {
        set_error("mcbgpu_gen_tree_shapes: invalid arguments");
        return MCBGPU_E_ARG;
    }
    *count = (int32_t)g->shapes.size();
    *chosen = g->chosen;
    for (int32_t i = 0; i < cap && i < *count; i++) {
        shapes[3 * i] = g->shapes[(size_t)i].threads;
        shapes[3 * i + 1] = g->shapes[(size_t)i].ctas_per_sm;
        shapes[3 * i + 2] = g->shapes[(size_t)i].delta_quarters;
        us_per_root[i] = (size_t)i < g->shape_us.size() ? g->shape_us[(size_t)i] : -1.0;
    }
    return MCBGPU_OK;
}

int64_t mcbgpu_gen_device_bytes(const mcbgpu_gen *g) {
    return g ? g->bytes + 4 * (g->K * 3) + 8 * (g->K + 1) + 4 * g->nnz + 8 * g->cand_cap : 0;
}

int mcbgpu_gen_destroy(mcbgpu_gen *g) {
    if (g) gen_free(g);
    return MCBGPU_OK;
}

}  // extern "C"
