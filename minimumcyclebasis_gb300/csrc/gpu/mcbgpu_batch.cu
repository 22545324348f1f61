// Batched de Pina solver: many independent problems (the biconnected components of
// one graph, or many graphs) solved in a persistent launch per cluster size.
//
// The reference solves one graph per process and, for a graph split into
// biconnected components, runs the whole driver once per component file
// (main.sh:19-32 loops `run.sh` over bicc's output).  Here every problem is a
// (N, candidates, coordinate lists) triple as mcbgpu_solver takes it; a cluster of csz
// CTAs owns one problem at a time and pulls the next from a device work counter
// (problems in order of decreasing N, so the longest start first).
//
// Per problem the cluster runs the blocked loop of mcbgpu_solver_run (64 iterations per
// block), every CTA with the block's state in its own shared memory:
//   1. T[c] = bits i of S_{e0+i}[c] for the block's rows (64x64 bit transposes; unit
//      bits for c in [e0, bound));
//   2. the rank-ordered scan, a chunk of candidates per round, a slice of it per CTA:
//      W_r = XOR of T over C_r's coordinates below the bound, reduced by the pivots
//      found so far (Four-Russians tables); what is left is compacted in rank order and
//      eliminated (mcbgpu_elim.cuh).  With several CTAs each one's pivots go to all of
//      them through distributed shared memory and are eliminated once more;
//   3. resolve: the reference's loop restricted to the block on 64-bit masks
//      (iteration k takes the first pivot with parity(W_p & m_k) = 1, later masks
//      with odd parity absorb m_k), which selects the reference's candidate for
//      every iteration (mcb/mcb_cycle_deg_two_remove.cpp:329-358);
//   4. the block's final rows S_{e0+k} = XOR_{l in m_k} S^0_{e0+l}, computed from T, a
//      share per CTA;
//   5. every later row j: D_j[k] = <C_sel_k, S_j>, beta = the sequential effect of
//      the 64 updates (a 64x64 GF(2) matrix applied to D), S_j ^= XOR_{k in beta}
//      S_{e0+k} (mcb/mcb_cycle_deg_two_remove.cpp:371-390 for 64 iterations), a residue
//      class of rows per warp.  A row that is still its unit vector and whose
//      coordinate lies on none of the block's cycles is not read.
// Clusters wait for nobody but themselves: the only shared word is the work counter.
#include <cooperative_groups.h>

#include <algorithm>
#include <vector>

#include "mcbgpu_elim.cuh"

using namespace mcbgpu;
using namespace mcbgpu::elim;
namespace cg = cooperative_groups;

namespace {

constexpr int kBThreads = kElimThreads;
constexpr int kBWarps = kBThreads / 32;
constexpr int kSmallQ = 2;               // candidates per thread and scan round, problems of N <= kSmallN
constexpr int kLargeQ = 4;               // the same for larger ones
constexpr int kSmallN = 1024;            // largest N of the small form (two CTAs per SM)
constexpr int kBChunk = 4;               // coordinates of each candidate loaded together beyond its head
constexpr int kBHead = 8;                // coordinates of a list's head (one aligned 32-byte slot per candidate)
constexpr int kBatchMaxN = 12288;        // largest N a CTA holds (T and the final rows in shared memory)
constexpr int kClasses = 4;              // launches of a batch: 8, 4, 2 or 1 CTAs per problem
constexpr unsigned kPairSmemMax = 8192;  // pairs kept in shared memory (more go to the CTA's global scratch)
constexpr size_t kSmemBudget = 214 * 1024;  // dynamic shared memory per CTA at most (static adds 12 KB)

constexpr int kBProf = 13;  // profile words per problem (mcbgpu_batch_profile)

// Words of the region that holds the scan's tables and row list and later the block's
// final rows.
constexpr size_t scan_words(int q) { return 2048 + (20 * (size_t)(kBThreads * q + 64) + 7) / 8; }

struct BatchGraph {
    long long cand;  // first candidate (index into weight / offsets)
    long long K;     // candidates
    long long srow;  // first word of the problem's support vectors (N rows of P words)
    long long sel;   // first entry of the problem in `selected`
    int N, P;
};

__device__ __forceinline__ int ffs64(uint64_t x) { return __ffsll((long long)x) - 1; }

// W of the kBQ candidates r0 + q * kBThreads (0 past `end`) from the block's T in shared
// memory.  The heads come in one coalesced read; the lists that go on below the bound
// are walked in lockstep, kBChunk coordinates of each per step, so kBQ x kBChunk
// independent loads are in flight per thread.  `walked` counts the bytes read.
template <int kBQ>
__device__ __forceinline__ void w_smem_q(long long r0, long long end, long long cand, const int64_t *__restrict__ off,
                                         const int32_t *__restrict__ coords, const int32_t *__restrict__ head,
                                         const uint64_t *T, int bound, uint64_t (&W)[kBQ], unsigned long long &walked) {
    long long ia[kBQ], ea[kBQ];
    int4 ha[kBQ], hb[kBQ];
#pragma unroll
    for (int q = 0; q < kBQ; q++) {
        const long long r = r0 + (long long)q * kBThreads;
        ha[q] = hb[q] = make_int4(0x7fffffff, 0x7fffffff, 0x7fffffff, 0x7fffffff);
        if (r < end) {
            const int4 *h = reinterpret_cast<const int4 *>(head + (size_t)(cand + r) * kBHead);
            ha[q] = __ldg(h);
            hb[q] = __ldg(h + 1);
            walked += 4 * kBHead;
        }
    }
    bool any = false;
#pragma unroll
    for (int q = 0; q < kBQ; q++) {
        const int c[kBHead] = {ha[q].x, ha[q].y, ha[q].z, ha[q].w, hb[q].x, hb[q].y, hb[q].z, hb[q].w};
        uint64_t w = 0;
#pragma unroll
        for (int t = 0; t < kBHead; t++)
            if (c[t] < bound) w ^= T[c[t]];
        W[q] = w;
        ia[q] = ea[q] = 0;
        if (c[kBHead - 1] < bound) {
            const long long r = cand + r0 + (long long)q * kBThreads;
            ia[q] = __ldg(off + r) + kBHead;
            ea[q] = __ldg(off + r + 1);
            walked += 16;
            any = true;
        }
    }
    while (any) {
        int cv[kBQ][kBChunk];
#pragma unroll
        for (int q = 0; q < kBQ; q++)
#pragma unroll
            for (int t = 0; t < kBChunk; t++) cv[q][t] = ia[q] + t < ea[q] ? __ldg(coords + ia[q] + t) : 0x7fffffff;
        any = false;
#pragma unroll
        for (int q = 0; q < kBQ; q++) {
            walked += 4ull * (unsigned long long)min((long long)kBChunk, ea[q] - ia[q] > 0 ? ea[q] - ia[q] : 0);
#pragma unroll
            for (int t = 0; t < kBChunk; t++)
                if (cv[q][t] < bound) W[q] ^= T[cv[q][t]];
            ia[q] = cv[q][kBChunk - 1] >= bound ? ea[q] : ia[q] + kBChunk;
            any |= ia[q] < ea[q];
        }
    }
}

// kBQ: candidates per thread in one scan round; kRowRegs: row words per lane in the
// update (ceil(largest N of the form / 2048)).
template <int kBQ, int kRowRegs, int kMinBlocks>
__global__ void __launch_bounds__(kBThreads, kMinBlocks) batch_solve_kernel(
    const BatchGraph *__restrict__ graphs, const int *__restrict__ order, int count, unsigned *next,
    const int32_t *__restrict__ weight, const int64_t *__restrict__ off, const int32_t *__restrict__ coords,
    const int32_t *__restrict__ head, const unsigned *__restrict__ bad, uint64_t *S, long long *selected,
    long long *total, unsigned *gstatus, unsigned *status, unsigned *pair_scratch, unsigned pair_cap, int ncap,
    unsigned pcap, long long *prof) {
    extern __shared__ __align__(16) uint64_t smem[];
    const int wcap = ncap >> 6;                       // ncap is a multiple of 64
    constexpr unsigned kListCap = kBThreads * kBQ + 64;
    constexpr size_t kScanWords = 2048 + (20 * (size_t)kListCap + 7) / 8;  // scan_words(kBQ)
    const size_t xw = kScanWords > (size_t)ncap ? kScanWords : (size_t)ncap;
    uint64_t *T = smem;                               // ncap words (the row buffers of the update alias it)
    uint64_t *F = smem + ncap;                        // 64 x wcap words: the block's final rows; before them:
    uint64_t(*tab)[256] = reinterpret_cast<uint64_t(*)[256]>(F);  // the pivots' tables
    RowList rows;                                     // and the rows of a round
    rows.w = F + 2048;
    uint64_t *row_w0 = rows.w + kListCap;      // their W as found
    rows.key = reinterpret_cast<unsigned *>(row_w0 + kListCap);
    unsigned *sPairs = (unsigned *)(F + xw);          // pcap pairs
    unsigned *gPairs = pair_scratch + (size_t)blockIdx.x * pair_cap;

    __shared__ ElimShared es;
    __shared__ uint64_t sBasis[64];  // reduced basis of the pivots, by pivot bit
    __shared__ uint64_t sPivW[64];   // W of the pivots, in rank order
    __shared__ int sPivR[64];        // their ranks
    __shared__ uint64_t sMask[64];   // final masks m_k
    __shared__ uint64_t sGcol[64];   // bit i of gcol[k] = <C_sel_k, S_{e0+i}> (i < k)
    __shared__ uint64_t sMrow[64];   // beta of a row = XOR of sMrow[k] over the k with D bit k
    __shared__ int sSel[64];         // rank selected at iteration e0 + k
    __shared__ unsigned sPre[65];    // pair offsets of the selected lists
    __shared__ __align__(8) unsigned sPart[kBQ * kBWarps];
    __shared__ uint64_t sRepV[2][64], sRepW[2][64];  // this CTA's report of a round: residuals, W's,
    __shared__ unsigned sRepKey[2][64], sRepN[2];    // ranks, number (by round parity)
    __shared__ uint32_t sUnit[kRowRegs * 64], sHit[kRowRegs * 64];  // bit j: S_j = e_j; j on a cycle of the block
    __shared__ int sGi[2];
    __shared__ unsigned sFail;
    // profile (thread 0 of the first CTA): cycles in T, scan, resolve, final rows, update;
    // candidates scanned; cycles of the scan's list walks; scan rounds; cycles of warp 0
    // in the update's D + beta and in its row writes
    __shared__ long long pc[10];
    __shared__ unsigned long long s_walked;

    cg::cluster_group cluster = cg::this_cluster();
    const unsigned csz = cluster.num_blocks(), crank = cluster.block_rank();
    auto cluster_sync = [&] {
        if (csz > 1) {
            asm volatile("barrier.cluster.arrive.release;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        } else {
            cta_sync();
        }
    };
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int gwarp = (int)crank * kBWarps + warp, nwarp = (int)csz * kBWarps;
    const unsigned full = 0xffffffffu;

    cluster_sync();  // every CTA of the cluster has started: its shared memory may be written
    for (unsigned turn = 0;; turn ^= 1) {
        if (crank == 0 && tid == 0) {
            const int g = (int)atomicAdd(next, 1u);
            for (unsigned i = 0; i < csz; i++) *cluster.map_shared_rank(&sGi[turn], i) = g;
        }
        cluster_sync();  // also: everyone is done with the previous problem
        const int gi = sGi[turn];
        if (gi >= count) break;
        const int gx = order[gi];
        const BatchGraph g = graphs[gx];
        const int N = g.N, P = g.P;
        const long long K = g.K, cand = g.cand;
        uint64_t *Sg = S + g.srow;

        // the problem's coordinate lists: ascending, in [0, N) (checked by the upload)
        if (bad[gx] || N > ncap) {
            if (crank == 0 && tid == 0) {
                gstatus[gx] |= ST_BAD_INPUT;
                atomicOr(status, ST_BAD_INPUT);
            }
            continue;  // the loop head's barrier separates the problems
        }
        // S_j = e_j; only words [0, j/64] of row j are ever read or written
        for (int j = gwarp; j < N; j += nwarp) {
            uint64_t *row = Sg + (size_t)j * P;
            for (int w = lane; w <= (j >> 6); w += 32) row[w] = w == (j >> 6) ? 1ull << (j & 63) : 0ull;
        }
        for (int i = tid; i < (N + 31) >> 5; i += kBThreads) sUnit[i] = 0xffffffffu;
        long long tot = 0;
        unsigned long long t_start = 0;
        unsigned long long walked = 0;  // this thread's list-walk bytes
        if (prof && tid == 0) s_walked = 0;
        if (prof && tid == 0) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_start));
        if (tid == 0) {
            sFail = 0;
            for (int q = 0; q < 10; q++) pc[q] = 0;
        }
        cluster_sync();

        for (int e0 = 0; e0 < N; e0 += 64) {
            const int b = min(64, N - e0), bound = e0 + b, wl = e0 >> 6, Wb = wl + 1;
            long long c0 = prof ? clock64() : 0;
            // ---- 1. T
            for (int c = e0 + tid; c < bound; c += kBThreads) T[c] = 1ull << (c - e0);
            for (int w = warp; w < wl; w += kBWarps) {
                const uint64_t *r0 = Sg + (size_t)(e0 + lane) * P + w;
                uint64_t x0 = lane < b ? __ldcg(r0) : 0ull;
                uint64_t x1 = lane + 32 < b ? __ldcg(r0 + (size_t)32 * P) : 0ull;
                warp_transpose64(x0, x1);
                T[(w << 6) + lane] = x0;
                T[(w << 6) + 32 + lane] = x1;
            }
            if (tid < 64) sBasis[tid] = 0;
            for (int i = tid; i < (N + 31) >> 5; i += kBThreads) sHit[i] = 0;
            cta_sync();
            if (prof && tid == 0) {
                const long long c = clock64();
                pc[0] += c - c0;
                c0 = c;
            }

            // ---- 2. pivots: the first b rank-ordered candidates with independent W
            int npiv = 0;
            const long long slice = (long long)kBThreads * kBQ;
            unsigned par = 0;
            for (long long base = 0; npiv < b; base += slice * csz, par ^= 1) {
                if (base >= K) {  // fewer than b independent candidates
                    if (tid == 0) sFail = 1;
                    break;
                }
                const long long mine = base + (long long)crank * slice;
                if (tid == 0) {  // the next slice's heads into L2 while this one is walked
                    const long long nb = mine + slice * csz;
                    if (nb < K) prefetch_l2(head + (size_t)(cand + nb) * kBHead, 4ull * kBHead * (unsigned long long)(min(nb + slice, K) - nb));
                }
                const long long cw = prof ? clock64() : 0;
                uint64_t W[kBQ], res[kBQ];
                w_smem_q<kBQ>(mine + tid, K, cand, off, coords, head, T, bound, W, walked);
                if (prof && tid == 0) {
                    pc[6] += clock64() - cw;
                    pc[7]++;
                }
                // what the pivots leave, in rank order
                unsigned nz[kBQ];
#pragma unroll
                for (int q = 0; q < kBQ; q++) {
                    res[q] = npiv > 0 && W[q] ? fr_reduce(W[q], tab) : W[q];
                    nz[q] = __ballot_sync(full, res[q] != 0);
                    if (lane == 0) sPart[q * kBWarps + warp] = __popc(nz[q]);
                }
                cta_sync();
                constexpr int kPer = kBQ * kBWarps / 32;  // counts per lane
                unsigned pc_[kPer], own = 0;
#pragma unroll
                for (int i = 0; i < kPer; i++) {
                    pc_[i] = own;
                    own += sPart[lane * kPer + i];
                }
                unsigned incl = own;
                for (int d = 1; d < 32; d <<= 1) {
                    const unsigned y = __shfl_up_sync(full, incl, d);
                    if (lane >= d) incl += y;
                }
                const unsigned cnt = __shfl_sync(full, incl, 31);
#pragma unroll
                for (int q = 0; q < kBQ; q++) {
                    unsigned at = 0;
#pragma unroll
                    for (int i = 0; i < kPer; i++) {
                        const unsigned v = __shfl_sync(full, incl - own + pc_[i], (q * kBWarps + warp) / kPer);
                        if ((q * kBWarps + warp) % kPer == i) at = v;
                    }
                    at += __popc(nz[q] & ((1u << lane) - 1u));
                    if (res[q]) {
                        rows.w[at] = res[q];
                        row_w0[at] = W[q];
                        rows.key[at] = (unsigned)(mine - base) + q * kBThreads + tid;
                    }
                }
                cta_sync();
                int nnew = cnt ? eliminate(rows, cnt, b - npiv, es) : 0;
                if (csz > 1) {
                    if (tid < nnew) {
                        sRepV[par][tid] = es.pw[tid];
                        sRepW[par][tid] = row_w0[es.pat[tid]];
                        sRepKey[par][tid] = es.pkey[tid];
                    }
                    if (tid == 0) sRepN[par] = (unsigned)nnew;
                    cluster_sync();
                    unsigned at = 0;
                    for (unsigned i = 0; i < csz; i++) {
                        const unsigned n = *cluster.map_shared_rank(&sRepN[par], i);
                        if ((unsigned)warp / 2 == i) {  // two warps per CTA of the cluster
                            const unsigned t = (unsigned)(warp & 1) * 32 + lane;
                            if (t < n) {
                                rows.w[at + t] = *cluster.map_shared_rank(&sRepV[par][t], i);
                                row_w0[at + t] = *cluster.map_shared_rank(&sRepW[par][t], i);
                                rows.key[at + t] = *cluster.map_shared_rank(&sRepKey[par][t], i);
                            }
                        }
                        at += n;
                    }
                    cta_sync();
                    nnew = at ? eliminate(rows, at, b - npiv, es) : 0;
                }
                if (nnew > 64 - npiv) nnew = 64 - npiv;
                if (tid < nnew) {
                    sPivW[npiv + tid] = row_w0[es.pat[tid]];
                    sPivR[npiv + tid] = (int)(base + es.pkey[tid]);
                }
                npiv += nnew;
                if (npiv < b && nnew > 0) {
                    if (warp == 0) basis_add(sBasis, nnew, es);
                    cta_sync();
                    fr_build(tab, sBasis);
                }
                cta_sync();
                if (tid == 0) pc[5] += slice * csz;
            }
            cta_sync();
            if (prof && tid == 0) {
                const long long c = clock64();
                pc[1] += c - c0;
                c0 = c;
            }
            if (sFail) break;

            // ---- 3. resolve (warp 0), gcol, the beta matrix, selected ranks, pair offsets
            if (warp == 0) {
                uint64_t a0 = lane < b ? sPivW[lane] : 0ull, a1 = lane + 32 < b ? sPivW[lane + 32] : 0ull, m0, m1;
                warp_transpose64(a0, a1);  // row j of A = bit j of every W
                int p0, p1;                // pivot of iteration lane / lane + 32
                const bool done = resolve_rows(b, a0, a1, m0, m1, p0, p1);
                sMask[lane] = lane < b ? m0 : 0ull;
                sMask[lane + 32] = lane + 32 < b ? m1 : 0ull;
                if (!done) {  // cannot happen for independent pivots; guards the indexing
                    if (lane == 0) sFail = 1;
                } else {
                    // gcol[k] bit i = A[i][p_k] (i < k) of the final rows
                    uint64_t col0 = a0, col1 = a1;
                    warp_transpose64(col0, col1);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int k = lane + 32 * h, p = h ? p1 : p0;
                        const uint64_t g0 = __shfl_sync(full, col0, p & 31), g1 = __shfl_sync(full, col1, p & 31);
                        sGcol[k] = k < b ? (p < 32 ? g0 : g1) & ((1ull << k) - 1ull) : 0ull;
                        if (k < b) sSel[k] = sPivR[p];
                    }
                    __syncwarp();
                    // beta for D = e_k: beta_i = 0 (i < k), 1 (i = k), parity(beta & gcol[i]) (i > k)
                    uint64_t bt0 = 1ull << lane, bt1 = 1ull << (lane + 32);
#pragma unroll 4
                    for (int i = 1; i < b; i++) {
                        const uint64_t gc = sGcol[i];
                        if (i > lane) bt0 |= (uint64_t)parity64(bt0 & gc) << i;
                        if (i > lane + 32) bt1 |= (uint64_t)parity64(bt1 & gc) << i;
                    }
                    sMrow[lane] = lane < b ? bt0 : 0ull;
                    sMrow[lane + 32] = lane + 32 < b ? bt1 : 0ull;
                    // pair offsets of the selected lists
                    long long l0 = 0, l1 = 0;
                    unsigned long long wt = 0;
                    if (lane < b) {
                        l0 = off[cand + sSel[lane] + 1] - off[cand + sSel[lane]];
                        wt += (unsigned long long)(long long)weight[cand + sSel[lane]];
                    }
                    if (lane + 32 < b) {
                        l1 = off[cand + sSel[lane + 32] + 1] - off[cand + sSel[lane + 32]];
                        wt += (unsigned long long)(long long)weight[cand + sSel[lane + 32]];
                    }
                    unsigned s0 = (unsigned)l0, s1 = (unsigned)l1;
                    for (int d = 1; d < 32; d <<= 1) {
                        const unsigned a0_ = __shfl_up_sync(full, s0, d), a1_ = __shfl_up_sync(full, s1, d);
                        if (lane >= d) {
                            s0 += a0_;
                            s1 += a1_;
                        }
                    }
                    const unsigned t0 = __shfl_sync(full, s0, 31);
                    sPre[lane + 1] = s0;
                    sPre[lane + 33] = t0 + s1;
                    if (lane == 0) sPre[0] = 0;
                    for (int d = 16; d > 0; d >>= 1) wt += __shfl_xor_sync(full, wt, d);
                    tot += (long long)wt;
                }
            }
            cta_sync();
            if (prof && tid == 0) {
                const long long c = clock64();
                pc[2] += c - c0;
                c0 = c;
            }
            if (sFail) break;
            const unsigned np = sPre[b];
            unsigned *pairs = np <= pcap ? sPairs : gPairs;

            // ---- 4. final rows of the block: a share per CTA into S (and F, alone), 5. pairs
            for (int item = gwarp; item < b * wl; item += nwarp) {
                const int k = item / wl, w = item - k * wl;
                const uint64_t mk = sMask[k];
                const unsigned lo = __ballot_sync(full, parity64(T[(w << 6) + lane] & mk));
                const unsigned hi = __ballot_sync(full, parity64(T[(w << 6) + 32 + lane] & mk));
                if (lane == 0) {
                    const uint64_t v = ((uint64_t)hi << 32) | lo;
                    if (csz == 1) F[k * Wb + w] = v;
                    Sg[(size_t)(e0 + k) * P + w] = v;
                }
            }
            for (int k = tid; k < b; k += kBThreads) {
                F[k * Wb + wl] = sMask[k];
                if (crank == 0) Sg[(size_t)(e0 + k) * P + wl] = sMask[k];
            }
            for (int k = warp; k < b; k += kBWarps) {
                const long long a = off[cand + sSel[k]], e = off[cand + sSel[k] + 1];
                const unsigned o = sPre[k];
                for (long long i = a + lane; i < e; i += 32) {
                    const unsigned c = (unsigned)coords[i];
                    pairs[o + (unsigned)(i - a)] = (c << 6) | (unsigned)k;
                    if ((int)c >= bound) atomicOr(&sHit[c >> 5], 1u << (c & 31));
                }
            }
            cluster_sync();
            if (csz > 1) {  // the other CTAs' shares
                for (int i = tid; i < b * wl; i += kBThreads) {
                    const int k = i / wl, w = i - k * wl;
                    F[k * Wb + w] = __ldcg(Sg + (size_t)(e0 + k) * P + w);
                }
                cta_sync();
            }
            if (prof && tid == 0) {
                const long long c = clock64();
                pc[3] += c - c0;
                c0 = c;
            }

            // ---- 6. later rows: one warp per row.  The row's words [0, Wb) are loaded
            // once (coalesced) into registers and, below e0, into the warp's row buffer
            // (T's storage, free until the next block); D_j from the pairs against the
            // buffer, beta = D_j x Mrow, then S_j ^= XOR_{k in beta} F_k.  Row j belongs to
            // warp j mod nwarp of the cluster throughout, which alone keeps its unit bit.
            uint64_t *rowbuf = T + (size_t)warp * wcap;
            for (int j = bound + ((gwarp - bound) % nwarp + nwarp) % nwarp; j < N; j += nwarp) {
                const bool unit = (sUnit[j >> 5] >> (j & 31)) & 1u;
                if (unit && !((sHit[j >> 5] >> (j & 31)) & 1u)) continue;  // D_j = 0
                const long long cu0 = prof ? clock64() : 0;
                uint64_t *Sj = Sg + (size_t)j * P;
                uint64_t v[kRowRegs];
#pragma unroll
                for (int i = 0; i < kRowRegs; i++) {
                    const int w = lane + 32 * i;
                    v[i] = w < Wb && !unit ? __ldcg(Sj + w) : 0ull;
                    if (w < wl) rowbuf[w] = v[i];
                }
                __syncwarp();
                uint64_t D = 0;
                for (unsigned i = lane; i < np; i += 32) {
                    const unsigned pr = pairs[i];
                    const int c = (int)(pr >> 6);
                    const uint64_t bit = c < e0 ? (rowbuf[c >> 6] >> (c & 63)) & 1ull : (uint64_t)(c == j);
                    D ^= bit << (pr & 63);
                }
                D = warp_xor64(D);
                uint64_t beta = ((D >> lane) & 1) ? sMrow[lane] : 0ull;
                if ((D >> (lane + 32)) & 1) beta ^= sMrow[lane + 32];
                beta = warp_xor64(beta);
                const long long cu1 = prof ? clock64() : 0;
                if (prof && tid == 0) pc[8] += cu1 - cu0;
                if (beta) {
                    if (unit && lane == 0) atomicAnd(&sUnit[j >> 5], ~(1u << (j & 31)));
#pragma unroll
                    for (int i = 0; i < kRowRegs; i++) {
                        const int w = lane + 32 * i;
                        if (w < Wb) {
                            uint64_t x = 0;
                            for (uint64_t bb = beta; bb; bb &= bb - 1) x ^= F[ffs64(bb) * Wb + w];
                            Sj[w] = v[i] ^ x;
                        }
                    }
                }
                if (prof && tid == 0) pc[9] += clock64() - cu1;
                __syncwarp();
            }
            if (crank == 0 && tid == 0)
                for (int k = 0; k < b; k++) selected[g.sel + e0 + k] = sSel[k];
            cluster_sync();
            if (prof && tid == 0) pc[4] += clock64() - c0;
        }
        if (crank == 0 && tid == 0) {
            if (sFail) {
                gstatus[gx] |= ST_RANK_DEFICIT;
                atomicOr(status, ST_RANK_DEFICIT);
            }
            total[gx] = sFail ? -1 : tot;  // tot lives in warp 0
        }
        if (prof) {
            atomicAdd(&s_walked, walked);
            cta_sync();
        }
        if (prof && crank == 0 && tid == 0) {
            unsigned long long t_end;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t_end));
            unsigned smid;
            asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
            long long *o = prof + (size_t)gx * kBProf;
            o[0] = (long long)(t_end - t_start);
            for (int q = 0; q < 6; q++) o[1 + q] = pc[q];
            o[7] = smid;
            o[8] = pc[6];
            o[9] = pc[7];
            o[10] = pc[8];
            o[11] = pc[9];
            o[12] = (long long)(s_walked * csz);  // the other CTAs walk as much
        }
    }
}

}  // namespace

namespace {

// The uploaded offsets: non-decreasing from 0 to nnz (out[0] = 1 if not); out[1] =
// the longest list (it sizes the pair scratch).
__global__ void batch_validate_kernel(const int64_t *__restrict__ off, long long K, long long nnz, unsigned *out) {
    unsigned long long mx = 0;
    unsigned bad = 0;
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < K; r += (long long)gridDim.x * blockDim.x) {
        const long long a = off[r], e = off[r + 1];
        if (e < a || a < 0 || e > nnz)
            bad = 1;
        else if ((unsigned long long)(e - a) > mx)
            mx = (unsigned long long)(e - a);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && (off[0] != 0 || off[K] != nnz)) bad = 1;
    if (mx > 0xffffffffull) mx = 0xffffffffull;
    unsigned m32 = (unsigned)mx;
    m32 = __reduce_max_sync(0xffffffffu, m32);
    bad = __reduce_or_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        if (m32) atomicMax(out + 1, m32);
        if (bad) atomicOr(out, 1u);
    }
}

// Behind it: each list's head (INT_MAX past its end), and bad[i] = 1 for a problem with
// a list that is not ascending in [0, N).  `first` holds the problems' first candidates
// (ascending; count entries).
__global__ void __launch_bounds__(256) batch_lists_kernel(const int64_t *__restrict__ off, const int32_t *__restrict__ coords,
                                                         long long K, const BatchGraph *__restrict__ graphs, int count,
                                                         int32_t *head, unsigned *bad) {
    for (long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x; r < K; r += (long long)gridDim.x * blockDim.x) {
        int lo = 0, hi = count - 1;  // the last problem that starts at or before r
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (graphs[mid].cand <= r)
                lo = mid;
            else
                hi = mid - 1;
        }
        const int N = graphs[lo].N;
        const int64_t a = off[r], e = off[r + 1];
        int v[kBHead], prev = -1;
        bool ok = true;
#pragma unroll
        for (int q = 0; q < kBHead; q++) v[q] = a + q < e ? coords[a + q] : 0x7fffffff;
#pragma unroll
        for (int q = 0; q < kBHead; q++)
            if (a + q < e) {
                ok &= v[q] > prev && v[q] < N;
                prev = v[q];
            }
        for (int64_t i = a + kBHead; i < e; i++) {
            const int c = coords[i];
            ok &= c > prev && c < N;
            prev = c;
        }
        if (!ok) bad[lo] = 1u;
        int4 *h = reinterpret_cast<int4 *>(head + (size_t)r * kBHead);
        h[0] = make_int4(v[0], v[1], v[2], v[3]);
        h[1] = make_int4(v[4], v[5], v[6], v[7]);
    }
}

}  // namespace

struct mcbgpu_batch {
    int count = 0;
    int sm_count = 0;
    long long total_K = 0, nnz = 0, total_N = 0, s_words = 0;
    unsigned pair_cap = 0;   // pair scratch words per CTA (64 x the longest list)
    std::vector<BatchGraph> graphs;
    std::vector<int> order;  // problems with coordinates, class by class, each by decreasing N
    struct Class {           // one launch: `cluster` CTAs per problem
        int cluster, at = 0, count = 0;  // its problems in `order`
        int ncap = 0;                    // largest N (rounded up to 64)
        bool small = false;              // every problem fits the small form
        int grid = 0, slab = 0;          // CTAs, and the first one's pair scratch
        cudaStream_t st = nullptr;       // every class but the first launched runs beside the caller's stream
        cudaEvent_t done = nullptr;
    } cls[kClasses] = {{8}, {4}, {2}, {1}};
    int slabs = 0;
    cudaEvent_t ev_fork = nullptr;
    BatchGraph *d_graphs = nullptr;
    int *d_order = nullptr;
    unsigned *d_next = nullptr;  // the classes' work counters
    int32_t *d_weight = nullptr;
    int64_t *d_off = nullptr;
    int32_t *d_coords = nullptr;
    int32_t *d_head = nullptr;   // kBHead per candidate
    uint64_t *d_S = nullptr;
    long long *d_selected = nullptr;
    long long *d_total = nullptr;
    unsigned *d_gstatus = nullptr;
    unsigned *d_bad = nullptr;    // per problem: its lists are malformed
    unsigned *d_status = nullptr;
    unsigned *d_check = nullptr;  // [bad offsets, longest list]
    unsigned *d_pairs = nullptr;
    long long *d_prof = nullptr;  // optional per-problem profile (count x kBProf)
    bool uploaded = false;
    long long launches = 0;
    long long device_bytes = 0;
};

namespace {

size_t batch_region_words(bool small, int ncap) {
    return std::max(scan_words(small ? kSmallQ : kLargeQ), (size_t)ncap);
}

// Pairs kept in shared memory next to T and the region of F.
unsigned batch_pair_smem(bool small, int ncap) {
    const size_t tf = 8 * ((size_t)ncap + batch_region_words(small, ncap));
    const size_t room = kSmemBudget > tf ? (kSmemBudget - tf) / 4 : 0;
    return (unsigned)std::min<size_t>(kPairSmemMax, room & ~(size_t)31);
}

size_t batch_smem_bytes(bool small, int ncap) {
    return 8 * ((size_t)ncap + batch_region_words(small, ncap)) + 4 * (size_t)batch_pair_smem(small, ncap);
}

void free_batch(mcbgpu_batch *b) {
    if (!b) return;
    cudaFree(b->d_graphs);
    cudaFree(b->d_order);
    cudaFree(b->d_next);
    cudaFree(b->d_weight);
    cudaFree(b->d_off);
    cudaFree(b->d_coords);
    cudaFree(b->d_head);
    cudaFree(b->d_S);
    cudaFree(b->d_selected);
    cudaFree(b->d_total);
    cudaFree(b->d_gstatus);
    cudaFree(b->d_bad);
    cudaFree(b->d_status);
    cudaFree(b->d_check);
    cudaFree(b->d_pairs);
    cudaFree(b->d_prof);
    for (auto &c : b->cls) {
        if (c.st) cudaStreamDestroy(c.st);
        if (c.done) cudaEventDestroy(c.done);
    }
    if (b->ev_fork) cudaEventDestroy(b->ev_fork);
    delete b;
}

using BatchKernel = void (*)(const BatchGraph *, const int *, int, unsigned *, const int32_t *, const int64_t *,
                            const int32_t *, const int32_t *, const unsigned *, uint64_t *, long long *, long long *,
                            unsigned *, unsigned *, unsigned *, unsigned, int, unsigned, long long *);

// A class is one queue in order of decreasing N: on the small form (two CTAs per SM)
// when every problem has N <= kSmallN, else on the large one.
BatchKernel batch_kernel(bool small) {
    return small ? (BatchKernel)batch_solve_kernel<kSmallQ, (kSmallN / 64 + 31) / 32, 2>
                 : (BatchKernel)batch_solve_kernel<kLargeQ, (kBatchMaxN / 64 + 31) / 32, 1>;
}

// CTAs per problem, as powers of two into `lg`.  One CTA each is the least work; but a
// long problem alone can take longer than the whole batch spread over the GPU, and then
// its scan and rows are split over a cluster.  With w = N x K (blocks times candidates)
// for a problem's time on one CTA, a cluster of 2, 4, 8 takes 0.62, 0.365, 0.23 of it
// (measured on problems of N = 5,700-6,400).  The least makespan M is sought for which
// every problem on its smallest sufficient cluster takes at most M and all of them
// together fill at most the GPU for M.  A CTA's slice of a scan round and some rows per
// warp must be left, so short problems stay on one CTA.  384 graphs of 50-5000 vertices:
// 69.5 ms on single CTAs (102 before), 43.0 / 25.3 / 32.9 with clusters of 2 / 4 / 8 for all,
// 17.7 this way; 4096 such graphs and the components of a block tree stay on single CTAs.
void choose_clusters(const std::vector<BatchGraph> &graphs, const std::vector<int> &order, int sms, std::vector<int> &lg) {
    const double time_of[kClasses] = {1.0, 0.62, 0.365, 0.23};
    lg.assign(graphs.size(), 0);
    double all = 0;
    auto weight = [&](int i) { return (double)graphs[i].N * (double)std::max<long long>(graphs[i].K, 2048); };
    for (int i : order) all += weight(i);
    for (double m = all / std::max(sms, 1);; m *= 1.1) {
        double load = 0, longest = 0;
        for (int i : order) {
            const long long slice = (long long)kBThreads * kLargeQ;
            int l = 0;
            while (l + 1 < kClasses && weight(i) * time_of[l] > m && graphs[i].K > (slice << (l + 1)) &&
                   graphs[i].N > (512 << l))
                l++;
            lg[i] = l;
            load += weight(i) * time_of[l] * (1 << l);
            longest = std::max(longest, weight(i) * time_of[l]);
        }
        // m has reached what the longest problem needs, or nothing can be split further
        if (load / std::max(sms, 1) <= m || longest >= all) return;
    }
}

void batch_launch_config(const mcbgpu_batch::Class &c, cudaLaunchConfig_t &cfg, cudaLaunchAttribute &at) {
    cfg = {};
    cfg.gridDim = dim3((unsigned)std::max(c.grid, c.cluster));
    cfg.blockDim = dim3(kBThreads);
    cfg.dynamicSmemBytes = batch_smem_bytes(c.small, c.ncap);
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)c.cluster;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
}

}  // namespace

extern "C" {

int mcbgpu_batch_max_coords(void) { return kBatchMaxN; }

int mcbgpu_batch_create(mcbgpu_batch **out, int32_t count, const int32_t *num_coords,
                        const int64_t *num_candidates, int64_t nnz) {
    if (!out || count < 0 || nnz < 0 || (count > 0 && (!num_coords || !num_candidates))) {
        set_error("mcbgpu_batch_create: invalid arguments");
        return MCBGPU_E_ARG;
    }
    *out = nullptr;
    for (int i = 0; i < count; i++) {
        if (num_coords[i] < 0 || num_coords[i] > kBatchMaxN || num_candidates[i] < 0 ||
            num_candidates[i] >= (1ll << 31)) {
            set_error("mcbgpu_batch_create: problem %d has N = %d, K = %lld (the batch takes N <= %d and "
                      "K < 2^31; solve larger problems with mcbgpu_solver)",
                      i, (int)num_coords[i], (long long)num_candidates[i], kBatchMaxN);
            return MCBGPU_E_ARG;
        }
    }
    mcbgpu_batch *b = new mcbgpu_batch();
    b->count = count;
    b->nnz = nnz;
    b->graphs.resize(count);
    for (int i = 0; i < count; i++) {
        BatchGraph &g = b->graphs[i];
        g.N = num_coords[i];
        g.P = (g.N + 63) / 64;
        g.K = num_candidates[i];
        g.cand = b->total_K;
        g.sel = b->total_N;
        g.srow = b->s_words;
        b->total_K += g.K;
        b->total_N += g.N;
        b->s_words += (long long)g.N * g.P;
    }
    // problems with no coordinate need no work; the rest by decreasing N
    for (int i = 0; i < count; i++)
        if (b->graphs[i].N > 0) b->order.push_back(i);
    std::stable_sort(b->order.begin(), b->order.end(),
                     [&](int x, int y) { return b->graphs[x].N > b->graphs[y].N; });
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&b->sm_count, cudaDevAttrMultiProcessorCount, dev);
    {
        std::vector<int> lg, sorted;
        choose_clusters(b->graphs, b->order, b->sm_count, lg);
        for (auto &c : b->cls) {
            c.at = (int)sorted.size();
            for (int i : b->order)
                if ((1 << lg[i]) == c.cluster) sorted.push_back(i);
            c.count = (int)sorted.size() - c.at;
            if (c.count > 0) c.ncap = (b->graphs[sorted[c.at]].N + 63) & ~63;
            c.small = c.ncap <= kSmallN;
        }
        b->order.swap(sorted);
    }
    long long bytes = 0;
#define ALLOC(ptr, sz)                                             \
    do {                                                           \
        size_t _b = (size_t)(sz);                                  \
        if (_b < 16) _b = 16;                                      \
        if (e == cudaSuccess) e = cudaMalloc((void **)&(ptr), _b); \
        bytes += (long long)_b;                                    \
    } while (0)
    ALLOC(b->d_graphs, sizeof(BatchGraph) * (size_t)count);
    ALLOC(b->d_order, sizeof(int) * b->order.size());
    ALLOC(b->d_next, sizeof(unsigned) * kClasses);
    ALLOC(b->d_weight, sizeof(int32_t) * (size_t)b->total_K);
    ALLOC(b->d_off, sizeof(int64_t) * (size_t)(b->total_K + 1));
    ALLOC(b->d_coords, sizeof(int32_t) * (size_t)nnz);
    ALLOC(b->d_head, sizeof(int32_t) * kBHead * (size_t)b->total_K);
    ALLOC(b->d_S, sizeof(uint64_t) * (size_t)b->s_words);
    ALLOC(b->d_selected, sizeof(long long) * (size_t)b->total_N);
    ALLOC(b->d_total, sizeof(long long) * (size_t)count);
    ALLOC(b->d_gstatus, sizeof(unsigned) * (size_t)count);
    ALLOC(b->d_bad, sizeof(unsigned) * (size_t)count);
    ALLOC(b->d_status, sizeof(unsigned));
    ALLOC(b->d_check, 2 * sizeof(unsigned));
#undef ALLOC
    if (e == cudaSuccess && count > 0)
        e = cudaMemcpy(b->d_graphs, b->graphs.data(), sizeof(BatchGraph) * (size_t)count, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && !b->order.empty())
        e = cudaMemcpy(b->d_order, b->order.data(), sizeof(int) * b->order.size(), cudaMemcpyHostToDevice);
    // the attribute is per kernel, shared by all handles: the form's largest need
    for (int k = 0; k < 2 && e == cudaSuccess; k++) {
        const int most = k ? kBatchMaxN : kSmallN;
        size_t need = batch_smem_bytes(!k, most);
        for (int n = 64; n < most; n += 64) need = std::max(need, batch_smem_bytes(!k, n));
        e = cudaFuncSetAttribute(batch_kernel(!k), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)need);
    }
    for (auto &c : b->cls) {
        if (e != cudaSuccess || c.count == 0) continue;
        // as many clusters as are resident at once, at most one per problem
        int clusters = 0;
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        batch_launch_config(c, cfg, at);
        e = cudaOccupancyMaxActiveClusters(&clusters, batch_kernel(c.small), &cfg);
        if (e == cudaSuccess && clusters < 1) e = cudaErrorInvalidConfiguration;
        c.grid = c.cluster * std::min(c.count, clusters);
        c.slab = b->slabs;
        b->slabs += c.grid;
        if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&c.st, cudaStreamNonBlocking);
        if (e == cudaSuccess) e = cudaEventCreateWithFlags(&c.done, cudaEventDisableTiming);
    }
    if (e == cudaSuccess) e = cudaEventCreateWithFlags(&b->ev_fork, cudaEventDisableTiming);
    if (e != cudaSuccess) {
        free_batch(b);
        return cuda_fail(e, "mcbgpu_batch_create");
    }
    b->device_bytes = bytes;
    *out = b;
    return MCBGPU_OK;
}

int mcbgpu_batch_upload(mcbgpu_batch *b, const int32_t *weight, const int64_t *offsets, const int32_t *coords,
                        void *stream) {
    if (!b || (b->total_K > 0 && (!weight || !offsets)) || (b->nnz > 0 && !coords)) {
        set_error("mcbgpu_batch_upload: NULL argument");
        return MCBGPU_E_ARG;
    }
    b->uploaded = false;
    cudaStream_t st = (cudaStream_t)stream;
    if (b->total_K > 0) {
        MCB_CUDA(cudaMemcpyAsync(b->d_weight, weight, sizeof(int32_t) * (size_t)b->total_K, cudaMemcpyHostToDevice,
                                 st));
        MCB_CUDA(cudaMemcpyAsync(b->d_off, offsets, sizeof(int64_t) * (size_t)(b->total_K + 1),
                                 cudaMemcpyHostToDevice, st));
    }
    if (b->nnz > 0)
        MCB_CUDA(cudaMemcpyAsync(b->d_coords, coords, sizeof(int32_t) * (size_t)b->nnz, cudaMemcpyHostToDevice, st));
    // offsets checked on the device (non-decreasing from 0 to nnz); the longest list
    // sizes the pair scratch; the coordinate lists are checked below (batch_lists_kernel)
    unsigned chk[2] = {0, 0};
    if (b->total_K > 0) {
        MCB_CUDA(cudaMemsetAsync(b->d_check, 0, sizeof chk, st));
        const int grid = (int)std::min<long long>((b->total_K + 255) / 256, (long long)std::max(b->sm_count, 1) * 8);
        batch_validate_kernel<<<grid, 256, 0, st>>>(b->d_off, b->total_K, b->nnz, b->d_check);
        MCB_CUDA(cudaGetLastError());
        MCB_CUDA(cudaMemcpyAsync(chk, b->d_check, sizeof chk, cudaMemcpyDeviceToHost, st));
    }
    MCB_CUDA(cudaStreamSynchronize(st));
    if (chk[0]) {
        set_error("mcbgpu_batch_upload: offsets must be non-decreasing from 0 to nnz");
        return MCBGPU_E_ARG;
    }
    const long long max_len = chk[1];
    if (max_len > kBatchMaxN) {  // a list has at most N distinct coordinates
        set_error("mcbgpu_batch_upload: a coordinate list is longer than N");
        return MCBGPU_E_ARG;
    }
    const unsigned cap = (unsigned)(64 * std::max<long long>(max_len, 1));
    if (cap > b->pair_cap) {  // one slab per CTA
        cudaFree(b->d_pairs);
        b->d_pairs = nullptr;
        b->pair_cap = 0;
        const size_t n = (size_t)cap * (size_t)std::max(b->slabs, 1);
        MCB_CUDA(cudaMalloc((void **)&b->d_pairs, sizeof(unsigned) * n));
        b->device_bytes += (long long)(sizeof(unsigned) * n);
        b->pair_cap = cap;
    }
    // the offsets are good: heads, and the coordinate lists checked problem by problem
    // (a bad one fails alone, when it is solved)
    if (b->count > 0) MCB_CUDA(cudaMemsetAsync(b->d_bad, 0, sizeof(unsigned) * (size_t)b->count, st));
    if (b->total_K > 0) {
        const int grid = (int)std::min<long long>((b->total_K + 255) / 256, (long long)std::max(b->sm_count, 1) * 16);
        batch_lists_kernel<<<grid, 256, 0, st>>>(b->d_off, b->d_coords, b->total_K, b->d_graphs, b->count, b->d_head,
                                                 b->d_bad);
        MCB_CUDA(cudaGetLastError());
    }
    MCB_CUDA(cudaStreamSynchronize(st));
    b->uploaded = true;
    return MCBGPU_OK;
}

int mcbgpu_batch_run(mcbgpu_batch *b, void *stream) {
    if (!b || !b->uploaded) {
        set_error("mcbgpu_batch_run: %s", b ? "upload first" : "NULL handle");
        return b ? MCBGPU_E_STATE : MCBGPU_E_ARG;
    }
    cudaStream_t st = (cudaStream_t)stream;
    MCB_CUDA(cudaMemsetAsync(b->d_next, 0, sizeof(unsigned) * kClasses, st));
    MCB_CUDA(cudaMemsetAsync(b->d_status, 0, sizeof(unsigned), st));
    if (b->count > 0) {
        MCB_CUDA(cudaMemsetAsync(b->d_gstatus, 0, sizeof(unsigned) * (size_t)b->count, st));
        MCB_CUDA(cudaMemsetAsync(b->d_total, 0, sizeof(long long) * (size_t)b->count, st));
    }
    // the classes side by side, the widest clusters first: the first on the caller's
    // stream, the others forked from it and joined
    MCB_CUDA(cudaEventRecord(b->ev_fork, st));
    cudaStream_t on = st;
    for (int k = 0; k < kClasses; k++) {
        const auto &c = b->cls[k];
        if (c.count == 0) continue;
        if (on != st) MCB_CUDA(cudaStreamWaitEvent(on = c.st, b->ev_fork, 0));
        cudaLaunchConfig_t cfg;
        cudaLaunchAttribute at;
        batch_launch_config(c, cfg, at);
        cfg.stream = on;
        MCB_CUDA(cudaLaunchKernelEx(&cfg, batch_kernel(c.small), (const BatchGraph *)b->d_graphs,
                                    (const int *)(b->d_order + c.at), c.count, b->d_next + k,
                                    (const int32_t *)b->d_weight, (const int64_t *)b->d_off,
                                    (const int32_t *)b->d_coords, (const int32_t *)b->d_head,
                                    (const unsigned *)b->d_bad, b->d_S, b->d_selected, b->d_total, b->d_gstatus,
                                    b->d_status, b->d_pairs + (size_t)c.slab * b->pair_cap, b->pair_cap, c.ncap,
                                    batch_pair_smem(c.small, c.ncap), b->d_prof));
        MCB_CUDA(cudaGetLastError());
        b->launches++;
        if (on != st) {
            MCB_CUDA(cudaEventRecord(c.done, on));
            MCB_CUDA(cudaStreamWaitEvent(st, c.done, 0));
        }
        on = c.st;
    }
    return MCBGPU_OK;
}

int mcbgpu_batch_results(mcbgpu_batch *b, int64_t *selected, int64_t *total_weight, uint32_t *problem_status,
                         void *stream) {
    if (!b) {
        set_error("mcbgpu_batch_results: NULL handle");
        return MCBGPU_E_ARG;
    }
    cudaStream_t st = (cudaStream_t)stream;
    unsigned v = 0;
    MCB_CUDA(cudaMemcpyAsync(&v, b->d_status, sizeof v, cudaMemcpyDeviceToHost, st));
    if (selected && b->total_N > 0)
        MCB_CUDA(cudaMemcpyAsync(selected, b->d_selected, sizeof(long long) * (size_t)b->total_N,
                                 cudaMemcpyDeviceToHost, st));
    if (total_weight && b->count > 0)
        MCB_CUDA(cudaMemcpyAsync(total_weight, b->d_total, sizeof(long long) * (size_t)b->count,
                                 cudaMemcpyDeviceToHost, st));
    if (problem_status && b->count > 0)
        MCB_CUDA(cudaMemcpyAsync(problem_status, b->d_gstatus, sizeof(unsigned) * (size_t)b->count,
                                 cudaMemcpyDeviceToHost, st));
    MCB_CUDA(cudaStreamSynchronize(st));
    if (v & ST_RANK_DEFICIT) {
        set_error("a problem's candidates do not span its cycle space (status 0x%x)", v);
        return MCBGPU_E_NO_CANDIDATE;
    }
    if (v) {
        set_error("a problem's coordinate lists are not ascending in [0, N) (status 0x%x)", v);
        return MCBGPU_E_ARG;
    }
    return MCBGPU_OK;
}

int mcbgpu_batch_get_support(mcbgpu_batch *b, int32_t problem, int32_t j, uint64_t *words, void *stream) {
    if (!b || problem < 0 || problem >= b->count || !words || j < 0 || j >= b->graphs[problem].N) {
        set_error("mcbgpu_batch_get_support: invalid arguments");
        return MCBGPU_E_ARG;
    }
    const BatchGraph &g = b->graphs[problem];
    cudaStream_t st = (cudaStream_t)stream;
    // words beyond j / 64 are never written: report them as zero
    for (int w = 0; w < g.P; w++) words[w] = 0;
    MCB_CUDA(cudaMemcpyAsync(words, b->d_S + g.srow + (size_t)j * g.P, sizeof(uint64_t) * (size_t)(j / 64 + 1),
                             cudaMemcpyDeviceToHost, st));
    MCB_CUDA(cudaStreamSynchronize(st));
    return MCBGPU_OK;
}

int mcbgpu_batch_set_profiling(mcbgpu_batch *b, int enable) {
    if (!b) {
        set_error("mcbgpu_batch_set_profiling: NULL handle");
        return MCBGPU_E_ARG;
    }
    if (enable && !b->d_prof) {
        MCB_CUDA(cudaMalloc((void **)&b->d_prof, sizeof(long long) * kBProf * (size_t)std::max(b->count, 1)));
        MCB_CUDA(cudaMemset(b->d_prof, 0, sizeof(long long) * kBProf * (size_t)std::max(b->count, 1)));
    } else if (!enable && b->d_prof) {
        MCB_CUDA(cudaFree(b->d_prof));
        b->d_prof = nullptr;
    }
    return MCBGPU_OK;
}

int mcbgpu_batch_profile(mcbgpu_batch *b, int64_t *out) {
    if (!b || !out || !b->d_prof) {
        set_error("mcbgpu_batch_profile: %s", b && b->d_prof ? "NULL output" : "profiling is off");
        return MCBGPU_E_ARG;
    }
    MCB_CUDA(cudaDeviceSynchronize());
    MCB_CUDA(cudaMemcpy(out, b->d_prof, sizeof(long long) * kBProf * (size_t)b->count, cudaMemcpyDeviceToHost));
    return MCBGPU_OK;
}

int64_t mcbgpu_batch_launches(const mcbgpu_batch *b) { return b ? b->launches : 0; }
int64_t mcbgpu_batch_device_bytes(const mcbgpu_batch *b) { return b ? b->device_bytes : 0; }

int mcbgpu_batch_destroy(mcbgpu_batch *b) {
    free_batch(b);
    return MCBGPU_OK;
}

int mcbgpu_batch_solve(int32_t count, const int32_t *num_coords, const int64_t *num_candidates,
                       const int32_t *weight, const int64_t *offsets, const int32_t *coords, int64_t *selected,
                       int64_t *total_weight) {
    long long totK = 0;
    for (int i = 0; i < count; i++) totK += num_candidates ? num_candidates[i] : 0;
    const int64_t nnz = totK > 0 && offsets ? offsets[totK] : 0;
    mcbgpu_batch *b = nullptr;
    int rc = mcbgpu_batch_create(&b, count, num_coords, num_candidates, nnz);
    if (rc) return rc;
    rc = mcbgpu_batch_upload(b, weight, offsets, coords, nullptr);
    if (!rc) rc = mcbgpu_batch_run(b, nullptr);
    if (!rc) rc = mcbgpu_batch_results(b, selected, total_weight, nullptr, nullptr);
    mcbgpu_batch_destroy(b);
    return rc;
}

}  // extern "C"
