// Rank-ordered elimination of 64-bit GF(2) rows and the resolve of a block, shared by
// the blocked solver's pivot search (mcbgpu_solver.cu) and the batched solver
// (mcbgpu_batch.cu).
#pragma once

#include "mcbgpu_internal.cuh"

namespace mcbgpu {
namespace elim {

constexpr int kElimThreads = 512;  // threads of a CTA that eliminates
constexpr int kElimWarps = kElimThreads / 32;

// Reduce W by the basis held as Four-Russians tables: tab[g][pat] = XOR of the basis
// vectors whose pivot bits form `pat` within byte g (0 for non-pivot bits).
__device__ __forceinline__ uint64_t fr_reduce(uint64_t W, const uint64_t (*tab)[256]) {
    uint64_t r = W;
#pragma unroll
    for (int g = 0; g < 8; g++) r ^= tab[g][(W >> (8 * g)) & 255];
    return r;
}

// Build tab from a reduced basis held by pivot bit (0: no vector has that pivot).
__device__ __forceinline__ void fr_build(uint64_t (*tab)[256], const uint64_t *by_bit) {
    for (int idx = threadIdx.x; idx < 8 * 256; idx += blockDim.x) {
        const int g = idx >> 8, pat = idx & 255;
        uint64_t v = 0;
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (pat & (1 << i)) v ^= by_bit[8 * g + i];
        tab[g][pat] = v;
    }
}

// Rows of an elimination in rank order: rank (relative to the step's first candidate)
// and residual, in shared memory.
struct RowList {
    uint64_t *w;
    unsigned *key;
};

// Shared scratch of eliminate().
struct ElimShared {
    ulonglong2 pick[64];  // chosen rows' residuals and pivot bits, in order of choice
    unsigned pos[64];     // their places in the row list
    int np[2];            // how many, after even and odd warps' turns
    uint64_t pw[64];      // the result in rank order: residuals,
    unsigned pkey[64];    // ranks
    unsigned pat[64];     // and places in the row list
};

__device__ __forceinline__ uint64_t join64(unsigned lo, unsigned hi) { return ((uint64_t)hi << 32) | lo; }

// Adds chosen row (v) with its pivot bit (low) to w if w has that bit.
__device__ __forceinline__ void add_pick(unsigned &wl, unsigned &wh, const ulonglong2 &p) {
    const unsigned hit = (wl & (unsigned)p.y) | (wh & (unsigned)(p.y >> 32));
    if (hit) {
        wl ^= (unsigned)p.x;
        wh ^= (unsigned)(p.x >> 32);
    }
}

// The rank-first basis of rows[0, n); returns its size (at most 64), with es.pw / es.pkey
// the chosen rows in rank order.  Every thread holds one row, every warp 32 consecutive
// ones.  Warp after warp chooses: first among the rows with a bit in the low half (the
// first such row is the next pivot and is added to the later rows with its lowest bit),
// then among those left with a bit in the high half (fewer columns have a subset of the
// pivots, so the low half may go first); then the later warps add the new pivots to
// theirs.  A pick is one chain of vote, shuffle and select on 32-bit words; the loop is
// kept short because a lone warp's time goes by the length of that chain (64-bit words,
// two rows per lane: 260 cycles a pick; eight rows fetched and reduced per turn: slower
// still, their code does not stay in the instruction buffer).
// Called by the whole CTA with a barrier since the rows were written; ends with one.
static __device__ __noinline__ int eliminate(const RowList rows, unsigned n, int most, ElimShared &es) {
    const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int np = 0;
    for (unsigned r0 = 0; r0 < n && np < most; r0 += kElimThreads) {
        const unsigned i = r0 + tid;
        const uint64_t w = i < n ? rows.w[i] : 0ull;
        unsigned wl = (unsigned)w, wh = (unsigned)(w >> 32);
        const unsigned nwarps = min((unsigned)kElimWarps, (n - r0 + 31) / 32);
        int added = 0;  // chosen rows already added to this warp's
        for (unsigned ch = 0; ch < nwarps; ch++) {
            if (warp >= ch) {
#pragma unroll 4
                for (; added < np; added++) add_pick(wl, wh, es.pick[added]);
            }
            if (warp == ch) {
                int q = np;
                for (unsigned m; (m = __ballot_sync(0xffffffffu, wl != 0)) != 0 && q < 64; q++) {
                    const int at = __ffs(m) - 1;
                    const unsigned vl = __shfl_sync(0xffffffffu, wl, at), vh = __shfl_sync(0xffffffffu, wh, at);
                    const unsigned low = vl & (0u - vl);
                    if (wl & low) {
                        wl ^= vl;
                        wh ^= vh;
                    }
                    if ((int)lane == at) {
                        es.pick[q] = make_ulonglong2(join64(vl, vh), low);
                        es.pos[q] = i;
                    }
                }
                for (unsigned m; (m = __ballot_sync(0xffffffffu, wh != 0)) != 0 && q < 64; q++) {
                    const int at = __ffs(m) - 1;
                    const unsigned vh = __shfl_sync(0xffffffffu, wh, at);
                    const unsigned low = vh & (0u - vh);
                    if (wh & low) wh ^= vh;
                    if ((int)lane == at) {
                        es.pick[q] = make_ulonglong2(join64(0u, vh), join64(0u, low));
                        es.pos[q] = i;
                    }
                }
                if (lane == 0) es.np[ch & 1] = q;
            }
            cta_sync();
            np = es.np[ch & 1];  // written again two barriers on
            if (np >= most) break;
        }
    }
    if ((int)tid < np) {  // in rank order
        const unsigned at = es.pos[tid];
        int place = 0;
        for (int j = 0; j < np; j++) place += es.pos[j] < at;
        es.pw[place] = es.pick[tid].x;
        es.pkey[place] = rows.key[at];
        es.pat[place] = at;
    }
    cta_sync();
    return np;
}

// Adds the np rows chosen last to a reduced basis held by pivot bit (every row was
// reduced by it before the elimination).  Warp 0.
static __device__ void basis_add(uint64_t *by_bit, int np, const ElimShared &es) {
    const int lane = threadIdx.x & 31;
    const uint64_t a0 = by_bit[lane], b0 = by_bit[lane + 32];
    unsigned al = (unsigned)a0, ah = (unsigned)(a0 >> 32), bl = (unsigned)b0, bh = (unsigned)(b0 >> 32);
#pragma unroll 4
    for (int q = 0; q < np; q++) {
        const ulonglong2 p = es.pick[q];
        add_pick(al, ah, p);
        add_pick(bl, bh, p);
        if (((unsigned)p.y >> lane) & 1u) {
            al = (unsigned)p.x;
            ah = (unsigned)(p.x >> 32);
        }
        if (((unsigned)(p.y >> 32) >> lane) & 1u) {
            bl = (unsigned)p.x;
            bh = (unsigned)(p.x >> 32);
        }
    }
    by_bit[lane] = join64(al, ah);
    by_bit[lane + 32] = join64(bl, bh);
}

// The block's b iterations on masks, by one warp: lane l holds rows l and l + 32 of A
// (A[j][p] = <m_j, W_p>, m_j = e_j at the start, so A is the transpose of the W's).
// Iteration k: p_k = the first unused p with A[k][p] = 1; every later row j with
// A[j][p_k] = 1 takes row k (m_j ^= m_k, and A[j] ^= A[k] with it).  Rows i < k are
// final, so gcol[k] bit i = <C_sel_k, S_{e0+i}> = A[i][p_k] of the rows left in a0 / a1.
// psel: lane l, the pivots of iterations l and l + 32.  False if an iteration has none.
__device__ __forceinline__ bool resolve_rows(int b, uint64_t &a0, uint64_t &a1, uint64_t &m0, uint64_t &m1, int &psel0,
                                             int &psel1) {
    const int lane = threadIdx.x & 31;
    // The loop is one chain per iteration (fetch row k, its first unused pivot as a bit,
    // add it to the later rows with that bit), so it works on 32-bit halves and bits
    // instead of indices; the selections stay in the lane of their iteration and gcol
    // is read off the final rows afterwards.
    unsigned al0 = (unsigned)a0, ah0 = (unsigned)(a0 >> 32), al1 = (unsigned)a1, ah1 = (unsigned)(a1 >> 32);
    unsigned ml0 = 1u << lane, mh0 = 0, ml1 = 0, mh1 = 1u << lane;
    unsigned freel = 0xffffffffu, freeh = 0xffffffffu;  // pivots not selected yet
    unsigned sl0 = 0, sh0 = 0, sl1 = 0, sh1 = 0;        // lane l: the pivots (bits) of iterations l and l + 32
    bool fail = false;
    const int b0 = b < 32 ? b : 32;
    for (int k = 0; k < b0; k++) {
        const unsigned rl = __shfl_sync(0xffffffffu, al0, k), rh = __shfl_sync(0xffffffffu, ah0, k);
        const unsigned nl = __shfl_sync(0xffffffffu, ml0, k), nh = __shfl_sync(0xffffffffu, mh0, k);
        const unsigned cl = rl & freel, chh = rh & freeh;
        const unsigned bl = cl & (0u - cl), bh = cl ? 0u : chh & (0u - chh);
        if (!(bl | bh)) {  // warp-uniform
            fail = true;
            break;
        }
        freel &= ~bl;
        freeh &= ~bh;
        if (lane == k) {
            sl0 = bl;
            sh0 = bh;
        }
        if (lane > k && ((al0 & bl) | (ah0 & bh))) {
            al0 ^= rl;
            ah0 ^= rh;
            ml0 ^= nl;
            mh0 ^= nh;
        }
        if ((al1 & bl) | (ah1 & bh)) {
            al1 ^= rl;
            ah1 ^= rh;
            ml1 ^= nl;
            mh1 ^= nh;
        }
    }
    for (int k = 0; k < b - 32 && !fail; k++) {
        const unsigned rl = __shfl_sync(0xffffffffu, al1, k), rh = __shfl_sync(0xffffffffu, ah1, k);
        const unsigned nl = __shfl_sync(0xffffffffu, ml1, k), nh = __shfl_sync(0xffffffffu, mh1, k);
        const unsigned cl = rl & freel, chh = rh & freeh;
        const unsigned bl = cl & (0u - cl), bh = cl ? 0u : chh & (0u - chh);
        fail = !(bl | bh);  // warp-uniform
        freel &= ~bl;
        freeh &= ~bh;
        if (lane == k) {
            sl1 = bl;
            sh1 = bh;
        }
        if (lane > k && ((al1 & bl) | (ah1 & bh))) {
            al1 ^= rl;
            ah1 ^= rh;
            ml1 ^= nl;
            mh1 ^= nh;
        }
    }
    a0 = join64(al0, ah0);
    a1 = join64(al1, ah1);
    m0 = join64(ml0, mh0);
    m1 = join64(ml1, mh1);
    psel0 = __ffsll((long long)join64(sl0, sh0)) - 1;
    psel1 = __ffsll((long long)join64(sl1, sh1)) - 1;
    return !fail;
}

}  // namespace elim
}  // namespace mcbgpu
