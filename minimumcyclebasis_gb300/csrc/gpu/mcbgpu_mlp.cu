// The learned proposal's network: a two-layer perceptron over per-candidate
// features, with its inference and training on the device.
//
//   h     = relu(W1 x + b1)        x: 16 features (bf16), W1: 64 x 16 (bf16), b1: 64
//   logit = w2 . h + b2            w2: 64 (bf16-rounded), b2: scalar
//
// Master parameters are fp32 (kept with their Adam moments); the forward pass uses
// bf16 copies of W1 and w2 and accumulates in fp32.  The first layer of the forward
// pass is a tensor-core matrix product: per tile of 128 candidates, one
// tcgen05.mma (kind::f16, M = 128, N = 64, K = 16) with the feature tile and W1 in
// shared memory (no-swizzle K-major core-matrix layout) and the 128 x 64 fp32
// accumulator in tensor memory, read back with tcgen05.ld for the bias, the ReLU
// and the second layer.  A training batch is one kernel per batch: the same forward
// tile, then the backward pass (binary cross-entropy with a positive weight, mean over
// the batch) of the tile on the CUDA cores with the hidden layer in shared memory.
//
// The network orders candidates for the proposal (minimumcyclebasis_gb300.learned);
// it never decides a result: the solve that uses its proposal checks itself and
// falls back to the full candidate list.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "mcbgpu_internal.cuh"

namespace mcbgpu {
namespace mlp {

constexpr int kIn = 16, kHid = 64;
constexpr int kParams = kHid * kIn + kHid + kHid + 1;  // W1, b1, w2, b2
constexpr int kTileRows = 128;
constexpr int kFwdThreads = 128;
constexpr uint32_t kTmemCols = 64;

__device__ __forceinline__ uint16_t f32_to_bf16(float f) {
    // round to nearest even (finite inputs)
    uint32_t u = __float_as_uint(f);
    u += 0x7fffu + ((u >> 16) & 1u);
    return (uint16_t)(u >> 16);
}
__device__ __forceinline__ float bf16_to_f32(uint16_t h) { return __uint_as_float((uint32_t)h << 16); }

// ---- tcgen05 / TMEM wrappers --------------------------------------------------
__device__ __forceinline__ void tmem_alloc(uint32_t *dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst_smem)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// D[tmem] (+)= A[smem] x B[smem]^T, bf16 inputs, fp32 accumulator; one thread issues.
__device__ __forceinline__ void umma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on `bar` once every tcgen05.mma this thread issued has completed.
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}
// 32 consecutive fp32 columns of this thread's TMEM lane; tmem_wait_ld() before use.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// A 16-lane x 64-column fp32 tile as a matrix fragment: thread l holds, for each of the
// eight groups g of 8 columns, columns 8g + 2 (l mod 4) and the next of lanes l / 4
// (r[4g], r[4g + 1]) and l / 4 + 8 (r[4g + 2], r[4g + 3]).
__device__ __forceinline__ void tmem_ld16x64(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.16x256b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor, no swizzle: start address, the byte distance
// between core matrices (8 rows x 16 bytes) adjacent along K (leading) and along
// M/N (stride), and the descriptor version bit.
__device__ __forceinline__ uint64_t smem_desc(const void *p, uint32_t lead_bytes, uint32_t stride_bytes) {
    uint64_t d = (uint64_t)((smem_addr(p) >> 4) & 0x3fffu);
    d |= (uint64_t)((lead_bytes >> 4) & 0x3fffu) << 16;
    d |= (uint64_t)((stride_bytes >> 4) & 0x3fffu) << 32;
    d |= 1ull << 46;
    return d;
}
// Instruction descriptor of kind::f16: fp32 accumulator, bf16 A and B, both K-major,
// N = 64, M = 128.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kHid >> 3) << 17) |
                            ((uint32_t)(kTileRows >> 4) << 24);

// Byte offset of element (row, k) of a rows x 16 bf16 matrix in the core-matrix
// layout: 8-row groups 256 bytes apart, the two 8-element K halves 128 bytes apart.
__device__ __forceinline__ uint32_t core_off(int row, int k) {
    return (uint32_t)((row >> 3) * 256 + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2);
}
constexpr uint32_t kLead = 128, kStride = 256;

// W1 (64 x 16 bf16, row = hidden unit) into the core-matrix layout, and the second
// layer's constants: {b1[2i], b1[2i+1], w2[2i], w2[2i+1]}.
__device__ __forceinline__ void load_weights(unsigned char *sB, float4 *s_bw, const uint16_t *__restrict__ w1,
                                             const float *__restrict__ b1, const float *__restrict__ w2) {
    for (int e = threadIdx.x; e < kHid * kIn; e += blockDim.x)
        *reinterpret_cast<uint16_t *>(sB + core_off(e / kIn, e % kIn)) = w1[e];
    for (int i = threadIdx.x; i < kHid / 2; i += blockDim.x)
        s_bw[i] = make_float4(b1[2 * i], b1[2 * i + 1], w2[2 * i], w2[2 * i + 1]);
}

// Forward pass over `count` candidates: logits[i].  304 MB per 8.4M candidates is 45 us at
// the copy rate; the second layer's 192 operations per candidate are about as much.  A
// tile used to be one chain (stage, barrier, multiply, wait, four TMEM reads, epilogue
// with the weights read from shared memory): 132 us.  Now the next tile is staged while
// this one is multiplied, its product is issued as soon as the accumulator is read, and
// the epilogue has the weights in registers: the fragment
// form of the TMEM read gives a thread the same 16 hidden units of every candidate (with
// all 64 per thread the broadcast reads of the weights kept shared memory 75% busy: 127
// us).  About 100 us: the arithmetic pipes, two thirds busy, and the tile's chain.
// (Packed fp32 pairs, and two TMEM buffers with the product an iteration ahead, were no
// faster: moves between registers, fewer CTAs.)
constexpr int kFwdCtas = 5;  // per SM (4: the same time, 6: spills, 1.4 times); 64 TMEM columns each
__global__ void __launch_bounds__(kFwdThreads, kFwdCtas) mlp_forward_kernel(
    const uint16_t *__restrict__ x, int64_t count, const uint16_t *__restrict__ w1, const float *__restrict__ b1,
    const float *__restrict__ w2, const float *__restrict__ b2p, float *__restrict__ logits, unsigned *status) {
    __shared__ __align__(1024) unsigned char sA[2][kTileRows * kIn * 2];
    __shared__ __align__(1024) unsigned char sB[kHid * kIn * 2];
    __shared__ __align__(16) float4 s_bw[kHid / 2];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t s_tmem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t ntiles = (count + kTileRows - 1) / kTileRows;
    // this thread's row of a tile: 16 bf16 = two 16-byte halves, loaded a tile ahead of
    // its staging
    uint4 lo, hi;
    auto load_row = [&](int64_t t) {
        const int64_t r = t * kTileRows + tid;
        lo = make_uint4(0, 0, 0, 0);
        hi = lo;
        if (t < ntiles && r < count) {
            const uint4 *src = reinterpret_cast<const uint4 *>(x + r * kIn);
            lo = __ldcs(src);
            hi = __ldcs(src + 1);
        }
    };
    auto stage_row = [&](int b) {
        *reinterpret_cast<uint4 *>(sA[b] + core_off(tid, 0)) = lo;
        *reinterpret_cast<uint4 *>(sA[b] + core_off(tid, 8)) = hi;
        fence_proxy_async_smem();  // generic-proxy writes -> visible to the tensor core
    };
    // on its way while the weights are read (one tile per CTA, 60k candidates: 7.3 -> 6.6 us)
    load_row(blockIdx.x);
    const float b2 = *b2p;
    if (warp == 0) tmem_alloc(&s_tmem, kTmemCols);
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    load_weights(sB, s_bw, w1, b1, w2);
    stage_row(0);
    load_row((int64_t)blockIdx.x + gridDim.x);
    tc_fence_before();
    cta_sync();
    tc_fence_after();
    if (warp == 0) tmem_relinquish();
    const uint32_t tmem = s_tmem;
    const uint64_t bdesc = smem_desc(sB, kLead, kStride);
    float4 bw[8];  // this thread's hidden units: 8g + 2 (lane mod 4) and the next
#pragma unroll
    for (int g = 0; g < 8; g++) bw[g] = s_bw[4 * g + (lane & 3)];
    uint32_t phase = 0;
    bool ok = true;
    if (tid == 0) {  // gridDim.x <= ntiles: every CTA has a first tile
        umma_bf16(tmem, smem_desc(sA[0], kLead, kStride), bdesc, kIdesc, 0);
        umma_commit(&bar);
    }
    int buf = 0;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t next = tile + gridDim.x;
        // the other buffer's product completed a tile ago
        if (next < ntiles) stage_row(buf ^ 1);
        load_row(next + gridDim.x);
        ok = mbar_wait_bounded(&bar, phase, 1u << 22);
        phase ^= 1u;
        __syncwarp();  // lanes leave the polls one by one; the aligned read wants the warp whole
        tc_fence_after();
        float z[4];  // candidates 32 warp + 8 i + lane / 4: the part of this thread's hidden units
        uint32_t acc[32];
        auto half = [&](int h) {
#pragma unroll
            for (int q = 0; q < 2; q++) {
                float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
                for (int g = 0; g < 8; g++) {
                    s0 = fmaf(bw[g].z, fmaxf(__uint_as_float(acc[4 * g + 2 * q]) + bw[g].x, 0.0f), s0);
                    s1 = fmaf(bw[g].w, fmaxf(__uint_as_float(acc[4 * g + 2 * q + 1]) + bw[g].y, 0.0f), s1);
                }
                z[2 * h + q] = s0 + s1;
            }
        };
        const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16);
        tmem_ld16x64(taddr, acc);
        tmem_wait_ld();
        half(0);
        tmem_ld16x64(taddr + (16u << 16), acc);
        tmem_wait_ld();
        tc_fence_before();
        ok = cta_sync_and(ok);  // the next tile is staged, this one's accumulator read
        if (!ok) break;
        if (tid == 0 && next < ntiles) {
            tc_fence_after();
            umma_bf16(tmem, smem_desc(sA[buf ^ 1], kLead, kStride), bdesc, kIdesc, 0);
            umma_commit(&bar);
        }
        half(1);
        // sum over the four threads of a candidate; thread i of them keeps candidate set i
        float k0 = (lane & 1) ? z[1] : z[0], k1 = (lane & 1) ? z[3] : z[2];
        k0 += __shfl_xor_sync(0xffffffffu, (lane & 1) ? z[0] : z[1], 1);
        k1 += __shfl_xor_sync(0xffffffffu, (lane & 1) ? z[2] : z[3], 1);
        const float sent = __shfl_xor_sync(0xffffffffu, (lane & 2) ? k0 : k1, 2);
        const int64_t row = tile * kTileRows + warp * 32 + 8 * (lane & 3) + (lane >> 2);
        if (row < count) __stcs(logits + row, b2 + (((lane & 2) ? k1 : k0) + sent));
        buf ^= 1;
    }
    if (!ok) {
        if (tid == 0) {
            atomicOr(status, ST_WAIT_TIMEOUT);
            mbar_wait_bounded(&bar, phase ^ 1u, 1u << 22);  // the MMA in flight, if any
        }
    }
    tc_fence_before();
    cta_sync();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

__device__ __forceinline__ float softplus(float z) { return fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z))); }

// Gradients of the mean weighted binary cross-entropy over `count` candidates into
// grads (kParams floats, accumulated with atomics) and the loss sum into *loss.
// Per tile of 128 candidates: the forward product, the epilogue by eight warps (each
// half of the hidden units of 32 candidates) into shared memory, then thread (s, j) adds
// hidden unit j's gradients of 32 candidates.  The hidden layer (fp32) never leaves the
// SM.  Batch of 16,384: forward and a backward that read one candidate per 64 threads
// and step from global memory took 36 us, this 9.4 us.
constexpr int kGradThreads = 256;
constexpr int kGradGroups = kGradThreads / kHid;            // candidates' groups of a tile
constexpr int kGradRows = kTileRows / kGradGroups;          // candidates per group
__global__ void __launch_bounds__(kGradThreads) mlp_grads_kernel(const uint16_t *__restrict__ x,
                                                                 const uint8_t *__restrict__ labels, int64_t count,
                                                                 float pos_weight, const uint16_t *__restrict__ w1,
                                                                 const float *__restrict__ b1,
                                                                 const float *__restrict__ w2,
                                                                 const float *__restrict__ b2p, float *grads, float *loss,
                                                                 unsigned *status) {
    __shared__ __align__(1024) unsigned char sA[kTileRows * kIn * 2];
    __shared__ __align__(1024) unsigned char sB[kHid * kIn * 2];
    __shared__ __align__(16) float4 s_bw[kHid / 2];
    __shared__ __align__(16) float s_h[kTileRows * (kHid + 1)];  // the hidden layer; at the end the sums
    __shared__ float s_z[2][kTileRows], s_dz[kTileRows], s_misc[kTileRows / 32][2];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t s_tmem;
    static_assert(kGradGroups * kHid * (kIn + 2) <= kTileRows * (kHid + 1), "the sums fit s_h");
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) tmem_alloc(&s_tmem, kTmemCols);
    if (tid == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    load_weights(sB, s_bw, w1, b1, w2);
    tc_fence_before();
    cta_sync();
    tc_fence_after();
    if (warp == 0) tmem_relinquish();
    const uint32_t tmem = s_tmem;
    const float b2 = *b2p, inv = 1.0f / (float)count;
    const int j = tid % kHid, s = tid / kHid;
    const float w2j = w2[j];
    float gw1[kIn];
#pragma unroll
    for (int i = 0; i < kIn; i++) gw1[i] = 0.0f;
    float gb1 = 0.0f, gw2 = 0.0f, gb2 = 0.0f, lsum = 0.0f;
    const int64_t ntiles = (count + kTileRows - 1) / kTileRows;
    uint32_t phase = 0;
    bool ok = true;
    for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int64_t row = tile * kTileRows + (tid & (kTileRows - 1));
        {  // two threads per candidate, 16 bytes each
            const int half = tid / kTileRows;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (row < count) v = __ldg(reinterpret_cast<const uint4 *>(x + row * kIn) + half);
            *reinterpret_cast<uint4 *>(sA + core_off(tid & (kTileRows - 1), 8 * half)) = v;
        }
        const int y = row < count ? labels[row] : 0;
        fence_proxy_async_smem();
        tc_fence_before();
        cta_sync();
        if (tid == 0) {
            tc_fence_after();
            umma_bf16(tmem, smem_desc(sA, kLead, kStride), smem_desc(sB, kLead, kStride), kIdesc, 0);
            umma_commit(&bar);
        }
        ok = mbar_wait_bounded(&bar, phase, 1u << 22);
        phase ^= 1u;
        ok = cta_sync_and(ok);
        if (!ok) break;
        tc_fence_after();
        {  // warp w: candidates 32 (w mod 4) .., hidden units 32 (w / 4) ..
            const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 32;
            uint32_t acc[32];
            tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0, acc);
            tmem_wait_ld();
            tc_fence_before();
            float s0 = 0.0f, s1 = 0.0f;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const float4 bw = s_bw[c0 / 2 + i];
                const float h0 = fmaxf(__uint_as_float(acc[2 * i]) + bw.x, 0.0f);
                const float h1 = fmaxf(__uint_as_float(acc[2 * i + 1]) + bw.y, 0.0f);
                s_h[r * (kHid + 1) + c0 + 2 * i] = h0;
                s_h[r * (kHid + 1) + c0 + 2 * i + 1] = h1;
                s0 = fmaf(bw.z, h0, s0);
                s1 = fmaf(bw.w, h1, s1);
            }
            s_z[warp >> 2][r] = s0 + s1;
        }
        cta_sync();
        if (tid < kTileRows) {
            const float z = b2 + (s_z[0][tid] + s_z[1][tid]);
            float dz = 0.0f;
            if (row < count) {
                const float wt = y ? pos_weight : 1.0f;
                const float sg = 1.0f / (1.0f + expf(-z));
                dz = (sg - (y ? 1.0f : 0.0f)) * wt * inv;
                gb2 += dz;
                lsum += wt * (y ? softplus(-z) : softplus(z));
            }
            s_dz[tid] = dz;
        }
        cta_sync();
#pragma unroll 4
        for (int i = 0; i < kGradRows; i++) {
            const int r = s * kGradRows + i;
            const float h = s_h[r * (kHid + 1) + j], dz = s_dz[r];
            gw2 = fmaf(dz, h, gw2);
            const float dh = h > 0.0f ? dz * w2j : 0.0f;
            gb1 += dh;
            uint32_t xv[8];
            *reinterpret_cast<uint4 *>(xv) = *reinterpret_cast<const uint4 *>(sA + core_off(r, 0));
            *reinterpret_cast<uint4 *>(xv + 4) = *reinterpret_cast<const uint4 *>(sA + core_off(r, 8));
#pragma unroll
            for (int q = 0; q < 8; q++) {
                gw1[2 * q] = fmaf(dh, __uint_as_float(xv[q] << 16), gw1[2 * q]);
                gw1[2 * q + 1] = fmaf(dh, __uint_as_float(xv[q] & 0xffff0000u), gw1[2 * q + 1]);
            }
        }
        cta_sync();  // the tile's candidates and hidden layer are overwritten by the next
    }
    if (ok) {
        // sum over the groups of each hidden unit in shared memory, then one atomic per
        // parameter and CTA
        float(*s_red)[kHid][kIn + 2] = reinterpret_cast<float(*)[kHid][kIn + 2]>(s_h);
#pragma unroll
        for (int i = 0; i < kIn; i++) s_red[s][j][i] = gw1[i];
        s_red[s][j][kIn] = gb1;
        s_red[s][j][kIn + 1] = gw2;
        for (int d = 16; d > 0; d >>= 1) {
            gb2 += __shfl_xor_sync(0xffffffffu, gb2, d);
            lsum += __shfl_xor_sync(0xffffffffu, lsum, d);
        }
        if (lane == 0 && warp < kTileRows / 32) {
            s_misc[warp][0] = gb2;
            s_misc[warp][1] = lsum;
        }
        cta_sync();
        for (int e = tid; e < kHid * (kIn + 2); e += kGradThreads) {
            const int u = e / (kIn + 2), i = e % (kIn + 2);
            float v = 0.0f;
            for (int k = 0; k < kGradGroups; k++) v += s_red[k][u][i];
            const int at = i < kIn ? u * kIn + i : i == kIn ? kHid * kIn + u : kHid * kIn + kHid + u;
            atomicAdd(&grads[at], v);
        }
        if (tid == 0) {
            float a = 0, l = 0;
            for (int k = 0; k < kTileRows / 32; k++) {
                a += s_misc[k][0];
                l += s_misc[k][1];
            }
            atomicAdd(&grads[kParams - 1], a);
            atomicAdd(loss, l);
        }
    } else if (tid == 0) {
        atomicOr(status, ST_WAIT_TIMEOUT);
        mbar_wait_bounded(&bar, phase ^ 1u, 1u << 22);  // the MMA in flight, if any
    }
    tc_fence_before();
    cta_sync();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, kTmemCols);
}

// The forward pass's weight copies: bf16 W1 and bf16-rounded w2 from the masters.
__global__ void mlp_weights_kernel(const float *params, uint16_t *w1_bf16, float *w2_round) {
    for (int e = threadIdx.x; e < kHid * kIn; e += blockDim.x) w1_bf16[e] = f32_to_bf16(params[e]);
    for (int j = threadIdx.x; j < kHid; j += blockDim.x)
        w2_round[j] = bf16_to_f32(f32_to_bf16(params[kHid * kIn + kHid + j]));
}

// One Adam step on every parameter, then the bf16 copies refreshed.
__global__ void mlp_adam_kernel(float *params, const float *grads, float *m1, float *m2, float lr, float beta1,
                                float beta2, float eps, float c1, float c2, uint16_t *w1_bf16, float *w2_round) {
    for (int e = threadIdx.x; e < kParams; e += blockDim.x) {
        const float g = grads[e];
        const float a = beta1 * m1[e] + (1.0f - beta1) * g;
        const float b = beta2 * m2[e] + (1.0f - beta2) * g * g;
        m1[e] = a;
        m2[e] = b;
        params[e] -= lr * (a / c1) / (sqrtf(b / c2) + eps);
    }
    cta_sync();
    for (int e = threadIdx.x; e < kHid * kIn; e += blockDim.x) w1_bf16[e] = f32_to_bf16(params[e]);
    for (int j = threadIdx.x; j < kHid; j += blockDim.x)
        w2_round[j] = bf16_to_f32(f32_to_bf16(params[kHid * kIn + kHid + j]));
}

}  // namespace mlp
}  // namespace mcbgpu

using namespace mcbgpu;
using namespace mcbgpu::mlp;

struct mcbgpu_mlp {
    float *d_params = nullptr, *d_m1 = nullptr, *d_m2 = nullptr, *d_w2r = nullptr;
    uint16_t *d_w1 = nullptr;
    // one block, read back with one copy: gradients | loss | status word
    float *d_grads = nullptr;
    float *d_loss = nullptr;
    unsigned *d_status = nullptr;
    float *h_out = nullptr;  // its pinned host copy
    int64_t steps = 0;
    int sm_count = 0;
};
constexpr int kOutWords = kParams + 2;

static void mlp_free(mcbgpu_mlp *m) {
    void *ps[] = {m->d_params, m->d_grads, m->d_m1, m->d_m2, m->d_w2r, m->d_w1};
    for (void *p : ps) cudaFree(p);
    if (m->h_out) cudaFreeHost(m->h_out);
    delete m;
}

// Reads back the last `words` words of the output block (the status word is the last)
// and waits for them; a status is reported and cleared.
static int mlp_read_back(mcbgpu_mlp *m, int words, cudaStream_t st, const char *what) {
    const int at = kOutWords - words;
    MCB_CUDA(cudaMemcpyAsync(m->h_out + at, m->d_grads + at, sizeof(float) * (size_t)words, cudaMemcpyDeviceToHost, st));
    MCB_CUDA(cudaStreamSynchronize(st));
    unsigned h = 0;
    std::memcpy(&h, m->h_out + kOutWords - 1, sizeof h);
    if (h) {
        MCB_CUDA(cudaMemsetAsync(m->d_status, 0, sizeof h, st));
        set_error("%s: device status 0x%x", what, h);
        return MCBGPU_E_DEVICE;
    }
    return MCBGPU_OK;
}

// The batch's gradients and loss sum into the output block.
static int mlp_grads(mcbgpu_mlp *m, const uint16_t *x, const uint8_t *labels, int64_t count, float pos_weight,
                     cudaStream_t st) {
    MCB_CUDA(cudaMemsetAsync(m->d_grads, 0, sizeof(float) * (kParams + 1), st));
    const int64_t tiles = (count + kTileRows - 1) / kTileRows;
    const int grid = (int)std::min<int64_t>(tiles, (int64_t)(m->sm_count > 0 ? m->sm_count : 148) * 2);
    mlp_grads_kernel<<<grid, kGradThreads, 0, st>>>(x, labels, count, pos_weight, m->d_w1, m->d_params + kHid * kIn,
                                                    m->d_w2r, m->d_params + kParams - 1, m->d_grads, m->d_loss,
                                                    m->d_status);
    MCB_CUDA(cudaGetLastError());
    return MCBGPU_OK;
}

extern "C" {

int mcbgpu_mlp_param_count(void) { return kParams; }

int mcbgpu_mlp_create(mcbgpu_mlp **out, const float *params) {
    if (!out || !params) {
        set_error("mcbgpu_mlp_create: NULL argument");
        return MCBGPU_E_ARG;
    }
    *out = nullptr;
    mcbgpu_mlp *m = new mcbgpu_mlp();
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&m->sm_count, cudaDevAttrMultiProcessorCount, dev);
    const size_t pb = sizeof(float) * kParams;
    if (e == cudaSuccess) e = cudaMalloc((void **)&m->d_params, pb);
    if (e == cudaSuccess) e = cudaMalloc((void **)&m->d_grads, sizeof(float) * kOutWords);
    if (e == cudaSuccess) e = cudaMallocHost((void **)&m->h_out, sizeof(float) * kOutWords);
    if (e == cudaSuccess) e = cudaMalloc((void **)&m->d_m1, pb);
    if (e == cudaSuccess) e = cudaMalloc((void **)&m->d_m2, pb);
    if (e == cudaSuccess) e = cudaMalloc((void **)&m->d_w2r, sizeof(float) * kHid);
    if (e == cudaSuccess) e = cudaMalloc((void **)&m->d_w1, sizeof(uint16_t) * kHid * kIn);
    m->d_loss = m->d_grads + kParams;
    m->d_status = reinterpret_cast<unsigned *>(m->d_grads + kParams + 1);
    if (e == cudaSuccess) e = cudaMemcpy(m->d_params, params, pb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(m->d_grads, 0, sizeof(float) * kOutWords);
    if (e == cudaSuccess) e = cudaMemset(m->d_m1, 0, pb);
    if (e == cudaSuccess) e = cudaMemset(m->d_m2, 0, pb);
    if (e == cudaSuccess) {
        mlp_weights_kernel<<<1, 256>>>(m->d_params, m->d_w1, m->d_w2r);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
        mlp_free(m);
        return cuda_fail(e, "mcbgpu_mlp_create");
    }
    *out = m;
    return MCBGPU_OK;
}

int mcbgpu_mlp_get_params(const mcbgpu_mlp *m, float *params) {
    if (!m || !params) {
        set_error("mcbgpu_mlp_get_params: NULL argument");
        return MCBGPU_E_ARG;
    }
    MCB_CUDA(cudaMemcpy(params, m->d_params, sizeof(float) * kParams, cudaMemcpyDeviceToHost));
    return MCBGPU_OK;
}

int mcbgpu_mlp_forward(mcbgpu_mlp *m, const uint16_t *x, int64_t count, float *logits, void *stream) {
    if (!m || count < 0 || (count > 0 && (!x || !logits))) {
        set_error("mcbgpu_mlp_forward: invalid arguments");
        return MCBGPU_E_ARG;
    }
    cudaStream_t st = (cudaStream_t)stream;
    if (count > 0) {
        const int64_t tiles = (count + kTileRows - 1) / kTileRows;
        const int grid = (int)std::min<int64_t>(tiles, (int64_t)(m->sm_count > 0 ? m->sm_count : 148) * kFwdCtas);
        mlp_forward_kernel<<<grid, kFwdThreads, 0, st>>>(x, count, m->d_w1, m->d_params + kHid * kIn, m->d_w2r,
                                                         m->d_params + kParams - 1, logits, m->d_status);
        MCB_CUDA(cudaGetLastError());
    }
    return mlp_read_back(m, 1, st, "mcbgpu_mlp_forward");
}

int mcbgpu_mlp_gradients(mcbgpu_mlp *m, const uint16_t *x, const uint8_t *labels, int64_t count, float pos_weight,
                         float *grads, float *loss, void *stream) {
    if (!m || count <= 0 || !x || !labels || !grads || !loss || !(pos_weight > 0.0f)) {
        set_error("mcbgpu_mlp_gradients: invalid arguments");
        return MCBGPU_E_ARG;
    }
    cudaStream_t st = (cudaStream_t)stream;
    int rc = mlp_grads(m, x, labels, count, pos_weight, st);
    if (rc) return rc;
    rc = mlp_read_back(m, kOutWords, st, "mcbgpu_mlp_gradients");
    std::memcpy(grads, m->h_out, sizeof(float) * kParams);
    *loss = m->h_out[kParams] / (float)count;
    return rc;
}

int mcbgpu_mlp_train_step(mcbgpu_mlp *m, const uint16_t *x, const uint8_t *labels, int64_t count, float pos_weight,
                          float lr, float *loss, void *stream) {
    if (!m || count <= 0 || !x || !labels || !(pos_weight > 0.0f) || !(lr > 0.0f)) {
        set_error("mcbgpu_mlp_train_step: invalid arguments");
        return MCBGPU_E_ARG;
    }
    cudaStream_t st = (cudaStream_t)stream;
    int rc = mlp_grads(m, x, labels, count, pos_weight, st);
    if (rc) return rc;
    m->steps++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.0f - powf(b1, (float)m->steps), c2 = 1.0f - powf(b2, (float)m->steps);
    mlp_adam_kernel<<<1, 256, 0, st>>>(m->d_params, m->d_grads, m->d_m1, m->d_m2, lr, b1, b2, 1e-8f, c1, c2, m->d_w1,
                                       m->d_w2r);
    MCB_CUDA(cudaGetLastError());
    if (loss) {
        rc = mlp_read_back(m, 2, st, "mcbgpu_mlp_train_step");
        *loss = m->h_out[kParams] / (float)count;
        return rc;
    }
    return MCBGPU_OK;
}

int mcbgpu_mlp_destroy(mcbgpu_mlp *m) {
    if (m) mlp_free(m);
    return MCBGPU_OK;
}

}  // extern "C"
