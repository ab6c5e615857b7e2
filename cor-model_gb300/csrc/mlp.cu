// mlp.cu -- the learned rigidity window's network (include/cor_window.h): a
// BF16 MLP whose every matrix product runs on the 5th-generation tensor cores.
//
// rows_kernel takes 128 rows of the batch through the whole network in one
// launch, by a cluster of four CTAs with a quarter of every hidden layer's
// columns each (or by one CTA, beside a scan stream: device_share.h): the
// activations stay in the shared memories from layer to layer, and the weights
// stream through a ring of shared-memory stages (a 64-deep K block of a CTA's
// columns, 8 KB, per cp.async.bulk).  For a training step it
// goes on through the loss and back through the layers (dZ of every layer), and
// leaves what the weight gradients need in global memory.  grad_kernel then
// takes the weight gradients (one CTA per 128 x 64 tile, K = the batch) and
// applies AdamW to its tile in the epilogue.
//
// Products: C[M][N] = A[M][K] . B[N][K]^T with A, B BF16 and K-major, C FP32 in
// tensor memory, one tcgen05.mma (M = 128, N up to 256, K = 16) per K slice.
// Operand tiles sit in shared memory in the no-swizzle K-major core-matrix
// layout (8 rows x 16 bytes per core matrix; LBO = 128 B between core matrices
// along K, SBO = 1024 B between 8-row groups), and everything a product reads
// from global memory is stored that way, K block by K block (`packed`), so a
// stage is one contiguous copy.  Transposed copies (for dW = dZ^T . X) come out
// of shared memory through ldmatrix.trans, core matrix by core matrix.
//
// Warps 0-15 are rows_kernel's epilogue (warp w owns rows 32 (w % 4) .. and
// columns 16 (w / 4) .. of the accumulator), warp 16 feeds the ring, warp 17
// issues the MMAs, warp 18 sends the CTA's columns to its peers.  Waits are
// bounded (about 2 s of SM clock); a wait that runs out sets the error word, every
// role leaves its loop, and the tile waits out what it issued and frees the TMEM.
//
// Measured: 2,664 rows forward 405 -> 43 us a call (kernel 22 us); a training
// step of 512 rows, its loss read back, 1,150 -> 113 us (rows_kernel 49,
// grad_kernel 16 us).  By one CTA to a tile 61 and 186 us, and 0.44 and 0.46 ms on
// the two SMs that a scan stream leaves.  One
// GEMM per launch had spent its time in synchronous stages (load, fence, MMA,
// wait: 5 to 7 us each), in epilogues that wrote rows with a stride, and in 25
// launches a step.  One CTA per 128 rows (without the cluster) took 38 and 111
// us: the SiLU of 128 x 256 elements alone is 3 us of issue slots a layer.  What
// bounds it now is the chain of the layers, about 4 us each way and layer: MMA,
// accumulator read, SiLU, exchange.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <math.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include "cor_trace.h"
#include "cor_window.h"
#include "device_share.h"
#include "mlp_schedule.h"

namespace mlp {

typedef __nv_bfloat16 bf16;

constexpr int kBM = 128;
constexpr int kBK = 64;
constexpr int kInPad = 64;      // 19 input features, zero-padded to one K block
constexpr int kOutPad = 16;     // 2 outputs, padded to the smallest N
constexpr int kH = COR_MLP_HIDDEN;
constexpr int kLayers = COR_MLP_LAYERS + 1;   // 5 weight matrices
constexpr long long kWaitCycles = 4000000000ll;

// Bytes of one K block of a packed matrix with `rows` rows.
__host__ __device__ constexpr uint32_t block_bytes(int rows) { return (uint32_t)rows * kBK * 2; }

// Byte offset of element (r, k) in a packed matrix with `rows` rows.
__host__ __device__ constexpr size_t packed_at(int rows, int r, int k) {
    return (size_t)(k / kBK) * rows * kBK * 2 + (size_t)(r >> 3) * 1024 + (size_t)((k % kBK) >> 3) * 128 + (r & 7) * 16 +
           (k & 7) * 2;
}

// ---- the weight stream of rows_kernel ------------------------------------------
__host__ __device__ constexpr int product_n(int p) { return p == 4 ? kOutPad : kH; }
__host__ __device__ constexpr size_t product_bytes(int p) { return (size_t)product_blocks(p) * block_bytes(product_n(p)); }
__host__ __device__ constexpr size_t product_offset(int p) {
    size_t o = 0;
    for (int i = 0; i < p; i++) o += product_bytes(i);
    return o;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor (tcgen05 "matrix descriptor"): start
// address, leading and stride byte offsets in 16-byte units, version 1,
// no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}

// instruction descriptor of kind::f16: D FP32, A and B BF16, both K-major.
__host__ __device__ constexpr uint32_t instr_desc(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
    const uint32_t a = smem_u32(bar);
    const long long t0 = clock64();
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
        if (clock64() - t0 > kWaitCycles) return false;
    }
}

// After a wait that ran out: copies and products that were issued and that
// nobody waits for any more end within microseconds.
constexpr long long kSettleCycles = 20000000ll;   // about 10 ms
__device__ __forceinline__ void settle() {
    const long long t0 = clock64();
    while (clock64() - t0 < kSettleCycles) {}
}

__device__ __forceinline__ float silu(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float silu_grad(float z) {
    const float s = 1.f / (1.f + expf(-z));
    return s * (1.f + z * (1.f - s));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
// One contiguous copy into shared memory (16-byte aligned, a multiple of 16 bytes).
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void commit_to(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// The four K = 16 products of one K block: A 128 rows at a0, B N rows at b0.
__device__ __forceinline__ void mma_block(uint32_t tmem, uint32_t a0, uint32_t b0, uint32_t idesc, bool first) {
#pragma unroll
    for (int s = 0; s < kBK / 16; s++) {
        const uint64_t ad = smem_desc(a0 + s * 256, 128, 1024);
        const uint64_t bd = smem_desc(b0 + s * 256, 128, 1024);
        const uint32_t acc = (!first || s > 0) ? 1u : 0u;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
            "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
    }
}

__device__ __forceinline__ void tmem_ld16(float* v, uint32_t taddr) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
        "[%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    return (uint32_t)__bfloat16_as_ushort(__float2bfloat16(a)) |
           ((uint32_t)__bfloat16_as_ushort(__float2bfloat16(b)) << 16);
}

// 16 values of one row, as BF16, to columns c0 .. c0+15 of a K block in shared memory.
__device__ __forceinline__ void put_row16(uint8_t* block, int row, int c0, const float* v) {
    uint32_t w[8];
#pragma unroll
    for (int i = 0; i < 8; i++) w[i] = pack_bf16(v[2 * i], v[2 * i + 1]);
    uint8_t* d = block + (row >> 3) * 1024 + (c0 >> 3) * 128 + (row & 7) * 16;
    *reinterpret_cast<uint4*>(d) = make_uint4(w[0], w[1], w[2], w[3]);
    *reinterpret_cast<uint4*>(d + 128) = make_uint4(w[4], w[5], w[6], w[7]);
}

// The transpose of this warp's 32 rows (quadrant q of the tile) and `cols`
// columns of a K block in shared memory, to the packed matrix [feature][batch]
// at `dst` with R features: features f0 .., batch b0 ...
__device__ __forceinline__ void put_transposed(uint8_t* dst, int R, int f0, int b0, const uint8_t* block, int q, int cols) {
    const int lane = threadIdx.x & 31;
    for (int c8 = 0; c8 < cols / 8; c8++) {
        // four core matrices: rows 32q .. 32q+31 of columns 8 c8 ..
        const uint32_t a = smem_u32(block + (4 * q + (lane >> 3)) * 1024 + c8 * 128 + (lane & 7) * 16);
        uint32_t r[4];
        asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(a)
                     : "memory");
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int b = b0 + 32 * q + 8 * k;
            *reinterpret_cast<uint32_t*>(dst + packed_at(R, f0 + 8 * c8, b) + lane * 4) = r[k];
        }
    }
}

constexpr int kEpiWarps = 16, kRowsThreads = 32 * (kEpiWarps + 3);
constexpr uint32_t kABlock = block_bytes(kBM);

// The two forms of rows_kernel: a tile of 128 rows by a cluster of four CTAs,
// with 64 columns of every hidden layer each, or by one.
template <int SPLIT>
struct Form {
    static constexpr int kOwn = kBlocks / SPLIT;   // K blocks of a hidden layer that a CTA computes
    static constexpr int kCols = kH / SPLIT;
    static constexpr int kSets = a_sets(SPLIT);
    static constexpr int kRing = SPLIT == 1 ? 4 : 8;
    static constexpr uint32_t kStage = block_bytes(kCols);
    static constexpr size_t kSmem = 1024 + (kSets * kBlocks + 1) * kABlock + kRing * kStage;
};
constexpr int kSplit = 4;
constexpr int kMaxRing = 8;

struct RowsArgs {
    const float* x;          // n x 19
    const float* target;     // n x 2 (training)
    int n;
    float* y;                // n x 2 (inference)
    const uint8_t* weights;  // the weight stream
    const float* bias[kLayers];
    // training
    float* z[COR_MLP_LAYERS];       // [tile][column][row]
    uint8_t* x0t;                   // packed [64][bt]
    uint8_t* ht[COR_MLP_LAYERS];    // packed [256][bt]
    uint8_t* dzt[COR_MLP_LAYERS];   // packed [256][bt]
    uint8_t* dyt;                   // packed [16][bt]
    float* gb[kLayers];             // bias gradients, zero at launch
    float* loss;                    // zero at launch
    int* err;
};

struct RowsShared {
    uint64_t full[kMaxRing], empty[kMaxRing], acc;
    uint64_t local;              // the single K block that this CTA fills itself (input, dY)
    // K block b of exchange x, in set x % kSets: this CTA's own written, or a
    // peer's copy landed.  As many sets as buffers: a peer sends x + 2 only
    // after this CTA has taken x, but it may send x + 1 before.
    uint64_t kready[2][kBlocks];
    uint32_t tmem;
    uint32_t failed;             // a CTA of the tile gave up
};
static_assert(sizeof(RowsShared) <= 1024, "rows_kernel header");

// Address of this CTA's shared-memory address `a` in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t peer_addr(uint32_t a, int rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}

// A barrier of the CTAs of one tile.
template <int SPLIT>
__device__ __forceinline__ void tile_sync() {
    if constexpr (SPLIT > 1)
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else
        __syncthreads();
}

// A cluster of four CTAs takes one tile of 128 rows: CTA r computes columns
// 64 r .. 64 r + 63 of every hidden layer, which are K block r of the next
// product's A, and copies them to its three peers' shared memory.  An epilogue
// of 128 x 64 elements by 16 warps takes a quarter of what the whole width
// does, and a weight block is a quarter of the size.  A has two buffers: a
// peer that writes exchange x has read exchange x - 1 of this CTA, which it
// sent after its products had read x - 2.  There is one accumulator: a product
// begins when this CTA's own blocks are complete, so its epilogue has read the
// product before (waits_for; tests/test_network_order.py checks both).
//
// SPLIT = 1: one CTA takes a tile alone, the same sums in the same order (the
// bits are the same), on any one SM.  A cluster needs four whole SMs of one GPC
// at a time, which a device that a scan stream holds does not have
// (device_share.h).
template <int SPLIT, bool TRAIN>
__global__ void __cluster_dims__(SPLIT, 1, 1) __launch_bounds__(kRowsThreads, 1) rows_kernel(const RowsArgs g) {
    using F = Form<SPLIT>;
    constexpr int kRing = F::kRing, kSets = F::kSets;
    extern __shared__ __align__(1024) uint8_t smem[];
    RowsShared& sh = *reinterpret_cast<RowsShared*>(smem);
    uint8_t* abuf = smem + 1024;                          // kSets x 4 K blocks
    uint8_t* single = abuf + kSets * kBlocks * kABlock;   // 1 K block
    uint8_t* ring = single + kABlock;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x % SPLIT, tile = blockIdx.x / SPLIT;
    const int m0 = tile * kBM;
    constexpr int kLast = TRAIN ? kProducts : kFwdProducts;
    constexpr uint32_t kCols = F::kCols;

    if (threadIdx.x == 0) {
        for (int k = 0; k < kRing; k++) {
            mbar_init(&sh.full[k], 1);
            mbar_init(&sh.empty[k], 1);
        }
        mbar_init(&sh.acc, 1);
        mbar_init(&sh.local, 32 * kEpiWarps);
        sh.failed = 0;
        for (int i = 0; i < kSets; i++)
            for (int b = 0; b < kBlocks; b++)
                mbar_init(&sh.kready[i][b], block_owner(SPLIT, b) == rank ? 32 * kEpiWarps : 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem)),
                     "r"(kCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    // every CTA's barriers are set up before a peer's copy can arrive
    tile_sync<SPLIT>();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh.tmem;
    bool ok = true;

    if (warp == kEpiWarps) {
        if (lane == 0) {
            int s = 0;
            for (int p = 0; p < kLast && ok; p++) {
                // the output layer's 16 rows go to every CTA; else this CTA's rows
                const uint32_t bytes = p == 4 ? block_bytes(kOutPad) : F::kStage;
                const uint8_t* src = g.weights + product_offset(p) + (p == 4 ? 0 : rank * F::kStage);
                for (int kb = 0; kb < product_blocks(p) && ok; kb++, s++) {
                    const int k = s % kRing;
                    if (s >= kRing) ok = mbar_wait(&sh.empty[k], (uint32_t)((s / kRing - 1) & 1));
                    if (!ok) break;
                    mbar_expect(&sh.full[k], bytes);
                    bulk_load(ring + k * F::kStage, src + (size_t)kb * block_bytes(product_n(p)), bytes, &sh.full[k]);
                }
            }
            if (!ok) {
                atomicExch(g.err, 1);
                // the copies in flight land before the block leaves
                for (int i = s > kRing ? s - kRing : 0; i < s; i++)
                    mbar_wait(&sh.full[i % kRing], (uint32_t)((i / kRing) & 1));
            }
        }
    } else if (warp == kEpiWarps + 1) {
        if (lane == 0) {
            int s = 0;
            for (int p = 0; p < kLast && ok; p++) {
                const uint32_t idesc = instr_desc(kBM, p == 4 ? kOutPad : F::kCols);
                const int x = exchange_into(p);
                if (x < 0) {
                    ok = mbar_wait(&sh.local, (uint32_t)(p == 5));
                } else {
                    for (int b = 0; b < kBlocks; b++)
                        if (block_owner(SPLIT, b) != rank) mbar_expect(&sh.kready[x % kSets][b], kABlock);
                }
                const uint8_t* a = x < 0 ? single : abuf + (x % kSets) * kBlocks * kABlock;
                for (int kb = 0; kb < product_blocks(p) && ok; kb++, s++) {
                    const int k = s % kRing;
                    for (int b = 0; x >= 0 && b < kBlocks && ok; b++)
                        if (waits_for(SPLIT, rank, kb, b))
                            ok = mbar_wait(&sh.kready[x % kSets][b], (uint32_t)((x / kSets) & 1));
                    ok = ok && mbar_wait(&sh.full[k], (uint32_t)((s / kRing) & 1));
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    mma_block(tmem, smem_u32(a + kb * kABlock), smem_u32(ring + k * F::kStage), idesc, kb == 0);
                    commit_to(&sh.empty[k]);
                }
                if (ok) commit_to(&sh.acc);
            }
            if (!ok) atomicExch(g.err, 1);
        }
    } else if (warp == kEpiWarps + 2) {
        if (SPLIT > 1 && lane == 0) {
            static_assert(SPLIT == 1 || F::kOwn == 1, "one block to send");
            // this CTA's K block to its peers
            for (int p = 0; p + 1 < kLast && ok; p++) {
                if (p == 4) continue;
                const int x = exchange_out(p);
                ok = mbar_wait(&sh.kready[x % kSets][rank], (uint32_t)((x / kSets) & 1));
                if (!ok) break;
                const uint32_t a = smem_u32(abuf + ((x % kSets) * kBlocks + rank) * kABlock);
                for (int i = 1; i < SPLIT; i++) {
                    const int r = (rank + i) % SPLIT;
                    asm volatile(
                        "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                            peer_addr(a, r)),
                        "r"(a), "r"(kABlock), "r"(peer_addr(smem_u32(&sh.kready[x % kSets][rank]), r))
                        : "memory");
                }
            }
            if (!ok) atomicExch(g.err, 1);
        }
    } else {
        const int q = warp & 3, cg = warp >> 2;
        const int row = 32 * q + lane;
        const int gr = m0 + row;
        const bool valid = gr < g.n;
        const uint32_t trow = tmem + ((uint32_t)(32 * q) << 16);
        float v[16];
        // the input: 16 columns per column group, in every CTA
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int c = 16 * cg + i;
            v[i] = valid && c < COR_MLP_IN ? g.x[(size_t)gr * COR_MLP_IN + c] : 0.f;
        }
        put_row16(single, row, 16 * cg, v);
        if (TRAIN && rank == 0) {
            __syncwarp();
            put_transposed(g.x0t, kInPad, 16 * cg, m0, single + 2 * cg * 128, q, 16);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive(&sh.local);
        for (int p = 0; p < kLast; p++) {
            ok = mbar_wait(&sh.acc, (uint32_t)(p & 1));
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (p == COR_MLP_LAYERS) {
                if (cg == 0) {
                    tmem_ld16(v, trow);
                    const float y0 = v[0] + g.bias[4][0], y1 = v[1] + g.bias[4][1];
                    if (!TRAIN) {
                        if (valid && rank == 0) {
                            g.y[2 * (size_t)gr] = y0;
                            g.y[2 * (size_t)gr + 1] = y1;
                        }
                    } else {
                        // mean squared error over the n rows and 2 outputs
                        const float scale = 2.f / (float)(g.n * COR_MLP_OUT);
                        float e0 = 0.f, e1 = 0.f;
                        if (valid) {
                            e0 = y0 - g.target[2 * (size_t)gr];
                            e1 = y1 - g.target[2 * (size_t)gr + 1];
                        }
                        float l = (e0 * e0 + e1 * e1) / (float)(g.n * COR_MLP_OUT);
                        float d0 = scale * e0, d1 = scale * e1;
#pragma unroll
                        for (int i = 0; i < 16; i++) v[i] = i == 0 ? d0 : i == 1 ? d1 : 0.f;
                        put_row16(single, row, 0, v);
                        v[0] = v[1] = 0.f;
                        for (int c0 = 16; c0 < 64; c0 += 16) put_row16(single, row, c0, v);
                        if (rank == 0) {
                            __syncwarp();
                            put_transposed(g.dyt, kOutPad, 0, m0, single, q, 16);
#pragma unroll
                            for (int o = 16; o > 0; o >>= 1) {
                                l += __shfl_xor_sync(0xffffffffu, l, o);
                                d0 += __shfl_xor_sync(0xffffffffu, d0, o);
                                d1 += __shfl_xor_sync(0xffffffffu, d1, o);
                            }
                            if (lane == 0) {
                                atomicAdd(g.loss, l);
                                atomicAdd(g.gb[4], d0);
                                atomicAdd(g.gb[4] + 1, d1);
                            }
                        }
                    }
                }
                if (TRAIN) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    mbar_arrive(&sh.local);
                }
                continue;
            }
            const int set = exchange_out(p) % kSets;
#pragma unroll 1
            for (int j = 0; j < F::kOwn; j++) {
                const int kb = rank * F::kOwn + j;
                const int col0 = 64 * kb + 16 * cg;   // this warp's 16 columns of the block
                uint8_t* block = abuf + (set * kBlocks + kb) * kABlock;
                tmem_ld16(v, trow + 64 * j + 16 * cg);
                if (p < COR_MLP_LAYERS) {
                    float z[16];
#pragma unroll
                    for (int i = 0; i < 16; i++) {
                        z[i] = v[i] + g.bias[p][col0 + i];
                        v[i] = silu(z[i]);
                    }
                    put_row16(block, row, 16 * cg, v);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    mbar_arrive(&sh.kready[set][kb]);
                    if (TRAIN) {
                        // what the way back needs, beside the next product
#pragma unroll
                        for (int i = 0; i < 16; i++) g.z[p][((size_t)tile * kH + col0 + i) * kBM + row] = z[i];
                        __syncwarp();
                        put_transposed(g.ht[p], kH, col0, m0, block + 2 * cg * 128, q, 16);
                    }
                } else {
                    const int l = kProducts - 1 - p;   // dZ of layer l + 1
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        v[i] = v[i] * silu_grad(g.z[l][((size_t)tile * kH + col0 + i) * kBM + row]);
                    put_row16(block, row, 16 * cg, v);
                    if (p + 1 < kLast) {
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        mbar_arrive(&sh.kready[set][kb]);
                    }
                    // column sums over the warp's 32 rows: lanes 2c and 2c+1 end with column c's
#pragma unroll
                    for (int o = 16, m = 8; m > 0; o >>= 1, m >>= 1) {
                        const bool up = (lane & o) != 0;
#pragma unroll
                        for (int i = 0; i < m; i++) {
                            const float give = up ? v[i] : v[i + m];
                            v[i] = (up ? v[i + m] : v[i]) + __shfl_xor_sync(0xffffffffu, give, o);
                        }
                    }
                    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
                    if ((lane & 1) == 0) atomicAdd(g.gb[l] + col0 + (lane >> 1), v[0]);
                    __syncwarp();
                    put_transposed(g.dzt[l], kH, col0, m0, block + 2 * cg * 128, q, 16);
                }
            }
        }
        if (!ok) atomicExch(g.err, 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    const int failed = __syncthreads_or(!ok);
    if (failed && threadIdx.x < SPLIT)
        asm volatile("st.shared::cluster.u32 [%0], 1;" ::"r"(peer_addr(smem_u32(&sh.failed), threadIdx.x)) : "memory");
    __syncwarp();
    // no CTA leaves while a peer's copy may still read or write shared memory:
    // where all went well, every copy was waited for; else they are waited out
    tile_sync<SPLIT>();
    if (*(volatile uint32_t*)&sh.failed) {
        settle();
        tile_sync<SPLIT>();
    }
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols));
}

// ---- weight gradients and AdamW ---------------------------------------------------
constexpr int kGradN = 64;                                   // columns of a tile
constexpr int kGradTiles = 2 + 3 * 2 * (kH / kGradN) + 2;    // W1: 2, W2-W4: 8 each, W5: 2
constexpr int kGradThreads = 32 * 10;                        // 8 epilogue warps, the ring's feeder, the MMAs' issuer
constexpr int kGradRing = 6;
constexpr uint32_t kGradStage = block_bytes(kBM) + block_bytes(kGradN);
constexpr size_t kGradSmem = 1024 + kGradRing * kGradStage;
static_assert(kBM * (kGradN + 1) * 4 <= 48 * 1024 && 48 * 1024 + kBM * kGradN * 2 <= kGradRing * kGradStage, "the tile");

struct GradArgs {
    const uint8_t* x0t;
    const uint8_t* ht[COR_MLP_LAYERS];
    const uint8_t* dzt[COR_MLP_LAYERS];
    const uint8_t* dyt;
    int blocks;              // K blocks: batch / 64
    float* w;                // parameters, moments: the packed parameter order
    float* m;
    float* v;
    const float* gb[kLayers];
    const float* loss;       // the batch's loss, copied to loss_out
    float* loss_out;
    float* grads;            // packed gradient export (may be null)
    uint8_t* weights;        // the weight stream
    float lr, b1c, b2c, decay;
    int update;
    int* err;
};

// Offsets of each tensor in the packed parameter order.
__host__ __device__ constexpr int layer_in(int l) { return l == 0 ? COR_MLP_IN : kH; }
__host__ __device__ constexpr int layer_out(int l) { return l == 4 ? COR_MLP_OUT : kH; }
__host__ __device__ constexpr int weight_at(int l) {
    int o = 0;
    for (int i = 0; i < l; i++) o += layer_out(i) * layer_in(i) + layer_out(i);
    return o;
}
__host__ __device__ constexpr int bias_at(int l) { return weight_at(l) + layer_out(l) * layer_in(l); }

// W(l) element (r, c) into the BF16 copies the products read.
__device__ __forceinline__ void store_weight(uint8_t* stream, int l, int r, int c, float w) {
    const bf16 b = __float2bfloat16(w);
    *reinterpret_cast<bf16*>(stream + product_offset(l) + packed_at(product_n(l), r, c)) = b;
    if (l > 0) *reinterpret_cast<bf16*>(stream + product_offset(9 - l) + packed_at(kH, c, r)) = b;
}

// AdamW with gradient gr: updates the moments, returns the new parameter.
__device__ __forceinline__ float adamw_step(const GradArgs& g, float gr, float& m, float& v, float w, float decay) {
    m = 0.9f * m + 0.1f * gr;
    v = 0.999f * v + 0.001f * gr * gr;
    return w - g.lr * ((m / g.b1c) / (sqrtf(v / g.b2c) + 1e-8f) + decay * w);
}

// The same on parameter i in place.
__device__ __forceinline__ float adamw(const GradArgs& g, int i, float gr, float decay) {
    float m = g.m[i], v = g.v[i];
    const float w = adamw_step(g, gr, m, v, g.w[i], decay);
    g.m[i] = m;
    g.v[i] = v;
    g.w[i] = w;
    return w;
}

// Whether `ok` holds for all 256 threads of grad_kernel's epilogue.  Each warp's
// wait has a limit of its own: what one of them found is not what the others
// did, and the barriers below count on all of them.
__device__ __forceinline__ bool epilogue_agrees(bool ok) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, 1, 256, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)ok)
        : "memory");
    return r != 0;
}

// One tile of a weight gradient (blocks 0 .. kGradTiles - 1), or the biases (the last block).
__global__ void __launch_bounds__(kGradThreads, 1) grad_kernel(const GradArgs g) {
    if (blockIdx.x == kGradTiles) {
        for (int l = 0; l < kLayers; l++)
            for (int r = threadIdx.x; r < layer_out(l); r += kGradThreads) {
                const float gr = g.gb[l][r];
                if (g.grads) g.grads[bias_at(l) + r] = gr;
                if (g.update) adamw(g, bias_at(l) + r, gr, 0.f);
            }
        if (threadIdx.x == 0) *g.loss_out = *g.loss;
        return;
    }
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t full[kGradRing], empty[kGradRing], accb;
    __shared__ uint32_t s_tmem;
    uint8_t* ring = smem + 1024;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // tile -> layer, M tile, N tile: C[m][n] = A[m][batch] . B[n][batch]^T
    int l, mt, n0 = 0, N = kGradN;
    const uint8_t *A, *B;
    int b_rows;
    if (blockIdx.x < 2) {
        l = 0;
        mt = blockIdx.x;
        A = g.dzt[0];
        B = g.x0t;
        b_rows = kInPad;
    } else if (blockIdx.x < kGradTiles - 2) {
        const int t = blockIdx.x - 2, per = 2 * (kH / kGradN);
        l = 1 + t / per;
        mt = (t % per) & 1;
        n0 = (t % per) / 2 * kGradN;
        A = g.dzt[l];
        B = g.ht[l - 1];
        b_rows = kH;
    } else {
        l = 4;
        mt = blockIdx.x - (kGradTiles - 2);
        A = g.ht[3];
        B = g.dyt;
        b_rows = kOutPad;
        N = kOutPad;
    }
    A += (size_t)mt * block_bytes(kBM);
    B += (size_t)n0 * kBK * 2;
    constexpr uint32_t kCols = 64;
    if (threadIdx.x == 0) {
        for (int k = 0; k < kGradRing; k++) {
            mbar_init(&full[k], 1);
            mbar_init(&empty[k], 1);
        }
        mbar_init(&accb, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                     "r"(kCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    bool ok = true;
    if (warp == 8) {
        if (lane == 0) {
            int s = 0;
            for (; s < g.blocks; s++) {
                const int k = s % kGradRing;
                if (s >= kGradRing) ok = mbar_wait(&empty[k], (uint32_t)((s / kGradRing - 1) & 1));
                if (!ok) break;
                mbar_expect(&full[k], block_bytes(kBM) + block_bytes(N));
                uint8_t* d = ring + k * kGradStage;
                bulk_load(d, A + (size_t)s * block_bytes(kH), block_bytes(kBM), &full[k]);
                bulk_load(d + block_bytes(kBM), B + (size_t)s * block_bytes(b_rows), block_bytes(N), &full[k]);
            }
            if (!ok) {
                atomicExch(g.err, 1);
                for (int i = s > kGradRing ? s - kGradRing : 0; i < s; i++)
                    mbar_wait(&full[i % kGradRing], (uint32_t)((i / kGradRing) & 1));
            }
        }
    } else if (warp == 9) {
        if (lane == 0) {
            const uint32_t idesc = instr_desc(kBM, N);
            for (int s = 0; s < g.blocks && ok; s++) {
                const int k = s % kGradRing;
                ok = mbar_wait(&full[k], (uint32_t)((s / kGradRing) & 1));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a0 = smem_u32(ring + k * kGradStage);
                mma_block(tmem, a0, a0 + block_bytes(kBM), idesc, s == 0);
                commit_to(&empty[k]);
            }
            if (ok) commit_to(&accb);
            else atomicExch(g.err, 1);
        }
    } else {
        ok = epilogue_agrees(mbar_wait(&accb, 0));
        if (!ok) {
            atomicExch(g.err, 1);
        } else {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int q = warp & 3, cg = warp >> 2;
            const int row = mt * kBM + 32 * q + lane;
            // the ring is free: the tile goes through it, so that parameters and
            // moments are read and written in whole lines
            float* tile = reinterpret_cast<float*>(ring);
            constexpr int kLd = kGradN + 1;
            uint8_t* block = ring + 48 * 1024;
            for (int c0 = 32 * cg; c0 < 32 * cg + 32 && c0 < N; c0 += 16) {
                float v[16];
                tmem_ld16(v, tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)c0);
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    const int col = n0 + c0 + i;
                    if (l < 4) {
                        tile[(32 * q + lane) * kLd + c0 + i] = v[i];
                    } else if (col < COR_MLP_OUT) {
                        const int at = weight_at(4) + col * kH + row;
                        if (g.grads) g.grads[at] = v[i];
                        if (g.update) store_weight(g.weights, 4, col, row, adamw(g, at, v[i], g.decay));
                    }
                }
            }
            if (l == 0) {
                // 128 rows of 19, contiguous
                asm volatile("bar.sync 1, 256;" ::: "memory");
                constexpr int kBatch = 10;
                static_assert(256 * kBatch >= kBM * COR_MLP_IN, "one batch");
                float m[kBatch], v[kBatch], w[kBatch];
                const int at0 = weight_at(0) + mt * kBM * COR_MLP_IN;
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    const int e = threadIdx.x + 256 * k;
                    if (e < kBM * COR_MLP_IN) {
                        m[k] = g.m[at0 + e];
                        v[k] = g.v[at0 + e];
                        w[k] = g.w[at0 + e];
                    }
                }
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    const int e = threadIdx.x + 256 * k, r = e / COR_MLP_IN, c = e % COR_MLP_IN;
                    if (e < kBM * COR_MLP_IN) {
                        const float gr = tile[r * kLd + c];
                        if (g.grads) g.grads[at0 + e] = gr;
                        if (g.update) {
                            const float nw = adamw_step(g, gr, m[k], v[k], w[k], g.decay);
                            g.m[at0 + e] = m[k];
                            g.v[at0 + e] = v[k];
                            g.w[at0 + e] = nw;
                            store_weight(g.weights, 0, mt * kBM + r, c, nw);
                        }
                    }
                }
            } else if (l < 4) {
                asm volatile("bar.sync 1, 256;" ::: "memory");
                // four float4 of each array in flight per thread
                constexpr int kBatch = 4;
                for (int e0 = threadIdx.x; e0 < kBM * kGradN / 4; e0 += 256 * kBatch) {
                    float4 m[kBatch], v[kBatch], w[kBatch];
                    int at[kBatch];
#pragma unroll
                    for (int k = 0; k < kBatch; k++) {
                        const int e = e0 + 256 * k;
                        at[k] = weight_at(l) + (mt * kBM + e / (kGradN / 4)) * kH + n0 + e % (kGradN / 4) * 4;
                        m[k] = *reinterpret_cast<const float4*>(g.m + at[k]);
                        v[k] = *reinterpret_cast<const float4*>(g.v + at[k]);
                        w[k] = *reinterpret_cast<const float4*>(g.w + at[k]);
                    }
#pragma unroll
                    for (int k = 0; k < kBatch; k++) {
                        const int e = e0 + 256 * k;
                        const int tr = e / (kGradN / 4), tc = e % (kGradN / 4) * 4;
                        const float* gr = tile + tr * kLd + tc;
                        if (g.grads) {
#pragma unroll
                            for (int i = 0; i < 4; i++) g.grads[at[k] + i] = gr[i];
                        }
                        if (g.update) {
                            w[k].x = adamw_step(g, gr[0], m[k].x, v[k].x, w[k].x, g.decay);
                            w[k].y = adamw_step(g, gr[1], m[k].y, v[k].y, w[k].y, g.decay);
                            w[k].z = adamw_step(g, gr[2], m[k].z, v[k].z, w[k].z, g.decay);
                            w[k].w = adamw_step(g, gr[3], m[k].w, v[k].w, w[k].w, g.decay);
                            *reinterpret_cast<float4*>(g.m + at[k]) = m[k];
                            *reinterpret_cast<float4*>(g.v + at[k]) = v[k];
                            *reinterpret_cast<float4*>(g.w + at[k]) = w[k];
                            const uint2 b = make_uint2(pack_bf16(w[k].x, w[k].y), pack_bf16(w[k].z, w[k].w));
                            *reinterpret_cast<uint2*>(g.weights + product_offset(l) +
                                                      packed_at(kH, mt * kBM + tr, n0 + tc)) = b;
                            *reinterpret_cast<uint2*>(block + packed_at(kBM, tr, tc)) = b;
                        }
                    }
                }
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (g.update)
                    put_transposed(g.weights + product_offset(9 - l), kH, n0 + 32 * cg, mt * kBM, block + 4 * cg * 128,
                                   q, 32);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (__syncthreads_or(!ok)) settle();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols));
}

// Every weight into its BF16 copies.
__global__ void cast_kernel(const float* __restrict__ w, uint8_t* __restrict__ weights) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    for (int l = 0; l < kLayers; l++) {
        const int n = layer_out(l) * layer_in(l);
        if (i < n) {
            store_weight(weights, l, i / layer_in(l), i % layer_in(l), w[weight_at(l) + i]);
            return;
        }
        i -= n;
    }
}

}  // namespace mlp

using namespace mlp;

struct cor_mlp {
    int device = 0;
    int max_bt = 0;
    char err[256] = {0};
    int step = 0;
    void* block = nullptr;      // one allocation holds every device buffer
    float *w, *mom, *vel;       // parameters and moments, the packed parameter order
    uint8_t* weights;           // BF16 copies in the order the products read them
    float* gb[kLayers];         // bias gradients, then the batch's loss
    float* loss;
    float* z[COR_MLP_LAYERS];
    uint8_t *x0t, *ht[COR_MLP_LAYERS], *dzt[COR_MLP_LAYERS], *dyt;
    bool can_cluster = false;   // the device (or this process's part of it) can place a cluster of rows_kernel
    int* err_h = nullptr;       // mapped: set by a wait that ran out
    int* err_d = nullptr;
};

static int mfail(cor_mlp* m, int code, const char* fmt, ...) {
    if (m) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(m->err, sizeof m->err, fmt, ap);
        va_end(ap);
    }
    return code;
}

#define MTRY(m, call)                                                                                  \
    do {                                                                                               \
        cudaError_t e_ = (call);                                                                       \
        if (e_ != cudaSuccess) return mfail((m), COR_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

static const size_t kGbBytes = sizeof(float) * (kLayers * kH + 64);

static RowsArgs rows_args(const cor_mlp* m, const float* x, int n) {
    RowsArgs g = {};
    g.x = x;
    g.n = n;
    g.weights = m->weights;
    for (int l = 0; l < kLayers; l++) {
        g.bias[l] = m->w + bias_at(l);
        g.gb[l] = m->gb[l];
    }
    for (int l = 0; l < COR_MLP_LAYERS; l++) {
        g.z[l] = m->z[l];
        g.ht[l] = m->ht[l];
        g.dzt[l] = m->dzt[l];
    }
    g.x0t = m->x0t;
    g.dyt = m->dyt;
    g.loss = m->loss;
    g.err = m->err_d;
    return g;
}

template <int SPLIT, bool TRAIN>
static bool set_rows_limit() {
    return cudaFuncSetAttribute(rows_kernel<SPLIT, TRAIN>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)Form<SPLIT>::kSmem) == cudaSuccess;
}
static bool set_rows_limits() {
    return set_rows_limit<1, false>() && set_rows_limit<1, true>() && set_rows_limit<kSplit, false>() &&
           set_rows_limit<kSplit, true>();
}

// Whether the current device, or this process's part of it, has room for a cluster at all.
static bool cluster_fits() {
    cudaLaunchAttribute dims = {};
    dims.id = cudaLaunchAttributeClusterDimension;
    dims.val.clusterDim = {kSplit, 1, 1};
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(kSplit);
    c.blockDim = dim3(kRowsThreads);
    c.dynamicSmemBytes = Form<kSplit>::kSmem;
    c.attrs = &dims;
    c.numAttrs = 1;
    int n = 0;
    const bool ok = cudaOccupancyMaxActiveClusters(&n, rows_kernel<kSplit, true>, &c) == cudaSuccess && n > 0;
    cudaGetLastError();
    return ok;
}

template <bool TRAIN>
static cudaError_t launch_rows(const RowsArgs& g, bool clusters, cudaStream_t s) {
    const int tiles = (g.n + kBM - 1) / kBM;
    if (clusters) rows_kernel<kSplit, TRAIN><<<kSplit * tiles, kRowsThreads, Form<kSplit>::kSmem, s>>>(g);
    else rows_kernel<1, TRAIN><<<tiles, kRowsThreads, Form<1>::kSmem, s>>>(g);
    return cudaGetLastError();
}

static int check_err(cor_mlp* m) {
    if (*(volatile int*)m->err_h) return mfail(m, COR_ERR_WATCHDOG, "a tensor-core wait ran out of time");
    return COR_OK;
}

extern "C" {

const char* cor_mlp_error(const cor_mlp* m) { return m ? m->err : "null network"; }

int cor_mlp_create(int device, int32_t max_batch, cor_mlp** out) {
    if (!out || max_batch < 1) return COR_ERR_INVALID;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        return COR_ERR_NODEV;
    }
    if (device < 0 || device >= ndev) return COR_ERR_INVALID;
    if (cudaSetDevice(device) != cudaSuccess) return COR_ERR_CUDA;
    cor_mlp* m = new cor_mlp();
    m->device = device;
    m->max_bt = (max_batch + kBM - 1) / kBM * kBM;
    const size_t bt = (size_t)m->max_bt;
    // sizes in bytes, each rounded to 256
    size_t total = 0;
    auto take = [&](size_t bytes) {
        const size_t o = total;
        total += (bytes + 255) & ~(size_t)255;
        return o;
    };
    const size_t ow = take(4 * COR_MLP_PARAMS), om = take(4 * COR_MLP_PARAMS), ov = take(4 * COR_MLP_PARAMS);
    const size_t owt = take(product_offset(kProducts));
    const size_t ogb = take(kGbBytes);
    size_t oz[COR_MLP_LAYERS], oht[COR_MLP_LAYERS], odz[COR_MLP_LAYERS];
    for (int l = 0; l < COR_MLP_LAYERS; l++) {
        oz[l] = take(4 * bt * kH);
        oht[l] = take(2 * bt * kH);
        odz[l] = take(2 * bt * kH);
    }
    const size_t ox = take(2 * bt * kInPad), ody = take(2 * bt * kOutPad);
    if (cudaMalloc(&m->block, total) != cudaSuccess) {
        delete m;
        return COR_ERR_NOMEM;
    }
    uint8_t* B = (uint8_t*)m->block;
    m->w = (float*)(B + ow);
    m->mom = (float*)(B + om);
    m->vel = (float*)(B + ov);
    m->weights = B + owt;
    for (int l = 0; l < kLayers; l++) m->gb[l] = (float*)(B + ogb) + l * kH;
    m->loss = (float*)(B + ogb) + kLayers * kH;
    for (int l = 0; l < COR_MLP_LAYERS; l++) {
        m->z[l] = (float*)(B + oz[l]);
        m->ht[l] = B + oht[l];
        m->dzt[l] = B + odz[l];
    }
    m->x0t = B + ox;
    m->dyt = B + ody;
    // the parameters, moments and BF16 copies (with their padding) start at zero
    if (cudaMemset(m->block, 0, ogb + kGbBytes) != cudaSuccess ||
        cudaHostAlloc((void**)&m->err_h, sizeof(int), cudaHostAllocMapped) != cudaSuccess ||
        cudaHostGetDevicePointer((void**)&m->err_d, m->err_h, 0) != cudaSuccess ||
        !set_rows_limits() ||
        cudaFuncSetAttribute(grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGradSmem) != cudaSuccess ||
        cudaDeviceSynchronize() != cudaSuccess) {
        cudaFree(m->block);
        if (m->err_h) cudaFreeHost(m->err_h);
        delete m;
        return COR_ERR_CUDA;
    }
    m->can_cluster = cluster_fits();
    *m->err_h = 0;
    *out = m;
    return COR_OK;
}

int cor_mlp_destroy(cor_mlp* m) {
    if (!m) return COR_OK;
    cudaSetDevice(m->device);
    cudaDeviceSynchronize();
    if (m->block) cudaFree(m->block);
    if (m->err_h) cudaFreeHost(m->err_h);
    delete m;
    return COR_OK;
}

int cor_mlp_set_params(cor_mlp* m, const float* params) {
    if (!m || !params) return COR_ERR_INVALID;
    MTRY(m, cudaSetDevice(m->device));
    MTRY(m, cudaMemcpy(m->w, params, sizeof(float) * COR_MLP_PARAMS, cudaMemcpyHostToDevice));
    MTRY(m, cudaMemset(m->mom, 0, sizeof(float) * COR_MLP_PARAMS));
    MTRY(m, cudaMemset(m->vel, 0, sizeof(float) * COR_MLP_PARAMS));
    cast_kernel<<<(COR_MLP_PARAMS + 255) / 256, 256>>>(m->w, m->weights);
    MTRY(m, cudaGetLastError());
    m->step = 0;
    MTRY(m, cudaDeviceSynchronize());
    return COR_OK;
}

int cor_mlp_get_params(cor_mlp* m, float* params) {
    if (!m || !params) return COR_ERR_INVALID;
    MTRY(m, cudaSetDevice(m->device));
    MTRY(m, cudaDeviceSynchronize());
    MTRY(m, cudaMemcpy(params, m->w, sizeof(float) * COR_MLP_PARAMS, cudaMemcpyDeviceToHost));
    return COR_OK;
}

int cor_mlp_forward(cor_mlp* m, const float* x_dev, int32_t n, float* y_dev, void* stream) {
    if (!m) return COR_ERR_INVALID;
    if (n < 0 || n > m->max_bt || (n > 0 && (!x_dev || !y_dev)))
        return mfail(m, COR_ERR_INVALID, "batch of %d outside [0, %d]", n, m->max_bt);
    if (n == 0) return COR_OK;
    MTRY(m, cudaSetDevice(m->device));
    cudaStream_t s = (cudaStream_t)stream;
    RowsArgs g = rows_args(m, x_dev, n);
    g.y = y_dev;
    const cor::NetworkTurn turn(m->device, m->can_cluster);   // until the call has waited for its kernel
    MTRY(m, launch_rows<false>(g, turn.clusters, s));
    MTRY(m, cudaStreamSynchronize(s));
    return check_err(m);
}

static int train(cor_mlp* m, const float* x, const float* t, int32_t n, float lr, float wd, float* loss,
                 float* grads, int do_update, void* stream) {
    if (!m) return COR_ERR_INVALID;
    if (n < 1 || n > m->max_bt || !x || !t || !loss)
        return mfail(m, COR_ERR_INVALID, "batch of %d outside [1, %d] or missing buffer", n, m->max_bt);
    MTRY(m, cudaSetDevice(m->device));
    cudaStream_t s = (cudaStream_t)stream;
    const int tiles = (n + kBM - 1) / kBM;
    MTRY(m, cudaMemsetAsync(m->gb[0], 0, kGbBytes, s));
    RowsArgs g = rows_args(m, x, n);
    g.target = t;
    const cor::NetworkTurn turn(m->device, m->can_cluster);
    MTRY(m, launch_rows<true>(g, turn.clusters, s));
    if (do_update) m->step++;
    GradArgs a = {};
    a.x0t = m->x0t;
    a.dyt = m->dyt;
    for (int l = 0; l < COR_MLP_LAYERS; l++) {
        a.ht[l] = m->ht[l];
        a.dzt[l] = m->dzt[l];
    }
    a.blocks = tiles * (kBM / kBK);
    a.w = m->w;
    a.m = m->mom;
    a.v = m->vel;
    for (int l = 0; l < kLayers; l++) a.gb[l] = m->gb[l];
    a.loss = m->loss;
    a.loss_out = loss;
    a.grads = grads;
    a.weights = m->weights;
    a.lr = lr;
    a.b1c = 1.f - powf(0.9f, (float)(m->step > 0 ? m->step : 1));
    a.b2c = 1.f - powf(0.999f, (float)(m->step > 0 ? m->step : 1));
    a.decay = wd;
    a.update = do_update;
    a.err = m->err_d;
    grad_kernel<<<kGradTiles + 1, kGradThreads, kGradSmem, s>>>(a);
    MTRY(m, cudaGetLastError());
    MTRY(m, cudaStreamSynchronize(s));
    return check_err(m);
}

int cor_mlp_train_step(cor_mlp* m, const float* x_dev, const float* t_dev, int32_t n, float lr, float weight_decay,
                       float* loss_dev, float* grads_dev, void* stream) {
    return train(m, x_dev, t_dev, n, lr, weight_decay, loss_dev, grads_dev, 1, stream);
}

int cor_mlp_gradient(cor_mlp* m, const float* x_dev, const float* t_dev, int32_t n, float* loss_dev,
                     float* grads_dev, void* stream) {
    if (!grads_dev) return mfail(m, COR_ERR_INVALID, "no gradient buffer");
    return train(m, x_dev, t_dev, n, 0.f, 0.f, loss_dev, grads_dev, 0, stream);
}

}  // extern "C"
