// Batched projection on the 5th-generation tensor cores: out[b][n] = sum_k trit[n][k] * act[b][k] for a batch of int8 activation
// vectors (prompt ingestion, batched decoding), the same integers as the batch-1 kernel of gemv_lut.cuh gives vector by vector.
//
// The reference has no batched path: its CPU runtime and its GPU decoder run a prompt token by token (quintrit-runtime/src/engine.rs
// forward_token, quintrit-runtime/src/gpu.rs:459-493), each token with its own activation scale. What is restated is the projection's
// definition (quintrit-runtime/src/layer.rs:123-177: the exact int32 sum, scaled afterwards), so a batch of B tokens gives B results
// that are bit-identical to B single-token projections.
//
// Shape on a B200. The batch-1 kernel streams velurex bytes (0.2 bytes per weight); turning those into int8 operands costs a table lookup and
// a byte transposition per weight byte, which would leave the tensor pipe waiting. This kernel therefore reads its own copy of the weights,
// made on the device the first time a matrix is used here: two bits per trit (0.25 bytes per weight), placed so that a mask, at most two shifts and one
// byte permute turn a quarter of a word into four int8 operands that are already in K order. The product runs as tcgen05.mma.kind::i8 on pairs of
// multiprocessors (cta_group::2) with the accumulator in tensor memory:
//   * a work item is 256 weight rows (the M of the instruction, 128 a block of the pair) times a range of 256-column stages (K) times up to 256 vectors (the N).
//     Each block of a pair holds half of the batch's activations, so a stage costs it n / 2 x 256 + 8192 bytes of shared memory and of L2 traffic: with a
//     block for itself (n x 256 + 8192) the activations' way through L2 would be longer than the products;
//   * sixteen warps decode, in four groups that take the stages round-robin: a thread takes a row's 64 bytes of a stage from shared memory and writes the row's
//     256 int8 operands into its lane of TENSOR MEMORY with tcgen05.st (64 columns a group). Operands that threads
//     store to shared memory need a proxy fence before the tensor cores may read them, and that fence was measured at more than a
//     thousand cycles a block; operands in tensor memory need none;
//   * two load warps, taking the stages in turn, fetch the tile's 8192 weight bytes (one bulk copy) and the matching activations (two
//     TMA boxes of n / 2 vectors x 128 bytes, 128-byte swizzle, in place from the caller's vectors where their pitch allows it). What a block loads completes on one
//     mbarrier of its own, but for the second block's activations: only the tensor cores read them, on the first block's command, so they complete on a barrier of the
//     first block (the cta_group::2 form of the copy), where a decode warp sees it before it hands its operand to the issuing thread;
//   * one thread of the pair's first block issues eight MMAs (256 x N x 32, A from tensor memory, B from shared memory) per stage and releases the stage
//     and the group's operand columns in both blocks with tcgen05.commit; a ring of 5 to 12 stages (as many as fit) keeps the loads ahead;
//   * the kernel is persistent: a pair takes items round-robin;
//   * at the end of an item the decode warps read the accumulator with tcgen05.ld (a row per thread, a quarter of the columns a group), release it and write
//     out[b][row] (when K was split over several items, so that matrices with few rows still fill the chip, each part writes its partial sums and the
//     consumer or a small second kernel adds the parts: exact integers in any order). A group decodes its first stage of the next item before that, so
//     the tensor cores wait for the reading of the accumulator only.
// Bound by the products at 256 vectors (1060 cycles a stage of 256 x 256 x 256, 1024 of them the tensor cores'), by what hands a stage on (about 700 cycles) at 32. Events around
// 24 launches of the Falcon3-10B shapes, weights from HBM, against the former kernel (a block a tile, 128-column stages, table lookups):
//   46080 x 3072, 256 vectors  59.7 -> 37.0 us;  32 vectors  43 -> 22.7 us
//   3072 x 23040, 256 vectors  27 -> 19.2 us;    32 vectors  21 -> 12.4 us
//   5120 x 3072, 256 vectors   22 -> 12.4 us;    32 vectors  10 -> 8.3 us
// Every wait on an mbarrier is bounded: after `spin_limit` polls the thread raises an abort flag that the other roles (of both blocks) see, the kernel
// sets its status word, waits (bounded) for its own copies in flight, frees its tensor memory and returns.
//
// Weight copy: the 16 bytes at ((tile * chunks + c) * 128 + r) * 16 hold columns 64 c .. 64 c + 63 of row r of a tile of 128 rows, 16 columns a
// 32-bit word: column k of a word as trit + 1 at bit 4 k for k < 8, at bit 4 (k - 8) + 2 for the others. Rows are padded to pairs of tiles and columns to
// whole stages with code 1 (trit 0).
#pragma once
#include <cstdint>

#include <cuda.h>
#include <cuda_runtime.h>

#include "gemm_turns.hpp"
#include "gemv_lut.cuh"

namespace qtb {

constexpr int kGemmM = 128;     // weight rows of a block; a pair takes two such tiles
constexpr int kGemmDecodeWarps = 16;
constexpr int kGemmGroups = 4;  // the decode warps work in groups of four; group g decodes the stages it, it + 4, ... of the pair's sequence on its own
constexpr int kGemmThreads = 32 * (kGemmDecodeWarps + 1 + kGemmLoadWarps);  // decode warps, the MMA warp, load warps
constexpr int kGemmMaxStages = 12;
constexpr int kGemmMaxN = 256;  // 256 accumulator columns + 4 x 64 operand columns are the 512 columns of tensor memory
constexpr int kGemmStageCols = 256;                            // columns (K) of one stage
constexpr int kGemmStageBytes = kGemmM * kGemmStageCols / 4;   // its weight bytes for one tile
constexpr unsigned int kGemmStatusTimeout = 4;

struct GemmArgs {
    const uint8_t* w;      // the two-bit copy
    int32_t* out;          // [batch][rows]; with K split over several items: the partial sums [part][batch][rows]
    unsigned int* status;  // set to kGemmStatusTimeout when a wait ran out
    int rows, pairs;       // weight rows; pairs of row tiles
    int blocks;            // stages (256 columns) of a row
    int ldo;               // elements between the results of consecutive vectors in `out` (rows, or more when the results go into a wider row)
    int n;                 // instruction N: vectors of a token tile, a multiple of 32
    int batch;             // activation vectors actually present
    int token_tiles;       // of n vectors each; the last may be ragged
    int blocks_per_item;   // stages of one work item (a pair of row tiles x a K part x a token tile)
    int stages;
    unsigned int spin_limit;
};

// Stages that fit the shared memory of an SM for a batch of n: as many as possible (at most kGemmMaxStages), because the stages in flight have to
// cover the latency of the weight bytes from HBM. Five at n = 256.
inline size_t gemm_stage_bytes(int n) { return size_t(n / 2) * kGemmStageCols + kGemmStageBytes; }
inline int gemm_stages_for(int n, size_t smem_limit) {
    const size_t fixed = 512 + 1024, fit = smem_limit > fixed ? (smem_limit - fixed) / gemm_stage_bytes(n) : 0;
    return static_cast<int>(fit < size_t(kGemmMaxStages) ? fit : size_t(kGemmMaxStages));
}
inline size_t gemm_smem_bytes(int n, int stages) { return size_t(stages) * gemm_stage_bytes(n) + 512 + 1024; }  // + barriers + alignment slack
inline size_t gemm_row_tiles(size_t rows) { return (rows + 2 * kGemmM - 1) / (2 * kGemmM) * 2; }
inline size_t gemm_blocks(size_t cols) { return (cols + kGemmStageCols - 1) / kGemmStageCols; }
inline size_t gemm_copy_bytes(size_t rows, size_t cols) { return gemm_row_tiles(rows) * gemm_blocks(cols) * kGemmStageBytes; }

// stream layout (gemv_lut.cuh) -> the two-bit copy, whose bytes are all 0x55 (code 1) before; `chunks` 16-byte units a row, `vblocks` 160-trit velurex blocks
// a row. The copy may be one of several matrices stacked row-wise into one (q | k | v, gate | up): its rows start at tile `tile0`. A warp takes a velurex
// block of 32 rows, a row a lane: 32 bytes in two 16-byte loads, a table lookup per byte for its five codes, ten words out. (A word a thread from single bytes took
// 4 ms longer over the four layers of a Falcon3-10B-shaped model's first prompt.)
__global__ void stream_to_two_bit_kernel(const uint4* __restrict__ stream, uint32_t* __restrict__ out, int rows, int cols, int chunks, int vblocks, int tiles, int tile0) {
    __shared__ unsigned short codes[256];  // byte -> its five codes, two bits each
    for (int v = threadIdx.x; v < 256; v += blockDim.x) {
        unsigned int d = 0x155;
        if (v <= 250) {
            const int d4 = v / 84, r4 = v - 84 * d4, d3 = r4 / 28, r3 = r4 - 28 * d3, d2 = r3 / 9, r2 = r3 - 9 * d2, d1 = r2 / 3;
            d = (r2 - 3 * d1) | d1 << 2 | d2 << 4 | d3 << 6 | d4 << 8;
        }
        codes[v] = static_cast<unsigned short>(d);
    }
    __syncthreads();
    const int lane = threadIdx.x & 31, warps = gridDim.x * (blockDim.x >> 5);
    for (int i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < vblocks * tiles; i += warps) {
        const int vb = i / tiles, t = i - vb * tiles, r = t * 32 + lane;
        const uint4* src = stream + (static_cast<size_t>(i) * 2) * 32 + lane;
        const uint4 x = src[0], y = src[32];
        const uint32_t words[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        uint32_t lo[5] = {0, 0, 0, 0, 0}, hi[5] = {0, 0, 0, 0, 0};  // columns 32 p .. 32 p + 15 and the sixteen behind them
#pragma unroll
        for (int k = 0; k < 32; ++k) {
            const unsigned int c = codes[(words[k >> 2] >> (8 * (k & 3))) & 0xffu];
            const int j = (k + lane) & 31, jj = j & 15, at = jj < 8 ? 4 * jj : 4 * (jj - 8) + 2;  // position k of a row holds planar byte (k + row) mod 32
#pragma unroll
            for (int p = 0; p < 5; ++p) {
                const uint32_t bits = ((c >> (2 * p)) & 3u) << at;
                lo[p] |= j < 16 ? bits : 0u;
                hi[p] |= j < 16 ? 0u : bits;
            }
        }
        if (r >= rows) continue;
        uint32_t* dst = out + (static_cast<size_t>(tile0 + r / kGemmM) * chunks * kGemmM + r % kGemmM) * 4;
#pragma unroll
        for (int w = 0; w < 10; ++w) {
            const int col = vb * 160 + w * 16, left = cols - col;
            uint32_t word = w & 1 ? hi[w >> 1] : lo[w >> 1];
            if (left <= 0) break;
            if (left < 16) {  // the columns behind the matrix stay code 1
                uint32_t keep = 0;
                for (int k = 0; k < left; ++k) keep |= 3u << (k < 8 ? 4 * k : 4 * (k - 8) + 2);
                word = (word & keep) | (0x55555555u & ~keep);
            }
            dst[static_cast<size_t>(col / 64) * (kGemmM * 4) + (col % 64) / 16] = word;
        }
    }
}

// out[i] = sum over the K parts of partial[part][i] (i over batch * rows): the second step of a projection whose K was split over several items
// (partial rows are dense, `rows` apart; the results of a vector are `ldo` apart in out)
__global__ void gemm_reduce_parts_kernel(const int32_t* __restrict__ partial, int32_t* __restrict__ out, size_t count, int parts, int rows, int ldo) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < count; i += size_t(gridDim.x) * blockDim.x) {
        int32_t sum = 0;
        for (int p = 0; p < parts; ++p) sum += partial[size_t(p) * count + i];
        out[(i / rows) * ldo + i % rows] = sum;
    }
}

// int8 activation vectors [batch][cols] -> the zero-padded matrix [n][whole stages of 256] the TMA reads
__global__ void gemm_pad_activations_kernel(const int8_t* __restrict__ act, int8_t* __restrict__ padded, int batch, int n, int cols, int k_pad) {
    const size_t total = size_t(n) * k_pad;
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < total; i += size_t(gridDim.x) * blockDim.x) {
        const int b = static_cast<int>(i / k_pad), c = static_cast<int>(i % k_pad);
        padded[i] = (b < batch && c < cols) ? act[size_t(b) * cols + c] : int8_t(0);
    }
}

namespace gemm_detail {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"  // the last operand: how long the hardware may park the thread per try
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(20000u)
        : "memory");
    return ok != 0;
}
// Bounded wait: false when the limit ran out or another role already gave up (the abort flag is then set).
// `heed_abort` false: keep waiting up to the limit although another role gave up (the wait for one's own copies in flight).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile unsigned int* abort_flag, unsigned int limit, bool heed_abort = true) {
    for (unsigned int i = 0; i < limit; ++i) {
        if (mbar_try(bar, parity)) return true;
        if (heed_abort && *abort_flag) return false;
    }
    *abort_flag = 1;
    return false;
}
// Plain bulk copy (no tensor map): `bytes` contiguous bytes, a multiple of 16, both addresses 16-byte aligned.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst), "l"(map), "r"(x), "r"(y),
                 "r"(z), "r"(bar)
                 : "memory");
}
// Shared-memory matrix descriptor of the tensor-core instruction (64 bits): start address, leading and stride byte offsets in
// 16-byte units, descriptor version 1 at bit 46, layout type in bits 61..63 (0 no swizzle, 6 32-byte swizzle).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes, uint32_t layout) {
    return uint64_t((addr & 0x3FFFFu) >> 4) | (uint64_t(lbo_bytes >> 4) << 16) | (uint64_t(sbo_bytes >> 4) << 32) | (uint64_t(1) << 46) | (uint64_t(layout) << 61);
}
// Instruction descriptor for kind::i8: S32 accumulator (2 at bit 4), signed 8-bit A and B (1 at bits 7 and 10), both K-major,
// N / 8 at bit 17, M / 16 at bit 24.
__device__ __forceinline__ uint32_t instr_desc_i8(int m, int n) { return (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n >> 3) << 17) | (uint32_t(m >> 4) << 24); }
__device__ __forceinline__ void mma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// ---- pairs of blocks (cta_group::2) ----
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The address, in the cluster's window, of what lies at `addr` in block `rank`'s shared memory.
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// An arrival at a barrier of either block. It orders nothing but what the tcgen05 fences and waits around it order (operands in tensor memory, accumulator reads), and nothing
// else is handed over by it: with .release.cluster an arrival, and .acquire.cluster a wait, cost about 3000 and 250 cycles.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void store_cluster(uint32_t addr, uint32_t value) { asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(value) : "memory"); }
__device__ __forceinline__ void raise_abort(uint32_t flag_addr, uint32_t rank) { store_cluster(cluster_addr(flag_addr, rank ^ 1), 1u); }  // in the other block too
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// The same with a barrier that may be the other block's (`bar`: an address in the cluster's window).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];" ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// 256 rows (128 in the tensor memory of either block) x N x 32; the first half of B's rows lies in the first block's shared memory, the rest in the second's.
__device__ __forceinline__ void mma_i8_ts_pair(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
        "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives at the barrier of that offset in both blocks once the MMAs issued so far are done.
__device__ __forceinline__ void mma_commit_pair(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(static_cast<uint16_t>(3)) : "memory");
}
// 16 columns of the two-bit copy -> four words of four int8 operands. A nibble of the masked word selects a byte of (-1, 0, 1, 0): its low two bits are a code, bit 2
// picks the second operand of the permute (the same word), bit 3 (sign fill) is masked away.
__device__ __forceinline__ void decode16(uint32_t w, uint32_t* v) {
    const uint32_t m0 = w & 0x77777777u, m1 = (w >> 2) & 0x77777777u;
    constexpr uint32_t kTrits = 0x000100FFu;
    asm("prmt.b32 %0, %1, %1, %2;" : "=r"(v[0]) : "r"(kTrits), "r"(m0));
    asm("prmt.b32 %0, %1, %1, %2;" : "=r"(v[1]) : "r"(kTrits), "r"(m0 >> 16));
    asm("prmt.b32 %0, %1, %1, %2;" : "=r"(v[2]) : "r"(kTrits), "r"(m1));
    asm("prmt.b32 %0, %1, %1, %2;" : "=r"(v[3]) : "r"(kTrits), "r"(m1 >> 16));
}
__device__ __forceinline__ void tmem_store32(uint32_t addr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, "
        "%29, %30, %31, %32};" ::"r"(addr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
        "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]),
        "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void tmem_load8(uint32_t addr, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(addr));
}

}  // namespace gemm_detail

// The end of an item: this thread's row of `own` (a multiple of eight) accumulator columns is read, the accumulator released, and the first `valid` of them written, `ldo` apart.
// Out of line: its 64 values would crowd the decoding loop's registers.
__device__ __noinline__ void gemm_write_out(uint32_t tmem, uint32_t released, int own, int32_t* dst, int ldo, int valid) {
    using namespace gemm_detail;
    constexpr int kMost = kGemmMaxN / kGemmGroups;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t v[kMost];
#pragma unroll
    for (int c = 0; c < kMost; c += 8)
        if (c < own) tmem_load8(tmem + c, v + c);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncwarp();
    if ((threadIdx.x & 31) == 0) mbar_arrive_cluster(released);
#pragma unroll
    for (int c = 0; c < kMost; c += 8) {
        if (c >= valid) break;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (c + i < valid) dst[static_cast<size_t>(static_cast<uint32_t>((c + i) * ldo))] = static_cast<int32_t>(v[c + i]);
    }
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kGemmThreads, 1) gemm_i8_tcgen05_kernel(const __grid_constant__ CUtensorMap act_map, GemmArgs a) {
    using namespace gemm_detail;
    extern __shared__ unsigned char gemm_smem_raw[];
    const uint32_t smem0 = (smem_u32(gemm_smem_raw) + 1023u) & ~1023u;  // the same offset in both blocks, as the descriptors want it
    unsigned char* smem = gemm_smem_raw + (smem0 - smem_u32(gemm_smem_raw));
    const int S = a.stages, n = a.n;
    const uint32_t act_bytes = uint32_t(n / 2) * kGemmStageCols;
    const uint32_t b_base = smem0;                                        // S stages of two tiles of n / 2 vectors x 128 bytes
    const uint32_t raw_base = smem0 + S * act_bytes;                      // S stages of the weight bytes of this block's tile
    const unsigned char* raw_tiles = smem + S * act_bytes;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S * (act_bytes + kGemmStageBytes));
    // barriers of each block: loaded[S] (its weight bytes of a stage, and in the first block the activations, have landed), empty[S] (the MMAs of the stage are done: it may be loaded
    // again, and the group may write its next operand), acc_full (those of an item); of the first block only: a_full[G] (group g's operand is written in both blocks), acc_empty (both
    // have read the accumulator), peer_acts[S] (the second block's activations have landed in its shared memory)
    const uint32_t bar0 = smem_u32(bars);
    auto loaded = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (kGemmMaxStages + s); };
    auto a_full = [&](int g) { return bar0 + 8u * (2 * kGemmMaxStages + g); };
    const uint32_t acc_full = bar0 + 8u * (2 * kGemmMaxStages + kGemmGroups), acc_empty = acc_full + 8u;
    auto peer_acts = [&](int s) { return acc_empty + 8u * (1 + s); };
    constexpr int kBarriers = 3 * kGemmMaxStages + kGemmGroups + 2;
    static_assert(kBarriers * 8 + 8 + 8 * kGemmLoadWarps <= 512, "the barriers and words do not fit their place");
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(bars + kBarriers);
    volatile unsigned int* abort_flag = reinterpret_cast<volatile unsigned int*>(tmem_slot + 1);
    volatile int* turn_until = reinterpret_cast<volatile int*>(tmem_slot + 2);  // how far the load warps came; in the first block, behind them: the second block's
    const uint32_t abort_addr = bar0 + 8u * kBarriers + 4u, peer_until_addr = abort_addr + 4u + 4u * kGemmLoadWarps;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_rank();
    // work items: (pair of row tiles, K part, token tile), taken round-robin by the pairs; an item is `per` stages of one pair of tiles. The token tiles of the
    // same weights are neighbours, so that HBM is read for one of them
    const int per = a.blocks_per_item, parts = (a.blocks + per - 1) / per, tiles = a.token_tiles, items = a.pairs * parts * tiles, first = blockIdx.x >> 1, step = gridDim.x >> 1;
    auto part_of = [&](int item) { return item / tiles % parts; };
    auto pair_of = [&](int item) { return item / (tiles * parts); };
    constexpr uint32_t kOperandCol = 256;  // tensor memory: the accumulator in columns [0, n), the operands of group g in 64 columns from 256 + 64 g

    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(loaded(s), 1);  // the expect_tx arrival of the loading thread
            mbar_init(empty(s), 1);   // tcgen05.commit
            mbar_init(peer_acts(s), 1);  // the expect_tx arrival of the first block's loading thread
        }
        for (int g = 0; g < kGemmGroups; ++g) mbar_init(a_full(g), 2 * kGemmDecodeWarps / kGemmGroups);  // one arrival per warp of the group in either block
        mbar_init(acc_full, 1);                      // tcgen05.commit after the last MMA of an item
        mbar_init(acc_empty, 2 * kGemmDecodeWarps);  // every warp that reads the accumulator has read its part
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(const_cast<uint32_t*>(tmem_slot))), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_sync_all();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = *tmem_slot;

    if (warp > kGemmDecodeWarps) {
        // ---- loads: one thread issues, but the warp stays together, so that addresses live in uniform registers ----
        const int mine = warp - kGemmDecodeWarps - 1;
        int it0 = 0, until = 0;  // stages of the sequence before this item; behind this warp's last issued stage
        const uint32_t own_bytes = rank == 0 ? kGemmStageBytes + act_bytes : kGemmStageBytes, acts_landed = rank == 0 ? loaded(0) : cluster_addr(peer_acts(0), 0);
        bool okay = true;
        for (int item = first; item < items && okay; item += step) {
            const int tile = pair_of(item) * 2 + static_cast<int>(rank), kb0 = part_of(item) * per, nkb = min(per, a.blocks - kb0);
            const uint8_t* src = a.w + (size_t(tile) * a.blocks + kb0) * kGemmStageBytes;
            for (int k = (mine - it0) & (kGemmLoadWarps - 1); k < nkb; k += kGemmLoadWarps) {
                const int it = it0 + k, s = it % S;
                if (!(okay = __all_sync(0xffffffffu, mbar_wait(empty(s), ((it / S) & 1) ^ 1, abort_flag, a.spin_limit)))) break;
                if (elect_one()) {
                    const uint32_t dst = b_base + s * act_bytes;
                    const int x = (kb0 + k) * kGemmStageCols, y = item % tiles * n + static_cast<int>(rank) * (n / 2);
                    // (the second block's copies may complete on peer_acts before the first one has announced them: the phase waits for the announcement's arrival)
                    const uint32_t acts = acts_landed + 8u * s;
                    mbar_expect_tx(loaded(s), own_bytes);
                    if (rank == 0) mbar_expect_tx(peer_acts(s), act_bytes);
                    bulk_load(raw_base + s * kGemmStageBytes, src + size_t(k) * kGemmStageBytes, kGemmStageBytes, loaded(s));
                    tma_load_2d_pair(dst, &act_map, x, y, acts);
                    tma_load_2d_pair(dst + act_bytes / 2, &act_map, x + 128, y, acts);
                }
                __syncwarp();
                until = it + 1;
            }
            it0 += nkb;
        }
        // its own copies in flight land before the block leaves (the second block's activations: at the end)
        turn_until[mine] = until;
        if (rank == 1 && lane == 0) store_cluster(cluster_addr(peer_until_addr + 4u * mine, 0), static_cast<uint32_t>(until));
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kGemmLoadWarps) : "memory");  // the load warps
        int furthest = until;
        for (int w = 0; w < kGemmLoadWarps; ++w) furthest = max(furthest, turn_until[w]);
        for (int it = gemm_drain_from(furthest, S); it < until; ++it)
            if ((it & (kGemmLoadWarps - 1)) == mine) okay &= mbar_wait(loaded(it % S), (it / S) & 1, abort_flag, a.spin_limit, false);
        if (!__all_sync(0xffffffffu, okay) && lane == 0) raise_abort(abort_addr, rank);
    } else if (warp == kGemmDecodeWarps) {
        // ---- tensor cores of both blocks: eight MMAs per stage (A from tensor memory, B from shared memory), issued by one thread of the first block. The warp
        // stays together around them, so that descriptors live in uniform registers (one lane alone took 80 cycles an instruction) ----
        if (rank == 0) {
            const uint32_t idesc = instr_desc_i8(2 * kGemmM, n);
            int j = 0, s = 0, it = 0;
            bool okay = true;
            // descriptor of stage 0, K tile 0 (128-byte swizzle, 8-row groups 1024 bytes apart); a stage or a tile further on only moves the start address field (16-byte units)
            const uint64_t b_desc0 = smem_desc(b_base, 16, 1024, 2);
            const uint32_t b_stage16 = act_bytes >> 4, b_half16 = act_bytes >> 5;
            for (int item = first; item < items && okay; item += step, ++j) {
                const int kb0 = part_of(item) * per, nkb = min(per, a.blocks - kb0);
                if (!(okay = __all_sync(0xffffffffu, mbar_wait(acc_empty, (j & 1) ^ 1, abort_flag, a.spin_limit)))) {  // the previous item's accumulator has been read
                    if (j > 0) mbar_wait(acc_full, (j - 1) & 1, abort_flag, a.spin_limit, false);  // its products are done before anyone leaves (their end is committed already)
                    break;
                }
                for (int k = 0; k < nkb; ++k, ++it) {
                    const int g = it & (kGemmGroups - 1);
                    // the arrivals of the first block's warps also stand for the activations of both blocks, which they have seen land
                    if (!(okay = __all_sync(0xffffffffu, mbar_wait(a_full(g), (it / kGemmGroups) & 1, abort_flag, a.spin_limit)))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t b_desc = b_desc0 + uint64_t(s * b_stage16);
                    const uint32_t a_tmem = tmem_base + kOperandCol + 64u * g;
                    if (elect_one()) {
#pragma unroll
                        for (int p = 0; p < 8; ++p) mma_i8_ts_pair(tmem_base, a_tmem + 8 * p, b_desc + uint64_t((p >> 2) * b_half16 + (p & 3) * 2), idesc, (k | p) != 0 ? 1u : 0u);
                        mma_commit_pair(empty(s));
                        if (k + 1 == nkb) mma_commit_pair(acc_full);  // arrives when every MMA issued so far has finished
                    }
                    __syncwarp();
                    if (++s == S) s = 0;
                }
                if (!okay) {  // what was issued is done before anyone leaves
                    if (elect_one()) mma_commit_pair(acc_full);
                    __syncwarp();
                    mbar_wait(acc_full, j & 1, abort_flag, a.spin_limit, false);
                }
            }
            if (!okay && lane == 0) raise_abort(abort_addr, rank);
        }
    } else {
        // ---- decode warps: a weight row (64 bytes of a stage = 256 int8 operands) per thread, in groups of four warps ----
        // Group g takes the stages g, g + 4, ... of the pair's sequence. A warp owns the 32 lanes of tensor memory that its index modulo 4
        // selects, so thread (warp, lane) takes row 32 (warp & 3) + lane of the tile and writes the row's operand into that lane with tcgen05.st:
        // no shared-memory store, so no proxy fence between the decode and the tensor cores.
        const int group = warp >> 2, quarter = warp & 3, r = quarter * 32 + lane;
        const uint32_t lanes = tmem_base + (uint32_t(quarter * 32) << 16), a_tmem = lanes + kOperandCol + 64u * group;
        const uint32_t to_full = cluster_addr(a_full(group), 0), to_empty = cluster_addr(acc_empty, 0);
        const bool sees_peer = rank == 0 && quarter == 0;  // one warp of a group waits for the second block's activations too (in the issuing warp, which every stage passes through, a step of 32 sequences took 3 % longer)
        const int own = n / kGemmGroups, c0 = group * own;  // accumulator columns (a multiple of eight) that this group writes out
        bool okay = true;
        auto finish = [&](int item, int j) {  // item `item`, the pair's j-th
            okay = __all_sync(0xffffffffu, mbar_wait(acc_full, j & 1, abort_flag, a.spin_limit));
            if (!okay) return;
            const int row = (pair_of(item) * 2 + static_cast<int>(rank)) * kGemmM + r, vector = item % tiles * n + c0;
            gemm_write_out(lanes + c0, to_empty, own, a.out + (size_t(part_of(item)) * a.batch + vector) * a.ldo + row, a.ldo, row < a.rows ? min(own, a.batch - vector) : 0);
        };
        int j = 0, it0 = 0, before = -1;  // `before`: the item whose accumulator has not been written out yet
        for (int item = first; item < items && okay; item += step, ++j) {
            const int nkb = min(per, a.blocks - part_of(item) * per);
            // A group decodes its first stage of an item before it writes out the item before. (All groups' reads before any store, or the reads first, or whichever is
            // ready first: 0 to 3 us slower of 37 at 46080 x 3072, 256 vectors.)
            bool owed = before >= 0;
            for (int k = (group - it0) & (kGemmGroups - 1); k < nkb && okay; k += kGemmGroups) {
                const int it = it0 + k, s = it % S;
                // The MMAs of this group's previous operand are done - and with them all loads up to that stage, so that the parity of the stage's barrier
                // is not mistaken - and the stage's bytes have landed. (S >= kGemmGroups: the barrier of that operand's stage cannot be a use further on.)
                const int last = it - kGemmGroups;
                if (!okay) break;
                okay = (last < 0 || mbar_wait(empty(last % S), (last / S) & 1, abort_flag, a.spin_limit)) && mbar_wait(loaded(s), (it / S) & 1, abort_flag, a.spin_limit) &&
                       (!sees_peer || mbar_wait(peer_acts(s), (it / S) & 1, abort_flag, a.spin_limit));
                okay = __all_sync(0xffffffffu, okay);
                if (!okay) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint4* raw = reinterpret_cast<const uint4*>(raw_tiles + s * kGemmStageBytes) + r;
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const uint4 x = raw[(2 * half) * kGemmM], y = raw[(2 * half + 1) * kGemmM];
                    uint32_t v[32];
                    decode16(x.x, v), decode16(x.y, v + 4), decode16(x.z, v + 8), decode16(x.w, v + 12);
                    decode16(y.x, v + 16), decode16(y.y, v + 20), decode16(y.z, v + 24), decode16(y.w, v + 28);
                    tmem_store32(a_tmem + 32 * half, v);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster(to_full);
                if (owed) finish(before, j - 1), owed = false;
            }
            if (owed && okay) finish(before, j - 1);
            before = item, it0 += nkb;
        }
        if (okay && before >= 0) finish(before, j - 1);
        if (!okay && lane == 0) raise_abort(abort_addr, rank);
    }
    // ---- leave: everyone is past its last use of tensor memory and of the other block's barriers ----
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (tid == 0 && *abort_flag) atomicExch(a.status, kGemmStatusTimeout);
    cluster_sync_all();
    if (*abort_flag) {  // the same in both blocks: who raised it raised it in both, before the barrier
        // the second block's activations in flight land before it leaves: the first block's barriers show it, once what it had not come to announce is announced
        if (rank == 0 && warp > kGemmDecodeWarps) {
            const int mine = warp - kGemmDecodeWarps - 1, until = turn_until[mine], theirs = turn_until[kGemmLoadWarps + mine];
            int furthest = theirs;
            for (int w = 0; w < kGemmLoadWarps; ++w) furthest = max(furthest, turn_until[kGemmLoadWarps + w]);
            for (int it = gemm_drain_from(furthest, S); it < theirs; ++it) {
                if ((it & (kGemmLoadWarps - 1)) != mine) continue;
                if (!gemm_announced(it, until) && elect_one()) mbar_expect_tx(peer_acts(it % S), act_bytes);
                __syncwarp();
                mbar_wait(peer_acts(it % S), (it / S) & 1, abort_flag, a.spin_limit, false);
            }
        }
        cluster_sync_all();
    }
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

}  // namespace qtb
