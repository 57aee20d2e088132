// Shared-memory plan of the token kernel (megakernel.cuh), and which models take that kernel: plain arithmetic, so that it can be followed without a device.
//
// Bytes from the dynamic base: attention region (its first 64 KiB double as the GEMV table) | y (floats) | a8 | small arrays | weights of the next norm | a row of the cos/sin
// table | the kernel's arguments | a descriptor per layer. The attention region holds whichever is largest: a scores unit (staged key block, the group's queries,
// the new key/value rows), a values unit for the longest chunk, or the output head's activations (floats).
#pragma once
#include <cstddef>

#ifdef __CUDACC__
#define QTB_PLAN_FN __host__ __device__ constexpr
#else
#define QTB_PLAN_FN constexpr
#endif

namespace qtb {

constexpr int kMegaThreads = 512;
constexpr int kMegaWarps = kMegaThreads / 32;
constexpr int kMegaMaxHeads = 64;
constexpr int kMegaCosSin = 256;  // floats of a row of the cos/sin table: rope_dims <= head_dim <= 256
constexpr int kAttnBlockPos = 128;                          // positions staged in shared memory at a time
constexpr int kAttnBlockBytes = kAttnBlockPos * 256 * 2;    // one staged block (head_dim <= 256 halves per row)
constexpr int kAttnSlice = 32;  // coordinates of a head that one values unit accumulates (one warp per query head)

constexpr int kV2Dims = 16;      // second form: coordinates per unit, two warps of eight coordinates x four chunks per query head
constexpr int kV2WarpsPerHead = kV2Dims / 8;
constexpr int kV2MaxCtx = 4096;
static_assert(kV2MaxCtx / 4 / 8 < 256, "a group's number fits the low byte of the table of next groups");
constexpr int kV2MaxGqa = 7;     // chain warps (two per head) + the warp of the sum chains must fit the 16 warps of the CTA

QTB_PLAN_FN size_t plan_up(size_t n, size_t unit) { return (n + unit - 1) / unit * unit; }

// Shared memory a values unit needs for chunks of `len` positions and `gqa` query heads per KV head.
QTB_PLAN_FN size_t values_unit_bytes(int len, int gqa) {
    return plan_up(static_cast<size_t>(len) * kAttnSlice * 2, 16) + static_cast<size_t>(2) * gqa * len * 4 + (kMegaWarps + 16) * 4 + plan_up(static_cast<size_t>(gqa) * ((len + 7) / 8 + 1) * 3, 16);
}
// Second form. Row length (floats) of the factor rows for chunks of `chunk` positions: a multiple of 8, at least `chunk`.
QTB_PLAN_FN int values2_clp(int chunk) { return (chunk + 7) / 8 * 8; }
// Positions per chunk in the staged V block: odd, so that the 32-byte pieces the four chunks' lanes read at one step fall into
// four different bank groups.
QTB_PLAN_FN int values2_clr(int chunk) { return values2_clp(chunk) + 1; }
QTB_PLAN_FN int values2_chunks(int ctx) { return ctx >= 512 ? 4 : 1; }
QTB_PLAN_FN int values2_chunk(int ctx) { return ctx >= 512 ? (ctx + 3) / 4 : ctx; }
// V block, factor rows, next groups, chunk-combine factors, M and S.
QTB_PLAN_FN size_t values2_rows_bytes(int ctx, int gqa) {
    const int nch = values2_chunks(ctx), chunk = values2_chunk(ctx), clp = values2_clp(chunk);
    return static_cast<size_t>(nch) * values2_clr(chunk) * kV2Dims * 2 + static_cast<size_t>(2) * gqa * nch * clp * 4 + static_cast<size_t>(gqa) * (clp / 8) * 4 + static_cast<size_t>(gqa) * 8 * 4 +
           static_cast<size_t>(gqa) * nch * 8 + 64;
}
// ... and a byte per (head, chunk, group of eight positions): where the maximum moves.
QTB_PLAN_FN size_t values2_bytes(int ctx, int gqa) { return values2_rows_bytes(ctx, gqa) + static_cast<size_t>(gqa) * values2_chunks(ctx) * (values2_clp(values2_chunk(ctx)) / 8); }

QTB_PLAN_FN size_t mega_region(int gqa, int head_dim, int hidden, size_t values, size_t least, size_t unit) {
    size_t need = static_cast<size_t>(kAttnBlockBytes) + static_cast<size_t>(gqa) * head_dim * 4 + static_cast<size_t>(head_dim) * 4 + 64;
    const size_t head = static_cast<size_t>(hidden) * 4;
    if (values > need) need = values;
    if (head > need) need = head;
    if (least > need) need = least;
    return plan_up(need, unit);
}
QTB_PLAN_FN size_t mega_values(int ctx, int gqa, bool v2) { return v2 ? values2_bytes(ctx, gqa) : values_unit_bytes(ctx < 512 ? ctx : (ctx + 3) / 4, gqa); }
QTB_PLAN_FN size_t mega_attn_region(int ctx, int gqa, int head_dim, int hidden, bool v2) { return mega_region(gqa, head_dim, hidden, mega_values(ctx, gqa, v2), 127 * 1024, 16); }

// The small arrays: one double and one float per warp, the exponential's table, four scales, a flag and the position.
constexpr size_t kMegaSmallSumF = kMegaWarps * 8, kMegaSmallExp = kMegaSmallSumF + kMegaWarps * 4, kMegaSmallScale = kMegaSmallExp + 32 * 8, kMegaSmallFlag = kMegaSmallScale + 16,
                 kMegaSmallPos = kMegaSmallFlag + 4, kMegaSmallBytes = (kMegaSmallPos + 4 + 15) / 16 * 16;
constexpr size_t kMegaArgsBytes = 464, kMegaLayerBytes = 192;  // sizeof(MegaArgs) in whole 16 bytes, sizeof(MegaLayer)
QTB_PLAN_FN size_t mega_smem_bytes(size_t attn_region, int maxvec, int hidden, int layers) {
    return attn_region + static_cast<size_t>(maxvec) * 4 + plan_up(maxvec, 16) + kMegaSmallBytes + plan_up(static_cast<size_t>(hidden) * 4, 16) + static_cast<size_t>(kMegaCosSin) * 4 + kMegaArgsBytes +
           static_cast<size_t>(layers) * kMegaLayerBytes;
}

// Whether a model takes the token kernel is not decided by the plan above but by this sum, which the plan never exceeds: what lies in shared memory has changed and may change
// again, and the models that take the kernel - without which tensor parallelism refuses them - are to stay the same. 4096 bytes stand for the small arrays, cos/sin row,
// arguments and moved positions, 200 for a layer. The region is charged 129 KiB at least: wider models (past 8 to 9 thousand values) have not been run through the kernel and
// take one kernel per step.
QTB_PLAN_FN size_t mega_charge(int ctx, int gqa, int head_dim, int hidden, int maxvec, int layers, bool v2) {
    const size_t values = v2 ? values2_rows_bytes(ctx, gqa) : mega_values(ctx, gqa, false);
    return mega_region(gqa, head_dim, hidden, values, 129 * 1024, 1024) + static_cast<size_t>(maxvec) * 4 + plan_up(maxvec, 16) + 4096 + plan_up(static_cast<size_t>(hidden) * 4, 16) +
           static_cast<size_t>(layers) * 200;
}

}  // namespace qtb
