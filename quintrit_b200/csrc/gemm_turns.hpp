// The order in which the load warps of the batched projection (gemm_tc.cuh) take the stages, as far as its exits need it: plain integers, so that it
// can be followed without a device.
#pragma once

#ifdef __CUDACC__
#define QTB_TURNS_FN __host__ __device__ inline constexpr
#else
#define QTB_TURNS_FN inline constexpr
#endif

namespace qtb {

constexpr int kGemmLoadWarps = 2;  // load warp w fetches the stages w, w + 2, ... of the pair's sequence: the fixed cost of a stage (about 600 cycles in one warp) would bound small batches

// The first stage whose copies a block's load warps wait for before it leaves; `until` is behind the last stage that any of them issued. That one was issued only after the
// products of the stage S before it, which lay in the same buffer, were done, and they read all stages up to it: of the stages before until - S nothing is in flight
// any more. From there on no buffer has been used again, so a stage's barrier is still in the phase behind its copies. It holds wherever the warps stopped, also in the middle of
// an item: what counts is how far they came, not where the item would have ended.
QTB_TURNS_FN int gemm_drain_from(int until, int stages) { return until > stages ? until - stages : 0; }

// Whether the first block has announced (expect_tx) the second one's activations of a stage: its load warp of the same turn, which came to `until`, does so when it issues its own.
QTB_TURNS_FN bool gemm_announced(int it, int until) { return it < until; }

}  // namespace qtb
