// Attention of a step of several sequences and of short prompt chunks (every token its own block per KV head and chunk of the cache) in the reference's
// arithmetic: per token and query head the operations of attention_kernel (decode.cuh), operation for operation (attention.rs:402-469). The
// query heads that share a KV head share one pass over its rows, in rounds of up to 256 positions:
//  A. half a warp holds four key rows as floats, two of the 32 accumulator lanes a thread, and scores them against every head with packed operations; the
//     lanes are added by halving exchanges (addition commutes, so the halves' sums have the bits of the reference's tree);
//  B. every warp turns some (head, 32 positions) into the factors ms / vs: maxima of the 32s first, then a scan inside each;
//  C. 128 threads run the value chains, two neighbouring coordinates packed, all heads of the group (hd = 256) or a part of them; a fifth warp the sums S.
// Key and value rows come as one sequence of 32-row stages through two buffers, so the first values are on their way while the factors are made.
//
// Bound by the instructions of the chains (F16 rounding after every operation: a multiply-add, a conversion and two widenings a pair of coordinates)
// and by HBM; four blocks a multiprocessor, each in another phase, hide one another's latencies. 32 sequences of 256 to 2048 positions, 12 / 4 heads of 256:
// 106 us a layer in attention_gqa_kernel (scalar steps, scores over whole warps, factors by one warp a head), 78 here.
#pragma once
#include "decode.cuh"
#include "packed_f32.cuh"
#include "prompt_attention.cuh"

namespace qtb {

constexpr int kRowAttnThreads = 160, kRowAttnChainThreads = 128, kRowAttnRound = 256, kRowAttnStage = 32, kRowAttnBuffers = 2;
__host__ __device__ constexpr int row_attn_stride(int hd) { return hd * 2 + 16; }  // bytes: the two halves of a warp read rows four apart, 64 bytes apart in the banks
__host__ __device__ constexpr size_t row_attn_smem(int g, int hd) {
    return static_cast<size_t>(kRowAttnBuffers) * kRowAttnStage * row_attn_stride(hd) + static_cast<size_t>(g) * (kRowAttnRound * 12 + hd * 4 + 40) + 32;
}

template <int G, int E, bool F32>  // query heads per KV head, head_dim / 32
__global__ void __launch_bounds__(kRowAttnThreads, 4) attention_rows_kernel(AttnArgs a) {
    constexpr int hd = 32 * E, kStride = row_attn_stride(hd), kStageBytes = kRowAttnStage * kStride, kRoundStages = kRowAttnRound / kRowAttnStage;
    constexpr int kPairs = hd / 2, kHeadStep = kRowAttnChainThreads / kPairs, kChains = (G + kHeadStep - 1) / kHeadStep;  // a chain thread takes heads tid / kPairs, + kHeadStep, ...
    extern __shared__ __align__(16) unsigned char rows_smem[];
    float2* s_vs = reinterpret_cast<float2*>(rows_smem + kRowAttnBuffers * kStageBytes);  // [G][256]: vs twice (packed operand); before that the score
    float* s_ms = reinterpret_cast<float*>(s_vs + G * kRowAttnRound);                   // [G][256]
    float* s_q = s_ms + G * kRowAttnRound;                                              // [G][hd]
    float* s_bm = s_q + G * hd;                                                         // [G][8]: maxima of 32 positions
    float* s_carry = s_bm + G * kRoundStages;                                           // [G] (two words a head in the plan above): the maximum before the round
    unsigned int* s_moved = reinterpret_cast<unsigned int*>(s_carry + 2 * G);           // [8]: positions at which some head's maximum moves by a factor other than one
    const int kvh = blockIdx.x, c = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h0 = kvh * G;
    const size_t z = blockIdx.z;
    const int seq_len = static_cast<int>(seq_position(a.seq, a.pos, blockIdx.z)) + 1;
    const int n_kv = min(max((seq_len + 255) / 256 * 256, 256), a.ctx);
    int start = 0, end = seq_len;
    if (n_kv >= 512) {
        const int chunk = (n_kv + 3) / 4;
        start = c * chunk, end = min(min(start + chunk, n_kv), seq_len);
    } else if (c > 0) {
        start = end;  // single-chunk case: chunks 1..3 are empty
    }
    const int len = end - start;
    float* my_ms = a.part_ms + z * a.b_ms + (static_cast<size_t>(h0) * 4 + c) * 2;
    if (len <= 0) {
        if (tid < G) my_ms[tid * 8] = -INFINITY, my_ms[tid * 8 + 1] = 0.0f;
        return;
    }
    const size_t first = seq_cache_offset(a.seq, blockIdx.z) + static_cast<size_t>(kvh) * hd + static_cast<size_t>(start) * a.kv_dim;
    const __half *kbase = a.k_cache + first, *vbase = a.v_cache + first;
    const int rounds = (len + kRowAttnRound - 1) / kRowAttnRound, last_stages = (len - (rounds - 1) * kRowAttnRound + kRowAttnStage - 1) / kRowAttnStage;
    const int total = (rounds - 1) * 2 * kRoundStages + 2 * last_stages;
    auto issue = [&](int s) {  // stage s: 32 key or value rows (always closes a copy group, so every thread counts the same groups)
        if (s < total) {
            const int round = s / (2 * kRoundStages), in = s % (2 * kRoundStages), n = round + 1 < rounds ? kRoundStages : last_stages;
            const int row0 = round * kRowAttnRound + (in < n ? in : in - n) * kRowAttnStage;
            const __half* src = (in < n ? kbase : vbase) + static_cast<size_t>(row0) * a.kv_dim;
            unsigned char* dst = rows_smem + (s % kRowAttnBuffers) * kStageBytes;
            constexpr int kPieces = hd / 8;  // 16-byte pieces of a row
            const int pieces = min(kRowAttnStage, len - row0) * kPieces;
            for (int i = tid; i < pieces; i += kRowAttnThreads) attn_cp16(dst + (i / kPieces) * kStride + (i % kPieces) * 16, src + static_cast<size_t>(i / kPieces) * a.kv_dim + (i % kPieces) * 8);
        }
        attn_cp_commit();
    };
#pragma unroll
    for (int k = 0; k < kRowAttnBuffers - 1; ++k) issue(k);
    for (int i = tid; i < G * hd; i += kRowAttnThreads) {
        const float v = a.q[z * a.b_q + h0 * hd + i];
        s_q[i] = F32 ? v : __half2float(__float2half_rn(v));
    }
    if (tid < G) s_carry[tid] = -INFINITY;
    const bool chain = warp < kRowAttnChainThreads / 32;
    const int pair = tid % kPairs, head0 = tid / kPairs;
    unsigned long long acc[kChains];
#pragma unroll
    for (int k = 0; k < kChains; ++k) acc[k] = 0ull;
    float S = 0.0f;
    const unsigned long long exp_entry = g_exp2_tab[lane];
    int s = 0;
    auto next_stage = [&]() -> const unsigned char* {  // its rows have landed; the buffer of the stage before is filled again
        asm volatile("cp.async.wait_group %0;" ::"n"(kRowAttnBuffers - 2) : "memory");
        __syncthreads();
        issue(s + kRowAttnBuffers - 1);
        return rows_smem + (s++ % kRowAttnBuffers) * kStageBytes;
    };
    for (int round = 0; round < rounds; ++round) {
        const int rows = min(kRowAttnRound, len - round * kRowAttnRound), stages = (rows + kRowAttnStage - 1) / kRowAttnStage;
        for (int t = 0; t < stages; ++t) {  // A (rows past the end give scores that nothing reads)
            const unsigned char* st = next_stage();
            if (!chain || t * kRowAttnStage + 8 * warp >= rows) continue;
            const int j = lane & 15, row0 = 8 * warp + 4 * (lane >> 4);  // accumulator lanes 2j, 2j + 1 of four rows
            unsigned long long kf[4][E];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int i = 0; i < E; ++i) kf[r][i] = widen_half2(*reinterpret_cast<const uint32_t*>(st + (row0 + r) * kStride + i * 64 + j * 4));
#pragma unroll 1
            for (int g = 0; g < G; ++g) {
                unsigned long long v[4] = {0ull, 0ull, 0ull, 0ull};
                const unsigned long long* q = reinterpret_cast<const unsigned long long*>(s_q + g * hd) + j;
#pragma unroll
                for (int i = 0; i < E; ++i) {
                    const unsigned long long x = q[i * 16];
#pragma unroll
                    for (int r = 0; r < 4; ++r) v[r] = fma_f32x2(kf[r][i], x, v[r]);
                }
                // lanes 16, 8, 4 apart, then neighbours (dot_lane_reduce_f16), or 8, 16, 4, 2 apart and neighbours (dot_lane_reduce_f16_f32)
                constexpr int kFirst = F32 ? 4 : 8, kSecond = F32 ? 8 : 4;
                halve_f32x2(v, 4, kFirst, (j & kFirst) != 0);
                halve_f32x2(v, 2, kSecond, (j & kSecond) != 0);
                v[0] = add_f32x2(v[0], shfl_xor_f32x2(v[0], 2));
                float score;
                if constexpr (F32) {
                    const float2 f = unpack_f32x2(add_f32x2(v[0], shfl_xor_f32x2(v[0], 1)));
                    score = __fadd_rn(f.x, f.y);
                } else {
                    const float2 f = unpack_f32x2(v[0]);
                    score = __fadd_rn(f.x, f.y);
                    score = __fadd_rn(score, __shfl_xor_sync(0xffffffffu, score, 1));
                }
                const int r = ((j & kFirst) != 0 ? 2 : 0) + ((j & kSecond) != 0 ? 1 : 0);  // which row the exchanges left here
                if ((j & 3) == 0) s_vs[g * kRowAttnRound + t * kRowAttnStage + row0 + r].x = __fmul_rn(score, a.scale);
            }
        }
        __syncthreads();
        // B: the running maximum is a prefix maximum, so maxima of the 32s and a scan inside each give the sequential values
        for (int t = warp; t < G * stages; t += kRowAttnThreads / 32) {
            const int g = t / stages, b = t - g * stages, p = b * 32 + lane;
            float m = p < rows ? s_vs[g * kRowAttnRound + p].x : -INFINITY;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (lane == 0) s_bm[g * kRoundStages + b] = m;
        }
        if (tid < kRoundStages) s_moved[tid] = 0u;
        __syncthreads();
        for (int t = warp; t < G * stages; t += kRowAttnThreads / 32) {
            const int g = t / stages, b = t - g * stages, p = b * 32 + lane;
            float carry = s_carry[g];
            for (int k = 0; k < b; ++k) carry = fmaxf(carry, s_bm[g * kRoundStages + k]);
            const float sc = p < rows ? s_vs[g * kRowAttnRound + p].x : -INFINITY;
            float incl = sc;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float up = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl = fmaxf(incl, up);
            }
            float excl = __shfl_up_sync(0xffffffffu, incl, 1);
            if (lane == 0) excl = -INFINITY;
            const float m_old = fmaxf(carry, excl);
            const bool up = sc > m_old;
            const float ex = device_expf_warp(up ? __fsub_rn(m_old, sc) : __fsub_rn(sc, m_old), exp_entry);
            if (p < rows) {
                s_ms[g * kRowAttnRound + p] = up ? ex : 1.0f;
                s_vs[g * kRowAttnRound + p] = up ? make_float2(1.0f, 1.0f) : make_float2(ex, ex);
            }
            const unsigned int moved = __ballot_sync(0xffffffffu, p < rows && up && ex != 1.0f);
            if (lane == 0 && moved != 0u) atomicOr(s_moved + b, moved);
        }
        for (int t = 0; t < stages; ++t) {  // C
            const unsigned char* st = next_stage();  // (the first one also publishes the factors)
            const int base = t * kRowAttnStage, n = min(kRowAttnStage, rows - base);
            if (chain) {
                const unsigned char* col = st + pair * 4;
                const float2* vs = s_vs + head0 * kRowAttnRound + base;
                const float* ms = s_ms + head0 * kRowAttnRound + base;
                const unsigned int moved = s_moved[t];
                auto add = [&](int r) {
                    const unsigned long long vf = widen_half2(*reinterpret_cast<const uint32_t*>(col + r * kStride));
#pragma unroll
                    for (int k = 0; k < kChains; ++k)
                        if (G % kHeadStep == 0 || head0 + k * kHeadStep < G)
                            acc[k] = value_round2<F32>(fma_f32x2(vf, *reinterpret_cast<const unsigned long long*>(vs + k * kHeadStep * kRowAttnRound + r), acc[k]));
                };
                int r = 0;
                while (r < n) {  // stretches without a moved maximum have no branch; at the positions between them the accumulators are rescaled first
                    const unsigned int later = moved >> r;
                    const int stop = later != 0u ? r + __ffs(static_cast<int>(later)) - 1 : n;
#pragma unroll 4
                    for (; r < stop; ++r) add(r);
                    if (r < n) {
#pragma unroll
                        for (int k = 0; k < kChains; ++k) {
                            if (G % kHeadStep == 0 || head0 + k * kHeadStep < G) {
                                const float m = ms[k * kHeadStep * kRowAttnRound + r];
                                if (m != 1.0f) acc[k] = value_round2<F32>(mul_f32x2(acc[k], pack_f32x2(m, m)));
                            }
                        }
                        add(r++);
                    }
                }
            } else if (lane < G) {
                const float2* vs = s_vs + lane * kRowAttnRound + base;
                const float* ms = s_ms + lane * kRowAttnRound + base;
#pragma unroll 8
                for (int r = 0; r < n; ++r) S = __fmaf_rn(S, ms[r], vs[r].x);  // attention.rs:466
                if (t == 0) {
                    float m = s_carry[lane];
                    for (int k = 0; k < stages; ++k) m = fmaxf(m, s_bm[lane * kRoundStages + k]);
                    s_carry[lane] = m;
                }
            }
        }
    }
    if (chain) {
        float* out = a.part_acc + z * a.b_acc + (static_cast<size_t>(h0) * 4 + c) * hd + 2 * pair;
#pragma unroll
        for (int k = 0; k < kChains; ++k)
            if (G % kHeadStep == 0 || head0 + k * kHeadStep < G) *reinterpret_cast<float2*>(out + static_cast<size_t>(head0 + k * kHeadStep) * 4 * hd) = unpack_f32x2(acc[k]);
    } else if (lane < G) {
        my_ms[lane * 8] = s_carry[lane], my_ms[lane * 8 + 1] = S;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The instantiation for a group size, head size and numerics, or nullptr where there is none.
inline AttnGqaKernel attention_rows_for(int gqa, int hd, bool f32_values) {
    auto pick = [&](auto g) -> AttnGqaKernel {
        constexpr int G = decltype(g)::value;
        switch (hd) {
            case 64: return f32_values ? attention_rows_kernel<G, 2, true> : attention_rows_kernel<G, 2, false>;
            case 128: return f32_values ? attention_rows_kernel<G, 4, true> : attention_rows_kernel<G, 4, false>;
            case 256: return f32_values ? attention_rows_kernel<G, 8, true> : attention_rows_kernel<G, 8, false>;
            default: return nullptr;
        }
    };
    switch (gqa) {
        case 1: return pick(std::integral_constant<int, 1>{});
        case 2: return pick(std::integral_constant<int, 2>{});
        case 3: return pick(std::integral_constant<int, 3>{});
        case 4: return pick(std::integral_constant<int, 4>{});
        default: return nullptr;
    }
}

}  // namespace qtb
