// Attention of a prompt chunk (many consecutive tokens of one sequence) in the reference's arithmetic: per token and query
// head the operations of attention_kernel (decode.cuh), operation for operation (attention.rs:402-469); only who does them
// differs. attention_gqa_kernel gives every token a block of its own, which reads the whole cache from L2 for one token,
// reduces every score over the lanes of a warp with five shuffles and runs the value chains of a coordinate in scalar steps.
// Here a block takes eight tokens of a KV head: the cache rows come to shared memory once for all of them, and
//  A. a warp holds eight key rows of a 64-row tile in registers (as floats, two of the 32 accumulator lanes per thread) and
//     scores them against every query of the block; the lanes are added by halving exchanges that reduce sixteen scores
//     with fifteen shuffles (addition commutes, so the halves' sums have the bits of the reference's tree);
//  B. a warp turns its own token's scores into the factors ms / vs with a warp scan;
//  C. the same warp runs all value chains of its token: a lane owns head_dim / 32 coordinates, two to a packed operation
//     (fma.rn.f32x2 rounds each half on its own; one conversion rounds both accumulators to F16).
// Bound by instruction issue and, in C, by the heavy half of the FMA pipe, which converts between F16 and F32 (ncu, 232 tokens at positions 768 to 999, 12 /
// 4 heads of 256: 201 us, while a multiprocessor is active 54 % of the issue slots and 58 % of that pipe; 40 warp instructions per token, head and
// position with the tiles' overhang, of which the source has 9 in a score and 22 in the chains). The 1000-token prompt of a 4-layer Falcon3-10B shape:
// 8.03 -> 6.11 ms against a block per token (attention_gqa_kernel). With all 1000 tokens in one launch, the last first: 580 -> 418 us a layer; still half the issue slots and half of the
// heavy side busy, 3.8 warps a scheduler (128 registers, 110 KB a block). Widening by mixed-precision additions, which either side takes: 3 % slower.
#pragma once
#include "decode.cuh"
#include "packed_f32.cuh"

namespace qtb {

constexpr int kTokenTile = 8, kTokenTileRows = 64, kTokenTileThreads = 256;
__host__ __device__ constexpr int attn_tile_key_stride(int hd) { return hd * 2 + 16; }  // bytes: the two half-warps of a warp read rows four apart, 64 bytes apart in the banks
__host__ __device__ constexpr size_t attn_tile_smem(int g, int hd) {
    return static_cast<size_t>(kTokenTileRows) * (attn_tile_key_stride(hd) + hd * 2) + static_cast<size_t>(kTokenTile) * g * (hd * 4 + kTokenTileRows * 12);
}

template <bool F32>
__device__ __forceinline__ unsigned long long value_round2(unsigned long long v) {  // value_round of both halves
    if constexpr (F32) return v;
    const float2 f = unpack_f32x2(v);
    const float2 r = __half22float2(__floats2half2_rn(f.x, f.y));
    return pack_f32x2(r.x, r.y);
}
// Grid (kv_heads, 4 chunks, token tiles). Token tiles are aligned to positions that are multiples of eight, so that the
// tokens of a tile agree on the division of the cache into chunks (it changes at multiples of 256).
template <int G, int E, bool F32>  // query heads per KV head, head_dim / 32
__global__ void __launch_bounds__(kTokenTileThreads, 2) attention_tile_kernel(AttnArgs a) {
    constexpr int hd = 32 * E, R = kTokenTile * G, kKeyStride = attn_tile_key_stride(hd);
    extern __shared__ __align__(16) unsigned char tile_smem[];
    unsigned char* s_k = tile_smem;                                                      // [64][kKeyStride bytes]
    __half* s_v = reinterpret_cast<__half*>(s_k + kTokenTileRows * kKeyStride);               // [64][hd]
    float* s_q = reinterpret_cast<float*>(s_v + kTokenTileRows * hd);                         // [R][hd]
    float2* s_vs = reinterpret_cast<float2*>(s_q + R * hd);                              // [R][64]: vs twice (packed operand); before that the score
    float* s_ms = reinterpret_cast<float*>(s_vs + R * kTokenTileRows);                        // [R][64]
    const int kvh = blockIdx.x, c = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h0 = kvh * G;
    const int pos0 = static_cast<int>(a.pos[0]), first = (pos0 / kTokenTile + static_cast<int>(gridDim.z - 1 - blockIdx.z)) * kTokenTile;  // the last tokens, whose rows are most, first
    const int last = min(first + kTokenTile, pos0 + a.tokens) - 1;  // the last position of the tile that is a token of the chunk
    if (last < first) return;
    const int n_kv = min(max((last + 1 + 255) / 256 * 256, 256), a.ctx);
    int start = 0, chunk_end = n_kv;
    if (n_kv >= 512) {
        const int chunk = (n_kv + 3) / 4;
        start = c * chunk, chunk_end = min(start + chunk, n_kv);
    } else if (c > 0) {
        chunk_end = 0;  // single-chunk case: chunks 1..3 are empty
    }
    const int p = first + warp, z = p - pos0;  // this warp's token
    const bool mine = z >= 0 && p <= last;
    const int len = mine ? min(chunk_end, p + 1) - start : 0, len_block = min(chunk_end, last + 1) - start;
    if (mine && len <= 0 && lane < G) {
        float* my_ms = a.part_ms + static_cast<size_t>(z) * a.b_ms + (static_cast<size_t>(h0 + lane) * 4 + c) * 2;
        my_ms[0] = -INFINITY, my_ms[1] = 0.0f;
    }
    if (len_block <= 0) return;
    const __half* kbase = a.k_cache + static_cast<size_t>(kvh) * hd + static_cast<size_t>(start) * a.kv_dim;
    const __half* vbase = a.v_cache + static_cast<size_t>(kvh) * hd + static_cast<size_t>(start) * a.kv_dim;
    constexpr int kPieces = hd / 8;  // 16-byte pieces of a row
    auto issue = [&](const __half* rows, int base, unsigned char* dst, int stride) {
        const int n = min(kTokenTileRows, len_block - base) * kPieces;
        for (int i = tid; i < n; i += kTokenTileThreads)
            attn_cp16(dst + (i / kPieces) * stride + (i % kPieces) * 16, rows + static_cast<size_t>(base + i / kPieces) * a.kv_dim + (i % kPieces) * 8);
        attn_cp_commit();
    };
    issue(kbase, 0, s_k, kKeyStride);
    issue(vbase, 0, reinterpret_cast<unsigned char*>(s_v), hd * 2);
    // queries: row t * G + g; positions of the tile that are no token of the chunk read as zeros
    for (int i = tid; i < R * hd; i += kTokenTileThreads) {
        const int t = i / (G * hd), zt = first + t - pos0;
        const float v = zt >= 0 && first + t <= last ? a.q[static_cast<size_t>(zt) * a.b_q + h0 * hd + i % (G * hd)] : 0.0f;
        s_q[i] = F32 ? v : __half2float(__float2half_rn(v));
    }
    unsigned long long acc[G][E / 2];
    float S[G], carry[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        S[g] = 0.0f, carry[g] = -INFINITY;
#pragma unroll
        for (int e = 0; e < E / 2; ++e) acc[g][e] = 0ull;
    }
    const unsigned long long exp_entry = g_exp2_tab[lane];
    const int j = lane & 15, row0 = 8 * warp + 4 * (lane >> 4);  // phase A: accumulator lanes 2j, 2j + 1 of four rows
    for (int base = 0; base < len_block; base += kTokenTileRows) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");  // the keys; the values may still be on their way
        __syncthreads();
        if (base + 8 * warp < len_block) {  // A (rows past the chunk's end give scores that nothing reads)
            unsigned long long kf[4][E];
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int i = 0; i < E; ++i) kf[r][i] = widen_half2(*reinterpret_cast<const uint32_t*>(s_k + (row0 + r) * kKeyStride + i * 64 + j * 4));
#pragma unroll 1
            for (int r0 = 0; r0 < R; r0 += 2) {
                unsigned long long v[8];
#pragma unroll
                for (int k = 0; k < 8; ++k) v[k] = 0ull;
                const unsigned long long* q0 = reinterpret_cast<const unsigned long long*>(s_q + r0 * hd) + j;
#pragma unroll
                for (int i = 0; i < E; ++i) {
                    const unsigned long long x0 = q0[i * 16], x1 = q0[hd / 2 + i * 16];
#pragma unroll
                    for (int r = 0; r < 4; ++r) v[r] = fma_f32x2(kf[r][i], x0, v[r]), v[4 + r] = fma_f32x2(kf[r][i], x1, v[4 + r]);
                }
                // lanes 16, 8, 4 apart, then neighbours (dot_lane_reduce_f16), or 8, 16, 4, 2 apart and neighbours (dot_lane_reduce_f16_f32)
                constexpr int kFirst = F32 ? 4 : 8, kSecond = F32 ? 8 : 4;
                halve_f32x2(v, 8, kFirst, (j & kFirst) != 0);
                halve_f32x2(v, 4, kSecond, (j & kSecond) != 0);
                halve_f32x2(v, 2, 2, (j & 2) != 0);
                float score;
                if constexpr (F32) {
                    const float2 f = unpack_f32x2(add_f32x2(v[0], shfl_xor_f32x2(v[0], 1)));
                    score = __fadd_rn(f.x, f.y);
                } else {
                    const float2 f = unpack_f32x2(v[0]);
                    score = __fadd_rn(f.x, f.y);
                    score = __fadd_rn(score, __shfl_xor_sync(0xffffffffu, score, 1));
                }
                // which of the eight values this thread ended with: bit 2 by the first exchange, bit 1 by the second, bit 0 by the third
                const int k = ((j & kFirst) != 0 ? 4 : 0) + ((j & kSecond) != 0 ? 2 : 0) + ((j & 2) != 0 ? 1 : 0);
                if ((j & 1) == 0) s_vs[(r0 + (k >> 2)) * kTokenTileRows + row0 + (k & 3)].x = __fmul_rn(score, a.scale);
            }
        }
        __syncthreads();
        if (base + kTokenTileRows < len_block)
            issue(kbase, base + kTokenTileRows, s_k, kKeyStride);
        else
            attn_cp_commit();  // (every thread counts the same groups)
        const int rows = min(kTokenTileRows, len - base);
        // B: the running maximum is a prefix maximum, so the scan gives the sequential values
        unsigned int moved[kTokenTileRows / 32];  // the positions at which some head's maximum moves (ms != 1): a few per token
#pragma unroll
        for (int b = 0; b < kTokenTileRows / 32; ++b) moved[b] = 0u;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float2* vs_g = s_vs + (warp * G + g) * kTokenTileRows;
            float* ms_g = s_ms + (warp * G + g) * kTokenTileRows;
#pragma unroll
            for (int b = 0; b < kTokenTileRows / 32; ++b) {
                const int r = 32 * b + lane;
                const float sc = r < rows ? vs_g[r].x : -INFINITY;
                float incl = sc;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const float up = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl = fmaxf(incl, up);
                }
                float excl = __shfl_up_sync(0xffffffffu, incl, 1);
                if (lane == 0) excl = -INFINITY;
                const float m_old = fmaxf(carry[g], excl);
                const bool up = sc > m_old;
                const float ex = device_expf_warp(up ? __fsub_rn(m_old, sc) : __fsub_rn(sc, m_old), exp_entry);
                if (r < rows) {
                    ms_g[r] = up ? ex : 1.0f;
                    vs_g[r] = up ? make_float2(1.0f, 1.0f) : make_float2(ex, ex);
                }
                moved[b] |= __ballot_sync(0xffffffffu, r < rows && up && ex != 1.0f);
                carry[g] = fmaxf(carry[g], __shfl_sync(0xffffffffu, incl, 31));
            }
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");  // the values
        __syncthreads();
        // C: stretches without a moved maximum have no branch; at the positions between them the accumulators are rescaled first
        {
            const unsigned long long* vs_w = reinterpret_cast<const unsigned long long*>(s_vs + warp * G * kTokenTileRows);
            const float* ms_w = s_ms + warp * G * kTokenTileRows;
            const __half* vrow = s_v + lane * E;
            auto add = [&](int r) {
                unsigned long long vf[E / 2];
                if constexpr (E == 8) {
                    const uint4 h = *reinterpret_cast<const uint4*>(vrow + r * hd);
                    vf[0] = widen_half2(h.x), vf[1] = widen_half2(h.y), vf[2] = widen_half2(h.z), vf[3] = widen_half2(h.w);
                } else if constexpr (E == 4) {
                    const uint2 h = *reinterpret_cast<const uint2*>(vrow + r * hd);
                    vf[0] = widen_half2(h.x), vf[1] = widen_half2(h.y);
                } else {
                    vf[0] = widen_half2(*reinterpret_cast<const uint32_t*>(vrow + r * hd));
                }
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const unsigned long long vs = vs_w[g * kTokenTileRows + r];
#pragma unroll
                    for (int e = 0; e < E / 2; ++e) acc[g][e] = value_round2<F32>(fma_f32x2(vf[e], vs, acc[g][e]));
                }
            };
            int r = 0;
            while (r < rows) {
                const unsigned long long later = (static_cast<unsigned long long>(moved[1]) << 32 | moved[0]) >> r;
                const int stop = later != 0ull ? r + __ffsll(static_cast<long long>(later)) - 1 : rows;
#pragma unroll 4
                for (; r < stop; ++r) {
                    add(r);
#pragma unroll
                    for (int g = 0; g < G; ++g) S[g] = __fadd_rn(S[g], s_vs[(warp * G + g) * kTokenTileRows + r].x);
                }
                if (r < rows) {
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        const float ms = ms_w[g * kTokenTileRows + r];
                        if (ms != 1.0f) {
                            const unsigned long long m2 = pack_f32x2(ms, ms);
#pragma unroll
                            for (int e = 0; e < E / 2; ++e) acc[g][e] = value_round2<F32>(mul_f32x2(acc[g][e], m2));
                        }
                        S[g] = __fmaf_rn(S[g], ms, s_vs[(warp * G + g) * kTokenTileRows + r].x);  // attention.rs:466
                    }
                    add(r++);
                }
            }
        }
        __syncthreads();
        if (base + kTokenTileRows < len_block)
            issue(vbase, base + kTokenTileRows, reinterpret_cast<unsigned char*>(s_v), hd * 2);
        else
            attn_cp_commit();
    }
    if (len > 0) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float* out = a.part_acc + static_cast<size_t>(z) * a.b_acc + (static_cast<size_t>(h0 + g) * 4 + c) * hd + lane * E;
#pragma unroll
            for (int e = 0; e < E / 2; ++e) *reinterpret_cast<float2*>(out + 2 * e) = unpack_f32x2(acc[g][e]);
            if (lane == 0) {
                float* my_ms = a.part_ms + static_cast<size_t>(z) * a.b_ms + (static_cast<size_t>(h0 + g) * 4 + c) * 2;
                my_ms[0] = carry[g], my_ms[1] = S[g];
            }
        }
    }
}

// The instantiation for a group size, head size and numerics, or nullptr where there is none.
inline AttnGqaKernel attention_tile_for(int gqa, int hd, bool f32_values) {
    auto pick = [&](auto g) -> AttnGqaKernel {
        constexpr int G = decltype(g)::value;
        switch (hd) {
            case 64: return f32_values ? attention_tile_kernel<G, 2, true> : attention_tile_kernel<G, 2, false>;
            case 128: return f32_values ? attention_tile_kernel<G, 4, true> : attention_tile_kernel<G, 4, false>;
            case 256: return f32_values ? attention_tile_kernel<G, 8, true> : attention_tile_kernel<G, 8, false>;
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
