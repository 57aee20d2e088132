// The steps between the projections of a prompt chunk or of a step of several sequences (per-tensor models), a token's vector at a time (and the norm of
// a block-scaled model's step):
// residual + norm + codes, combination of the KV chunks + codes, activation + codes. Operation for operation those of norm_quant_kernel,
// attn_finish_kernel and act_quant_kernel (decode.cuh), which single steps use; here a thread takes four neighbouring elements at a time and
// keeps them in registers from the load to the codes.
//
// What bounds them is latency: a token is 12 to 180 KB, and the sums of a projection whose K was split come as up to eight parts. The elements'
// loads, parts included, are all requested before the first is used (one element at a time in a loop that stores to the residual stream, the parts
// of an element were fetched one after another), block-wide results take two rounds of shuffles, codes leave four to a store. 256 tokens of the
// Falcon3-10B shape (12 heads of 256, 23040 channels), by ncu: norm 17.5 -> 7.4 us, KV chunks 16.2 -> 9.9 us, activation 71 -> 30 us.
//
// Longer vectors, events around 20 launches, 32 tokens, against the kernels of decode.cuh: norm of 8192 / 16384 values 9.4 -> 6.6 / 12.4 -> 10.4 us; KV
// chunks of 8192 / 10240 / 16384 values 23 -> 8.3 / 29 -> 14.4 / 41 -> 14.5 us; 256 tokens of 16384 25 -> 17 and 70 -> 30 us. (At 1024 threads the long
// forms spill: 16 bytes a thread of the norm with four turns, 64 and 288 of the KV chunks with two and four. They are ahead all the same.)
#pragma once
#include "decode.cuh"

namespace qtb {

// Four neighbouring sums (i a multiple of four, as are the row lengths: the batched paths take multiples of 32 only).
__device__ __forceinline__ int4 acc_view_read4(const AccView& v, size_t z, int i) {
    const int32_t* p = v.base + z * v.ld + i;
    int4 s = *reinterpret_cast<const int4*>(p), t[kAccPartsMax - 1];
#pragma unroll
    for (int k = 1; k < kAccPartsMax; ++k) t[k - 1] = k < v.parts ? *reinterpret_cast<const int4*>(p + static_cast<size_t>(k) * v.part_stride) : make_int4(0, 0, 0, 0);
#pragma unroll
    for (int k = 0; k < kAccPartsMax - 1; ++k) s.x += t[k].x, s.y += t[k].y, s.z += t[k].z, s.w += t[k].w;
    return s;
}

// Block-wide results for every thread; `sh` holds 32 values and is used once.
__device__ __forceinline__ double row_sum_f64(double v, double* sh) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31;
    if (lane == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    v = lane < static_cast<int>(blockDim.x >> 5) ? sh[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float row_max_f32(float v, float* sh) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    const int lane = threadIdx.x & 31;
    if (lane == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    v = lane < static_cast<int>(blockDim.x >> 5) ? sh[lane] : 0.0f;
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// Per-tensor int8 codes of four values (ops.rs:241-267), packed in order.
__device__ __forceinline__ uint32_t quantize4(const float (&y)[4], float amax, float s) {
    uint32_t out = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        float q = 0.0f;
        if (amax > 0.0f) {
            q = roundf(__fmul_rn(y[e], s));
            q = q != q ? 0.0f : fminf(fmaxf(q, -128.0f), 127.0f);
        }
        out |= (static_cast<uint32_t>(static_cast<int>(q)) & 0xffu) << (8 * e);
    }
    return out;
}
__device__ __forceinline__ float inverse_rms(double sum, int n, float eps) {
    const float mean = __double2float_rn(sum / static_cast<double>(n));
    return __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(mean, eps)));
}

// Threads of a block for vectors of n elements, and how many turns of four elements each of them takes (0: too long for these kernels).
inline int row_threads(int n) { return std::min(1024, (n / 4 + 31) / 32 * 32); }
inline int row_turns(int n) {
    const int turns = (n / 4 + row_threads(n) - 1) / row_threads(n);
    return turns <= 4 ? turns : 0;
}

// Q8_0 codes (quantize_q8_0_block) of four neighbouring values: eight neighbouring lanes hold a block of 32. Every lane of the warp calls it.
__device__ __forceinline__ uint32_t quantize_q8_0_4(const float (&y)[4], bool store_scale, float* scale) {
    float m = 0.0f;
#pragma unroll
    for (int e = 0; e < 4; ++e) m = fmaxf(m, fabsf(y[e]));  // (f32::max ignores a NaN, and so does fmaxf)
    for (int o = 4; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (store_scale) *scale = __half2float(__float2half_rn(__fdiv_rn(m, 127.0f)));
    const float id = m != 0.0f ? __fdiv_rn(127.0f, m) : 0.0f;
    uint32_t out = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float r = rintf(__fmul_rn(y[e], id));
        const int q = r == r ? static_cast<int>(fminf(fmaxf(r, -128.0f), 127.0f)) : 0;
        out |= (static_cast<uint32_t>(q) & 0xffu) << (8 * e);
    }
    return out;
}

// Grid (1, 1, tokens). a.v_prev holds the previous projection's sums where there is one (a.acc_prev only says that there is). BLOCKS: a step of a
// block-scaled model, whose projections leave floats (a.acc_prev) and take Q8_0 blocks.
template <int TURNS, bool BLOCKS = false>
__global__ void __launch_bounds__(1024) norm_quant_rows_kernel(const __grid_constant__ NormQuantArgs a) {
    __shared__ double sh_d[32];
    __shared__ float sh_f[32];
    const size_t z = blockIdx.z;
    const bool prev = a.acc_prev != nullptr;
    float* x = a.x + z * a.b_x;
    float4 xv[TURNS], wv[TURNS];
    int4 sums[TURNS];
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const int i = (threadIdx.x + k * blockDim.x) * 4;
        const bool there = i < a.n;
        xv[k] = there ? *reinterpret_cast<const float4*>(x + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        wv[k] = there ? *reinterpret_cast<const float4*>(a.norm_w + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        sums[k] = !prev || !there ? make_int4(0, 0, 0, 0) : BLOCKS ? *reinterpret_cast<const int4*>(a.acc_prev + z * a.b_acc + i) : acc_view_read4(a.v_prev, z, i);
    }
    float post = 0.0f;
    bool live = false;
    if (prev && !BLOCKS) {
        const float s = a.scale_prev[a.b_scale ? z : 0];
        live = s > 0.0f;  // layer.rs:148-150: a zero activation scale gives a zero projection
        post = live ? __fdiv_rn(a.ws_prev, s) : 0.0f;
    }
    float y[TURNS][4];
    double sum = 0.0;
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const int i = (threadIdx.x + k * blockDim.x) * 4;
        y[k][0] = xv[k].x, y[k][1] = xv[k].y, y[k][2] = xv[k].z, y[k][3] = xv[k].w;
        if (prev) {
            const int c[4] = {sums[k].x, sums[k].y, sums[k].z, sums[k].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) y[k][e] = __fadd_rn(y[k][e], BLOCKS ? __int_as_float(c[e]) : live ? __fmul_rn(static_cast<float>(c[e]), post) : 0.0f);
            if (i < a.n) *reinterpret_cast<float4*>(x + i) = make_float4(y[k][0], y[k][1], y[k][2], y[k][3]);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) sum += static_cast<double>(__fmul_rn(y[k][e], y[k][e]));
    }
    const float inv = inverse_rms(row_sum_f64(sum, sh_d), a.n, a.eps);
    float amax = 0.0f;
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const float w[4] = {wv[k].x, wv[k].y, wv[k].z, wv[k].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            y[k][e] = __fmul_rn(__fmul_rn(y[k][e], inv), w[e]);
            amax = fmaxf(amax, fabsf(y[k][e]));
        }
    }
    if (a.q_out == nullptr) {
#pragma unroll
        for (int k = 0; k < TURNS; ++k) {
            const int i = (threadIdx.x + k * blockDim.x) * 4;
            if (i >= a.n) continue;
            unsigned short h[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) h[e] = a.y16_bf16 ? float_to_bf16_bits(y[k][e]) : __half_as_ushort(__float2half_rn(y[k][e]));
            *reinterpret_cast<ushort4*>(a.y16_out + z * a.b_y16 + i) = make_ushort4(h[0], h[1], h[2], h[3]);
        }
        return;
    }
    if constexpr (BLOCKS) {
#pragma unroll
        for (int k = 0; k < TURNS; ++k) {
            const int i = (threadIdx.x + k * blockDim.x) * 4;
            const uint32_t codes = quantize_q8_0_4(y[k], i < a.n && (threadIdx.x & 7) == 0, a.q8_d + i / 32);
            if (i < a.n) *reinterpret_cast<uint32_t*>(a.q_out + z * a.b_q + i) = codes;
        }
        return;
    }
    amax = row_max_f32(amax, sh_f);
    const float s = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const int i = (threadIdx.x + k * blockDim.x) * 4;
        if (i < a.n) *reinterpret_cast<uint32_t*>(a.q_out + z * a.b_q + i) = quantize4(y[k], amax, s);
    }
    if (threadIdx.x == 0) a.scale_out[a.b_scale ? z : 0] = s;
}

// Rotation of queries and keys and the cache's new rows (rope_kv_kernel's operations) for many tokens: eight elements a thread - eight neighbours, or with NEOX pairing
// four neighbours and their four partners - in 16-byte loads and stores. Grid (blocks of 128 threads over a token's elements, 1, tokens). Bound by its instructions where
// an element a thread was divided, scaled and looked up by itself (1000 tokens of 12 + 2 x 4 heads of 256: 30 us at 75 % of the issue slots; see rope_rows_fit).
constexpr int kRopeThreads = 128;
inline bool rope_rows_fit(const RopeKvArgs& a) { return !a.block_scaled && a.v_q.base != nullptr && a.rope_dims % 8 == 0 && a.head_dim % 8 == 0; }
__device__ __forceinline__ void scaled4(const AccView& v, int i, float post, bool live, float (&x)[4]) {
    const int4 s = acc_view_read4(v, blockIdx.z, i);
    x[0] = live ? __fmul_rn(static_cast<float>(s.x), post) : 0.0f, x[1] = live ? __fmul_rn(static_cast<float>(s.y), post) : 0.0f;
    x[2] = live ? __fmul_rn(static_cast<float>(s.z), post) : 0.0f, x[3] = live ? __fmul_rn(static_cast<float>(s.w), post) : 0.0f;
}
__device__ __forceinline__ uint2 halves4(const float (&x)[4]) {
    const __half2 lo = __floats2half2_rn(x[0], x[1]), hi = __floats2half2_rn(x[2], x[3]);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}
__global__ void __launch_bounds__(kRopeThreads) rope_kv_rows_kernel(const __grid_constant__ RopeKvArgs a) {
    const size_t z = blockIdx.z;
    const int qk = (a.q_dim + a.kv_dim) / 8, t = blockIdx.x * kRopeThreads + threadIdx.x;
    if (t >= qk + a.kv_dim / 8) return;
    const float s = a.act_scale[a.b_scale ? z : 0];
    const bool live = s > 0.0f;
    const uint32_t pos = seq_position(a.seq, a.pos, blockIdx.z);
    const size_t row = seq_cache_offset(a.seq, blockIdx.z) + static_cast<size_t>(pos) * a.kv_dim;
    float x[4], y[4];
    if (t >= qk) {  // values: scale and append
        const int i = (t - qk) * 8;
        const float post = live ? __fdiv_rn(a.ws_v, s) : 0.0f;
        scaled4(a.v_v, i, post, live, x), scaled4(a.v_v, i + 4, post, live, y);
        *reinterpret_cast<uint2*>(a.v_cache + row + i) = halves4(x);
        *reinterpret_cast<uint2*>(a.v_cache + row + i + 4) = halves4(y);
        return;
    }
    const int per_head = a.head_dim / 8, h = t / per_head, item = t - h * per_head, base = h * a.head_dim;
    const bool is_q = base < a.q_dim, rot = item < a.rope_dims / 8;
    const float post = live ? __fdiv_rn(is_q ? a.ws_q : a.ws_k, s) : 0.0f;
    // where x and y lie in the head: neighbours, or (NEOX, rotated part) half the rotated dimensions apart
    const bool apart = a.neox && rot;
    const int d0 = apart ? item * 4 : item * 8, d1 = apart ? d0 + a.rope_dims / 2 : d0 + 4;
    const AccView& v = is_q ? a.v_q : a.v_k;
    const int from = is_q ? base : base - a.q_dim;
    scaled4(v, from + d0, post, live, x), scaled4(v, from + d1, post, live, y);
    if (rot) {
        const float* cs = a.cos_sin + static_cast<size_t>(pos) * a.rope_dims;
        auto turn = [](float& p, float& q, float c, float sn) {
            const float r0 = __fmaf_rn(p, c, -__fmul_rn(q, sn)), r1 = __fmaf_rn(p, sn, __fmul_rn(q, c));
            p = r0, q = r1;
        };
        if (apart) {
            const float4 c0 = *reinterpret_cast<const float4*>(cs + 2 * d0), c1 = *reinterpret_cast<const float4*>(cs + 2 * d0 + 4);
            turn(x[0], y[0], c0.x, c0.y), turn(x[1], y[1], c0.z, c0.w), turn(x[2], y[2], c1.x, c1.y), turn(x[3], y[3], c1.z, c1.w);
        } else {
            const float4 c0 = *reinterpret_cast<const float4*>(cs + d0), c1 = *reinterpret_cast<const float4*>(cs + d1);
            turn(x[0], x[1], c0.x, c0.y), turn(x[2], x[3], c0.z, c0.w), turn(y[0], y[1], c1.x, c1.y), turn(y[2], y[3], c1.z, c1.w);
        }
    }
    if (is_q) {
        float* q = a.q_out + z * a.b_q + base;
        *reinterpret_cast<float4*>(q + d0) = make_float4(x[0], x[1], x[2], x[3]);
        *reinterpret_cast<float4*>(q + d1) = make_float4(y[0], y[1], y[2], y[3]);
    } else {
        *reinterpret_cast<uint2*>(a.k_cache + row + from + d0) = halves4(x);
        *reinterpret_cast<uint2*>(a.k_cache + row + from + d1) = halves4(y);
    }
}

// The factors of a head's four chunks (attn_combine_chunks), which are the same for all its coordinates.
struct ChunkFactors {
    float older[4], newer[4], inv;
    unsigned int used;  // bit c: chunk c is not empty
};

// Grid (1, 1, tokens); head_dim a multiple of four; dynamic shared memory: a ChunkFactors per head.
template <int TURNS>
__global__ void __launch_bounds__(1024) attn_finish_rows_kernel(const __grid_constant__ AttnFinishArgs a) {
    __shared__ double sh_d[32];
    __shared__ float sh_f[32];
    extern __shared__ __align__(16) unsigned char finish_sm[];
    ChunkFactors* f = reinterpret_cast<ChunkFactors*>(finish_sm);
    const int hd = a.head_dim, n = a.q_heads * hd;
    const size_t z = blockIdx.z;
    const int seq_len = static_cast<int>(seq_position(a.seq, a.pos, z)) + 1;
    const bool four = min(max((seq_len + 255) / 256 * 256, 256), a.ctx) >= 512;  // the cache is divided into four chunks
    float4 pa[TURNS][4], wv[TURNS];
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const int i = (threadIdx.x + k * blockDim.x) * 4;
        const float* p = a.part_acc + z * a.b_acc + static_cast<size_t>(i / hd) * 4 * hd + i % hd;
#pragma unroll
        for (int c = 0; c < 4; ++c) pa[k][c] = i < n && (c == 0 || four) ? *reinterpret_cast<const float4*>(p + c * hd) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        wv[k] = a.sub_norm_w != nullptr && i < n ? *reinterpret_cast<const float4*>(a.sub_norm_w + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    for (int h = threadIdx.x; h < a.q_heads; h += blockDim.x) {
        const float* ms = a.part_ms + z * a.b_ms + static_cast<size_t>(h) * 8;
        const float4 lo = *reinterpret_cast<const float4*>(ms);
        ChunkFactors r;
        r.used = 1u;
        if (four) {
            const float4 hi = *reinterpret_cast<const float4*>(ms + 4);
            const float m[4] = {lo.x, lo.z, hi.x, hi.z}, s[4] = {lo.y, lo.w, hi.y, hi.w};
            float m_final = -INFINITY, s_final = 0.0f;
            r.used = 0u;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if (s[c] == 0.0f) continue;  // empty or fully masked chunk
                const float m_new = fmaxf(m_final, m[c]);
                r.older[c] = device_expf(__fsub_rn(m_final, m_new));
                r.newer[c] = device_expf(__fsub_rn(m[c], m_new));
                s_final = __fmaf_rn(s_final, r.older[c], __fmul_rn(s[c], r.newer[c]));
                m_final = m_new;
                r.used |= 1u << c;
            }
            r.inv = s_final != 0.0f ? __fdiv_rn(1.0f, s_final) : 1.0f;  // (a sum of zero leaves the zeros as they are)
        } else {
            r.inv = lo.y == 0.0f ? 0.0f : __fdiv_rn(1.0f, lo.y);
        }
        f[h] = r;
    }
    __syncthreads();
    float y[TURNS][4];
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const int i = (threadIdx.x + k * blockDim.x) * 4;
        const ChunkFactors& r = f[min(i / hd, a.q_heads - 1)];
        float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (four) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                if ((r.used >> c & 1u) == 0u) continue;
                const float v[4] = {pa[k][c].x, pa[k][c].y, pa[k][c].z, pa[k][c].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[e] = __fmaf_rn(acc[e], r.older[c], __fmul_rn(v[e], r.newer[c]));
            }
        } else {
            acc[0] = pa[k][0].x, acc[1] = pa[k][0].y, acc[2] = pa[k][0].z, acc[3] = pa[k][0].w;
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) y[k][e] = i < n ? __fmul_rn(acc[e], r.inv) : 0.0f;
    }
    if (a.sub_norm_w != nullptr) {
        double sum = 0.0;
#pragma unroll
        for (int k = 0; k < TURNS; ++k)
#pragma unroll
            for (int e = 0; e < 4; ++e) sum += static_cast<double>(__fmul_rn(y[k][e], y[k][e]));
        const float inv = inverse_rms(row_sum_f64(sum, sh_d), n, a.eps);
#pragma unroll
        for (int k = 0; k < TURNS; ++k) {
            const float w[4] = {wv[k].x, wv[k].y, wv[k].z, wv[k].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) y[k][e] = __fmul_rn(__fmul_rn(y[k][e], inv), w[e]);
        }
    }
    float amax = 0.0f;
#pragma unroll
    for (int k = 0; k < TURNS; ++k)
#pragma unroll
        for (int e = 0; e < 4; ++e) amax = fmaxf(amax, fabsf(y[k][e]));
    amax = row_max_f32(amax, sh_f);
    const float s = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const int i = (threadIdx.x + k * blockDim.x) * 4;
        if (i < n) *reinterpret_cast<uint32_t*>(a.q_out + z * a.b_q + i) = quantize4(y[k], amax, s);
    }
    if (threadIdx.x == 0) a.scale_out[a.b_scale ? z : 0] = s;
}

// The activation step is the longest vector by far: a cluster of eight blocks takes a token, each block an eighth of it, and the two results over
// the whole vector (sum of squares for the sub-norm, maximum for the scale) go through distributed shared memory. Grid (8, 1, tokens);
// a.v_gate and a.v_up hold the sums.
constexpr int kActClusterSize = 8;
__host__ __device__ constexpr int act_cluster_slice(int n) { return (n / 4 + kActClusterSize - 1) / kActClusterSize * 4; }

template <int TURNS, int THREADS>
__global__ void __cluster_dims__(kActClusterSize, 1, 1) __launch_bounds__(THREADS) act_quant_rows_kernel(const __grid_constant__ ActQuantArgs a) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ double sh_d[32];
    __shared__ float sh_f[32];
    __shared__ double x_sum;
    __shared__ float x_max;
    const size_t z = blockIdx.z;
    const int rank = static_cast<int>(cluster.block_rank()), other = threadIdx.x & (kActClusterSize - 1);
    const int per = act_cluster_slice(a.n), first = min(a.n, rank * per), end = min(a.n, first + per);
    const float s_in = a.act_scale[a.b_scale ? z : 0];
    const bool live = s_in > 0.0f;
    const float pg = live ? __fdiv_rn(a.ws_gate, s_in) : 0.0f, pu = live ? __fdiv_rn(a.ws_up, s_in) : 0.0f;
    float y[TURNS][4];
    int4 g[TURNS], u[TURNS];
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const int i = first + (threadIdx.x + k * THREADS) * 4;
        if (a.v_gate.parts == 1 && a.v_up.parts == 1) {  // (the usual case: so many rows need no split of K)
            g[k] = i < end ? *reinterpret_cast<const int4*>(a.v_gate.base + z * a.v_gate.ld + i) : make_int4(0, 0, 0, 0);
            u[k] = i < end ? *reinterpret_cast<const int4*>(a.v_up.base + z * a.v_up.ld + i) : make_int4(0, 0, 0, 0);
        } else {
            g[k] = i < end ? acc_view_read4(a.v_gate, z, i) : make_int4(0, 0, 0, 0);
            u[k] = i < end ? acc_view_read4(a.v_up, z, i) : make_int4(0, 0, 0, 0);
        }
    }
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const int cg4[4] = {g[k].x, g[k].y, g[k].z, g[k].w}, cu4[4] = {u[k].x, u[k].y, u[k].z, u[k].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float gv = live ? __fmul_rn(static_cast<float>(cg4[e]), pg) : 0.0f, uv = live ? __fmul_rn(static_cast<float>(cu4[e]), pu) : 0.0f;
            if (a.relu2) {
                const float p = gv > 0.0f ? gv : 0.0f;
                y[k][e] = __fmul_rn(__fmul_rn(p, p), uv);
            } else {
                y[k][e] = __fmul_rn(ggml_silu(gv), uv);
            }
        }
    }
    if (a.sub_norm_w != nullptr) {
        float4 wv[TURNS];
        double sum = 0.0;
#pragma unroll
        for (int k = 0; k < TURNS; ++k) {
            const int i = first + (threadIdx.x + k * THREADS) * 4;
            wv[k] = i < end ? *reinterpret_cast<const float4*>(a.sub_norm_w + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int e = 0; e < 4; ++e) sum += i < end ? static_cast<double>(__fmul_rn(y[k][e], y[k][e])) : 0.0;
        }
        sum = row_sum_f64(sum, sh_d);
        if (threadIdx.x == 0) x_sum = sum;
        cluster.sync();
        double total = *cluster.map_shared_rank(&x_sum, other);
        for (int o = 1; o < kActClusterSize; o <<= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        const float inv = inverse_rms(total, a.n, a.eps);
#pragma unroll
        for (int k = 0; k < TURNS; ++k) {
            const float w[4] = {wv[k].x, wv[k].y, wv[k].z, wv[k].w};
#pragma unroll
            for (int e = 0; e < 4; ++e) y[k][e] = __fmul_rn(__fmul_rn(y[k][e], inv), w[e]);
        }
    }
    float amax = 0.0f;
#pragma unroll
    for (int k = 0; k < TURNS; ++k)
#pragma unroll
        for (int e = 0; e < 4; ++e) amax = first + static_cast<int>(threadIdx.x + k * THREADS) * 4 < end ? fmaxf(amax, fabsf(y[k][e])) : amax;
    amax = row_max_f32(amax, sh_f);
    if (threadIdx.x == 0) x_max = amax;
    cluster.sync();
    amax = *cluster.map_shared_rank(&x_max, other);
    for (int o = 1; o < kActClusterSize; o <<= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float s = amax > 0.0f ? __fdiv_rn(127.0f, amax) : 0.0f;
#pragma unroll
    for (int k = 0; k < TURNS; ++k) {
        const int i = first + (threadIdx.x + k * THREADS) * 4;
        if (i < end) *reinterpret_cast<uint32_t*>(a.q_out + z * a.b_q + i) = quantize4(y[k], amax, s);
    }
    if (rank == 0 && threadIdx.x == 0) a.scale_out[a.b_scale ? z : 0] = s;
    cluster.sync();  // no block leaves while its partial results may still be read
}

// ---- launches: n tokens, all lengths multiples of 32 -----------------------------------------------------------------
inline void launch_norm_quant_rows(const NormQuantArgs& a, int n, cudaStream_t s) {
    auto go = [&](auto kernel) { kernel<<<dim3(1, 1, n), row_threads(a.n), 0, s>>>(a); };
    switch (row_turns(a.n)) {
        case 1: return go(norm_quant_rows_kernel<1>);
        case 2: return go(norm_quant_rows_kernel<2>);
        case 3: case 4: return go(norm_quant_rows_kernel<4>);
        default: norm_quant_kernel<<<dim3(1, 1, n), kRowThreads, a.n * sizeof(float), s>>>(a);
    }
}
// One token of a block-scaled model (hidden a multiple of 32). One block's chain of reads, sums and codes: 3072 values: a step of two layers (five of them)
// 284 -> 277 us.
inline void launch_norm_blocks(const NormQuantArgs& a, cudaStream_t s) {
    switch (row_turns(a.n)) {
        case 1: norm_quant_rows_kernel<1, true><<<1, row_threads(a.n), 0, s>>>(a); return;
        case 2: norm_quant_rows_kernel<2, true><<<1, row_threads(a.n), 0, s>>>(a); return;
        case 3: case 4: norm_quant_rows_kernel<4, true><<<1, row_threads(a.n), 0, s>>>(a); return;
        default: norm_quant_kernel<<<1, kRowThreads, a.n * sizeof(float), s>>>(a);
    }
}
inline void launch_attn_finish_rows(const AttnFinishArgs& a, int n, cudaStream_t s) {
    const int q_dim = a.q_heads * a.head_dim;
    auto go = [&](auto kernel) { kernel<<<dim3(1, 1, n), row_threads(q_dim), a.q_heads * sizeof(ChunkFactors), s>>>(a); };
    switch (a.head_dim % 4 == 0 && a.q_heads * sizeof(ChunkFactors) <= 40960 ? row_turns(q_dim) : 0) {
        case 1: return go(attn_finish_rows_kernel<1>);
        case 2: return go(attn_finish_rows_kernel<2>);
        case 3: case 4: return go(attn_finish_rows_kernel<4>);
        default: attn_finish_kernel<<<dim3(1, 1, n), kRowThreads, q_dim * sizeof(float), s>>>(a);
    }
}
inline void launch_act_quant_rows(const ActQuantArgs& a, int n, cudaStream_t s) {
    // Turns of 256 threads with four elements each. Past four, blocks of 512 threads: eight turns a thread do not fit the registers (36864 channels,
    // 32 tokens: 35 us against 12.4; 256 tokens: 192 against 66). A model's vector is at most 51200 long, seven turns; longer ones take the
    // general kernel.
    const int turns = (act_cluster_slice(a.n) + 1023) / 1024;
    auto go = [&](auto kernel, int threads) { kernel<<<dim3(kActClusterSize, 1, n), threads, 0, s>>>(a); };
    if (turns <= 1) go(act_quant_rows_kernel<1, 256>, 256);
    else if (turns == 2) go(act_quant_rows_kernel<2, 256>, 256);
    else if (turns == 3) go(act_quant_rows_kernel<3, 256>, 256);
    else if (turns == 4) go(act_quant_rows_kernel<4, 256>, 256);
    else if (turns <= 8) go(act_quant_rows_kernel<4, 512>, 512);
    else act_quant_kernel<<<dim3(1, 1, n), kRowThreads, a.n * sizeof(float), s>>>(a);
}

}  // namespace qtb
