// spl_elementwise.cuh — embedding, RMSNorm, SiLU gate, row gather and arg-max.
#pragma once
#include "spl_common.cuh"
#include "spl_gemm_tc.cuh"

// Embedding: gather a q4 row per token and dequantise it, h = scale * nibble + bias in fp32
// (Sources/Shaders/engine.metal:39-57). The embedding keeps the MLX row-major layout.
// Grid (rows), any block size.
__global__ void spl_embed_q4_kernel(const uint32_t *__restrict__ packed, const uint16_t *__restrict__ scales,
                                    const uint16_t *__restrict__ biases, const uint32_t *__restrict__ tokens, float *out, int hidden) {
    spl_grid_begin();
    const int row = blockIdx.x;
    const uint32_t token = tokens[row];
    const int words = hidden / 8, groups = hidden / 64;
    for (int w = threadIdx.x; w < words; w += blockDim.x) {
        const uint32_t word = packed[size_t(token) * words + w];
        const float s = spl_bf16_to_float(scales[size_t(token) * groups + (w >> 3)]);
        const float b = spl_bf16_to_float(biases[size_t(token) * groups + (w >> 3)]);
        float v[8];
#pragma unroll
        for (int nib = 0; nib < 8; ++nib) v[nib] = __fmaf_rn(s, float((word >> (4 * nib)) & 0xFu), b);
        float4 *dst = reinterpret_cast<float4 *>(out + size_t(row) * hidden + w * 8);
        dst[0] = make_float4(v[0], v[1], v[2], v[3]);
        dst[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
}

// RMSNorm into a GEMM operand (layout: SplOperand in spl_gemm_tc.cuh): bf16(x * rsqrt(mean x^2 + eps) * w) and the
// per-64 sums of the rounded values, the stored weight applied directly (engine.metal:159-178, 1609-1640; operand
// rounding engine_na.metal:42-57). When `index` is not
// null row r of the output reads input row index[r] (the logit-row gather, engine.metal:273-281).
// Grid (rows), a multiple of 32 threads up to 1,024.
__global__ void __launch_bounds__(1024)
spl_rmsnorm_kernel(const float *input, int in_ld, const uint16_t *__restrict__ weight, const uint32_t *__restrict__ index,
                   SplOperand out, int dim, float eps) {
    spl_grid_begin();
    __shared__ float part[32];
    const int stride = blockDim.x * 4, warps = blockDim.x >> 5;
    const int row = blockIdx.x;
    const float *x = input + size_t(index ? index[row] : row) * in_ld;
    float ss = 0.0f;
    for (int i = threadIdx.x * 4; i < dim; i += stride) {
        const float4 v = *reinterpret_cast<const float4 *>(x + i);
        ss += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
    ss = spl_warp_sum(ss);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = ss;
    __syncthreads();
    float total = 0.0f;
    for (int i = 0; i < warps; ++i) total += part[i];
    const float inv = 1.0f / sqrtf(total / float(dim) + eps);
    for (int base = 0; base < dim; base += stride) {
        const int i = base + threadIdx.x * 4;
        float r0 = 0.f, r1 = 0.f, r2 = 0.f, r3 = 0.f;
        if (i < dim) {
            const float4 v = *reinterpret_cast<const float4 *>(x + i);
            const uint2 w = *reinterpret_cast<const uint2 *>(weight + i);
            const uint16_t b0 = spl_float_to_bf16(v.x * inv * spl_bf16_to_float(uint16_t(w.x)));
            const uint16_t b1 = spl_float_to_bf16(v.y * inv * spl_bf16_to_float(uint16_t(w.x >> 16)));
            const uint16_t b2 = spl_float_to_bf16(v.z * inv * spl_bf16_to_float(uint16_t(w.y)));
            const uint16_t b3 = spl_float_to_bf16(v.w * inv * spl_bf16_to_float(uint16_t(w.y >> 16)));
            r0 = spl_bf16_to_float(b0); r1 = spl_bf16_to_float(b1); r2 = spl_bf16_to_float(b2); r3 = spl_bf16_to_float(b3);
            *reinterpret_cast<uint2 *>(out.values + out.at(row, i)) = spl_operand_pack4(r0, r1, r2, r3);
        }
        // Per-64 sums of the rounded values: sixteen consecutive threads hold one group.
        float gsum = (r0 + r1) + (r2 + r3);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) gsum += __shfl_xor_sync(0xffffffffu, gsum, o);
        if (i < dim && (threadIdx.x & 15) == 0) out.put_sum(row, i / 64, gsum);
    }
}

// Arg-max over [0, limit) per logit row, first index on ties (vDSP_maxvi, Sampler.swift:11-16;
// the vocabulary limit Sampler.swift:94-96). Grid (rows), 1024 threads.
__global__ void __launch_bounds__(1024)
spl_argmax_kernel(const float *__restrict__ logits, int ld, int limit, int32_t *ids) {
    __shared__ float best_v[32];
    __shared__ int best_i[32];
    const float *x = logits + size_t(blockIdx.x) * ld;
    float bv = -INFINITY; int bi = 0x7fffffff;
    // Sixteen-byte loads, four of them in flight a thread (rows start on 16-byte boundaries: the vocabulary is a multiple
    // of 16); ascending i per thread, so strict > keeps the first.
    const int quads = limit / 4;
    int q = threadIdx.x;
    for (; q + 3 * int(blockDim.x) < quads; q += 4 * blockDim.x) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = reinterpret_cast<const float4 *>(x)[q + u * blockDim.x];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = 4 * (q + u * int(blockDim.x));
            if (v[u].x > bv) { bv = v[u].x; bi = i; }
            if (v[u].y > bv) { bv = v[u].y; bi = i + 1; }
            if (v[u].z > bv) { bv = v[u].z; bi = i + 2; }
            if (v[u].w > bv) { bv = v[u].w; bi = i + 3; }
        }
    }
    for (; q < quads; q += blockDim.x) {
        const float4 v = reinterpret_cast<const float4 *>(x)[q];
        const int i = 4 * q;
        if (v.x > bv) { bv = v.x; bi = i; }
        if (v.y > bv) { bv = v.y; bi = i + 1; }
        if (v.z > bv) { bv = v.z; bi = i + 2; }
        if (v.w > bv) { bv = v.w; bi = i + 3; }
    }
    for (int i = 4 * quads + threadIdx.x; i < limit; i += blockDim.x) {
        const float v = x[i];
        if (v > bv) { bv = v; bi = i; }
    }
    if (bi == 0x7fffffff) { bv = -INFINITY; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    if ((threadIdx.x & 31) == 0) { best_v[threadIdx.x >> 5] = bv; best_i[threadIdx.x >> 5] = bi; }
    __syncthreads();
    if (threadIdx.x < 32) {
        bv = best_v[threadIdx.x]; bi = best_i[threadIdx.x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
        }
        // A row of NaNs or -inf never beats the initial value: index 0, as a scan from 0 would give.
        if (threadIdx.x == 0) ids[blockIdx.x] = bi == 0x7fffffff ? 0 : bi;
    }
}

// The k largest of [0, limit) per logit row in descending order, the lower index first among equal values
// (TopK.select, Sampler.swift:19-52), in two kernels, so that a row is many blocks' work and is read once. A warp keeps a
// stretch of 1,024 values in registers as order-preserving keys (32 a lane, in four groups with a maximum each) and picks k
// times: two warp-wide reductions find the best key and its lowest index, and the lane that held it looks for its next
// best in one group. A block merges its eight sorted lists; the second kernel merges a row's blocks the same way, a lane a
// list. Bound: the row's one trip from HBM for many rows, the chain of k picks for few.
// One block a row scanning it k times (what this replaced) took 1.31-1.34 ms for k = 20 of 248,077 at 12 to 64 rows; a
// twelve-row decode step with its top-k went from 9.07 to 7.76 ms.
//
// A key is the float's bits made to order as unsigned numbers, minus zero taken as zero (the two are equal values, so the lower
// index goes first); 0 stands for what is never picked: NaN, -inf and what lies past the limit.
#define SPL_TOPK_WARP 1024               // values of a warp
#define SPL_TOPK_STRETCH (8 * SPL_TOPK_WARP)
#define SPL_TOPK_MAX 64
// Floats of device scratch a top-k takes at most: the rows' lists and their picks (ids, then values).
inline size_t spl_topk_floats(int rows, int vocab) { return size_t(rows) * (size_t(vocab + SPL_TOPK_STRETCH - 1) / SPL_TOPK_STRETCH + 1) * SPL_TOPK_MAX * 2; }
__device__ __forceinline__ uint32_t spl_topk_key(float v) {
    if (!(v > -INFINITY)) return 0u;
    const uint32_t b = __float_as_uint(v + 0.0f);
    return b ^ (uint32_t(int32_t(b) >> 31) | 0x80000000u);
}
// k rounds of a merge of sorted lists by one warp: list n is lists[n * k ...] (key, index), ended by key 0 or by its k-th
// entry; a lane walks the lists lane, lane + 32, ... Round r's pick (key 0: none left) goes to emit(r, key, index) on lane 0.
template <typename Emit>
__device__ __forceinline__ void spl_topk_merge_lists(const uint2 *lists, int count, int k, uint8_t *cursor, Emit emit) {
    const int lane = threadIdx.x & 31;
    uint2 head = make_uint2(0u, 0xffffffffu); int mine = -1;
    auto next = [&]() {                                       // the best head of this lane's lists
        head = make_uint2(0u, 0xffffffffu); mine = -1;
        for (int n = lane; n < count; n += 32) {
            const int at = cursor[n];
            if (at >= k) continue;
            const uint2 c = lists[size_t(n) * k + at];
            if (c.x > head.x || (c.x == head.x && c.y < head.y)) { head = c; mine = n; }
        }
    };
    next();
    for (int round = 0; round < k; ++round) {
        const uint32_t key = __reduce_max_sync(0xffffffffu, head.x);
        const uint32_t index = __reduce_min_sync(0xffffffffu, head.x == key ? head.y : 0xffffffffu);
        if (lane == 0) emit(round, key, index);
        if (key != 0u && head.x == key && head.y == index) { ++cursor[mine]; next(); }
    }
}
// Grid (stretches, rows), 256 threads; lists [rows][stretches][k] of (key, index).
__global__ void __launch_bounds__(256)
spl_topk_stretch_kernel(const float *__restrict__ logits, int ld, int limit, int k, uint2 *lists) {
    __shared__ uint2 own[8 * SPL_TOPK_MAX];
    __shared__ uint8_t cursor[8];
    spl_grid_begin();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int base = int(blockIdx.x) * SPL_TOPK_STRETCH + warp * SPL_TOPK_WARP + lane;
    const float *x = logits + size_t(blockIdx.y) * ld;
    float v[32];
#pragma unroll
    for (int e = 0; e < 32; ++e) v[e] = base + 32 * e < limit ? x[base + 32 * e] : -INFINITY;
    uint32_t key[32];
#pragma unroll
    for (int e = 0; e < 32; ++e) key[e] = spl_topk_key(v[e]);
    uint32_t taken = 0u;                                      // this lane's elements that have been picked
    auto group = [&](int q) {
        uint32_t m = 0u;
#pragma unroll
        for (int e = 0; e < 8; ++e) m = max(m, (taken >> (8 * q + e) & 1u) ? 0u : key[8 * q + e]);
        return m;
    };
    // (the groups are spelt out: a loop over them becomes an indexed array in local memory)
    uint32_t top0 = group(0), top1 = group(1), top2 = group(2), top3 = group(3);
    uint2 *list = own + warp * k;
    for (int round = 0; round < k; ++round) {
        const uint32_t best = max(max(top0, top1), max(top2, top3));
        const uint32_t all = __reduce_max_sync(0xffffffffu, best);
        if (all == 0u) {                                      // nothing left: the list ends here
            if (lane == 0) list[round] = make_uint2(0u, 0xffffffffu);
            break;
        }
        // The lowest element of this lane that has the key (elements ascend in index), and the lowest index of the warp.
        int e0 = 32;
        if (best == all) {
#pragma unroll
            for (int e = 31; e >= 0; --e) e0 = (key[e] == all && !(taken >> e & 1u)) ? e : e0;
        }
        const uint32_t at = uint32_t(base + 32 * e0);
        const uint32_t first = __reduce_min_sync(0xffffffffu, e0 < 32 ? at : 0xffffffffu);
        if (e0 < 32 && at == first) {
            list[round] = make_uint2(all, first);
            taken |= 1u << e0;
            if (e0 < 16) { if (e0 < 8) top0 = group(0); else top1 = group(1); }
            else { if (e0 < 24) top2 = group(2); else top3 = group(3); }
        }
    }
    if (lane == 0) cursor[warp] = 0;
    __syncthreads();
    if (warp != 0) return;
    // A list that ended early has key 0 at its end and is not read beyond it: a pick never has key 0.
    uint2 *out = lists + (size_t(blockIdx.y) * gridDim.x + blockIdx.x) * k;
    spl_topk_merge_lists(own, 8, k, cursor, [&](int round, uint32_t picked, uint32_t index) { out[round] = make_uint2(picked, index); });
}
// Grid (rows), 32 threads; ids and values [rows][k]. Dynamic shared memory: a cursor byte a list, after the row's lists where
// `staged` (they fit the default 48 KB up to 95 stretches at k = 64: the k picks then wait for shared memory instead of L2).
// Fewer than k selectable values (a short row, NaNs, -inf) leave the reference's untouched slots, id 0 at -inf.
__global__ void __launch_bounds__(32)
spl_topk_merge_kernel(const float *__restrict__ logits, int ld, const uint2 *lists, int count, int k, int staged, int32_t *ids, float *values) {
    extern __shared__ uint2 spl_topk_smem[];
    spl_grid_begin();
    const int lane = threadIdx.x;
    const uint2 *row_lists = lists + size_t(blockIdx.x) * count * k;
    uint8_t *cursor = reinterpret_cast<uint8_t *>(spl_topk_smem + (staged ? count * k : 0));
    if (staged) for (int i = lane; i < count * k; i += 32) spl_topk_smem[i] = row_lists[i];
    for (int n = lane; n < count; n += 32) cursor[n] = 0;
    __syncwarp();
    spl_topk_merge_lists(staged ? spl_topk_smem : row_lists, count, k, cursor, [&](int round, uint32_t picked, uint32_t index) {
        const size_t at = size_t(blockIdx.x) * k + round;
        ids[at] = picked ? int32_t(index) : 0;
        values[at] = picked ? logits[size_t(blockIdx.x) * ld + index] : -INFINITY;
    });
}

// Fill helpers for synthetic contexts.
__global__ void spl_fill_codes_kernel(uint64_t *words, size_t count, uint64_t seed) {
    for (size_t idx = blockIdx.x * size_t(blockDim.x) + threadIdx.x; idx < count; idx += size_t(gridDim.x) * blockDim.x)
        words[idx] = spl_splitmix_at(seed, idx);
}
__global__ void spl_fill_float_kernel(float *data, size_t count, float value) {
    for (size_t idx = blockIdx.x * size_t(blockDim.x) + threadIdx.x; idx < count; idx += size_t(gridDim.x) * blockDim.x) data[idx] = value;
}
__global__ void spl_fill_uniform_kernel(float *data, size_t count, uint64_t seed, float lo, float hi) {
    for (size_t idx = blockIdx.x * size_t(blockDim.x) + threadIdx.x; idx < count; idx += size_t(gridDim.x) * blockDim.x)
        data[idx] = lo + (hi - lo) * (float(spl_splitmix_at(seed, idx) >> 40) * (1.0f / 16777216.0f));
}
