// spl_gemm_narrow.cuh — the MLX affine-4 dequant-GEMM for steps of up to 64 rows (decode and verify steps).
//
// Contract, weight layout and arithmetic are those of spl_gemm_tc.cuh: exact fp16 weights scale * (code - 8) formed by converting warps in tensor
// memory, two issuing warps with an accumulator each, the second term (bias + 8 scale) * sum(a) from split means. What is different is how a block's
// roles meet. Such a GEMM is a stream of weights from HBM, and what bounds it is neither bytes nor instructions but the pace of its hand-overs: on this
// part a wait on an mbarrier costs 106-126 cycles even when the phase is complete, an arrive reaches a waiting warp in 150-190, and a thread that feeds a
// ring needs 250 cycles a copy and 550 for two copies and a wait in a row. Clock stamps of every role of a block in the middle of the grid said, in turn:
//   * the copier of activations was the pace-setter (950 of a converting warp's 2,200 cycles a unit were spent waiting for it): it now brings a stage
//     of four groups and its split means with two lanes side by side, and two lanes wait for the two units that had the place;
//   * the issuing warps came next (three waits a unit: means, activations, converted weights): the split means lie with the stage, and the first warp of
//     a converting set answers for the activations, so an issuing warp waits once a unit;
//   * waits that are nearly always over are asked about ahead (mbarrier.test_wait) and looked at after other work;
//   * of a block's 27K cycles 9K were set-up, first copies and output. Blocks of tiles that are not cut stay and take the next tile, whose weights are
//     on their way while a tile's sums are written; nobody waits for the copier's first copies any more; the SiLU
//     gate's rows are taken several at a time, everything they need asked for first, and what the other outputs need is asked for before the sums are there.
// The blocks of a cut tile are a cluster: the cluster's warps add the blocks' sums through distributed shared memory and write the output, with the
// residual and the next deferred norm's operand. (They used to leave partial sums in global memory for a second kernel.)
// Measured before and after, with those second kernels and the kernel that forms the operand: 5,120 x 6,144 at one row 13.5 -> 11.0 us, at 64 rows 16.6 -> 14.2;
// 34,816 x 5,120 36.8 -> 28.4 and 40.0 -> 35.5; 1,024 x 5,120 9.2 -> 8.0 and 11.0 -> 10.4. A step of the 27B shape with one row 6,590 -> 5,489 us, twelve rows
// 7,739 -> 6,584, 64 rows 11,191 -> 10,736.
#pragma once
#include "spl_gemm_tc.cuh"

#define SPL_NARROW_THREADS SPL_TC_THREADS
#define SPL_NARROW_CLUSTER 8               // the most pieces a tile is cut in (the portable cluster size)
__host__ __device__ constexpr int spl_narrow_cstages(int rn) { return rn >= 64 ? 4 : 6; }        // stages (four groups) of codes with their scale/bias words
#define SPL_NARROW_SLOTS 5                 // operand slots in tensor memory, a unit (two groups, 64 columns) each, with 8 columns each for the second term
__host__ __device__ constexpr int spl_narrow_bstages(int rn) { return rn >= 64 ? 3 : rn >= 32 ? 5 : 6; }        // stages of activations with their split means
__host__ __device__ constexpr size_t spl_narrow_smem_bytes(int rn) {
    return 1024 /* alignment slack */ + size_t(spl_narrow_cstages(rn)) * 4 * (4096 + 512) + size_t(spl_narrow_bstages(rn)) * rn * (512 + 32) + rn * 16 + size_t(rn) * 512 + 2048;
}

struct SplNarrowArgs {
    const unsigned char *codes, *sb;       // the weight (SplQ4Dev)
    const unsigned char *act, *means;      // the operand (SplOperand, one row block) and its tiles of split means
    float *out;
    const float *residual;
    int out_ld, rows, groups, tiles, splits, interleave, fuse, drop;
    int wide;                              // out and residual lie on 8-byte boundaries (a caller's may lie on any float): two columns an access
    int *error_flag;
    const float *in_squares; int in_groups; float in_dim, eps;
    SplOperand act_out;                    // fuse: the SiLU-gated activation, the next GEMM's operand
    const uint16_t *emit_weight; SplOperand emit_out; float *emit_squares;
};

// The barriers of this kernel, a block's and a cluster's, are instructions of whole converged warps (.aligned): where a warp has branched by lane since it last
// met, a __syncwarp stands in front of them. Nothing else promises that its lanes have come together again.
// A part in a barrier of the block without waiting for it.
template <int ID, int COUNT> __device__ __forceinline__ void spl_named_arrive() { asm volatile("bar.arrive %0, %1;\n" ::"n"(ID), "n"(COUNT) : "memory"); }
// K-major without swizzle: core matrices of eight rows of 16 bytes, `k_step` bytes from the first eight of a k16 to the last eight, 128 from eight rows to the next.
__device__ __forceinline__ uint64_t spl_tc_desc_plain(uint32_t smem_byte_addr, uint32_t k_step) {
    return uint64_t((smem_byte_addr & 0x3FFFFu) >> 4) | uint64_t((k_step & 0x3FFFFu) >> 4) << 16 | uint64_t(128 >> 4) << 32 | uint64_t(1) << 46;
}
// Whether a phase is complete, without waiting: asked ahead of the work in front of a wait, so that the answer's hundred cycles pass under it.
__device__ __forceinline__ bool spl_mbar_test(uint64_t *bar, uint32_t parity) {
    uint32_t done;
    asm volatile("{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(done) : "r"(spl_smem_addr(bar)), "r"(parity) : "memory");
    return done != 0;
}
__device__ __forceinline__ void spl_cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ uint32_t spl_cluster_map(uint32_t addr, uint32_t rank) {
    uint32_t out;
    asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(out) : "r"(addr), "r"(rank));
    return out;
}
__device__ __forceinline__ float2 spl_shared_load2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ float2 spl_cluster_load2(uint32_t addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
    return v;
}

// Two neighbouring columns of the output or the residual.
__device__ __forceinline__ float2 spl_columns_load(const float *p, bool wide) {
    return wide ? *reinterpret_cast<const float2 *>(p) : make_float2(p[0], p[1]);
}
__device__ __forceinline__ void spl_columns_store(float *p, float2 v, bool wide) {
    if (wide) *reinterpret_cast<float2 *>(p) = v;
    else { p[0] = v.x; p[1] = v.y; }
}

// A converting thread's two columns of its warp's output items, and what they need that can be asked for before the sums are there: the residual of the
// first item, the weight of the next norm.
struct SplNarrowColumns { int n; bool inside; float2 res; uint32_t weight; };

// What follows a tile's sum where a row's columns have to meet (SiLU gate, next operand) or the tile is cut, by all converting warps of the blocks that hold its pieces: the pieces' sums are added in the order of the contraction
// (through distributed shared memory where a tile is cut).
template <int RN>
__device__ __forceinline__ void spl_narrow_output(const SplNarrowArgs &a, const float *plane, int tile, int split, int S, int warp, int lane, const SplNarrowColumns &at) {
    constexpr int WARPS = SPL_TC_SETS * 4;
    if (a.fuse) {
        constexpr int PRE = RN / 16;          // rows a warp takes at a time, everything asked for before any is worked on
        const uint32_t base = spl_smem_addr(plane);
        // A fused gate|up tensor: in each run of 32 columns of a tile the first sixteen are gate columns and the next sixteen the up columns of the same
        // elements. act = bf16(silu(gate) * up) (Sources/Shaders/engine.metal:200-219) into the next GEMM's operand, a warp a row.
        const int e = 2 * lane, gc = (e >> 4) * 32 + (e & 15);
#pragma unroll 1
        for (int k0 = 0; warp + k0 * WARPS < a.rows; k0 += PRE) {          // (never of a cut tile)
            float2 g[PRE], u[PRE];
#pragma unroll
            for (int k = 0; k < PRE; ++k) {
                const uint32_t at = base + uint32_t(min(warp + (k0 + k) * WARPS, RN - 1) * 128 + gc) * 4;
                g[k] = spl_shared_load2(at); u[k] = spl_shared_load2(at + 64);
            }
#pragma unroll
            for (int k = 0; k < PRE; ++k) {
                const int row = warp + (k0 + k) * WARPS;
                const float v0 = spl_bf16_to_float(spl_float_to_bf16(spl_silu_exact(g[k].x) * u[k].x)), v1 = spl_bf16_to_float(spl_float_to_bf16(spl_silu_exact(g[k].y) * u[k].y));
                // The sum in one fixed order: neighbours, then a butterfly over the rest.
                float s = v0 + v1;
                s += __shfl_xor_sync(0xffffffffu, s, 1);
#pragma unroll
                for (int o = 16; o > 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (row < a.rows) {
                    *reinterpret_cast<__half2 *>(reinterpret_cast<__half *>(a.act_out.values) + a.act_out.at(row, tile * 64 + e)) = __halves2half2(__float2half_rn(v0), __float2half_rn(v1));
                    if (lane == 0) a.act_out.put_sum(row, tile, s);
                }
            }
        }
        return;
    }
    // An item is a row's 64 columns, every WARPS x S-th of a tile's a warp's: all of the same half of the tile. What bounds this stage is instruction fetches
    // and trips to the other blocks' memory. The body therefore stands here once (a block comes here once, and pays for every instruction's first use), a
    // warp reads what it has items for and no more, and four blocks' sums are on their way at a time. Taking RN / 16 items at a time, the last one again where
    // there were fewer, a block after the other: 1,024 x 5,120 at 64 rows 13.7 us with its operand, now 10.4; 128 x 4,096 13.3, now 9.0; 5,120 x 6,144 at one
    // row 11.1, now 11.0, at 24 rows 12.2, now 11.7.
    const int step = WARPS * S, n = at.n;
    const uint32_t plane_at = spl_smem_addr(plane) + uint32_t((warp & 1) * 64 + 2 * lane) * 4;
    float2 res = at.res;
#pragma unroll 1
    for (int item = split * WARPS + warp; item < a.rows * 2; item += step) {
        const int row = item >> 1;
        float2 next = make_float2(0.0f, 0.0f);
        if (a.residual && at.inside && item + step < a.rows * 2) next = spl_columns_load(a.residual + size_t(row + step / 2) * a.out_ld + n, a.wide);
        // The pieces' sums in the order of the contraction, four blocks asked at a time.
        float2 x = make_float2(0.0f, 0.0f);
#pragma unroll 1
        for (int r0 = 0; r0 < S; r0 += 4) {
            if (S == 1) { x = spl_shared_load2(plane_at + uint32_t(row) * 512); break; }
            float2 p[4];
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (r0 + r < S) p[r] = spl_cluster_load2(spl_cluster_map(plane_at + uint32_t(row) * 512, r0 + r));
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (r0 + r < S) x = r0 + r == 0 ? p[r] : make_float2(x.x + p[r].x, x.y + p[r].y);
        }
        if (at.inside) {
            if (a.residual) { x.x += res.x; x.y += res.y; }
            spl_columns_store(a.out + size_t(row) * a.out_ld + n, x, a.wide);
        } else x = make_float2(0.0f, 0.0f);
        res = next;
        if (a.emit_weight) {
            // The output feeds a deferred norm (Sources/Shaders/engine_na.metal:365-415): bf16(x * w) as the next operand, its per-64 sum, and the
            // squares of x per 64 columns. Both sums are butterflies over the warp: one fixed order.
            const float v0 = spl_bf16_to_float(spl_float_to_bf16(x.x * spl_bf16_to_float(uint16_t(at.weight & 0xFFFFu))));
            const float v1 = spl_bf16_to_float(spl_float_to_bf16(x.y * spl_bf16_to_float(uint16_t(at.weight >> 16))));
            if (at.inside) *reinterpret_cast<__half2 *>(reinterpret_cast<__half *>(a.emit_out.values) + a.emit_out.at(row, n)) = __halves2half2(__float2half_rn(v0), __float2half_rn(v1));
            const float vs = spl_warp_sum(v0 + v1), sq = spl_warp_sum(x.x * x.x + x.y * x.y);
            const int group = tile * 2 + (warp & 1);
            if (lane == 0 && group * 64 < a.out_ld) { a.emit_out.put_sum(row, group, vs); a.emit_squares[size_t(row) * (a.out_ld / 64) + group] = sq; }
        }
    }
}

// Grid (tiles x splits), the splits of a tile a cluster.
template <int RN>
__global__ void __launch_bounds__(SPL_NARROW_THREADS, 1)
spl_gemm_q4_narrow_kernel(const __grid_constant__ SplNarrowArgs a) {
    constexpr int SG = SPL_TC_SUPER, BST = spl_narrow_bstages(RN), CST = spl_narrow_cstages(RN), AUN = SPL_NARROW_SLOTS, SETS = SPL_TC_SETS, WARPS = SETS * 4;
    constexpr int BTILE = SG * RN * 128, TTILE = RN * 32, WSTAGE = SG * 4096, QSTAGE = SG * 512;
    // A set meets every second stage, and has to meet every phase of a slot of codes it waits on: an mbarrier's wait tells two phases apart and no more, so with an
    // odd ring the wait for a slot's next-but-one phase would be answered by the last one. (The ring of activations may be odd: before a set waits for stage s it
    // has seen the units of stage s - BST multiplied, through the wait for its operand slot, as long as the ring has no more stages than there are slots.)
    static_assert(CST % 2 == 0, "a set meets every second stage");
    static_assert(BST % 2 == 0 || BST <= AUN, "see above");
    extern __shared__ unsigned char spl_tc_smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(spl_tc_smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char *b_ring = smem, *w_ring = b_ring + size_t(BST) * BTILE, *q_ring = w_ring + size_t(CST) * WSTAGE, *t_ring = q_ring + size_t(CST) * QSTAGE, *zeros = t_ring + size_t(BST) * TTILE;
    float *plane = reinterpret_cast<float *>(zeros + RN * 16);          // [RN][128] a tile's sums
    uint64_t *bars = reinterpret_cast<uint64_t *>(plane + RN * 128);
    uint64_t *full_c = bars, *empty_c = full_c + CST, *full_b = empty_c + CST, *full_u = full_b + BST, *done = full_u + 2 * AUN, *finished = done + 16, *drained = finished + 1;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drained + 1);
    int *abort_word = reinterpret_cast<int *>(tmem_slot + 1);
    const volatile int *abort = abort_word;
    float *row_factor = reinterpret_cast<float *>(bars) + 256;          // [RN] at byte 1,024 of the control area

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int W_COPY = WARPS, W_MMA0 = W_COPY + 1, W_COPYB = W_COPY + 2, W_MMA1 = W_COPY + 3;
    const bool direct = a.splits == 1 && !a.fuse && !a.emit_weight;
    const int S = a.splits, split = S == 1 ? 0 : int(blockIdx.x) % S, tile0 = S == 1 ? int(blockIdx.x) : int(blockIdx.x) / S, tile_step = S == 1 ? int(gridDim.x) : a.tiles;
    const int stages_all = a.groups / SG, per = S == 1 ? stages_all : (stages_all + S - 1) / S, s_first = split * per, stages = min(per, stages_all - s_first), units = 2 * stages;
    // Every block of a GEMM reads the same activation lines. Blocks therefore walk the contraction from different starting points (a fixed function
    // of the tile), so that at any moment they ask L2 for different lines.
    auto rotation = [&](int tile) { return stages > 1 ? int((uint32_t(tile) * 2654435761u >> 12) % uint32_t(stages)) : 0; };
    if (warp == 0) {
        const int total = int(drained + 1 - bars);
        for (int b = lane + CST; b < total; b += 32) {
            uint64_t *bar = bars + b;
            const uint32_t count = bar < full_b ? 8u                  // empty_c: the two sets (four warps each) that take the stage's units
                                 : bar < full_u ? 1u                  // full_b: the copies' bytes
                                 : bar < done ? 4u                    // full_u: the four warps of a set
                                 : bar < finished ? 1u                // done: the commit of the issuing warp that took the unit
                                 : bar < drained ? 2u                 // finished: both issuing warps
                                 : uint32_t(WARPS);                   // drained: the converting warps
            spl_mbar_init(bar, count);
        }
        if (lane == 0) *abort_word = 0;
        for (int z = lane; z < RN; z += 32) reinterpret_cast<uint4 *>(zeros)[z] = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");        // the tensor core reads them
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == W_MMA0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(spl_smem_addr(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    // The warp that copies weights sets up its own barriers and asks for the first stages at once; the others wait for its barriers, not for its copies, and
    // it for theirs only when the ring is full.
    if (warp == W_COPY) {
        if (lane < CST) spl_mbar_init(&full_c[lane], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        __syncwarp();
        spl_named_arrive<2, SPL_NARROW_THREADS>();
    } else {
        spl_tc_fence_before();
        __syncwarp();
        spl_named_barrier<2, SPL_NARROW_THREADS>();
        spl_tc_fence_after();
        spl_named_arrive<3, SPL_NARROW_THREADS>();
    }
    const uint32_t tmem = warp == W_COPY ? 0u : *tmem_slot;
    // Two accumulators of RN columns, one per issuing warp; the operand slots; the second terms' operands.
    const uint32_t tmem_d = tmem, tmem_a = tmem + 128, tmem_aq = tmem_a + AUN * 64;
    bool ok = true;
    int issued_c = 0, issued_b = 0;
    if (warp == W_COPY) {
        // ---- copies of the weight: lane 0 the codes, lane 1 the scale/bias words. They are nobody's output: the ring is filled before the wait for the
        // kernels in front, and the next tile's stages are on their way while a tile's sums are written.
        unsigned char *dst = lane == 0 ? w_ring : q_ring;
        const uint32_t bytes = lane == 0 ? WSTAGE : QSTAGE;
        int slot = 0, n = 0;
        uint32_t parity = 1;
        for (int tile = tile0; tile < a.tiles && ok; tile += tile_step) {
            const unsigned char *src = (lane == 0 ? a.codes : a.sb) + (size_t(tile) * stages_all + s_first) * bytes;
            const int rot = rotation(tile);
            for (int i = 0; i < stages; ++i, ++n) {
                if (n == CST) { __syncwarp(); spl_named_barrier<3, SPL_NARROW_THREADS>(); spl_grid_begin(); }
                if (n >= CST) ok = spl_mbar_wait_warp(&empty_c[slot], parity, abort);
                if (!ok) { if (!*abort && lane == 0) spl_note_wait(a.error_flag, 10, i); break; }
                issued_c = n + 1;
                if (i != a.drop) {
                    if (lane == 0) spl_mbar_expect_tx(&full_c[slot], WSTAGE + QSTAGE);
                    __syncwarp();
                    if (lane < 2) spl_bulk_g2s(dst + slot * bytes, src + size_t(i + rot < stages ? i + rot : i + rot - stages) * bytes, bytes, &full_c[slot]);
                }
                if (++slot == CST) { slot = 0; parity ^= 1u; }
            }
        }
        if (n <= CST && ok) { __syncwarp(); spl_named_barrier<3, SPL_NARROW_THREADS>(); spl_grid_begin(); }
    } else if (warp == W_COPYB) {
        // ---- copies of activations (lane 0) and of their split means (lane 1), a stage at a time; a lane each waits for one of the units that had the place.
        {
            const unsigned char *src = lane == 0 ? a.act + size_t(s_first) * BTILE : a.means + size_t(s_first) * TTILE;
            unsigned char *dst = lane == 0 ? b_ring : t_ring;
            const uint32_t bytes = lane == 0 ? BTILE : TTILE;
            int slot = 0, n = 0;
            spl_grid_begin();
            for (int tile = tile0; tile < a.tiles && ok; tile += tile_step) {
                const int rot = rotation(tile);
                for (int i = 0; i < stages; ++i, ++n) {
                    if (n >= BST) { const int un = 2 * (n - BST) + (lane & 1); ok = spl_mbar_wait_warp(&done[un & 15], (un >> 4) & 1, abort); }
                    if (!ok) { if (!*abort && lane == 0) spl_note_wait(a.error_flag, 21, i); break; }
                    issued_b = n + 1;
                    if (lane == 0) spl_mbar_expect_tx(&full_b[slot], BTILE + TTILE);
                    __syncwarp();
                    if (lane < 2) spl_bulk_g2s(dst + slot * bytes, src + size_t(i + rot < stages ? i + rot : i + rot - stages) * bytes, bytes, &full_b[slot]);
                    if (++slot == BST) slot = 0;
                }
            }
        }
    } else if (warp == W_MMA0 || warp == W_MMA1) {
        const int m = warp == W_MMA0 ? 0 : 1;
        constexpr uint32_t idesc = spl_tc_idesc(RN);
        const uint64_t b_desc0 = spl_tc_desc_sw128(spl_smem_addr(b_ring));
        const uint32_t t0 = spl_smem_addr(t_ring), z0 = spl_smem_addr(zeros), d_mine = tmem_d + m * RN;
        int slot = m, fu = m, bs = 0, un = m, t = 0;
        uint32_t a_parity = 0;
        spl_grid_begin();
        for (int tile = tile0; tile < a.tiles && ok; tile += tile_step, ++t) {
            // The tile's first unit overwrites this warp's accumulator: the sums of the tile before have to be out of it.
            if (t > 0) { ok = spl_mbar_wait_warp(drained, (t - 1) & 1, abort); if (!ok) { if (!*abort && lane == 0) spl_note_wait(a.error_flag, 38 + m, t); break; } }
            for (int i = 0; i < stages; ++i, un += 2) {
                const uint32_t t_at = t0 + bs * TTILE + m * (RN * 16);
                const uint64_t b_desc = b_desc0 + uint64_t((bs * BTILE + m * 2 * RN * 128) >> 4), t_desc = spl_tc_desc_plain(t_at, z0 - t_at);
                const uint32_t a_base = tmem_a + slot * 64, aq_base = tmem_aq + slot * 8;
                ok = spl_mbar_wait_warp(&full_u[fu], a_parity, abort);
                if (!ok) { if (!*abort && lane == 0) spl_note_wait(a.error_flag, 36 + m, un); break; }
                spl_tc_fence_after();
                if (spl_elect_one()) {
                    if (i > 0) spl_tc_mma_ts_acc(d_mine, a_base, b_desc, idesc);
                    else spl_tc_mma_ts(d_mine, a_base, b_desc, idesc, 0u);
#pragma unroll
                    for (int q = 1; q < 8; ++q) spl_tc_mma_ts_acc(d_mine, a_base + q * 8, b_desc + uint64_t(((q >> 2) * RN * 128 + (q & 3) * 32) >> 4), idesc);
                    spl_tc_mma_ts_acc(d_mine, aq_base, t_desc, idesc);
                    spl_tc_commit(&done[un & 15]);
                    if (i + 1 == stages) spl_tc_commit(finished);
                }
                __syncwarp();
                slot += 2; if (slot >= AUN) slot -= AUN;
                if (++bs == BST) bs = 0;
                fu += 2; if (fu >= 2 * AUN) { fu -= 2 * AUN; a_parity ^= 1u; }
            }
        }
    } else {
        const int quarter = warp & 3, col = quarter * 32 + lane, set = warp >> 2, half = set & 1;
        const uint32_t lane_base = uint32_t(quarter * 32) << 16;
        constexpr int FROWS = (RN + 15) / 16;
        float part[FROWS];
        spl_grid_begin();
#pragma unroll
        for (int f = 0; f < FROWS; ++f) part[f] = 0.0f;
        if (a.in_squares)
            for (int g0 = lane; g0 < a.in_groups; g0 += 128) {
                float v[FROWS][4];
#pragma unroll
                for (int f = 0; f < FROWS; ++f)
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int row = warp + 16 * f, g = g0 + 32 * u;
                        v[f][u] = (row < a.rows && g < a.in_groups) ? a.in_squares[size_t(row) * a.in_groups + g] : 0.0f;
                    }
#pragma unroll
                for (int f = 0; f < FROWS; ++f) part[f] += (v[f][0] + v[f][1]) + (v[f][2] + v[f][3]);
            }
        // A second-term operand has four data columns; the other four meet zeros, but have to be numbers: written once.
        for (int z = set; z < AUN; z += SETS) spl_tc_st4(tmem_aq + lane_base + z * 8 + 4, 0u, 0u, 0u, 0u);
        const unsigned char *codes0 = w_ring + half * 8192 + col * 16, *codes1 = codes0 + 2048, *sb0 = q_ring + half * 1024 + col * 4;
        int sc = set >> 1, slot = set, fu = set, bs = set >> 1;
        uint32_t c_parity = 0, b_parity = 0;
        bool ready_c = false;
        int un = set, t = 0;
#pragma unroll 1
        for (int tile = tile0; tile < a.tiles; tile += tile_step, ++t) {
        const int un_end = (t + 1) * units;
#pragma unroll 1
        for (; un < un_end && ok; un += SETS) {
            if (!__all_sync(0xffffffffu, ready_c)) ok = spl_mbar_wait_warp(&full_c[sc], c_parity, abort);
            if (!ok) { if (!*abort && lane == 0) spl_note_wait(a.error_flag, 41, un); break; }
            // The slot's last tenant has to have been multiplied: asked now, looked at when the codes are in registers.
            const bool ready_d = un < AUN || spl_mbar_test(&done[(un - AUN) & 15], ((un - AUN) >> 4) & 1);
            const uint4 lo[2] = {*reinterpret_cast<const uint4 *>(codes0 + sc * WSTAGE), *reinterpret_cast<const uint4 *>(codes0 + sc * WSTAGE + 4096)};
            const uint4 hi[2] = {*reinterpret_cast<const uint4 *>(codes1 + sc * WSTAGE), *reinterpret_cast<const uint4 *>(codes1 + sc * WSTAGE + 4096)};
            const uint32_t sbw[2] = {*reinterpret_cast<const uint32_t *>(sb0 + sc * QSTAGE), *reinterpret_cast<const uint32_t *>(sb0 + sc * QSTAGE + 512)};
            __syncwarp();
            if (lane == 0) spl_mbar_arrive(&empty_c[sc]);
            sc += 2; if (sc >= CST) { sc -= CST; c_parity ^= 1u; }
            if (!__all_sync(0xffffffffu, ready_d)) ok = spl_mbar_wait_warp(&done[(un - AUN) & 15], ((un - AUN) >> 4) & 1, abort);
            if (!ok) { if (!*abort && lane == 0) spl_note_wait(a.error_flag, 42, un); break; }
            spl_tc_fence_after();
            ready_c = spl_mbar_test(&full_c[sc], c_parity);
            uint32_t aq[4];
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const float sf = __uint_as_float(sbw[v] << 16), bf = __uint_as_float(sbw[v] & 0xFFFF0000u);
                const __half2 s2h = __float2half2_rn(sf), m24h = __hmul2(s2h, __float2half2_rn(-24.0f)), q2 = __hmul2(s2h, __float2half2_rn(512.0f)), q1 = __float2half2_rn(bf * 64.0f);
                const uint32_t s2 = *reinterpret_cast<const uint32_t *>(&s2h), m24 = *reinterpret_cast<const uint32_t *>(&m24h);
                aq[2 * v] = *reinterpret_cast<const uint32_t *>(&q1); aq[2 * v + 1] = *reinterpret_cast<const uint32_t *>(&q2);
#pragma unroll
                for (int part2 = 0; part2 < 2; ++part2) {
                    const uint4 src = part2 == 0 ? lo[v] : hi[v];
                    const uint32_t w4[4] = {src.x, src.y, src.z, src.w};
                    uint32_t r[16];
#pragma unroll
                    for (int w = 0; w < 4; ++w)
                        asm("{\n .reg .b32 xa, xb, xc, xd;\n"
                            " shr.b32 xb, %4, 4;\n prmt.b32 xc, %4, 0, 0x0321;\n shl.b32 xd, %4, 4;\n"
                            " lop3.b32 xa, %4, 0x03C003C0, 0x4C004C00, 0xEA;\n"
                            " lop3.b32 xb, xb, 0x03C003C0, 0x4C004C00, 0xEA;\n"
                            " lop3.b32 xc, xc, 0x03C003C0, 0x4C004C00, 0xEA;\n"
                            " lop3.b32 xd, xd, 0x03C003C0, 0x4C004C00, 0xEA;\n"
                            " fma.rn.f16x2 %0, xa, %5, %6;\n fma.rn.f16x2 %1, xb, %5, %6;\n"
                            " fma.rn.f16x2 %2, xc, %5, %6;\n fma.rn.f16x2 %3, xd, %5, %6;\n}\n"
                            : "=r"(r[4 * w]), "=r"(r[4 * w + 1]), "=r"(r[4 * w + 2]), "=r"(r[4 * w + 3])
                            : "r"(w4[w]), "r"(s2), "r"(m24));
                    spl_tc_st16(tmem_a + lane_base + slot * 64 + v * 32 + part2 * 16, r);
                }
            }
            spl_tc_st4(tmem_aq + lane_base + slot * 8, aq[0], aq[1], aq[2], aq[3]);
            // The set's first warp answers for the unit's activations as well: the issuing warps' waits are what the whole block keeps pace with, so they
            // get one barrier a unit.
            if (quarter == 0) {
                ok = spl_mbar_wait_warp(&full_b[bs], b_parity, abort);
                if (!ok) { if (!*abort && lane == 0) spl_note_wait(a.error_flag, 34, un); break; }
            }
            bs += 2; if (bs >= BST) { bs -= BST; b_parity ^= 1u; }
            spl_tc_st_wait();
            spl_tc_fence_before();
            __syncwarp();
            if (lane == 0) spl_mbar_arrive(&full_u[fu]);
            slot = slot == 0 ? AUN - 1 : slot - 1;          // four on, of five
            fu += SETS; if (fu >= 2 * AUN) fu -= 2 * AUN;
        }
        // ---- the tile's sums. Every converting warp comes here whatever happened to it before: the barriers cannot be left waiting.
        if (!ok) *abort_word = 1;
        if (t == 0 && a.in_squares)
#pragma unroll
            for (int f = 0; f < FROWS; ++f) {
                // The rows' factors of a deferred norm, the squares in one fixed order: a lane's groups, then a butterfly.
                const float ss = spl_warp_sum(part[f]);
                if (lane == 0) row_factor[warp + 16 * f] = 1.0f / sqrtf(ss / a.in_dim + a.eps);
            }
        // A load asked for now comes while the last products are formed.
        SplNarrowColumns at = {tile * 128 + (warp & 1) * 64 + 2 * lane, false, make_float2(0.0f, 0.0f), 0u};
        at.inside = at.n < a.out_ld;
        if (a.interleave > 0) {
            const int c2 = (warp & 1) * 64 + 2 * lane, e = tile * 64 + (c2 >> 5) * 16 + (c2 & 15);
            at.n = ((c2 & 16) ? a.interleave : 0) + e; at.inside = e < a.interleave;
        }
        {
            const int row = (split * WARPS + warp) >> 1;
            if (a.residual && at.inside && row < a.rows) at.res = spl_columns_load(a.residual + size_t(row) * a.out_ld + at.n, a.wide);
            if (a.emit_weight && at.inside) at.weight = *reinterpret_cast<const uint32_t *>(a.emit_weight + at.n);
        }
        __syncwarp();
        spl_named_barrier<1, SETS * 128>();
        if (ok && !spl_mbar_wait_warp(finished, t & 1, abort)) { ok = false; if (!*abort && lane == 0) spl_note_wait(a.error_flag, 40, t); }
        if (ok && set * 16 < RN) {
            spl_tc_fence_after();
            uint32_t v0[16], v1[16];
            spl_tc_ld16(v0, tmem_d + lane_base + set * 16);
            spl_tc_ld16(v1, tmem_d + lane_base + RN + set * 16);
            spl_tc_fence_before();
            // A cut tile's partial sums are scaled one by one, so their sum is.
            float x[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                x[r] = __uint_as_float(v0[r]) + __uint_as_float(v1[r]);
                if (a.in_squares) x[r] *= row_factor[set * 16 + r];
            }
            if (direct) {
                // A whole tile's plain output goes from the registers to its place, a column a thread (any float address will do): nobody else has to see
                // it. Through the plane, as the other outputs go, 17,408 x 5,120 at 64 rows took 21.4 us with its operand, and takes 20.3.
                const int e = tile * 64 + (col >> 5) * 16 + (col & 15), n = a.interleave > 0 ? ((col & 16) ? a.interleave : 0) + e : tile * 128 + col;
                if (a.interleave > 0 ? e < a.interleave : n < a.out_ld) {
                    const int last = a.rows - set * 16;
                    const size_t first = size_t(set * 16) * a.out_ld + n;
#pragma unroll
                    for (int r0 = 0; r0 < 16; r0 += 4) {
                        float res[4];
#pragma unroll
                        for (int r = 0; r < 4; ++r) res[r] = a.residual && r0 + r < last ? a.residual[first + size_t(r0 + r) * a.out_ld] : 0.0f;
#pragma unroll
                        for (int r = 0; r < 4; ++r)
                            if (r0 + r < last) a.out[first + size_t(r0 + r) * a.out_ld] = a.residual ? __fadd_rn(x[r0 + r], res[r]) : x[r0 + r];
                    }
                }
            } else
#pragma unroll
                for (int r = 0; r < 16; ++r) plane[(set * 16 + r) * 128 + col] = x[r];
        }
        __syncwarp();
        if (lane == 0) spl_mbar_arrive(drained);
        if (direct) continue;
        __syncwarp();
        if (S > 1) { spl_cluster_barrier(); } else spl_named_barrier<1, SETS * 128>();
        if (!*abort) spl_narrow_output<RN>(a, plane, tile, split, S, warp, lane, at);
        __syncwarp();
        if (S == 1) spl_named_barrier<1, SETS * 128>();        // the sums have been read: the next tile's may come
        }
    }
    if (!ok) { *abort_word = 1; atomicExch(a.error_flag, 1 + warp); }
    __syncwarp();
    if (S > 1 && warp >= WARPS) spl_cluster_barrier();          // every thread of a cluster's blocks meets the barrier the converting warps met above
    spl_tc_fence_before();
    __syncthreads();
    if (warp == W_MMA0) {
        spl_tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512) : "memory");
    }
    // A block that gave up may have copies in flight that nobody waited for: the copying threads wait (bounded) for the last one they asked for in
    // every ring slot before the block's shared memory is handed on.
    if (*abort_word && lane == 0) {
        if (warp == W_COPY)
            for (int q = 0; q < CST && q < issued_c; ++q) { const int i = q + (issued_c - 1 - q) / CST * CST; if (i % stages != a.drop) spl_mbar_wait(&full_c[q], (i / CST) & 1); }
        if (warp == W_COPYB)
            for (int q = 0; q < BST && q < issued_b; ++q) { const int i = q + (issued_b - 1 - q) / BST * BST; spl_mbar_wait(&full_b[q], (i / BST) & 1); }
    }
    __syncwarp();
    if (S > 1) spl_cluster_barrier();        // no block leaves while another may still read its sums
}
