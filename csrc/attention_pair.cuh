// Causal flash-prefill over the paged fp16 cache with TWO query tiles a block (attention_tc.cuh has one).
//
// Bound by the tensor cores and the exponentials, each some 1,024 clocks for 128 queries x 128 keys x 128 dims, if they work at the same time.
// With one tile they take turns: the P.V of a tile of keys needs its softmax.  Here a block owns two tiles - the same 128 queries of two query
// heads that share a key / value head, or (odd group sizes) 256 queries of one head -, and while the four softmax warps of one tile work, the
// MMAs of the other run.  K and V are fetched once for both.  The softmax weights go back to TENSOR MEMORY as fp16, over the scores they came
// from, and enter P.V from there (tcgen05.mma with A in tensor memory): no shared memory for P, no proxy fences.
//   tensor memory: scores and weights of tile s in [128 s, + 128), outputs in [256 + 128 s, + D)
//   order of the one MMA thread:  QK0(0) QK1(0) | PV0(i) QK0(i+1) PV1(i) QK1(i+1) | ...   MMAs of a block complete in order, so the arrival
//   of scores i + 1 also says that P.V of tile i has read its weights and updated the output.
// The output is rescaled only when a row maximum has grown by more than 2^8 since the last time (weights up to 256: the same relative rounding).
// 32 query heads over 8, D = 128, in us: 2,048 queries behind 4,096 keys 191 (0.90 PFLOP/s; one tile a block 370), 953 behind 6,144 120 (0.86),
// 2,048 from the start 65.
#pragma once
#include "attention_tc.cuh"
#include "gemm_quant_small.cuh"

namespace dlp {

template <int D>
struct FpCfg {
    static constexpr int BM = 128, BN = 128, KB = D / 64;
    static constexpr int TILE = 128 * D * 2;                     // one Q, K or V tile
    static constexpr int SMEM_BYTES = 6 * TILE + 1024 + 256;     // Q of two tiles, two stages of K and V
    static constexpr int THREADS = 320;
};

template <int D>
__global__ void __launch_bounds__(320, 1)
attn_prefill_pair_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                         const FaParams p, const int by_head) {
    using Cfg = FpCfg<D>;
    constexpr int BM = Cfg::BM, BN = Cfg::BN, KB = Cfg::KB, TILE = Cfg::TILE;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t *sm_q = smem, *sm_k = smem + 2 * TILE, *sm_v = sm_k + 2 * TILE;      // [tile or stage][KB][128 rows][128 B]
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 6 * TILE);
    uint64_t *q_full = bars, *k_full = bars + 1, *v_full = bars + 3, *k_empty = bars + 5, *v_empty = bars + 7, *s_full = bars + 9, *p_full = bars + 11, *o_done = bars + 13;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 15);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int qt = gridDim.x - 1 - blockIdx.x;                   // heaviest (latest) queries first
    int hq[2], t0[2], n[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
        hq[s] = by_head ? 2 * blockIdx.y + s : blockIdx.y;
        t0[s] = (by_head ? qt : 2 * qt + s) * BM;
        n[s] = t0[s] < p.T ? (p.pos0 + min(t0[s] + BM, p.T) + BN - 1) / BN : 0;
    }
    const int kvh = hq[0] / (p.Hq / p.Hkv), n_max = max(n[0], n[1]);

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_v);
        mbar_init(q_full, 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(&k_full[s], 1); mbar_init(&v_full[s], 1); mbar_init(&k_empty[s], 1); mbar_init(&v_empty[s], 1);
            mbar_init(&s_full[s], 1); mbar_init(&p_full[s], 4); mbar_init(&o_done[s], 1);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();

    if (warp == 0) {
        if (elect_one()) {
            mbar_expect_tx(q_full, (n[1] > 0 ? 2 : 1) * TILE);
#pragma unroll
            for (int s = 0; s < 2; ++s)
                for (int kb = 0; kb < KB && n[s] > 0; ++kb) tma_load_2d(sm_q + s * TILE + kb * (BM * 128), &tm_q, q_full, hq[s] * D + kb * 64, t0[s]);
            const int ps = p.page_size, chunks = BN / ps;
            for (int i = 0; i < n_max; ++i) {
                const int s = i & 1;
                const uint32_t ph = (uint32_t)(i >> 1) & 1u;
                auto row_of = [&](int pc) { return (p.bt_row[min((i * BN + pc * ps) / ps, p.max_pages - 1)] * p.Hkv + kvh) * ps; };
                mbar_wait_b(&k_empty[s], ph ^ 1);
                mbar_expect_tx(&k_full[s], TILE);
                for (int pc = 0; pc < chunks; ++pc) {
                    const int row = row_of(pc);
                    for (int kb = 0; kb < KB; ++kb) tma_load_2d(sm_k + s * TILE + kb * (BN * 128) + pc * (ps * 128), &tm_k, &k_full[s], kb * 64, row);
                }
                mbar_wait_b(&v_empty[s], ph ^ 1);
                mbar_expect_tx(&v_full[s], TILE);
                for (int pc = 0; pc < chunks; ++pc) {
                    const int row = row_of(pc);
                    for (int kb = 0; kb < KB; ++kb) tma_load_2d(sm_v + s * TILE + kb * (BN * 128) + pc * (ps * 128), &tm_v, &v_full[s], kb * 64, row);
                }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc_s = make_idesc_f16(BM, BN, 0);
            constexpr uint32_t idesc_o = make_idesc_f16_bmn(BM, D, 0);
            auto scores = [&](int s, int i) {                    // S_s = Q_s . K_i^T
                mbar_wait_b(&k_full[i & 1], (uint32_t)(i >> 1) & 1u);
                tc_fence_after();
#pragma unroll
                for (int kb = 0; kb < KB; ++kb) {
                    const uint64_t da = make_smem_desc_sw128(smem_u32(sm_q + s * TILE + kb * (BM * 128)));
                    const uint64_t db = make_smem_desc_sw128(smem_u32(sm_k + (i & 1) * TILE + kb * (BN * 128)));
#pragma unroll
                    for (int k = 0; k < 4; ++k) tc_mma_f16(tmem_base + s * 128, da + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc_s, (kb > 0 || k > 0) ? 1u : 0u);
                }
                tc_commit(&s_full[s]);
            };
            mbar_wait_b(q_full, 0);
#pragma unroll
            for (int s = 0; s < 2; ++s)
                if (n[s] > 0) scores(s, 0);
            tc_commit(&k_empty[0]);
            for (int i = 0; i < n_max; ++i) {
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    if (i >= n[s]) continue;
                    mbar_wait_b(&v_full[i & 1], (uint32_t)(i >> 1) & 1u);
                    mbar_wait_b(&p_full[s], (uint32_t)i & 1u);
                    tc_fence_after();
#pragma unroll
                    for (int kk = 0; kk < BN / 16; ++kk)
                        tc_mma_f16_ts(tmem_base + 256 + s * 128, tmem_base + s * 128 + kk * 8,
                                      make_smem_desc_sw128_mn(smem_u32(sm_v + (i & 1) * TILE + kk * 16 * 128), BN * 128), idesc_o, (i > 0 || kk > 0) ? 1u : 0u);
                    if (i + 1 < n[s]) scores(s, i + 1);
                    else tc_commit(&o_done[s]);
                }
                tc_commit(&v_empty[i & 1]);
                if (i + 1 < n_max) tc_commit(&k_empty[(i + 1) & 1]);
            }
        }
    } else {
        const int s = (warp - 2) >> 2, q4 = warp & 3, r = q4 * 32 + lane;
        const int n_s = s ? n[1] : n[0], t0_s = s ? t0[1] : t0[0], hq_s = s ? hq[1] : hq[0];
        const int pos_t = p.pos0 + t0_s, q_pos = pos_t + r;      // this row sees keys 0 .. q_pos
        const uint32_t s_addr = tmem_base + ((uint32_t)(q4 * 32) << 16) + s * 128, o_addr = s_addr + 256;
        constexpr float LOG2E = 1.4426950408889634f;
        float m = -INFINITY, l = 0.f;                            // the maximum that the weights are relative to
        for (int i = 0; i < n_s; ++i) {
            const int n0 = i * BN;
            mbar_wait_b(&s_full[s], (uint32_t)i & 1u);
            tc_fence_after();
            uint32_t sv[BN];
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) tmem_ld_32x32(s_addr + c * 32, *reinterpret_cast<uint32_t(*)[32]>(&sv[c * 32]));
            tc_wait_ld();
            if (n0 + BN - 1 > pos_t) {                           // some (query, key) pairs are masked
#pragma unroll
                for (int j = 0; j < BN; ++j)
                    if (n0 + j > q_pos) sv[j] = __float_as_uint(-INFINITY);
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int j = 0; j < BN; ++j) mx[j & 3] = fmaxf(mx[j & 3], __uint_as_float(sv[j]));
            const float top = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            const bool grow = m == -INFINITY ? top != -INFINITY : (top - m) * LOG2E > 8.f;
            if (__any_sync(0xffffffffu, grow)) {
                const float mn = fmaxf(m, top);
                const float alpha = m == -INFINITY ? 0.f : exp2f((m - mn) * LOG2E);
                m = mn;
                l *= alpha;
                if (i > 0) {
#pragma unroll 1
                    for (int c = 0; c < D / 32; ++c) {
                        uint32_t o[32];
                        tmem_ld_32x32(o_addr + c * 32, o);
                        tc_wait_ld();
#pragma unroll
                        for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
                        tmem_st_32x32(o_addr + c * 32, o);
                    }
                }
            }
            const float ms = m == -INFINITY ? 0.f : m * LOG2E;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
            // the weights replace the scores in registers: fp16 pairs in the lower half of sv
#pragma unroll
            for (int j = 0; j < BN; j += 2) {
                const float p0 = exp2f(fmaf(__uint_as_float(sv[j]), LOG2E, -ms)), p1 = exp2f(fmaf(__uint_as_float(sv[j + 1]), LOG2E, -ms));
                const __half2 h = __floats2half2_rn(p0, p1);
                const float2 hf = __half22float2(h);              // the sum uses the rounded values that the tensor cores will see
                sum[(j >> 1) & 3] += hf.x + hf.y;
                sv[j / 2] = *reinterpret_cast<const uint32_t*>(&h);
            }
            l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
#pragma unroll
            for (int c = 0; c < BN / 64; ++c) tmem_st_32x32(s_addr + c * 32, *reinterpret_cast<const uint32_t(*)[32]>(&sv[c * 32]));
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[s]);
        }
        pdl_launch_dependents();
        if (n_s > 0) {
            mbar_wait_b(&o_done[s], 0);
            tc_fence_after();
            const float inv = l > 0.f ? 1.f / l : 0.f;
            const int t = t0_s + r;
#pragma unroll 1
            for (int c = 0; c < D / 32; ++c) {
                uint32_t o[32];
                tmem_ld_32x32(o_addr + c * 32, o);
                tc_wait_ld();
                if (t < p.T) {
                    __half* orow = reinterpret_cast<__half*>(p.out) + (size_t)t * p.ldo + (size_t)hq_s * D;
#pragma unroll
                    for (int j = 0; j < 32; j += 8) {
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const __half2 h = __floats2half2_rn(__uint_as_float(o[j + 2 * e]) * inv, __uint_as_float(o[j + 2 * e + 1]) * inv);
                            w[e] = *reinterpret_cast<const uint32_t*>(&h);
                        }
                        *reinterpret_cast<uint4*>(orow + c * 32 + j) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
                __syncwarp();
            }
        }
    }
    gemm_wait_aftermath();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        __syncwarp();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace dlp
