// Dense GEMM for prompts:  Y[T, N] (op)= X[T, K] . W[N, K]^T  (fp16 or bf16, fp32 sums) on PAIRS of SMs (tcgen05 cta_group::2).
//
// Bound by the tensor cores.  gemm_tcgen05_kernel (one SM, 128 x 256 tiles, a block per tile) reads 48 KB and receives 48 KB of shared memory
// per 512 clocks of MMA - more than the 128 bytes a clock that an SM has - and its epilogue stands alone at the end of every tile.  Here
//   * two blocks of a cluster share a tile of 256 features x BT tokens: each loads its 128 rows of W and HALF of the tokens, and the pair's MMA
//     reads both halves (64 KB per 512 clocks);
//   * the grid is one pair per two SMs and walks the tiles; with one accumulator of at most 256 columns the next tile's products go to the other
//     half of tensor memory while eight warps drain the first (gate + up of 256 tokens fill it: there the drain stands alone);
//   * the token tile (16 .. 256 in steps of 16) and with the residual epilogue the split of K are chosen by the host so that the last wave is
//     full (pair_plan).
// fp16, times in us before (gemm_tcgen05_kernel) and now, in brackets the rate now: 512 tokens x 6144 x 4096 36 -> 22.7 (1.14 PFLOP/s),
// gate and up 14336 x 4096 120 -> 104 (1.15); 2,048 tokens: 6144 x 4096 75 (1.37), 4096 x 4096 45 (1.54), gate and up 364 (1.32),
// 4096 x 14336 182 (1.32; about 290 before).
#pragma once
#include "gemm_tcgen05.cuh"

namespace dlp {

__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ uint32_t leader_addr(const void* p) {       // the same place in the shared memory of the pair's first block
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void pair_tma_2d(void* smem_dst, const void* desc, uint32_t leader_bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(desc), "r"(leader_bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void pair_mma_f16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void pair_commit(uint64_t* bar) {           // arrives at this barrier of both blocks when the MMAs so far are done
    asm volatile(
        "{\n\t.reg .b16 m;\n\t"
        "mov.b16 m, 3;\n\t"
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], m;\n\t}"
        ::"r"(smem_u32(bar)) : "memory");
}

struct PairPlan { int bt, splits, tiles_n, tiles_t, kb_per_split; };

template <int NA>
struct PairCfg {
    static constexpr int A_BYTES = GEMM_BM * GEMM_BK * 2, B_BYTES = 128 * GEMM_BK * 2;      // of one block; B: up to 128 tokens
    static constexpr int STAGE = NA * A_BYTES + B_BYTES;
    static constexpr int STAGES = NA == 2 ? 4 : 6;
    static constexpr int SMEM_BYTES = STAGES * STAGE + 1024 + 256;
};

template <int NA, int AB_FMT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(320, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tm_w0, const __grid_constant__ CUtensorMap tm_w1, const __grid_constant__ CUtensorMap tm_x,
                 const GemmParams p, const PairPlan pl) {
    using Cfg = PairCfg<NA>;
    constexpr int STAGES = Cfg::STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE);
    uint64_t *full = bars, *empty = bars + STAGES, *acc_full = bars + 2 * STAGES, *acc_empty = acc_full + 2;      // full and acc_empty: the first block's
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int bt = pl.bt, half = bt / 2;
    const int n_buf = NA * bt <= 256 ? 2 : 1;                      // accumulator sets in the 512 columns
    const int up_col = NA == 2 ? (n_buf == 2 ? 128 : 256) : 0;
    const uint32_t stage_tx = 2u * (NA * Cfg::A_BYTES + half * GEMM_BK * 2);      // both blocks' loads

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tm_w0);
        if (NA == 2) tma_prefetch_desc(&tm_w1);
        tma_prefetch_desc(&tm_x);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 16); }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                            // both blocks' barriers are up
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();

    const bool grouped = p.grp.tile_expert != nullptr;
    const int tiles_t = grouped ? *p.grp.n_tiles : pl.tiles_t;
    const int items = tiles_t * pl.tiles_n * pl.splits;
    const int total_kb = (p.K + GEMM_BK - 1) / GEMM_BK;
    struct Item { int n_out, n_w, t0, t_end, kb0, kb1; };
    auto item_of = [&](int i) {                                    // tokens fastest: the pairs at work share a few tiles of W and of X
        Item it;
        const int tt = i % tiles_t, rest = i / tiles_t, tn = rest % pl.tiles_n, z = rest / pl.tiles_n;
        it.n_out = it.n_w = tn * 2 * GEMM_BM + (int)rank * GEMM_BM;
        it.t0 = tt * bt;
        it.t_end = min(p.T, it.t0 + bt);
        if (grouped) {
            it.n_w += p.grp.tile_expert[tt] * p.grp.rows_per_expert;
            it.t0 = p.grp.tile_row0[tt];
            it.t_end = it.t0 + p.grp.tile_rows[tt];
        }
        it.kb0 = z * pl.kb_per_split;
        it.kb1 = min(total_kb, it.kb0 + pl.kb_per_split);
        return it;
    };
    const int i0 = blockIdx.x >> 1, step = gridDim.x >> 1;

    if (warp == 0) {
        // ===== TMA: this block's rows of W and its half of the tokens; the bytes count at the first block's barrier =====
        if (elect_one()) {      // (elect.sync: with lane == 0 the compiler issues TMA and MMAs through a loop over the lanes, 100 clocks each)
            int s = 0;
            uint32_t ph = 0;
            for (int i = i0; i < items; i += step) {
                const Item it = item_of(i);
                for (int kb = it.kb0; kb < it.kb1; ++kb) {
                    mbar_wait_b<true>(&empty[s], ph ^ 1);
                    if (rank == 0) mbar_expect_tx(&full[s], stage_tx);
                    const uint32_t bar = leader_addr(&full[s]);
                    uint8_t* st = smem + s * Cfg::STAGE;
                    pair_tma_2d(st, &tm_w0, bar, kb * GEMM_BK, it.n_w);
                    if (NA == 2) pair_tma_2d(st + Cfg::A_BYTES, &tm_w1, bar, kb * GEMM_BK, it.n_w);
                    pair_tma_2d(st + NA * Cfg::A_BYTES, &tm_x, bar, kb * GEMM_BK, it.t0 + (int)rank * half);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        // ===== MMA: one thread of the first block issues for both =====
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = make_idesc_f16(2 * GEMM_BM, bt, AB_FMT);
            int s = 0, n = 0;
            uint32_t ph = 0;
            for (int i = i0; i < items; i += step, ++n) {
                const Item it = item_of(i);
                const int b = n_buf == 2 ? n & 1 : 0;
                const uint32_t use = (uint32_t)(n_buf == 2 ? n >> 1 : n);
                mbar_wait_b<true>(&acc_empty[b], (use & 1) ^ 1);
                tc_fence_after();
                const uint32_t d = tmem_base + b * 256;
                for (int kb = it.kb0; kb < it.kb1; ++kb) {
                    mbar_wait_b<true>(&full[s], ph);
                    tc_fence_after();
                    const uint32_t st = smem_u32(smem + s * Cfg::STAGE);
                    const uint64_t da0 = make_smem_desc_sw128(st), da1 = make_smem_desc_sw128(st + Cfg::A_BYTES), db = make_smem_desc_sw128(st + NA * Cfg::A_BYTES);
#pragma unroll
                    for (int k = 0; k < GEMM_BK / 16; ++k) {
                        const uint32_t acc = (kb > it.kb0 || k > 0) ? 1u : 0u;
                        pair_mma_f16(d, da0 + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, acc);
                        if (NA == 2) pair_mma_f16(d + up_col, da1 + (uint64_t)(2 * k), db + (uint64_t)(2 * k), idesc, acc);
                    }
                    pair_commit(&empty[s]);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
                pair_commit(&acc_full[b]);
            }
        }
    } else {
        // ===== epilogue: warps 2-5 and 6-9 take turns over chunks of 32 tokens; lane quarter warp % 4 holds 32 of this block's features =====
        const int q = warp & 3, group = (warp - 2) >> 2;
        int n = 0;
        for (int i = i0; i < items; i += step, ++n) {
            const Item it = item_of(i);
            const int b = n_buf == 2 ? n & 1 : 0;
            const uint32_t use = (uint32_t)(n_buf == 2 ? n >> 1 : n);
            const int col = it.n_out + q * 32 + lane;
            const float bias = p.epilogue == EPI_TAIL_BF16 && p.tail.bias != nullptr && col < p.N ? p.tail.bias[col] : 0.f;
            mbar_wait_b<true>(&acc_full[b], use & 1);
            tc_fence_after();
            const uint32_t addr = tmem_base + ((uint32_t)(q * 32) << 16) + b * 256;
#pragma unroll 1
            for (int c = group; c * 32 < it.t_end - it.t0; c += 2) {
                uint32_t r0[32], r1[32];
                tmem_ld_32x32(addr + c * 32, r0);
                if (NA == 2) tmem_ld_32x32(addr + up_col + c * 32, r1);
                tc_wait_ld();
                if (col < p.N) {
                    const int tb = it.t0 + c * 32;
                    switch (p.epilogue) {
                        case EPI_STORE_F16: if (NA == 1) epi_loop<EPI_STORE_F16, 32>(p, r0, r1, tb, col, it.t_end); break;
                        case EPI_STORE_BF16: if (NA == 1) epi_loop<EPI_STORE_BF16, 32>(p, r0, r1, tb, col, it.t_end); break;
                        case EPI_STORE_F32: if (NA == 1) epi_loop<EPI_STORE_F32, 32>(p, r0, r1, tb, col, it.t_end); break;
                        case EPI_ATOMIC_ADD_F32: if (NA == 1) epi_loop<EPI_ATOMIC_ADD_F32, 32>(p, r0, r1, tb, col, it.t_end); break;
                        case EPI_SWIGLU_F16: if (NA == 2) epi_loop<EPI_SWIGLU_F16, 32>(p, r0, r1, tb, col, it.t_end); break;
                        case EPI_GEGLU_BF16: if (NA == 2 && AB_FMT == 1) epi_loop<EPI_GEGLU_BF16, 32>(p, r0, r1, tb, col, it.t_end); break;
                        case EPI_SWIGLU_BF16: if (NA == 2 && AB_FMT == 1) epi_loop<EPI_SWIGLU_BF16, 32>(p, r0, r1, tb, col, it.t_end); break;
                        case EPI_RELU2_BF16: if (NA == 1 && AB_FMT == 1) epi_loop<EPI_RELU2_BF16, 32>(p, r0, r1, tb, col, it.t_end); break;
                        case EPI_TAIL_BF16: if (NA == 1 && AB_FMT == 1) epi_loop<EPI_TAIL_BF16, 32>(p, r0, r1, tb, col, it.t_end, bias); break;
                    }
                }
                __syncwarp();
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(leader_addr(&acc_empty[b])) : "memory");
        }
        pdl_launch_dependents();
    }
    gemm_wait_aftermath();
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();                                            // neither block leaves while the other may still read its shared memory or arrive at its barriers
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

}  // namespace dlp
