// Dense GEMM on pairs of SMs (kernel: gemm_pair.cuh).
#include "gemm_pair.cuh"

namespace dlp {

// Wider than the token tiles that the workspace splits and the narrow tiles of gemm_tcgen05_kernel are for.  At 96 tokens both stream the weights
// (4096 x 14336: 25 us); from 128 on the pairs gain (256 tokens x 4096 x 14336: 30 us against 48).  Routed experts: tiles of at least 64 tokens.
bool gemm_pair_takes(int T, const GemmGroup* grp) { return grp ? grp->bt >= 64 : T > 64; }

// Token tile and split of K by a model of the launch in nanoseconds, fitted to sweeps of both at 512 and 2,048 tokens: full waves of pairs, each
// tile its blocks of 64 columns.  Up to some 128 tokens a block costs what its way through L2 and shared memory costs, then the products take
// over (one accumulator: 210 ns at 64 tokens, 246 at 128, 303 at 192, 383 at 256; gate and up: 330, 430, 590, 810 with the drain that stands alone).
static PairPlan pair_plan(int T, int N, int K, int na, bool split, const GemmGroup* grp) {
    const int pairs = sm_count() / 2, total_kb = (K + GEMM_BK - 1) / GEMM_BK, tiles_n = (N + 2 * GEMM_BM - 1) / (2 * GEMM_BM);
    PairPlan best = {};
    if (grp) return {grp->bt, 1, tiles_n, grp->max_tiles, total_kb};
    double best_cost = -1;
    for (int bt = 256; bt >= 32; bt -= 16) {
        if (bt > 32 && bt - 16 >= T) continue;
        const double per_kb = na == 2 ? 300 + 0.0078 * bt * bt : 200 + 0.0028 * bt * bt;
        for (int z = 1; z <= (split ? 8 : 1); ++z) {
            if (z > 1 && total_kb / z < 16) break;
            const int tiles_t = (T + bt - 1) / bt, kb = (total_kb + z - 1) / z;
            const long waves = ((long)tiles_n * tiles_t * z + pairs - 1) / pairs;
            const double cost = waves * (kb * per_kb + 1500 + (z > 1 ? 4.0 * bt : 0));      // (split: the sums meet in L2)
            if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = {bt, z, tiles_n, tiles_t, kb}; }
        }
    }
    return best;
}

template <int NA, int AB_FMT>
static int launch_pair(const CUtensorMap& tw0, const CUtensorMap& tw1, const CUtensorMap& tx, const GemmParams& p, const PairPlan& pl, cudaStream_t stream) {
    auto kern = gemm_pair_kernel<NA, AB_FMT>;
    if (first_use_on_device((const void*)kern))
        DLP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg<NA>::SMEM_BYTES));
    const long items = (long)pl.tiles_n * pl.tiles_t * pl.splits, pairs = sm_count() / 2;
    DLP_CHECK_CUDA(launch_pdl(kern, dim3(2 * (unsigned)(items < pairs ? items : pairs)), dim3(320), PairCfg<NA>::SMEM_BYTES, stream, tw0, tw1, tx, p, pl));
    return 0;
}

int gemm_pair(const GemmParams& p, const void* w0, const void* w1, int ldw, const void* x, int ldx, int is_bf16, int na, int split_k, cudaStream_t stream) {
    const GemmGroup* grp = p.grp.tile_expert ? &p.grp : nullptr;
    const PairPlan pl = pair_plan(p.T, p.N, p.K, na, p.epilogue == EPI_ATOMIC_ADD_F32 && split_k <= 0 && gemm_add_may_split(p.T, p.N, (p.K + GEMM_BK - 1) / GEMM_BK), grp);
    const uint64_t w_rows = grp ? (uint64_t)grp->rows_per_expert * grp->n_expert : (uint64_t)p.N;
    CUtensorMap tw0, tw1, tx;
    int rc;
    if ((rc = make_tmap_2d(&tw0, w0, is_bf16, w_rows, p.K, ldw, GEMM_BM))) return rc;
    tw1 = tw0;
    if (na == 2 && (rc = make_tmap_2d(&tw1, w1, is_bf16, w_rows, p.K, ldw, GEMM_BM))) return rc;
    if ((rc = make_tmap_2d(&tx, x, is_bf16, p.T, p.K, ldx, pl.bt / 2))) return rc;
#ifdef DLP_LAYERS_ONLY
    return na == 2 ? launch_pair<2, 1>(tw0, tw1, tx, p, pl, stream) : launch_pair<1, 1>(tw0, tw1, tx, p, pl, stream);
#else
    if (is_bf16) return na == 2 ? launch_pair<2, 1>(tw0, tw1, tx, p, pl, stream) : launch_pair<1, 1>(tw0, tw1, tx, p, pl, stream);
    return na == 2 ? launch_pair<2, 0>(tw0, tw1, tx, p, pl, stream) : launch_pair<1, 0>(tw0, tw1, tx, p, pl, stream);
#endif
}

}  // namespace dlp
