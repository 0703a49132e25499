// tcgen05 GEMM with the block-quant decode fused into the A-operand producer (kernel: gemm_tcgen05.cuh).
#include "gemm_tcgen05.cuh"

namespace dlp {

bool gemm_quant_small_takes(const QWeight& w, int wtype);
int gemm_quant_small(const QWeight& w0, const QWeight& w1, int na, int wtype, int bt, const CUtensorMap& tx, const GemmParams& p, int split_k, void* ws,
                     size_t ws_bytes, cudaStream_t stream);

// ---- prompts: unpack a piece of the weights to fp16, multiply it on pairs of SMs ---------------------------------------------------
// gemm_tcgen05_kernel unpacks its rows again for every 256 tokens and waits for them.  Here every weight is unpacked once, into pieces of
// scratch that L2 (126 MB) mostly holds until the GEMM behind has read them.  Llama-8B in Q4_K, 1,021 tokens, us: gate and up 634 -> 242 (the
// GEMM alone 185), 4096 x 14336 190 -> 119, 4096 x 4096 39.
template <int WT>
__global__ void __launch_bounds__(256) unpack_rows_kernel(const QWeight w0, const QWeight w1, int row0, int rows, __half* __restrict__ out) {
    const int nchunk = w0.K / 32;
    const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
    const int r = (int)(i / nchunk), c = (int)(i - (long)r * nchunk);
    QChunk ch;
    if (r < rows) load_chunk<WT>(blockIdx.y ? w1 : w0, row0 + r, c, ch);      // weights are static: requested before the predecessor has finished
    pdl_wait();                                                                // (which may still read the scratch)
    pdl_launch_dependents();
    if (r >= rows) return;
    __half* dst = out + ((size_t)blockIdx.y * rows + r) * w0.K;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
        uint32_t o[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const float2 f = __half22float2(ch.q[g][j]);
            const __half2 h = __floats2half2_rn(fmaf(ch.scale[g], f.x, ch.bias[g]), fmaf(ch.scale[g], f.y, ch.bias[g]));
            o[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        uint4* p = reinterpret_cast<uint4*>(dst + ch.k[g]);
        p[0] = make_uint4(o[0], o[1], o[2], o[3]);
        p[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
}

int gemm_quant_pieces(const QWeight& w0, const QWeight* w1, int wtype, const void* x, void* y, int ldy, int T, int epilogue, void* scratch,
                      size_t scratch_bytes, cudaStream_t stream) {
    const int N = w0.N, K = w0.K, na = epilogue == EPI_SWIGLU_F16 ? 2 : 1;
    DLP_REQUIRE(na == 1 || w1 != nullptr, "gemm_quant: SwiGLU epilogue needs the up-projection weight");
    const long most = (long)(scratch_bytes / ((size_t)K * 2 * na)) / 256 * 256;      // whole row tiles
    DLP_REQUIRE(most >= 256 && (reinterpret_cast<uintptr_t>(scratch) & 15) == 0, "gemm_quant: scratch of %zu bytes at %p for rows of %d columns", scratch_bytes, scratch, K);
    const int pieces = (int)((N + most - 1) / most), per = ((N + pieces - 1) / pieces + 255) / 256 * 256;
    const QWeight up = w1 ? *w1 : w0;
    for (int n0 = 0; n0 < N; n0 += per) {
        const int rows = N - n0 < per ? N - n0 : per;
        const dim3 grid((unsigned)(((long)rows * (K / 32) + 255) / 256), na);
        __half* out = (__half*)scratch;
        switch (wtype) {
            case W_Q8_0: DLP_CHECK_CUDA(launch_pdl(unpack_rows_kernel<W_Q8_0>, grid, dim3(256), 0, stream, w0, up, n0, rows, out)); break;
            case W_Q4_K: DLP_CHECK_CUDA(launch_pdl(unpack_rows_kernel<W_Q4_K>, grid, dim3(256), 0, stream, w0, up, n0, rows, out)); break;
            case W_Q5_K: DLP_CHECK_CUDA(launch_pdl(unpack_rows_kernel<W_Q5_K>, grid, dim3(256), 0, stream, w0, up, n0, rows, out)); break;
            case W_Q6_K: DLP_CHECK_CUDA(launch_pdl(unpack_rows_kernel<W_Q6_K>, grid, dim3(256), 0, stream, w0, up, n0, rows, out)); break;
            default: DLP_REQUIRE(false, "gemm_quant: unsupported weight type %d", wtype);
        }
        const size_t size = epilogue == EPI_STORE_F16 || epilogue == EPI_SWIGLU_F16 ? 2 : 4;
        // (the launch before this one makes the operand: not static)
        const int rc = gemm_f16(out, na == 2 ? out + (size_t)rows * K : nullptr, K, x, K, (uint8_t*)y + (size_t)n0 * size, ldy, T, rows, K, epilogue, 0, 0, false, stream);
        if (rc) return rc;
    }
    return 0;
}

// Y[T,N] (op)= X[T,K] . dequant(W)[N,K]^T with the block-quant decode fused into the A-operand producer.
int gemm_quant(const QWeight& w0, const QWeight* w1, int wtype, const void* x, int ldx, void* y, int ldy, int T, int epilogue,
               int split_k, cudaStream_t stream, const GemmCollective* coll, const GemmGroup* grp, void* ws, size_t ws_bytes) {
    // grouped: w0 / w1 describe the stack of all experts (w0.N = n_expert * rows_per_expert); one expert's width tiles the grid
    const int N = grp ? grp->rows_per_expert : w0.N, K = w0.K;
    DLP_REQUIRE(T > 0 && N > 0 && K > 0 && K % 256 == 0, "gemm_quant: bad problem T=%d N=%d K=%d", T, N, K);
    DLP_REQUIRE(grp == nullptr || (grp->tile_expert && grp->tile_row0 && grp->tile_rows && grp->n_tiles && grp->max_tiles > 0 && split_k <= 1 &&
                                   epilogue != EPI_RS_PUSH_F32 && epilogue != EPI_ATOMIC_ADD_F32 && w0.N == grp->rows_per_expert * grp->n_expert),
                "gemm_quant: bad grouped descriptor");
    const int na = (epilogue == EPI_SWIGLU_F16) ? 2 : 1;
    DLP_REQUIRE(na == 1 || w1 != nullptr, "gemm_quant: SwiGLU epilogue needs the up-projection weight");
    const int total_kb = K / GEMM_BK;
    int splits = split_k;
    if (splits <= 0) {
        splits = 1;
        if (epilogue == EPI_ATOMIC_ADD_F32) {
            const int bt_guess = T <= 16 ? 16 : T <= 32 ? 32 : T <= 64 ? 64 : T <= 128 ? 128 : 256;
            const long tiles = (long)((N + GEMM_BM - 1) / GEMM_BM) * ((T + bt_guess - 1) / bt_guess);
            const int sms = sm_count();
            while (tiles * splits * 2 <= sms && total_kb / (splits * 2) >= 8) splits *= 2;
        }
    }
    DLP_REQUIRE(splits == 1 || epilogue == EPI_ATOMIC_ADD_F32, "gemm_quant: split-K needs the atomic-add epilogue or a workspace");
    if (splits > total_kb) splits = total_kb;
    GemmParams p;
    memset(&p, 0, sizeof(p));
    if (coll) p.coll = *coll;
    DLP_REQUIRE(epilogue != EPI_RS_PUSH_F32 || (coll && coll->rs_rows > 0 && coll->rs_done && coll->rs_tp >= 1 && coll->rs_tp <= 8 && splits == 1),
                "gemm: the reduce-scatter epilogue needs a collective descriptor and no atomic split-K");
    p.y = y; p.T = T; p.N = N; p.K = K; p.ldy = ldy; p.epilogue = epilogue; p.w_static = true;
    if (grp) p.grp = *grp;
    int bt = grp ? grp->bt : (T <= 16 ? 16 : T <= 32 ? 32 : T <= 64 ? 64 : T <= 128 ? 128 : 256);
    const QWeight up = w1 ? *w1 : QWeight();
    // Token tiles of up to 64 stream the weights' bytes (gemm_quant_small.cuh); wider ones are bound by the MMAs.  At 64 tokens the
    // bytes still bound it (Q8_0 gate and up of Llama-8B: 35 us, 7 tokens 34), up to 192 some tiles of 64 are mostly faster than unpacking the
    // weights for one pass.  192 tokens in tiles / 193 in one pass, us: gate and up of 14336 x 4096 in Q8_0 88 / 143, Q4_K 119 / 138, Q5_K 132 / 140, Q6_K
    // 132 / 130; 4096 x 14336 38 / 63, 45 / 61, 50 / 62, 84 / 57; 2048 x 2048 6.9 / 12.1, 8.6 / 11.7, 9.2 / 11.8, 8.4 / 11.4.  Four tiles of 64 in Q4_K: 160 / 143.
    if ((bt <= 64 || (grp == nullptr && T <= 192)) && coll == nullptr && epilogue != EPI_RS_PUSH_F32 && gemm_quant_small_takes(w0, wtype) && (na == 1 || gemm_quant_small_takes(up, wtype))) {
        if (bt > 64) bt = 64;
        CUtensorMap tx;
        if (int rc = make_tmap_2d(&tx, x, 0, T, K, ldx, bt)) return rc;
        return gemm_quant_small(w0, up, na, wtype, bt, tx, p, split_k, ws, ws_bytes, stream);
    }
    if (splits == 1)
        splits = auto_split_ws(epilogue, split_k, (long)((N + GEMM_BM - 1) / GEMM_BM) * (grp ? grp->max_tiles : (T + bt - 1) / bt), total_kb, na, bt,
                               ws, ws_bytes, p);
    p.k_blocks_per_split = (total_kb + splits - 1) / splits;
    splits = (total_kb + p.k_blocks_per_split - 1) / p.k_blocks_per_split;
    if (splits == 1) { p.ws = nullptr; p.ws_counters = nullptr; }
    CUtensorMap tx;
    int rc;
    if ((rc = make_tmap_2d(&tx, x, 0, T, K, ldx, bt))) return rc;
#define DLP_QG_BT(WT_, BT_)                                                                                   \
    case BT_:                                                                                                 \
        return na == 2 ? launch_gemm<BT_, 2, 0, WT_>(tx, tx, tx, p, splits, stream, w0, up)                   \
                       : launch_gemm<BT_, 1, 0, WT_>(tx, tx, tx, p, splits, stream, w0, up);
#define DLP_QG_TYPE(WT_)                                                                                      \
    case WT_:                                                                                                 \
        switch (bt) { DLP_QG_BT(WT_, 16) DLP_QG_BT(WT_, 32) DLP_QG_BT(WT_, 64) DLP_QG_BT(WT_, 128) DLP_QG_BT(WT_, 256) } \
        break;
    switch (wtype) {
        DLP_QG_TYPE(W_Q8_0)
        DLP_QG_TYPE(W_Q4_K)
        DLP_QG_TYPE(W_Q5_K)
        DLP_QG_TYPE(W_Q6_K)
    }
#undef DLP_QG_TYPE
#undef DLP_QG_BT
    DLP_REQUIRE(false, "gemm_quant: unsupported weight type %d", wtype);
}

}  // namespace dlp
