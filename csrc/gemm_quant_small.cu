// Block-quantised weights x up to 64 tokens a tile (kernel: gemm_quant_small.cuh).
#include "gemm_quant_small.cuh"

namespace dlp {

// Whether the TMA maps of this kernel can describe the weight (16-byte planes; its row strides are multiples of 16 for K % 256 == 0)
bool gemm_quant_small_takes(const QWeight& w, int wtype) {
    auto ok = [](const void* p, int a) { return (reinterpret_cast<uintptr_t>(p) & (a - 1)) == 0; };
    return ok(w.base, 16) && (wtype != W_Q8_0 || ok(w.aux0, 8)) && (wtype != W_Q6_K || (ok(w.aux0, 16) && ok(w.aux1, 16)));
}

int gemm_quant_small(const QWeight& w0, const QWeight& w1, int na, int wtype, int bt, const CUtensorMap& tx, const GemmParams& p, int split_k, void* ws,
                     size_t ws_bytes, cudaStream_t stream) {
#define DLP_QS_BT(WT_, BT_)                                                                                          \
    case BT_:                                                                                                        \
        return na == 2 ? launch_quant_small<BT_, 2, WT_>(w0, w1, tx, p, split_k, ws, ws_bytes, stream)               \
                       : launch_quant_small<BT_, 1, WT_>(w0, w1, tx, p, split_k, ws, ws_bytes, stream);
#define DLP_QS_TYPE(WT_)                                                                                             \
    case WT_:                                                                                                        \
        switch (bt) { DLP_QS_BT(WT_, 16) DLP_QS_BT(WT_, 32) DLP_QS_BT(WT_, 64) }                                     \
        break;
    switch (wtype) {
        DLP_QS_TYPE(W_Q8_0)
        DLP_QS_TYPE(W_Q4_K)
        DLP_QS_TYPE(W_Q5_K)
        DLP_QS_TYPE(W_Q6_K)
    }
#undef DLP_QS_TYPE
#undef DLP_QS_BT
    DLP_REQUIRE(false, "gemm_quant: unsupported weight type %d or token tile %d", wtype, bt);
}

}  // namespace dlp
