// Prompt portions of grouped-query attention: the tcgen05 flash kernel of attention_tc.cuh on tiles of 128 tokens.
#include "attention_tc.cuh"
#include "layers.cuh"

namespace dlp {

template <int D1, int D2>
static int launch_tiles(const GqaArgs& a, FaParams p, cudaStream_t s) {
    using Cfg = FaCfg<D1, D2, FA_TILES>;
    static_assert(Cfg::SMEM_BYTES <= 227 * 1024, "flash staging");
    CUtensorMap tq, tk, tv;
    int rc;
    const uint64_t rows = (uint64_t)a.n_pages * a.G * a.page_size;
    if ((rc = make_tmap_2d(&tq, a.q, 1, (uint64_t)a.T, (uint64_t)a.H * a.Dc, (uint64_t)a.H * a.Dc, Cfg::BM))) return rc;
    if ((rc = make_tmap_2d(&tk, a.kc, 1, rows * a.maps, a.Dc, a.Dc, (uint32_t)a.page_size))) return rc;
    if ((rc = make_tmap_2d(&tv, a.vc, 1, rows, a.Vc, a.Vc, (uint32_t)a.page_size))) return rc;
    auto kern = attn_prefill_tc_kernel<D1, D2, FA_TILES>;
    if (first_use_on_device((const void*)kern)) DLP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    kern<<<dim3(a.n_tiles, a.H), Cfg::THREADS, Cfg::SMEM_BYTES, s>>>(tq, tk, tv, p);
    DLP_LAUNCH_CHECK();
    return 0;
}

// queries prepared, keys and values cached; a tile is up to 128 consecutive tokens of one request
int gqa_flash(const GqaArgs& a, cudaStream_t s) {
    DLP_REQUIRE(a.q && a.kc && a.vc && a.block_table && a.tok_slot && a.pos && a.out && a.tile_row0 && a.tile_rows && a.n_tiles > 0, "gqa_flash: null argument");
    DLP_REQUIRE(a.H % a.G == 0 && a.Dc <= 128 && a.Vc <= 128 && a.Dc % 16 == 0 && a.Vc % 16 == 0 && a.V <= a.Vc && a.window >= 1 && a.keep >= 0 && a.chunk >= 0 && a.n_pages > 0 &&
                (a.maps == 1 || a.maps == 2) && (a.H / a.G) % a.maps == 0,
                "gqa_flash: heads of %d and %d", a.Dc, a.Vc);
    DLP_REQUIRE(a.page_size % 8 == 0 && a.page_size <= 128 && 128 % a.page_size == 0, "gqa_flash: page size %d (multiple of 8 that divides 128)", a.page_size);
    FaParams p;
    memset(&p, 0, sizeof(p));
    p.out = a.out; p.T = a.T; p.Hq = a.H; p.Hkv = a.G; p.page_size = a.page_size; p.max_pages = a.max_pages; p.ldo = a.ldo; p.V = a.V; p.scale = a.scale;
    p.q_head = a.Dc; p.tile_row0 = a.tile_row0; p.tile_rows = a.tile_rows; p.pos = a.pos; p.tok_slot = a.tok_slot; p.block_table = a.block_table; p.window = a.window; p.keep = a.keep;
    p.chunk = a.chunk; p.maps = a.maps; p.out_f32 = a.maps > 1;
    if (a.Dc <= 64) return a.Vc <= 64 ? launch_tiles<64, 64>(a, p, s) : launch_tiles<64, 128>(a, p, s);
    return a.Vc <= 64 ? launch_tiles<128, 64>(a, p, s) : launch_tiles<128, 128>(a, p, s);
}

}  // namespace dlp
