// Block-quantised weights x few tokens (decode batches, token tiles of routed experts): Y[T, N] (op)= X[T, K] . dequant(W)[N, K]^T, T <= 64 a tile.
//
// Bound by the bytes of W, if only enough of them are in flight and unpacking keeps up.  So the GGUF bytes arrive by TMA in a ring of units
// (256 columns of 128 rows; 128 columns of Q8_0) that is requested ahead - in plain launches before the predecessor has finished -, and the
// unpacking warps (two groups of four, slices in turn; thread r owns row r) turn 64 columns from shared memory into fp16 pairs in registers and store these to TENSOR
// MEMORY, from where tcgen05.mma takes its A operand: no fp16 copy of the weights goes through shared memory, whose bandwidth (written by
// the warps, read by the MMA) would be spent first (4-bit weights: 256 of 330 clocks of a slice).  Unpacking costs some 3 instructions a
// weight: a byte is placed in the mantissa of 256.0f by one PRMT, one FMA applies scale and offset in fp32, one F2FP rounds two values.
// The values are the fp16 ones that gemm_tcgen05_kernel unpacks.  Two blocks an SM where shared memory allows, so that one's start-up
// and epilogue hide behind the other's stream.
// Llama-8B shapes in us, 7 tokens: Q8_0 gate and up 123 -> 34 (floor of the bytes 19), 4096 x 14336 53 -> 16.5 (9.6), 128256 x 4096 109 (86);
// Q4_K gate and up 38 (10), 4096 x 14336 20 (5), 128256 x 4096 120 (45): unpacking bounds the 4- and 6-bit types (some 5 instructions a weight
// with one group of unpacking warps and unpacked FMAs: 150).  Mixtral gate and up of 8 experts in Q4_K, 16 tokens: 1,104 -> 189.
#pragma once
#include "gemm_tcgen05.cuh"

namespace dlp {

int make_tmap_bytes(CUtensorMap* out, const void* base, uint64_t rows, uint64_t row_bytes, uint32_t box_bytes, int swizzle);

__device__ __forceinline__ void tc_mma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st_a(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
          "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]),
          "r"(r[30]), "r"(r[31])
        : "memory");
}

template <int WT> struct QsFmt;      // PARTS: byte planes of a unit, COLS: columns of it, RAW: bytes of its 128 rows
template <> struct QsFmt<W_Q8_0> { static constexpr int PARTS = 1, COLS = 128, RAW = 128 * 128; };
template <> struct QsFmt<W_Q4_K> { static constexpr int PARTS = 1, COLS = 256, RAW = 128 * 144; };
template <> struct QsFmt<W_Q5_K> { static constexpr int PARTS = 1, COLS = 256, RAW = 128 * 176; };
template <> struct QsFmt<W_Q6_K> { static constexpr int PARTS = 3, COLS = 256, RAW = 128 * (128 + 64 + 16); };      // low nibbles | high bits | scales

template <int BT, int NA, int WT>
struct QsCfg {
    static constexpr int COLS = QsFmt<WT>::COLS, SLICES = COLS / 64;
    static constexpr int X_BYTES = SLICES * BT * 128;
    static constexpr int STAGE = NA * QsFmt<WT>::RAW + X_BYTES;          // multiples of 1024 all
    static constexpr int A_STAGES = NA == 2 ? 3 : 4;
    static constexpr int A_COL = NA * BT <= 32 ? 32 : NA * BT;           // tensor memory: accumulators, then A slices of 32 columns
    static constexpr int COLS_USED = A_COL + A_STAGES * NA * 32;
    static constexpr int TMEM_COLS = COLS_USED <= 256 ? 256 : 512;
    static constexpr int PAIR = TMEM_COLS == 256 ? (110 * 1024) / STAGE : 0;
    static constexpr int STAGES_RAW = PAIR >= 2 ? PAIR : (220 * 1024) / STAGE;
    static constexpr int STAGES = STAGES_RAW > 6 ? 6 : STAGES_RAW;
    static constexpr int PER_SM = PAIR >= 2 ? 2 : 1;
    static constexpr int SMEM_BYTES = STAGES * STAGE + 1024 /*align*/ + 256 /*barriers*/;
    static_assert(STAGES >= 2 && STAGE % 1024 == 0 && COLS_USED <= 512, "gemm_quant_small: tile");
};

struct QsMaps { CUtensorMap m[3]; };      // byte planes of one matrix

// 64 weights of this thread's row -> fp16 pairs.  `st` = the unit's bytes, r = row, j = slice of the unit; d: what the thread fetched itself
// (Q8_0: the fp16 scales of the unit's 4 blocks; Q6_K: the fp16 super-block scale)
__device__ __forceinline__ float byte_256(uint32_t bytes, int k) {        // 256 + 2 b_k for bytes of the form 0x80 | b
    return __uint_as_float(__byte_perm(bytes, 0x00000043u, 0x4055 | (k << 8)));
}
__device__ __forceinline__ uint32_t fma2_h2(float a, float b, float2 s, float2 o) {        // two FMAs in one instruction, then one rounding to fp16 each
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\t"
        "mov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
        "fma.rn.f32x2 x, x, y, z;\n\tmov.b64 {%0, %1}, x;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a), "f"(b), "f"(s.x), "f"(s.y), "f"(o.x), "f"(o.y));
    const __half2 h = __floats2half2_rn(r.x, r.y);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ void unpack4(uint32_t bytes, float scale, float off, uint32_t* out, float c = 0.f) {
    const float2 s = make_float2(scale, scale), o = make_float2(off, off);
    float f[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) { f[k] = byte_256(bytes, k); if (c != 0.f) f[k] += c; }
    out[0] = fma2_h2(f[0], f[1], s, o);
    out[1] = fma2_h2(f[2], f[3], s, o);
}
// a + b, and whether that is exact (taking the larger one away again leaves exactly the rest; NaN: no)
__device__ __forceinline__ bool sum_exact(float a, float b, float& s) {
    s = __fadd_rn(a, b);
    return __fsub_rn(s, a) == b && __fsub_rn(s, b) == a;
}
template <int WT>
__device__ __forceinline__ void unpack_slice(const uint8_t* st, int r, int j, uint2 d, uint32_t (&out)[32]) {
    if constexpr (WT == W_Q8_0) {
        const __half2 sub = __float2half2_rn(1152.f);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const uint32_t pair = j == 0 ? d.x : d.y;
            const __half2 s = __half2half2(__ushort_as_half((unsigned short)(b ? pair >> 16 : pair & 0xffffu)));
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const uint4 v = *reinterpret_cast<const uint4*>(st + r * 128 + (((j * 4 + b * 2 + c) ^ (r & 7)) << 4));
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    __half2 lo, hi;
                    bytes4_to_h2(w[i] ^ 0x80808080u, sub, lo, hi);
                    lo = __hmul2(lo, s);                                  // the product of an 8-bit integer and an fp16 scale, rounded once
                    hi = __hmul2(hi, s);
                    out[b * 16 + c * 8 + i * 2] = *reinterpret_cast<const uint32_t*>(&lo);
                    out[b * 16 + c * 8 + i * 2 + 1] = *reinterpret_cast<const uint32_t*>(&hi);
                }
            }
        }
    } else if constexpr (WT == W_Q6_K) {
        const int half = j >> 1, up = j & 1;                             // 128 columns; their low (first 64) or high nibbles
        const uint8_t *ql = st, *qh = st + 128 * 128, *sc = qh + 128 * 64;
        const float dd = __half2float(__ushort_as_half((unsigned short)d.x));
        const uint32_t s4 = *reinterpret_cast<const uint32_t*>(sc + r * 16 + half * 8 + up * 4);      // scales of four groups of 16
        uint32_t h[8];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const uint4 v = *reinterpret_cast<const uint4*>(qh + r * 64 + (((half * 2 + c) ^ ((r >> 1) & 3)) << 4));
            h[c * 4] = v.x; h[c * 4 + 1] = v.y; h[c * 4 + 2] = v.z; h[c * 4 + 3] = v.w;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {                                    // group of 16: nibbles of 16 bytes, two high bits of 16 bytes
            const uint4 v = *reinterpret_cast<const uint4*>(ql + r * 128 + (((half * 4 + c) ^ (r & 7)) << 4));
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            const float s = dd * (float)(int8_t)(s4 >> (8 * c)), off = -160.f * s;      // (exact: 11 + 8 + 3 bits)  256 + 2 (q + 32)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t lo = (w[i] >> (4 * up)) & 0x0F0F0F0Fu, hb = ((h[(c & 1) * 4 + i] >> (4 * up + 2 * (c >> 1))) & 0x03030303u) << 4;
                unpack4(lo | hb | 0x80808080u, 0.5f * s, off, out + c * 8 + i * 2);
            }
        }
    } else {
        constexpr int PITCH = WT == W_Q5_K ? 176 : 144, QS = WT == W_Q5_K ? 48 : 16;
        const uint8_t* row = st + r * PITCH;
        const uint4 hdr = *reinterpret_cast<const uint4*>(row);
        const float2 dm = h2_to_f2(hdr.x);
        // the 6-bit scales and mins of four sub-blocks at a time (the packing of scale_min_k4), then the two of this slice as 256 + 2 v
        const uint32_t sc4 = (j < 2 ? hdr.y & 0x3F3F3F3Fu : (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u)) | 0x80808080u;
        const uint32_t mn4 = (j < 2 ? hdr.z & 0x3F3F3F3Fu : ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u)) | 0x80808080u;
        const uint32_t sc = sc4 >> (16 * (j & 1)), mn = mn4 >> (16 * (j & 1));
        const float s0 = dm.x * fmaf(byte_256(sc, 0), 0.5f, -128.f), s1 = dm.x * fmaf(byte_256(sc, 1), 0.5f, -128.f);
        const float m0 = dm.y * fmaf(byte_256(mn, 0), 0.5f, -128.f), m1 = dm.y * fmaf(byte_256(mn, 1), 0.5f, -128.f);
        // A 4-bit (5-bit) value at the top of the mantissa is 16 (16 + q) (8 (32 + q)): one FMA with scale / 16 and - 16 scale - min gives scale q - min,
        // rounded once, if that offset is exact in fp32 - as it is unless min and scale are more than some 2^3 or 2^6 apart.  Then q by itself.
        constexpr float BIAS = WT == W_Q5_K ? 32.f : 16.f, INV = WT == W_Q5_K ? 0.125f : 0.0625f;
        constexpr int UP = WT == W_Q5_K ? 2 : 3;                  // bits that a value is moved up in its byte
        float o0, o1;
        const bool exact0 = sum_exact(-BIAS * s0, -m0, o0), exact1 = sum_exact(-BIAS * s1, -m1, o1);
        auto all = [&](float c, float p0, float p1) {             // c: what the placed bytes still have to lose
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const uint4 v = *reinterpret_cast<const uint4*>(row + QS + j * 32 + k * 16);
                const uint32_t w[4] = {v.x, v.y, v.z, v.w};
                uint32_t h[4] = {0u, 0u, 0u, 0u};
                if constexpr (WT == W_Q5_K) {
                    const uint4 x = *reinterpret_cast<const uint4*>(row + 16 + k * 16);
                    h[0] = x.x; h[1] = x.y; h[2] = x.z; h[3] = x.w;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    constexpr uint32_t MASK = 0x0F0F0F0Fu << UP;
                    uint32_t lo = ((w[i] << UP) & MASK) | 0x80808080u, hi = ((w[i] >> (4 - UP)) & MASK) | 0x80808080u;
                    if constexpr (WT == W_Q5_K) {
                        lo |= ((h[i] >> (2 * j)) & 0x01010101u) << 6;
                        hi |= ((h[i] >> (2 * j + 1)) & 0x01010101u) << 6;
                    }
                    unpack4(lo, INV * s0, p0, out + k * 8 + i * 2, c);
                    unpack4(hi, INV * s1, p1, out + 16 + k * 8 + i * 2, c);
                }
            }
        };
        if (exact0 && exact1) all(0.f, o0, o1);
        else all(-256.f, -m0, -m1);
    }
}

template <int BT, int NA, int WT>
__global__ void __launch_bounds__(320, (QsCfg<BT, NA, WT>::PER_SM))
gemm_quant_small_kernel(const __grid_constant__ QsMaps tw0, const __grid_constant__ QsMaps tw1, const __grid_constant__ CUtensorMap tm_x,
                        const GemmParams p, const QWeight qw0, const QWeight qw1) {
    using Cfg = QsCfg<BT, NA, WT>;
    using Fmt = QsFmt<WT>;
    constexpr int STAGES = Cfg::STAGES, SLICES = Cfg::SLICES, AS = Cfg::A_STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE);
    uint64_t *raw_full = bars, *raw_empty = bars + STAGES, *a_full = bars + 2 * STAGES, *a_empty = a_full + AS, *done = a_empty + AS;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_out0 = blockIdx.x * GEMM_BM;
    int n0 = n_out0, t0 = blockIdx.y * BT, t_end = p.T;
    const bool grouped = p.grp.tile_expert != nullptr;
    if (grouped) {
        pdl_wait();                                             // the table is a predecessor's
        if ((int)blockIdx.y >= *p.grp.n_tiles) return;          // (uniform over the block, before any barrier / TMEM allocation)
        n0 += p.grp.tile_expert[blockIdx.y] * p.grp.rows_per_expert;
        t0 = p.grp.tile_row0[blockIdx.y];
        t_end = t0 + p.grp.tile_rows[blockIdx.y];
    }
    const int total = p.K / 64, u_begin = blockIdx.z * p.k_blocks_per_split / SLICES;
    const int units = (min(total, (int)(blockIdx.z + 1) * p.k_blocks_per_split)) / SLICES - u_begin;      // (host: whole units, at least one)

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tm_x);
        for (int i = 0; i < Fmt::PARTS; ++i) { tma_prefetch_desc(&tw0.m[i]); if (NA == 2) tma_prefetch_desc(&tw1.m[i]); }
        for (int s = 0; s < STAGES; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], 9); }      // 8 unpacking warps, the MMAs that read X
        for (int s = 0; s < AS; ++s) { mbar_init(&a_full[s], 4); mbar_init(&a_empty[s], 1); }
        mbar_init(done, 1);
        mbar_fence_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, Cfg::TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (elect_one()) {      // (elect.sync: with lane == 0 the compiler issues TMA and MMAs through a loop over the lanes, 100 clocks each)
            auto load_w = [&](int u, int s) {
                uint8_t* st = smem + s * Cfg::STAGE;
                const int uu = u_begin + u;
#pragma unroll
                for (int a = 0; a < NA; ++a, st += Fmt::RAW) {
                    const CUtensorMap* m = a ? tw1.m : tw0.m;
                    if (WT == W_Q6_K) {
                        tma_load_2d(st, &m[0], &raw_full[s], uu * 128, n0);
                        tma_load_2d(st + 128 * 128, &m[1], &raw_full[s], uu * 64, n0);
                        tma_load_2d(st + 128 * 192, &m[2], &raw_full[s], uu * 16, n0);
                    } else {
                        tma_load_2d(st, &m[0], &raw_full[s], uu * (Fmt::RAW / 128), n0);
                    }
                }
            };
            auto load_x = [&](int u, int s) {
                uint8_t* st = smem + s * Cfg::STAGE + NA * Fmt::RAW;
#pragma unroll
                for (int j = 0; j < SLICES; ++j) tma_load_2d(st + j * BT * 128, &tm_x, &raw_full[s], (u_begin + u) * Cfg::COLS + j * 64, t0);
            };
            const int first = min(STAGES, units);
            for (int u = 0; u < first; ++u) {                   // weights are static: requested before the predecessor has finished
                mbar_expect_tx(&raw_full[u], Cfg::STAGE);
                load_w(u, u);
            }
            if (!grouped) pdl_wait();
            for (int u = 0; u < first; ++u) load_x(u, u);
            int s = 0;
            uint32_t ph = 0;
            for (int u = first; u < units; ++u) {
                mbar_wait_b(&raw_empty[s], ph);
                mbar_expect_tx(&raw_full[s], Cfg::STAGE);
                load_w(u, s);
                load_x(u, s);
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        if (elect_one()) {
            constexpr uint32_t idesc = make_idesc_f16(GEMM_BM, BT, 0);
            int s = 0, as = 0;
            uint32_t ph = 0, aph = 0;
            if (!grouped) pdl_wait();                               // (X comes after that; the limit of the waits counts from there)
            for (int u = 0; u < units; ++u) {
                mbar_wait_b(&raw_full[s], ph);
                const uint32_t xs = smem_u32(smem + s * Cfg::STAGE + NA * Fmt::RAW);
                for (int j = 0; j < SLICES; ++j) {
                    mbar_wait_b(&a_full[as], aph);
                    tc_fence_after();
                    const uint64_t db = make_smem_desc_sw128(xs + j * BT * 128);
                    const uint32_t ta = tmem_base + Cfg::A_COL + as * (NA * 32);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t acc = (u > 0 || j > 0 || k > 0) ? 1u : 0u;
                        tc_mma_f16_ts(tmem_base, ta + k * 8, db + (uint64_t)(2 * k), idesc, acc);
                        if (NA == 2) tc_mma_f16_ts(tmem_base + BT, ta + 32 + k * 8, db + (uint64_t)(2 * k), idesc, acc);
                    }
                    tc_commit(&a_empty[as]);
                    if (++as == AS) { as = 0; aph ^= 1; }
                }
                tc_commit(&raw_empty[s]);
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
            tc_commit(done);
        }
    } else {
        const int q = warp & 3, r = q * 32 + lane;
        const size_t row = min(n0 + r, qw0.N - 1);              // (rows behind the last: zeros from the maps)
        auto scales = [&](const QWeight& w, int u) {
            uint2 d = make_uint2(0u, 0u);
            u = u_begin + min(u, units - 1);
            if constexpr (WT == W_Q8_0) d = __ldg(reinterpret_cast<const uint2*>(w.aux0 + (row * (w.K >> 5) + (size_t)u * 4) * 2));
            if constexpr (WT == W_Q6_K) d.x = __ldg(reinterpret_cast<const unsigned short*>(w.aux2) + row * (w.K >> 8) + u);
            return d;
        };
        uint2 d0 = scales(qw0, 0), d1 = make_uint2(0u, 0u);
        if (NA == 2) d1 = scales(qw1, 0);
        const int group = (warp - 2) >> 2;                      // every other slice
        int s = 0, as = group;
        uint32_t ph = 0, aph = 0;
        if (!grouped) pdl_wait();                                   // (as above; the epilogue reads and writes what a predecessor may still use)
        for (int u = 0; u < units; ++u) {
            const uint2 e0 = scales(qw0, u + 1), e1 = NA == 2 ? scales(qw1, u + 1) : d1;      // (a unit ahead)
            mbar_wait_b(&raw_full[s], ph);
            const uint8_t* st = smem + s * Cfg::STAGE;
#pragma unroll 1
            for (int j = group; j < SLICES; j += 2) {
                uint32_t w0[32], w1[32];
                unpack_slice<WT>(st, r, j, d0, w0);
                if (NA == 2) unpack_slice<WT>(st + Fmt::RAW, r, j, d1, w1);
                mbar_wait_b(&a_empty[as], aph ^ 1);
                tc_fence_after();
                const uint32_t ta = tmem_base + ((uint32_t)(q * 32) << 16) + Cfg::A_COL + as * (NA * 32);
                tmem_st_a(ta, w0);
                if (NA == 2) tmem_st_a(ta + 32, w1);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[as]);
                as += 2;
                if (as >= AS) { as -= AS; aph ^= 1; }
            }
            if (lane == 0) mbar_arrive(&raw_empty[s]);
            if (++s == STAGES) { s = 0; ph ^= 1; }
            d0 = e0;
            d1 = e1;
        }
        pdl_launch_dependents();
        if (group == 0) {
            mbar_wait_b(done, 0);
            gemm_drain<BT, NA, 0>(p, tmem_base, done, true, n_out0, t0, t_end);
        }
    }
    gemm_wait_aftermath();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        __syncwarp();
        tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
    }
}

// Byte planes of 128-row units
template <int WT>
static int quant_maps(const QWeight& w, uint64_t rows, QsMaps& m) {
    const uint64_t K = w.K;
    int rc = 0;
    if (WT == W_Q8_0) rc = make_tmap_bytes(&m.m[0], w.base, rows, K, 128, 128);
    else if (WT == W_Q6_K) {
        if ((rc = make_tmap_bytes(&m.m[0], w.base, rows, K / 2, 128, 128))) return rc;
        if ((rc = make_tmap_bytes(&m.m[1], w.aux0, rows, K / 4, 64, 64))) return rc;
        rc = make_tmap_bytes(&m.m[2], w.aux1, rows, K / 16, 16, 0);
    } else rc = make_tmap_bytes(&m.m[0], w.base, rows, K / 256 * (QsFmt<WT>::RAW / 128), QsFmt<WT>::RAW / 128, 0);
    return rc;
}

// Splits of K: enough blocks for every slot of the machine, each with at least two units to stream
static int quant_small_splits(long tiles, int units, int slots) {
    long s = tiles > 0 ? slots / tiles : 1;
    if (s > 16) s = 16;
    while (s > 1 && units / s < 2) --s;
    return s < 1 ? 1 : (int)s;
}

template <int BT, int NA, int WT>
static int launch_quant_small(const QWeight& w0, const QWeight& w1, const CUtensorMap& tx, GemmParams p, int split_k, void* ws, size_t ws_bytes,
                              cudaStream_t stream) {
    using Cfg = QsCfg<BT, NA, WT>;
    QsMaps m0, m1;
    int rc;
    if ((rc = quant_maps<WT>(w0, w0.N, m0))) return rc;
    m1 = m0;
    if (NA == 2 && (rc = quant_maps<WT>(w1, w1.N, m1))) return rc;
    const int units = p.K / Cfg::COLS;
    const long tiles_n = (p.N + GEMM_BM - 1) / GEMM_BM, tiles_t = p.grp.tile_expert ? p.grp.max_tiles : (p.T + BT - 1) / BT, tiles = tiles_n * tiles_t;
    int splits = split_k > 0 ? split_k : 1;
    bool by_ws = false;
    p.ws = nullptr;
    p.ws_counters = nullptr;
    if (split_k <= 0 && p.epilogue == EPI_ATOMIC_ADD_F32 && gemm_add_may_split(p.T, p.N, p.K / GEMM_BK)) splits = quant_small_splits(tiles, units, sm_count() * Cfg::PER_SM);
    else if (split_k <= 0 && ws != nullptr && tiles <= (long)GEMM_WS_COUNTERS && p.epilogue != EPI_RS_PUSH_F32) {
        // (grouped: the table decides how many tiles there are; most routings of few tokens fill about half of the bound)
        splits = quant_small_splits(p.grp.tile_expert ? (tiles + 1) / 2 : tiles, units, sm_count() * Cfg::PER_SM);
        if (splits > 8) splits = 8;
        const size_t per = (size_t)NA * BT * GEMM_BM * sizeof(float);
        while (splits > 1 && GEMM_WS_COUNTERS * 4 + (size_t)tiles * splits * per > ws_bytes) --splits;
        by_ws = true;
    }
    if (splits > units) splits = units;
    const int per_split = (units + splits - 1) / splits;
    splits = (units + per_split - 1) / per_split;
    p.k_blocks_per_split = per_split * Cfg::SLICES;
    if (splits > 1 && by_ws) {
        p.ws_counters = reinterpret_cast<unsigned*>(ws);
        p.ws = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(ws) + GEMM_WS_COUNTERS * 4);
    }
    auto kern = gemm_quant_small_kernel<BT, NA, WT>;
    if (first_use_on_device((const void*)kern))
        DLP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES));
    DLP_CHECK_CUDA(launch_pdl(kern, dim3(tiles_n, tiles_t, splits), dim3(320), Cfg::SMEM_BYTES, stream, m0, m1, tx, p, w0, w1));
    return 0;
}

}  // namespace dlp
