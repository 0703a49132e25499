// Paged-KV attention for decode / small query counts: split-KV flash-decoding + LSE combine.
//
// Reference counterparts: `flash_attn_ext_vec` (llama.cpp/ggml/src/ggml-cuda/fattn-vec.cuh) with
// `parallel_blocks` split-KV and `flash_attn_combine_results` (fattn-common.cuh:721-772).  The reference
// cache is a contiguous ring per stream; here K/V live in fixed-size pages
// [n_pages][Hkv][page_size][D] addressed through a block table, so sequences grow without copies and
// TP ranks own disjoint KV heads.  One CTA = (split, kv head [x q-head group], query); the query heads that
// share a KV head are processed together so each K/V byte is read once per group.
#include "kernels.cuh"
#include <cooperative_groups.h>

namespace dlp {

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool pred) {
    const uint32_t s = smem_u32(smem);
    const int sz = pred ? 16 : 0;  // src-size 0 => zero fill
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(gmem), "r"(sz) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* smem) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(smem)));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* smem) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(smem)));
}
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t movmatrix(uint32_t a) {      // 8 x 8 halves, two of a row per lane, transposed
    uint32_t d;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}
// two fp32 values as fp16 pairs: value and remainder (23 bits together), or with `rest` what is left of those as well (all 24)
__device__ __forceinline__ void split_h2(float a, float b, uint32_t& hi, uint32_t& lo, uint32_t* rest = nullptr) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    lo = *reinterpret_cast<const uint32_t*>(&l);
    if (rest != nullptr) {
        const float2 g = __half22float2(l);
        *rest = pack_h2((a - f.x) - g.x, (b - f.y) - g.y);
    }
}

// ---- split-KV attention on the tensor cores ------------------------------------------------------------------------------
// Bound by the bytes of K and V: one CTA = (split of the keys, KV head, query); the query heads that share the KV head are the 8 columns of
// mma.sync m16n8k16 (a query has too few heads for a tcgen05 tile), 16 keys (then 16 dims of V, transposed by ldmatrix) its rows, so every
// K / V byte is read once.  (Heads as the 16 rows: half of the tile is padding, twice the MMAs.)  Each of the 4 warps streams its own tiles of 16 keys through a private ring of
// 3 stages (cp.async, 8 KB a stage at D = 128; 2 CTAs an SM: 128 KB in flight) and keeps its own running maximum; page ids are fetched one
// tile ahead; the warps are merged through shared memory, the splits by the last CTA of the (query, head) to finish.
// Scores and sums are fp32.  The softmax weights (and with ROPE the rotated fp32 queries) enter the tensor cores as two (three) fp16 parts, value
// and remainder, 23 (24) bits together, scaled by powers of two so that no part overflows or goes subnormal where it counts: weights in units of
// 2^-15, a head's queries by its largest one.  What an MMA adds is cut off, not rounded, at the size of its largest term, so no MMA adds to a
// sum that is kept: each takes 16 products from zero, parts apart, and the sums over them are rounded fp32 additions.  Error against 64 bits
// before the output's rounding, 32 heads over 8, D = 128, keys of deviation 1.5: 700 keys 2.4e-7 (fp32 FMA per key 2.4e-7, sums kept in the MMAs
// 4.1e-7), 32,000 3.1e-7 (3.4e-7, 8.3e-7).
// 32,000 keys of 8 KV heads of 4 query heads, D = 128 (131 MB): 28.7 us (4.6 TB/s; 108 us with fp32 FMA per key in 128 CTAs); 32 queries
// of 2,000 keys each (262 MB): 42 us (172 us).
//   ROPE: takes the fp32 row of the QKV mat-vec, rotates q in registers, writes the new token's K and V and uses them from shared memory.
constexpr int ATTN_KEYS_MIN = 128;      // keys a split is worth: 2 tiles per warp, all requested before the dependency wait (700 keys in a
                                        // decode step: as fast as the cluster form; with 256 keys 1.7 us slower)
constexpr int ATTN_KEYS_WHOLE = 320;    // no split up to here: joining costs some 3 us, 64 keys 0.7 (300 keys, 32 heads over 8: 6.5 us whole, 7.2 in three)
constexpr int ATTN_JOIN_MAX = 40;       // ranges of a query that are worth joining (300 + 8,000 keys, 32 heads over 4, D = 64: 11.9 us with the long one in 22, 12.5 in
                                        // 30, 14.1 in 46, 16.2 in 63; 300 + 32,000: 19.6 in 31, 20.1 in 47, 21.8 in 73)
constexpr int ATTN_POOL_NQ = 256;       // (more queries: prompts token by token, not worth a look at every length)
// Splits of the keys.  One query takes up to n_splits.  Several share a pool (attn_pool): all are cut into ranges of the same length, the
// shortest that the pool has room for, so that a long sequence among short ones is spread over the machine as it would be alone (32,000 keys
// beside 31 x 300, 32 heads over 8, D = 128: 44 us; 154 with 16 ranges for every query, 218 with 2).  Places in the pool are those of the ranges' partial results.
struct AttnRange { int qi, first, eff, begin, end, len; };      // query (-1: no such range), place of its first range, ranges; keys of this one; keys of the query
__device__ __forceinline__ int attn_per(int len, int n) {         // keys of a range when `len` keys are cut into n: whole tiles
    return max(16, ((len + n - 1) / n + 15) & ~15);
}
__device__ __forceinline__ int attn_pieces(int len, int per) { return len <= max(per, ATTN_KEYS_WHOLE) ? 1 : (len + per - 1) / per; }
// The range at `place`, or (place < 0) the first one of query `qi`.  All lanes of a warp call it and get the same.
__device__ __forceinline__ AttnRange attn_range(const AttnParams& p, int place, int qi, int lane) {
    AttnRange r;
    int per = 0;
    if (p.pool == 0) {
        r.qi = place < 0 ? qi : place / p.n_splits;
        r.first = r.qi * p.n_splits;
        r.len = p.kv_len[r.qi];
        per = attn_per(r.len, min(min(p.n_splits, ATTN_JOIN_MAX), max(1, (r.len + ATTN_KEYS_MIN - 1) / ATTN_KEYS_MIN)));
        r.eff = attn_pieces(r.len, per);
        if (place >= 0 && place - r.first >= r.eff) r.qi = -1;
    } else {
        const int mine = lane < p.nq ? p.kv_len[lane] : 0;
        auto len_of = [&](int b) { return b == 0 ? mine : b + lane < p.nq ? p.kv_len[b + lane] : 0; };
        int total = 0, most = 0;
        for (int b = 0; b < p.nq; b += 32) {
            total += __reduce_add_sync(0xffffffffu, len_of(b));
            most = max(most, __reduce_max_sync(0xffffffffu, len_of(b)));
        }
        // no query is cut that is about as long as what every slot of the machine has to do anyway
        const int share = max(ATTN_KEYS_MIN, attn_per(total + total / 5, p.wave));
        if (most <= max(share, ATTN_KEYS_WHOLE)) {                // every query is a range of its own
            r.qi = r.first = place < 0 ? qi : place < p.nq ? place : -1;
            if (r.qi < 0) return r;
            r.eff = 1;
            r.len = p.nq <= 32 ? __shfl_sync(0xffffffffu, mine, r.qi) : p.kv_len[r.qi];
        } else {
            per = max(share, max(attn_per(total, p.pool - p.nq / 2), attn_per(most, ATTN_JOIN_MAX)));
            const int enough = attn_per(total, p.pool - p.nq);      // (last ranges are short: at most nq places more than total / per)
            while (per < enough) {
                int used = 0;
                for (int b = 0; b < p.nq; b += 32) used += __reduce_add_sync(0xffffffffu, b + lane < p.nq ? attn_pieces(len_of(b), per) : 0);
                if (used <= p.pool) break;
                per = min(enough, (per + (per >> 3) + 15) & ~15);
            }
            r.qi = -1;
            for (int b = 0, at = 0; b < p.nq; b += 32) {
                const int len = len_of(b), n = b + lane < p.nq ? attn_pieces(len, per) : 0;
                int upto = n;                                     // ranges of the queries up to this lane's
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int x = __shfl_up_sync(0xffffffffu, upto, o);
                    if (lane >= o) upto += x;
                }
                const unsigned hit = __ballot_sync(0xffffffffu, place < 0 ? b + lane == qi : place >= at + upto - n && place < at + upto);
                if (hit) {
                    const int src = __ffs(hit) - 1;
                    r.qi = b + src;
                    r.eff = __shfl_sync(0xffffffffu, n, src);
                    r.first = at + __shfl_sync(0xffffffffu, upto, src) - r.eff;
                    r.len = __shfl_sync(0xffffffffu, len, src);
                    break;
                }
                at += __shfl_sync(0xffffffffu, upto, 31);
            }
            if (r.qi < 0) return r;
        }
    }
    r.begin = r.eff == 1 || place < 0 ? 0 : (place - r.first) * per;
    r.end = r.eff == 1 ? r.len : min(r.len, r.begin + per);
    return r;
}
struct AttnRope {
    const float* qkv;          // [nq][(Hq + 2 Hkv) * D], not rotated
    const float* inv_freq;     // [D / 2], or
    const float2* cs;          // [nq][D / 2] (cos, sin)
    __half* kc_w;
    __half* vc_w;
    int neox;
    float q_scale;
};

// One warp joins the partials of `eff` splits of one (query, head): a lane takes D / 32 dims, its loads of 8 splits in flight at a time.
// (One thread per dim, splits one after the other: 45 us instead of 28.5 for 32,000 keys in 37 splits.)
template <int D>
__device__ __forceinline__ void attn_join(const AttnParams& p, int qi, int hq, int first, int eff, int lane) {
    constexpr int E = D / 32;
    constexpr float LOG2E = 1.4426950408889634f;
    const size_t pi0 = (size_t)hq * p.nq * p.n_splits + first, head = (size_t)qi * p.Hq + hq;
    const float* ml = p.part_ml + pi0 * 2;
    float mn = -INFINITY, ls = 0.f, acc[E];
#pragma unroll
    for (int i = 0; i < E; ++i) acc[i] = 0.f;
    for (int s = lane; s < eff; s += 32) mn = fmaxf(mn, __ldcg(ml + 2 * s));
    mn = warp_max(mn);
    for (int s0 = 0; s0 < eff; s0 += 32) {
        const float2 v = s0 + lane < eff ? make_float2(__ldcg(ml + 2 * (s0 + lane)), __ldcg(ml + 2 * (s0 + lane) + 1)) : make_float2(-INFINITY, 0.f);
        const float a = v.x == -INFINITY ? 0.f : exp2f((v.x - mn) * LOG2E);
        ls += v.y * a;
        const int n = min(32, eff - s0);
        for (int s = 0; s < n; s += 8) {
            float x[8][E];
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float* src = p.part_o + (pi0 + s0 + min(s + u, n - 1)) * D + lane;
#pragma unroll
                for (int i = 0; i < E; ++i) x[u][i] = __ldcg(src + 32 * i);
            }
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                const float w = __shfl_sync(0xffffffffu, a, min(s + u, 31));
#pragma unroll
                for (int i = 0; i < E; ++i) if (s + u < n) acc[i] = fmaf(x[u][i], w, acc[i]);
            }
        }
    }
    ls = warp_sum(ls);
    const float inv = ls > 0.f ? 1.f / ls : 0.f;
#pragma unroll
    for (int i = 0; i < E; ++i) p.out[head * D + lane + 32 * i] = __float2half_rn(acc[i] * inv);
}

template <int D> constexpr int attn_split_smem() { return 4 * 3 * 2 * 16 * D * 2; }      // warps x stages x (K, V) x keys x D (the merge needs 4 x 16 x (D + 2) floats of it)

template <int D, int NH, bool ROPE>      // NH: groups of 8 query heads in use
__global__ void __launch_bounds__(128, 2) attn_split_kernel(const AttnParams p, const AttnRope ra) {
    constexpr int STAGES = 3, KS = D / 16, CPR = D / 8, TILE = 16 * D * 2;      // k steps, 16-byte chunks per row, bytes of one K or V tile
    constexpr float LOG2E = 1.4426950408889634f, UP = 32768.f;
    extern __shared__ __align__(128) uint8_t as_smem[];
    const int gqa = p.Hq / p.Hkv, R = 8 * NH, groups = (gqa + R - 1) / R;
    const int kvh = blockIdx.y / groups, h0 = (blockIdx.y % groups) * R, G = min(R, gqa - h0), hq0 = kvh * gqa + h0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    trace_event(p.trace, TR_ATTN | TR_BEGIN);
    // ROPE: length, pages and the cached rows were written at least two launches back (the immediate predecessor is the QKV mat-vec), so
    // the first tiles are requested before the dependency wait.  Otherwise the predecessor wrote the newest K / V row.
    if (!ROPE) pdl_wait();
    const int place = blockIdx.z * gridDim.x + blockIdx.x;
    const AttnRange rg = attn_range(p, place, 0, lane);
    if (rg.qi < 0) return;
    const int qi = rg.qi, n_old = rg.len - 1;
    const int n_tiles = (rg.end - rg.begin + 15) >> 4, n_mine = n_tiles > warp ? (n_tiles - warp + 3) >> 2 : 0;
    const int* bt = p.block_table + (size_t)(p.bt_row ? p.bt_row[qi] : qi) * p.max_pages;
    uint8_t* ring = as_smem + warp * (STAGES * 2 * TILE);
    auto rows_of = [&](int j) {              // lane r < 16: element offset of row r of this warp's tile j (-1: not a cached key)
        const int tok = rg.begin + ((j * 4 + warp) << 4) + (lane & 15);
        if (j >= n_mine || tok >= (ROPE ? min(rg.end, n_old) : rg.end)) return (long long)-1;
        const int pg = tok / p.page_size;
        return (((long long)bt[pg] * p.Hkv + kvh) * p.page_size + (tok - pg * p.page_size)) * D;
    };
    auto issue = [&](int j, long long where) {
        if (j < n_mine) {
            uint8_t* st = ring + (j % STAGES) * (2 * TILE);
#pragma unroll
            for (int i = 0; i < CPR / 2; ++i) {
                const int e = i * 32 + lane, r = e / CPR, c = e % CPR;
                const long long o = __shfl_sync(0xffffffffu, where, r);
                const int at = r * (D * 2) + ((c ^ (r & 7)) << 4);
                cp_async16(st + at, p.kc + (o < 0 ? 0 : o + c * 8), o >= 0);
                cp_async16(st + TILE + at, p.vc + (o < 0 ? 0 : o + c * 8), o >= 0);
            }
        }
        cp_async_commit();
    };
    issue(0, rows_of(0));
    issue(1, rows_of(1));
    long long where = rows_of(2);
    if (ROPE) {
        pdl_wait();
        if (p.pdl_early) pdl_launch_dependents();
    }
    trace_event(p.trace, TR_ATTN | TR_WAITED);

    // queries as B fragments: head g, dims ks * 16 + 2t, + 1 and + 8, + 9
    uint32_t qh[KS][NH][2], ql[ROPE ? KS : 1][NH][2], qr[ROPE ? KS : 1][NH][2];
    float unscale[NH][2];                    // ROPE: what brings the scores of heads 2t and 2t + 1 back to the queries' own size (a power of two)
    const float2* cs_tab = ROPE && ra.cs ? ra.cs + (size_t)qi * (D / 2) : nullptr;
    auto angle = [&](int i) {               // (cos, sin) of pair i
        if (cs_tab) return cs_tab[i];
        float2 v;
        sincosf((float)n_old * ra.inv_freq[i], &v.y, &v.x);
        return v;
    };
    const float* row = ROPE ? ra.qkv + (size_t)qi * (p.Hq + 2 * p.Hkv) * D : nullptr;
#pragma unroll
    for (int nh = 0; nh < NH; ++nh) {
        const int r = nh * 8 + g;
        if constexpr (ROPE) {
            const float* src = row + (size_t)(hq0 + min(r, G - 1)) * D;
            float2 x[KS][2];
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                for (int e = 0; e < 2; ++e) x[ks][e] = *reinterpret_cast<const float2*>(src + ks * 16 + e * 8 + 2 * t);
            if (ra.neox) {
#pragma unroll
                for (int ks = 0; ks < KS / 2; ++ks)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float2 a = angle(ks * 16 + e * 8 + 2 * t), b = angle(ks * 16 + e * 8 + 2 * t + 1), u = x[ks][e], v = x[ks + KS / 2][e];
                        x[ks][e] = make_float2(u.x * a.x - v.x * a.y, u.y * b.x - v.y * b.y);
                        x[ks + KS / 2][e] = make_float2(v.x * a.x + u.x * a.y, v.y * b.x + u.y * b.y);
                    }
            } else {
#pragma unroll
                for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float2 a = angle(ks * 8 + e * 4 + t), u = x[ks][e];
                        x[ks][e] = make_float2(u.x * a.x - u.y * a.y, u.x * a.y + u.y * a.x);
                    }
            }
            float top = 0.f;
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const float sc = r < G ? ra.q_scale : 0.f;
                    x[ks][e] = make_float2(x[ks][e].x * sc, x[ks][e].y * sc);
                    top = fmaxf(top, fmaxf(fabsf(x[ks][e].x), fabsf(x[ks][e].y)));
                }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            const int up = top > 0.f ? max(-100, min(100, 141 - (int)(__float_as_uint(top) >> 23))) : 0;      // the head's largest |q|: 2^14 .. 2^15
            const float f = __uint_as_float((uint32_t)(127 + up) << 23), back = __uint_as_float((uint32_t)(127 - up) << 23);
#pragma unroll
            for (int h = 0; h < 2; ++h) unscale[nh][h] = __shfl_sync(0xffffffffu, back, (2 * t + h) * 4);
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                for (int e = 0; e < 2; ++e) split_h2(x[ks][e].x * f, x[ks][e].y * f, qh[ks][nh][e], ql[ks][nh][e], &qr[ks][nh][e]);
        } else {
            const __half* src = p.q + ((size_t)qi * p.Hq + hq0 + min(r, G - 1)) * D;
#pragma unroll
            for (int ks = 0; ks < KS; ++ks)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const uint32_t v = *reinterpret_cast<const uint32_t*>(src + ks * 16 + e * 8 + 2 * t);
                    qh[ks][nh][e] = r < G ? v : 0u;
                }
        }
    }
    float o[D / 16][NH][4];                  // dims g and g + 8 of a group of 16, heads 2t and 2t + 1
#pragma unroll
    for (int i = 0; i < D / 16; ++i)
#pragma unroll
        for (int nh = 0; nh < NH; ++nh) { o[i][nh][0] = o[i][nh][1] = o[i][nh][2] = o[i][nh][3] = 0.f; }
    float m[NH][2], l[NH][2];
#pragma unroll
    for (int nh = 0; nh < NH; ++nh) { m[nh][0] = m[nh][1] = -INFINITY; l[nh][0] = l[nh][1] = 0.f; }
    const int mat = lane >> 3, r8 = lane & 7;
    for (int j = 0; j < n_mine; ++j) {
        const long long next = rows_of(j + 3);
        issue(j + 2, where);                 // (its stage was read in iteration j - 1)
        where = next;
        cp_async_wait_group<2>();
        __syncwarp();
        uint8_t* sK = ring + (j % STAGES) * (2 * TILE);
        uint8_t* sV = sK + TILE;
        const int tok0 = rg.begin + ((j * 4 + warp) << 4);
        if (ROPE && n_old >= tok0 && n_old < min(tok0 + 16, rg.end)) {      // the new token: rotate K, round K and V to the cache's type, into the tile and into the page
            constexpr int E = D / 32;
            const float* ks_ = row + (size_t)(p.Hq + kvh) * D + lane * E;
            const float* vs_ = ks_ + (size_t)p.Hkv * D;
            float kx[E], vx[E];
#pragma unroll
            for (int i = 0; i < E; ++i) { kx[i] = ks_[i]; vx[i] = vs_[i]; }
            if (ra.neox) {
#pragma unroll
                for (int i = 0; i < E; ++i) {
                    const float other = __shfl_xor_sync(0xffffffffu, kx[i], 16);
                    const float2 a = angle((lane & 15) * E + i);
                    kx[i] = lane < 16 ? kx[i] * a.x - other * a.y : kx[i] * a.x + other * a.y;
                }
            } else {
#pragma unroll
                for (int i = 0; i < E; i += 2) {
                    const float2 a = angle((lane * E + i) >> 1);
                    const float u = kx[i], v = kx[i + 1];
                    kx[i] = u * a.x - v * a.y;
                    kx[i + 1] = u * a.y + v * a.x;
                }
            }
            const int r = n_old - tok0, pg = n_old / p.page_size;
            const int at = r * (D * 2) + ((((lane * E) >> 3) ^ (r & 7)) << 4) + ((lane * E) & 7) * 2;
            const size_t gl = (((size_t)bt[pg] * p.Hkv + kvh) * p.page_size + (n_old - pg * p.page_size)) * D + lane * E;
#pragma unroll
            for (int i = 0; i < E; i += 2) {
                const uint32_t kk = pack_h2(kx[i], kx[i + 1]), vv = pack_h2(vx[i], vx[i + 1]);
                *reinterpret_cast<uint32_t*>(sK + at + i * 2) = kk;
                *reinterpret_cast<uint32_t*>(sV + at + i * 2) = vv;
                if (h0 == 0) {
                    *reinterpret_cast<uint32_t*>(ra.kc_w + gl + i) = kk;
                    *reinterpret_cast<uint32_t*>(ra.vc_w + gl + i) = vv;
                }
            }
            __syncwarp();
        }
        // scores: keys g (0, 1) and g + 8 (2, 3), heads 2t (even) and 2t + 1; `low`: of the queries' remainders, 2^-12 of the others (what is cut off
        // there does not count), in independent chains, since an MMA waits for the one before it in its chain
        constexpr int CHAINS = NH == 1 ? 2 : 1;
        float part[NH][KS / 2][4], low[NH][2 * CHAINS][4];
#pragma unroll
        for (int nh = 0; nh < NH; ++nh)
#pragma unroll
            for (int c = 0; c < 2 * CHAINS; ++c) { low[nh][c][0] = low[nh][c][1] = low[nh][c][2] = low[nh][c][3] = 0.f; }
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            uint32_t ka[4];
            const int kr = (mat & 1) * 8 + r8, c = ks * 2 + (mat >> 1);
            ldmatrix_x4(ka, sK + kr * (D * 2) + ((c ^ (kr & 7)) << 4));
#pragma unroll
            for (int nh = 0; nh < NH; ++nh) {
                float x[4] = {0.f, 0.f, 0.f, 0.f};
                mma_16816(x, ka, qh[ks][nh][0], qh[ks][nh][1]);
                if constexpr (ROPE) {
                    mma_16816(low[nh][ks % CHAINS * 2], ka, ql[ks][nh][0], ql[ks][nh][1]);
                    mma_16816(low[nh][ks % CHAINS * 2 + 1], ka, qr[ks][nh][0], qr[ks][nh][1]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) part[nh][ks / 2][e] = ks & 1 ? part[nh][ks / 2][e] + x[e] : x[e];
            }
        }
#pragma unroll
        for (int n = KS / 4; n >= 1; n /= 2)
#pragma unroll
            for (int nh = 0; nh < NH; ++nh)
#pragma unroll
                for (int i = 0; i < n; ++i)
#pragma unroll
                    for (int e = 0; e < 4; ++e) part[nh][i][e] += part[nh][i + n][e];
        uint32_t ph[NH][2], pl[NH][2];       // weights as B fragments: head g, keys 2t, 2t + 1 and + 8, + 9
        float alpha[NH][2];
#pragma unroll
        for (int nh = 0; nh < NH; ++nh) {
            float v[4], pr[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float x = part[nh][0][e];
                if constexpr (ROPE) {
                    float y = low[nh][0][e] + low[nh][1][e];
                    if constexpr (CHAINS == 2) y += low[nh][2][e] + low[nh][3][e];
                    x = (x + y) * unscale[nh][e & 1];
                }
                v[e] = tok0 + g + (e >> 1) * 8 < rg.end ? x : -INFINITY;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float mx = fmaxf(v[h], v[2 + h]);
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                const float mn = fmaxf(m[nh][h], mx), off = mn == -INFINITY ? 0.f : mn;
                alpha[nh][h] = m[nh][h] == -INFINITY ? 0.f : exp2f((m[nh][h] - mn) * LOG2E);
                m[nh][h] = mn;
                pr[h] = exp2f((v[h] - off) * LOG2E);
                pr[2 + h] = exp2f((v[2 + h] - off) * LOG2E);
                l[nh][h] = l[nh][h] * alpha[nh][h] + (pr[h] + pr[2 + h]);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                uint32_t hi, lo;
                split_h2(pr[2 * e] * UP, pr[2 * e + 1] * UP, hi, lo);
                ph[nh][e] = movmatrix(hi);
                pl[nh][e] = movmatrix(lo);
            }
        }
#pragma unroll
        for (int i = 0; i < D / 16; ++i) {
            uint32_t va[4];
            const int vr = (mat >> 1) * 8 + r8, c = i * 2 + (mat & 1);
            ldmatrix_x4_trans(va, sV + vr * (D * 2) + ((c ^ (vr & 7)) << 4));
#pragma unroll
            for (int nh = 0; nh < NH; ++nh) {
                float hi[4] = {0.f, 0.f, 0.f, 0.f}, lo[4] = {0.f, 0.f, 0.f, 0.f};
                mma_16816(hi, va, ph[nh][0], ph[nh][1]);
                mma_16816(lo, va, pl[nh][0], pl[nh][1]);
#pragma unroll
                for (int e = 0; e < 4; ++e) o[i][nh][e] = fmaf(o[i][nh][e], alpha[nh][e & 1], hi[e] + lo[e]);
            }
        }
        __syncwarp();
    }
    cp_async_wait_all();
    trace_event(p.trace, TR_ATTN | TR_MAIN_DONE);
    pdl_launch_dependents();
    __syncthreads();                         // every ring has been read: its memory takes the warps' results
    float* sm_o = reinterpret_cast<float*>(as_smem);       // [4][R][D]
    float* sm_ml = sm_o + 4 * R * D;                       // [4][R][2]
#pragma unroll
    for (int nh = 0; nh < NH; ++nh)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float ls = l[nh][h];
            ls += __shfl_xor_sync(0xffffffffu, ls, 4);
            ls += __shfl_xor_sync(0xffffffffu, ls, 8);
            ls += __shfl_xor_sync(0xffffffffu, ls, 16);
            const int r = nh * 8 + 2 * t + h;
            if (r < G) {
#pragma unroll
                for (int i = 0; i < D / 16; ++i) {
                    float* dst = sm_o + ((size_t)warp * R + r) * D + i * 16 + g;
                    dst[0] = o[i][nh][h] * (1.f / UP);
                    dst[8] = o[i][nh][2 + h] * (1.f / UP);
                }
                if (g == 0) { sm_ml[(warp * R + r) * 2] = m[nh][h]; sm_ml[(warp * R + r) * 2 + 1] = ls; }
            }
        }
    __syncthreads();
    for (int idx = threadIdx.x; idx < G * D; idx += 128) {
        const int r = idx / D, d = idx % D, hq = hq0 + r;
        float mn = -INFINITY, acc = 0.f, ls = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w) mn = fmaxf(mn, sm_ml[(w * R + r) * 2]);
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            const float mw = sm_ml[(w * R + r) * 2], a = mw == -INFINITY ? 0.f : exp2f((mw - mn) * LOG2E);
            acc += sm_o[((size_t)w * R + r) * D + d] * a;
            ls += sm_ml[(w * R + r) * 2 + 1] * a;
        }
        if (rg.eff == 1) {
            p.out[((size_t)qi * p.Hq + hq) * D + d] = __float2half_rn(ls > 0.f ? acc / ls : 0.f);
        } else {
            const size_t pi = (size_t)hq * p.nq * p.n_splits + place;
            p.part_o[pi * D + d] = acc;
            if (d == 0) { p.part_ml[pi * 2] = mn; p.part_ml[pi * 2 + 1] = ls; }
        }
    }
    trace_event(p.trace, TR_ATTN | TR_END);       // (CTA 0 is rarely the combining CTA: its END marks the partial write)
    if (rg.eff == 1 || p.counters == nullptr) return;
    // the last split CTA of this (query, head group) to finish merges all partials - no second launch
    __shared__ int is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        int* ctr = p.counters + (size_t)qi * gridDim.y + blockIdx.y;
        const int prev = atomicAdd(ctr, 1);
        is_last = (prev == rg.eff - 1);
        if (is_last) *ctr = 0;   // ready for the next launch
    }
    __syncthreads();
    if (!is_last) return;
    __threadfence();
    for (int r = warp; r < G; r += 4) attn_join<D>(p, qi, hq0 + r, rg.first, rg.eff, lane);
}

// ---------------------------------------------------------------------------------------------
// Decode step in ONE launch for callers without a workspace (attn_split_kernel is faster from 64 keys on: 3.4 against 7.5 us there, 6.6 against
// 8.3 at 512, 7.6 against 13 at 2,048): RoPE on Q and on the new token's K, paged write of that token's K/V, split-KV attention over the
// cache, and the split combine through distributed shared memory.
//
//   * The splits of one (query, KV-head group) form a thread-block CLUSTER (grid.x = cluster size = n_splits <= 16): partial
//     (o, m, l) triples are stored straight into the leader CTA's shared memory (st.shared::cluster through
//     cluster.map_shared_rank) and merged after one cluster barrier - no global workspace, no __threadfence + atomic ticket,
//     no L2 round trips, no second kernel.
//   * Q arrives un-rotated as the fp32 output row of the fused QKV mat-vec; every lane rotates the 16 dims it owns (the
//     half-split "neox" partner dim sits 4 lanes away: one shuffle).  The new token (position kv_len-1) is not in the cache
//     yet: the CTA that owns the tail of the key range rotates K, writes K/V to the page and folds the token in from
//     registers, so the separate RoPE + KV-write launch of the unfused path (rope_kv_kernel) disappears from the decode step.
// Reference counterparts: ggml_rope_ext + ggml_set_rows (K/V cache write) + flash_attn_ext_vec + flash_attn_combine_results -
// four graph nodes / launches per layer in `llama.cpp/src/models/llama.cpp:60-110`, `ggml-cuda/fattn-vec.cuh`.
template <int D, int G>
__global__ void __launch_bounds__(128) attn_decode_rope_kernel(const AttnParams p, const float* __restrict__ qkv,
                                                               const float* __restrict__ inv_freq,
                                                               const float2* __restrict__ rope_cs, __half* __restrict__ kc_w,
                                                               __half* __restrict__ vc_w, int neox, float q_scale) {
    namespace cg = cooperative_groups;
    constexpr int DL = D / 8;     // dims per lane (8 lanes share one token)
    constexpr int NV = DL / 8;    // 16-byte loads per lane and tensor
    constexpr int MAXS = 16;
    static_assert(DL % 8 == 0, "head dim must be a multiple of 64");
    cg::cluster_group cluster = cg::this_cluster();
    const int split = blockIdx.x;                      // == rank in the cluster (cluster dims = (gridDim.x, 1, 1))
    const int gqa = p.Hq / p.Hkv;
    const int groups_per_kv = gqa / G;
    const int kvh = blockIdx.y / groups_per_kv;
    const int hq0 = kvh * gqa + (blockIdx.y % groups_per_kv) * G;
    const int qi = blockIdx.z;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int grp = lane >> 3, sub = lane & 7;
    const int H = p.Hq + 2 * p.Hkv;

    // (a variant that staged 64-key K/V tiles in 64 KB of dynamic shared memory with cp.async measured slower: the large
    // carve-out keeps the kernel from sharing an SM with the neighbouring mat-vecs and costs the PDL overlap)
    __shared__ float sm_m[4][G], sm_l[4][G];
    __shared__ float sm_o[4][G][D];
    __shared__ float cl_o[MAXS][G][D];                 // leader only: landing zone of the splits' partial outputs
    __shared__ float cl_ml[MAXS][G][2];

    trace_event(p.trace, TR_ATTN | TR_BEGIN);
    // Everything the previous kernel (the QKV mat-vec) did NOT write is fetched before the dependency wait: sequence length,
    // block table and the step's rotation table come from the bookkeeping kernel at the start of the step (at least two launches
    // back, hence complete once this grid may start), the cached K/V rows from earlier steps.  Only `qkv` needs the wait, so the
    // dependent chain length -> page id -> K/V row runs under the predecessor's tail instead of after it.
    const int len = p.kv_len[qi];                      // keys visible to this query, the new token included
    const int n_old = len - 1;                         // ... of which this many are already in the cache
    const int eff = min((int)gridDim.x, max(1, (len + p.keys_per_split - 1) / p.keys_per_split));
    if (eff == 1 && split > 0) return;                 // uniform over the cluster: nobody waits on a barrier in that case
    const bool active = split < eff;
    const int per = (len + eff - 1) / eff;
    const int begin = split * per, end = min(len, begin + per);
    const int end_c = min(end, n_old);                 // cached part of this CTA's key range
    const bool owns_new = active && end == len;
    const int* bt = p.block_table + (size_t)(p.bt_row ? p.bt_row[qi] : qi) * p.max_pages;
    const float* row = qkv + (size_t)qi * H * D;
    uint4 kr[NV], vr[NV], kn[NV], vn[NV];
    auto fetch = [&](int tok0, uint4 (&kd)[NV], uint4 (&vd)[NV]) {
        const int tok = min(tok0 + grp, end_c - 1);
        const int page = bt[tok / p.page_size], off = tok % p.page_size;
        const size_t base = (((size_t)page * p.Hkv + kvh) * p.page_size + off) * D + sub * DL;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            kd[i] = ldg_nc_v4(p.kc + base + i * 8);
            vd[i] = ldg_nc_v4(p.vc + base + i * 8);
        }
    };
    const int t_first = begin + warp * 4;
    if (active && t_first < end_c) fetch(t_first, kr, vr);
    pdl_wait();
    if (p.pdl_early) pdl_launch_dependents();
    trace_event(p.trace, TR_ATTN | TR_WAITED);

    if (active) {

        // rotation terms of the DL dims this lane owns (shared by the G query heads and the new key): the per-step table
        // [nq][D/2] of (cos, sin) written by advance_rope_kernel once for all layers, or computed here
        float cs[DL], sn[DL];
        if (rope_cs != nullptr) {
            const float2* tab = rope_cs + (size_t)qi * (D / 2);
            if (neox) {
#pragma unroll
                for (int i = 0; i < DL; i += 2) {
                    const float4 v = *reinterpret_cast<const float4*>(tab + (sub & 3) * DL + i);
                    cs[i] = v.x; sn[i] = v.y; cs[i + 1] = v.z; sn[i + 1] = v.w;
                }
            } else {
#pragma unroll
                for (int i = 0; i < DL; i += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(tab + sub * (DL / 2) + i / 2);
                    cs[i] = cs[i + 1] = v.x; sn[i] = sn[i + 1] = v.y;
                    cs[i + 2] = cs[i + 3] = v.z; sn[i + 2] = sn[i + 3] = v.w;
                }
            }
        } else {
            const float pos = (float)n_old;
#pragma unroll
            for (int i = 0; i < DL; ++i) {
                const int d = sub * DL + i;
                const int fi = neox ? (d % (D / 2)) : (d >> 1);
                sincosf(pos * inv_freq[fi], &sn[i], &cs[i]);
            }
        }
        auto rotate = [&](float (&x)[DL]) {
            if (neox) {
#pragma unroll
                for (int i = 0; i < DL; ++i) {
                    const float other = __shfl_xor_sync(0xffffffffu, x[i], 4);     // dim d +- D/2 lives in lane sub ^ 4
                    x[i] = sub < 4 ? x[i] * cs[i] - other * sn[i] : x[i] * cs[i] + other * sn[i];
                }
            } else {
#pragma unroll
                for (int i = 0; i < DL; i += 2) {
                    const float a = x[i], b = x[i + 1];
                    x[i] = a * cs[i] - b * sn[i];
                    x[i + 1] = a * sn[i] + b * cs[i];
                }
            }
        };
        auto load_row = [&](const float* src, float (&x)[DL]) {
#pragma unroll
            for (int i = 0; i < DL; i += 4) {
                const float4 v = *reinterpret_cast<const float4*>(src + sub * DL + i);
                x[i] = v.x; x[i + 1] = v.y; x[i + 2] = v.z; x[i + 3] = v.w;
            }
        };
        float q[G][DL];
        float kf_new[DL], vf_new[DL];
        const bool do_new = owns_new && warp == 0;     // the new token's K/V rows travel with the Q rows: one L2 round trip
        if (do_new) {
            load_row(row + (size_t)(p.Hq + kvh) * D, kf_new);
            load_row(row + (size_t)(p.Hq + p.Hkv + kvh) * D, vf_new);
        }
#pragma unroll
        for (int g = 0; g < G; ++g) load_row(row + (size_t)(hq0 + g) * D, q[g]);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            rotate(q[g]);
#pragma unroll
            for (int i = 0; i < DL; ++i) q[g][i] *= q_scale;
        }
        float m[G], l[G], o[G][DL];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            m[g] = -INFINITY;
            l[g] = 0.f;
#pragma unroll
            for (int i = 0; i < DL; ++i) o[g][i] = 0.f;
        }
        auto accumulate = [&](const float (&kf)[DL], const float (&vf)[DL], bool valid) {
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float sc = 0.f;
#pragma unroll
                for (int i = 0; i < DL; ++i) sc = fmaf(q[g][i], kf[i], sc);
                sc += __shfl_xor_sync(0xffffffffu, sc, 1);
                sc += __shfl_xor_sync(0xffffffffu, sc, 2);
                sc += __shfl_xor_sync(0xffffffffu, sc, 4);
                if (!valid) continue;
                const float mn = fmaxf(m[g], sc);
                const float alpha = __expf(m[g] - mn), pr = __expf(sc - mn);
                m[g] = mn;
                l[g] = l[g] * alpha + pr;
#pragma unroll
                for (int i = 0; i < DL; ++i) o[g][i] = fmaf(pr, vf[i], o[g][i] * alpha);
            }
        };

        if (do_new) {
            // the new token first (online softmax does not care about order): rotate K, round K/V to the cache precision,
            // write the page slot, fold it in (lane group 0)
            rotate(kf_new);
            uint32_t kh[DL / 2], vh[DL / 2];
#pragma unroll
            for (int i = 0; i < DL; i += 2) {
                const __half2 a = __floats2half2_rn(kf_new[i], kf_new[i + 1]), b = __floats2half2_rn(vf_new[i], vf_new[i + 1]);
                kh[i / 2] = *reinterpret_cast<const uint32_t*>(&a);
                vh[i / 2] = *reinterpret_cast<const uint32_t*>(&b);
                const float2 af = __half22float2(a), bf = __half22float2(b);
                kf_new[i] = af.x; kf_new[i + 1] = af.y; vf_new[i] = bf.x; vf_new[i + 1] = bf.y;
            }
            if (grp == 0 && blockIdx.y % groups_per_kv == 0) {
                const int page = bt[n_old / p.page_size], off = n_old % p.page_size;
                const size_t base = (((size_t)page * p.Hkv + kvh) * p.page_size + off) * D + sub * DL;
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    *reinterpret_cast<uint4*>(kc_w + base + i * 8) = make_uint4(kh[4 * i], kh[4 * i + 1], kh[4 * i + 2], kh[4 * i + 3]);
                    *reinterpret_cast<uint4*>(vc_w + base + i * 8) = make_uint4(vh[4 * i], vh[4 * i + 1], vh[4 * i + 2], vh[4 * i + 3]);
                }
            }
            accumulate(kf_new, vf_new, grp == 0);
        }
        for (int tok0 = t_first; tok0 < end_c; tok0 += 16) {
            const bool valid = tok0 + grp < end_c;
            const bool more = tok0 + 16 < end_c;
            if (more) fetch(tok0 + 16, kn, vn);
            float kf[DL], vf[DL];
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const uint32_t kw[4] = {kr[i].x, kr[i].y, kr[i].z, kr[i].w}, vw[4] = {vr[i].x, vr[i].y, vr[i].z, vr[i].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 a = h2_to_f2(kw[j]), b = h2_to_f2(vw[j]);
                    kf[i * 8 + 2 * j] = a.x; kf[i * 8 + 2 * j + 1] = a.y;
                    vf[i * 8 + 2 * j] = b.x; vf[i * 8 + 2 * j + 1] = b.y;
                }
            }
            accumulate(kf, vf, valid);
            if (more) {
#pragma unroll
                for (int i = 0; i < NV; ++i) { kr[i] = kn[i]; vr[i] = vn[i]; }
            }
        }
        trace_event(p.trace, TR_ATTN | TR_MAIN_DONE);
        pdl_launch_dependents();
        // merge the 4 lane groups of the warp, then the 4 warps of the CTA
#pragma unroll
        for (int g = 0; g < G; ++g) {
#pragma unroll
            for (int off = 8; off <= 16; off <<= 1) {
                const float m2 = __shfl_xor_sync(0xffffffffu, m[g], off);
                const float l2 = __shfl_xor_sync(0xffffffffu, l[g], off);
                const float mn = fmaxf(m[g], m2);
                const float a1 = (m[g] == -INFINITY) ? 0.f : __expf(m[g] - mn);
                const float a2 = (m2 == -INFINITY) ? 0.f : __expf(m2 - mn);
#pragma unroll
                for (int i = 0; i < DL; ++i) {
                    const float o2 = __shfl_xor_sync(0xffffffffu, o[g][i], off);
                    o[g][i] = o[g][i] * a1 + o2 * a2;
                }
                l[g] = l[g] * a1 + l2 * a2;
                m[g] = mn;
            }
            if (grp == 0) {
#pragma unroll
                for (int i = 0; i < DL; ++i) sm_o[warp][g][sub * DL + i] = o[g][i];
                if (sub == 0) { sm_m[warp][g] = m[g]; sm_l[warp][g] = l[g]; }
            }
        }
        __syncthreads();
        float* dst_o = eff == 1 ? nullptr : cluster.map_shared_rank(&cl_o[0][0][0], 0);
        float* dst_ml = eff == 1 ? nullptr : cluster.map_shared_rank(&cl_ml[0][0][0], 0);
        for (int idx = threadIdx.x; idx < G * D; idx += blockDim.x) {
            const int g = idx / D, d = idx % D;
            float mn = -INFINITY;
#pragma unroll
            for (int w = 0; w < 4; ++w) mn = fmaxf(mn, sm_m[w][g]);
            float acc = 0.f, ls = 0.f;
#pragma unroll
            for (int w = 0; w < 4; ++w) {
                const float a = (sm_m[w][g] == -INFINITY) ? 0.f : __expf(sm_m[w][g] - mn);
                acc += sm_o[w][g][d] * a;
                ls += sm_l[w][g] * a;
            }
            if (eff == 1) {
                p.out[((size_t)qi * p.Hq + hq0 + g) * D + d] = __float2half_rn(ls > 0.f ? acc / ls : 0.f);
            } else {
                dst_o[((size_t)split * G + g) * D + d] = acc;
                if (d == 0) { dst_ml[(split * G + g) * 2] = mn; dst_ml[(split * G + g) * 2 + 1] = ls; }
            }
        }
    } else {
        pdl_launch_dependents();
    }
    if (eff == 1) { trace_event(p.trace, TR_ATTN | TR_END); return; }
    cluster.sync();                                    // release/acquire at cluster scope: the partials are visible in rank 0
    if (split != 0) return;
    for (int idx = threadIdx.x; idx < G * D; idx += blockDim.x) {
        const int g = idx / D, d = idx % D;
        float mn = -INFINITY;
        for (int sp = 0; sp < eff; ++sp) mn = fmaxf(mn, cl_ml[sp][g][0]);
        float acc = 0.f, ls = 0.f;
        for (int sp = 0; sp < eff; ++sp) {
            const float ms = cl_ml[sp][g][0];
            const float a = (ms == -INFINITY) ? 0.f : __expf(ms - mn);
            acc += cl_o[sp][g][d] * a;
            ls += cl_ml[sp][g][1] * a;
        }
        p.out[((size_t)qi * p.Hq + hq0 + g) * D + d] = __float2half_rn(ls > 0.f ? acc / ls : 0.f);
    }
    trace_event(p.trace, TR_ATTN | TR_END);
}

static int attn_pdl_early() {
    static int early = -1;
    if (early < 0) { const char* e = getenv("DLP_PDL_EARLY"); early = (e && e[0] == '0') ? 0 : 1; }
    return early;
}

template <int D, int G>
static int launch_attn_rope_g(const AttnParams& p, const float* qkv, const float* inv_freq, const float2* rope_cs, __half* kc_w,
                              __half* vc_w, int neox, float q_scale, cudaStream_t s) {
    auto kern = attn_decode_rope_kernel<D, G>;
    if (first_use_on_device((const void*)kern))   // cluster sizes above 8 are "non-portable": opt in once per device
        DLP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    const int gqa = p.Hq / p.Hkv;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.n_splits, p.Hkv * (gqa / G), p.nq);
    cfg.blockDim = dim3(128);
    cfg.dynamicSmemBytes = 0;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = p.n_splits;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    DLP_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kern, p, qkv, inv_freq, rope_cs, kc_w, vc_w, neox, q_scale));
    return 0;
}

template <int D>
static int launch_attn_rope(const AttnParams& p, const float* qkv, const float* inv_freq, const float2* rope_cs, __half* kc_w,
                            __half* vc_w, int neox, float q_scale, cudaStream_t s) {
    const int gqa = p.Hq / p.Hkv;
    if (gqa % 4 == 0) return launch_attn_rope_g<D, 4>(p, qkv, inv_freq, rope_cs, kc_w, vc_w, neox, q_scale, s);
    if (gqa % 2 == 0) return launch_attn_rope_g<D, 2>(p, qkv, inv_freq, rope_cs, kc_w, vc_w, neox, q_scale, s);
    return launch_attn_rope_g<D, 1>(p, qkv, inv_freq, rope_cs, kc_w, vc_w, neox, q_scale, s);
}

int attn_decode_rope(const AttnParams& p_in, const float* qkv, const float* inv_freq, const float2* rope_cs, __half* kc_w,
                     __half* vc_w, int D, int neox, float q_scale, cudaStream_t s) {
    AttnParams p = p_in;
    p.trace = trace_buffer();
    static int kps = 0;
    if (kps == 0) {
        const char* k = getenv("DLP_ATTN_KEYS_PER_SPLIT");
        kps = k ? atoi(k) : 32;
        if (kps < 16) kps = 16;
    }
    p.pdl_early = attn_pdl_early();
    p.keys_per_split = kps;
    DLP_REQUIRE(inv_freq != nullptr || rope_cs != nullptr, "attn_decode_rope: need inv_freq or a (cos, sin) table");
    DLP_REQUIRE(p.nq > 0 && p.Hq % p.Hkv == 0, "attn_decode_rope: bad head configuration Hq=%d Hkv=%d", p.Hq, p.Hkv);
    DLP_REQUIRE(p.n_splits >= 1 && p.n_splits <= 16, "attn_decode_rope: cluster size %d outside 1..16", p.n_splits);
    if (D == 64) return launch_attn_rope<64>(p, qkv, inv_freq, rope_cs, kc_w, vc_w, neox, q_scale, s);
    if (D == 128) return launch_attn_rope<128>(p, qkv, inv_freq, rope_cs, kc_w, vc_w, neox, q_scale, s);
    DLP_REQUIRE(false, "attn_decode_rope: head dim %d unsupported (64, 128)", D);
}

template <int D>
__global__ void attn_combine_kernel(const AttnParams p) {
    const int hq = blockIdx.x, qi = blockIdx.y;
    pdl_wait();
    pdl_launch_dependents();
    const AttnRange rg = attn_range(p, -1, qi, threadIdx.x);
    if (rg.eff == 1) return;   // the single range already wrote the final output
    attn_join<D>(p, qi, hq, rg.first, rg.eff, threadIdx.x);
}

// Ranges that several queries share: one wave of the kernel's two CTAs an SM, or half a wave more than there are queries - as far as the
// workspace goes -, so that queries of equal length stay whole where cutting them would only start a second wave (32 x 2,000 keys, 32 heads over 8:
// 42 us whole, 51 in two each; 16: 26.8 in two, 35 in three; 8: 14.1 in four, 22 in five).  0: every query has its n_splits.
static void attn_pool(AttnParams& p, int groups) {
    p.pool = 0;
    if (p.n_splits <= 1 || p.nq <= 1 || p.nq > ATTN_POOL_NQ) return;
    p.wave = max(1, 2 * sm_count() / (p.Hkv * groups));
    p.pool = min(p.nq * p.n_splits, max(p.wave, p.nq + max(1, p.wave / 2)));
}

template <int D, int NH, bool ROPE>
static int launch_attn_split(AttnParams p, const AttnRope& ra, cudaStream_t s) {
    auto kern = attn_split_kernel<D, NH, ROPE>;
    if (first_use_on_device((const void*)kern))
        DLP_CHECK_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, attn_split_smem<D>()));
    const int gqa = p.Hq / p.Hkv, groups = (gqa + 8 * NH - 1) / (8 * NH);
    attn_pool(p, groups);
    const dim3 grid(p.pool ? p.pool : p.n_splits, p.Hkv * groups, p.pool ? 1 : p.nq);
    DLP_CHECK_CUDA(launch_pdl(kern, grid, dim3(128), attn_split_smem<D>(), s, p, ra));
    if (p.n_splits > 1 && p.counters == nullptr)
        DLP_CHECK_CUDA(launch_pdl(attn_combine_kernel<D>, dim3(p.Hq, p.nq), dim3(32), 0, s, p));
    return 0;
}
template <int D, bool ROPE>
static int launch_attn(const AttnParams& p, const AttnRope& ra, cudaStream_t s) {
    return p.Hq / p.Hkv <= 8 ? launch_attn_split<D, 1, ROPE>(p, ra, s) : launch_attn_split<D, 2, ROPE>(p, ra, s);
}

// The one-launch form for long contexts: RoPE, K / V write and split-KV attention with the splits joined through the caller's workspace.
int attn_decode_split(const AttnParams& p_in, const float* qkv, const float* inv_freq, const float2* rope_cs, __half* kc_w, __half* vc_w, int D,
                      int neox, float q_scale, cudaStream_t s) {
    AttnParams p = p_in;
    p.trace = trace_buffer();
    p.pdl_early = attn_pdl_early();
    DLP_REQUIRE(inv_freq != nullptr || rope_cs != nullptr, "attn_decode_split: need inv_freq or a (cos, sin) table");
    DLP_REQUIRE(p.nq > 0 && p.Hq % p.Hkv == 0, "attn_decode_split: bad head configuration Hq=%d Hkv=%d", p.Hq, p.Hkv);
    DLP_REQUIRE(p.n_splits >= 1 && (p.n_splits == 1 || (p.part_o && p.part_ml && p.counters)), "attn_decode_split: split-KV needs a workspace");
    const AttnRope ra = {qkv, inv_freq, rope_cs, kc_w, vc_w, neox, q_scale};
    if (D == 64) return launch_attn<64, true>(p, ra, s);
    if (D == 128) return launch_attn<128, true>(p, ra, s);
    DLP_REQUIRE(false, "attn_decode_split: head dim %d unsupported (64, 128)", D);
}

int attn_paged(const AttnParams& p_in, int D, cudaStream_t s) {
    AttnParams p = p_in;
    p.trace = trace_buffer();
    DLP_REQUIRE(p.nq > 0 && p.Hq % p.Hkv == 0, "attn: bad head configuration Hq=%d Hkv=%d", p.Hq, p.Hkv);
    DLP_REQUIRE(p.n_splits >= 1 && (p.n_splits == 1 || (p.part_o && p.part_ml)), "attn: split-KV needs a workspace");
    const AttnRope none = {};
    if (D == 64) return launch_attn<64, false>(p, none, s);
    if (D == 128) return launch_attn<128, false>(p, none, s);
    DLP_REQUIRE(false, "attn: head dim %d unsupported (64, 128)", D);
}

}  // namespace dlp

// =================================================================================================
// Causal flash-prefill over the paged cache (one sequence chunk).
//
// Reference counterpart: `flash_attn_ext_f16` (ggml-cuda/fattn-mma-f16.cuh).  FlashAttention-2 schedule:
// one CTA = 64 query rows of one head (4 warps x 16 rows), K/V streamed page-by-page through shared
// memory with cp.async, scores and P.V on the legacy tensor-core path (mma.sync m16n8k16, fp32
// accumulate), online softmax in registers.  Attention is ~1% of prefill FLOPs at the benchmark shapes
// (the linear layers run on tcgen05), so this kernel favours simplicity; a TMEM-resident variant is the
// planned upgrade.
namespace dlp {


template <int D>
__global__ void __launch_bounds__(128) attn_prefill_kernel(const __half* __restrict__ q, const __half* __restrict__ kc,
                                                           const __half* __restrict__ vc, const int* __restrict__ bt,
                                                           __half* __restrict__ out, int T, int pos0, int Hq, int Hkv, int PS) {
    constexpr int LD = D + 8;      // padded row (halves) -> conflict-free ldmatrix
    constexpr int BQ = 64, BKV = 64;
    extern __shared__ __align__(16) uint8_t att_smem[];
    __half* sQ = reinterpret_cast<__half*>(att_smem);
    __half* sKV = sQ + BQ * LD;              // two stages of (K tile | V tile): the next tile lands while this one is consumed
    // heaviest query tiles first: under the causal mask the last tile has the most key tiles to walk
    const int q0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * BQ, hq = blockIdx.y, kvh = hq / (Hq / Hkv);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    constexpr int CPR = D / 8;  // 16-byte chunks per row

    for (int i = tid; i < BQ * CPR; i += 128) {
        const int r = i / CPR, c = i % CPR;
        const bool ok = q0 + r < T;
        cp_async16(sQ + r * LD + c * 8, q + ((size_t)(ok ? q0 + r : 0) * Hq + hq) * D + c * 8, ok);
    }
    const int n_kv = pos0 + min(q0 + BQ, T);
    const int n_tiles = (n_kv + BKV - 1) / BKV;

    uint32_t qf[D / 16][4];
    float o[D / 8][4];
#pragma unroll
    for (int i = 0; i < D / 8; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};
    constexpr float LOG2E = 1.4426950408889634f;

    auto load_kv = [&](int kt) {
        __half* dK = sKV + (kt & 1) * 2 * BKV * LD;
        __half* dV = dK + BKV * LD;
        for (int i = tid; i < BKV * CPR; i += 128) {
            const int r = i / CPR, c = i % CPR;
            const int tok = kt * BKV + r;
            const bool ok = tok < n_kv;
            const int tk = ok ? tok : 0;
            const size_t src = (((size_t)bt[tk / PS] * Hkv + kvh) * PS + tk % PS) * D + c * 8;
            cp_async16(dK + r * LD + c * 8, kc + src, ok);
            cp_async16(dV + r * LD + c * 8, vc + src, ok);
        }
        cp_async_commit();
    };
    load_kv(0);                                // (commits the Q rows requested above with it)
    for (int kt = 0; kt < n_tiles; ++kt) {
        __syncthreads();                       // tile kt-1 fully consumed: its stage may be refilled
        if (kt + 1 < n_tiles) { load_kv(kt + 1); cp_async_wait_group<1>(); } else { cp_async_wait_group<0>(); }
        __syncthreads();                       // tile kt (and Q) visible to every warp
        const __half* sK = sKV + (kt & 1) * 2 * BKV * LD;
        const __half* sV = sK + BKV * LD;
        if (kt == 0) {
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks)
                ldmatrix_x4(qf[ks], sQ + (warp * 16 + (lane & 15)) * LD + ks * 16 + (lane >> 4) * 8);
        }
        // ---- S = Q K^T (16 x 64 per warp) ----
        float s[BKV / 8][4];
#pragma unroll
        for (int i = 0; i < BKV / 8; ++i) { s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f; }
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
#pragma unroll
            for (int np = 0; np < BKV / 16; ++np) {
                uint32_t kb[4];
                const int mat = lane >> 3, r = lane & 7;
                ldmatrix_x4(kb, sK + (np * 16 + (mat >> 1) * 8 + r) * LD + ks * 16 + (mat & 1) * 8);
                mma_16816(s[np * 2], qf[ks], kb[0], kb[1]);
                mma_16816(s[np * 2 + 1], qf[ks], kb[2], kb[3]);
            }
        }
        // ---- causal mask + online softmax (rows g and g+8 of this warp's 16) ----
        const int qpos0 = pos0 + q0 + warp * 16 + g;
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int nt = 0; nt < BKV / 8; ++nt) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int kpos = kt * BKV + nt * 8 + t4 * 2 + (e & 1);
                const int qpos = qpos0 + (e >> 1) * 8;
                if (kpos > qpos) s[nt][e] = -INFINITY;
                mx[e >> 1] = fmaxf(mx[e >> 1], s[nt][e]);
            }
        }
        float alpha[2], msc[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
            mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2));
            const float mn = fmaxf(m_run[h], mx[h]);
            alpha[h] = (m_run[h] == -INFINITY) ? 0.f : exp2f((m_run[h] - mn) * LOG2E);
            msc[h] = (mn == -INFINITY) ? 0.f : mn * LOG2E;
            m_run[h] = mn;
        }
        float rs[2] = {0.f, 0.f};
#pragma unroll
        for (int nt = 0; nt < BKV / 8; ++nt) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float pv = exp2f(s[nt][e] * LOG2E - msc[e >> 1]);  // exp2(-inf) = 0 for masked keys
                s[nt][e] = pv;
                rs[e >> 1] += pv;
            }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) l_run[h] = l_run[h] * alpha[h] + rs[h];
#pragma unroll
        for (int i = 0; i < D / 8; ++i) {
            o[i][0] *= alpha[0]; o[i][1] *= alpha[0];
            o[i][2] *= alpha[1]; o[i][3] *= alpha[1];
        }
        // ---- O += P V ----
#pragma unroll
        for (int kk = 0; kk < BKV / 16; ++kk) {
            uint32_t pa[4];
            pa[0] = pack_h2(s[2 * kk][0], s[2 * kk][1]);
            pa[1] = pack_h2(s[2 * kk][2], s[2 * kk][3]);
            pa[2] = pack_h2(s[2 * kk + 1][0], s[2 * kk + 1][1]);
            pa[3] = pack_h2(s[2 * kk + 1][2], s[2 * kk + 1][3]);
#pragma unroll
            for (int dp = 0; dp < D / 16; ++dp) {
                uint32_t vb[4];
                const int mat = lane >> 3, r = lane & 7;
                ldmatrix_x4_trans(vb, sV + (kk * 16 + (mat & 1) * 8 + r) * LD + dp * 16 + (mat >> 1) * 8);
                mma_16816(o[dp * 2], pa, vb[0], vb[1]);
                mma_16816(o[dp * 2 + 1], pa, vb[2], vb[3]);
            }
        }
    }
    // ---- finalise: row sums live per-quad; reduce then normalise and store ----
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 1);
        l_run[h] += __shfl_xor_sync(0xffffffffu, l_run[h], 2);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int row = q0 + warp * 16 + g + h * 8;
        if (row < T) {
            const float inv = l_run[h] > 0.f ? 1.f / l_run[h] : 0.f;
            __half* op = out + ((size_t)row * Hq + hq) * D;
#pragma unroll
            for (int i = 0; i < D / 8; ++i) {
                const uint32_t v = pack_h2(o[i][h * 2] * inv, o[i][h * 2 + 1] * inv);
                *reinterpret_cast<uint32_t*>(op + i * 8 + t4 * 2) = v;
            }
        }
    }
}

int attn_prefill(const __half* q, const __half* kc, const __half* vc, const int* bt_row, __half* out, int T, int pos0,
                 int Hq, int Hkv, int D, int page_size, cudaStream_t s) {
    DLP_REQUIRE(T > 0 && Hq % Hkv == 0, "attn_prefill: bad shape");
    dim3 grid((T + 63) / 64, Hq);
    if (D == 128) {
        const int smem = 5 * 64 * (128 + 8) * 2;   // Q + 2 stages x (K, V)
        if (first_use_on_device((const void*)attn_prefill_kernel<128>))
            DLP_CHECK_CUDA(cudaFuncSetAttribute(attn_prefill_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        attn_prefill_kernel<128><<<grid, 128, smem, s>>>(q, kc, vc, bt_row, out, T, pos0, Hq, Hkv, page_size);
    } else if (D == 64) {
        const int smem = 5 * 64 * (64 + 8) * 2;
        if (first_use_on_device((const void*)attn_prefill_kernel<64>))
            DLP_CHECK_CUDA(cudaFuncSetAttribute(attn_prefill_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        attn_prefill_kernel<64><<<grid, 128, smem, s>>>(q, kc, vc, bt_row, out, T, pos0, Hq, Hkv, page_size);
    } else {
        DLP_REQUIRE(false, "attn_prefill: head dim %d unsupported (64, 128)", D);
    }
    DLP_LAUNCH_CHECK();
    return 0;
}

}  // namespace dlp

// =================================================================================================
// Split-KV paged attention without a caller-provided workspace.
//
// Some hosts of this library are not in a position to hand us scratch memory: a serving process that carved
// the whole HBM into weights + KV pages at start-up and then froze its allocator, a plug-in running under a
// "no device allocation after init" rule, or code sitting between cudaStreamBeginCapture / EndCapture where
// cudaMalloc is illegal.  For them the split-KV partial results (the only scratch `attn_paged` needs) live in
// a fixed array inside this module's device image.  Costs and rules, all of which the header repeats:
//   * the array is ATTN_STATIC_SCRATCH_FLOATS floats (4 MiB) on every GPU that loads the library, until exit;
//   * a launch needs nq * Hq * n_splits * (D + 2) floats and is refused with an error beyond that;
//   * every call on a device shares the same array, so calls that overlap on the GPU (different streams, or
//     graphs replayed concurrently) race - serialise them;
//   * nothing has to start at zero: the combine kernel reads the slots of the ranges that the partial kernel had
//     keys for and wrote, so stale contents of an earlier call are never observed.
// In host code the array's name is only a handle: the device address is obtained once per device with
// cudaGetSymbolAddress (device current, return code checked) on the first call there, which therefore must
// happen outside stream capture.
namespace dlp {

constexpr size_t ATTN_STATIC_SCRATCH_FLOATS = size_t(1) << 20;  // keep in sync with DLP_ATTN_STATIC_SCRATCH_FLOATS
static __device__ __align__(256) float g_attn_static_scratch[ATTN_STATIC_SCRATCH_FLOATS];

int attn_paged_static(AttnParams p, int D, cudaStream_t s) {
    DLP_REQUIRE(p.nq > 0 && p.Hq > 0 && p.n_splits >= 1 && D > 0, "attn_paged_static: bad shape");
    const size_t n_part = (size_t)p.nq * p.Hq * p.n_splits;
    const size_t need = p.n_splits > 1 ? n_part * (size_t)(D + 2) : 0;
    DLP_REQUIRE(need <= ATTN_STATIC_SCRATCH_FLOATS,
                "attn_paged_static: nq*Hq*n_splits*(D+2) = %zu floats exceeds the built-in scratch of %zu floats; "
                "lower n_splits / batch or use dlp_attn_paged with your own workspace",
                need, (size_t)ATTN_STATIC_SCRATCH_FLOATS);
    constexpr int MAX_DEV = 64;
    static float* dev_ptr[MAX_DEV] = {nullptr};
    int dev = -1;
    DLP_CHECK_CUDA(cudaGetDevice(&dev));
    DLP_REQUIRE(dev >= 0 && dev < MAX_DEV, "attn_paged_static: device ordinal %d out of range", dev);
    float* ptr = dev_ptr[dev];
    if (ptr == nullptr) {  // once per device, with that device current (racing first calls store the same value)
        DLP_CHECK_CUDA(cudaGetSymbolAddress((void**)&ptr, g_attn_static_scratch));
        DLP_REQUIRE(ptr != nullptr, "attn_paged_static: cudaGetSymbolAddress returned a null address");
        dev_ptr[dev] = ptr;
    }
    p.counters = nullptr;                // this entry point keeps the two-kernel combine
    p.part_o = ptr;                      // [Hq, nq * n_splits, D]
    p.part_ml = ptr + n_part * (size_t)D;  // [Hq, nq * n_splits, 2]
    return attn_paged(p, D, s);
}

}  // namespace dlp
