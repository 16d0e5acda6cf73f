// attention_prefill_tc.cu — causal prefill attention over the paged KV cache on the 5th-generation tensor cores.
//
// Three kernels with one order of a row's sums, so one result; prefill_attention_kernel_of() at the end of the file chooses by the batch: one head a CTA (few short items),
// two heads a CTA (short query tiles, odd groups of heads of 128) and, for most batches, one head a CTA whose softmax warpgroups take the key tiles in turn, on
// pairs of CTAs for heads of 128.
//
// The first.  One CTA = 128 query rows of one (sequence, head); KV is consumed in tiles of 128 tokens (two 64-token pages):
//   warp 0    : TMA producer — Q tile once, then the K pages of a KV tile and the V pages of the one before it.  K and V have SEPARATE
//               2-stage rings: K_j is released as soon as S_j has been computed, V_j only after P_j·V_j, so the K load of tile
//               j+2 gets a full tile period of slack instead of being exposed behind the second MMA
//   warp 1    : tcgen05.mma issuer —  S_j = Q · K_j^T   (M=128, N=128, K=D;   A, B K-major)        -> TMEM S[j&1]
//                                     O  += P_j · V_j   (M=128, N=D,   K=128; A K-major, B MN-major: V[kv, d] as stored)  -> TMEM O
//   warps 2-5 : one query row per thread.  tcgen05.ld S_j once (128 values), causal mask, P_j = 2^(s - m_ref) rounded to bf16 into
//               swizzled shared memory (the A operand of the second MMA).  O stays in TMEM for the whole KV sweep: the reference
//               maximum m_ref is only raised — and O, l rescaled via tcgen05.ld/st — when a row's maximum exceeds it by more than
//               2^8 (lazy rescaling), so the common tile costs one TMEM read, 128 exp2 and 16 shared-memory stores per thread and
//               overlaps the tensor-core work of its neighbours (S and P are double-buffered).
// Row sums use the unrounded p, P·V the bf16-rounded p — the rounding points the oracle mirrors.  TMEM: 2x128 (S) + D (O).

#include <algorithm>

#include "common.cuh"
#include "cta_pair.cuh"
#include "kernels.hpp"

namespace oa {

static constexpr int KV_TILE = 128;

// One warp: 64 columns of O of its 32 rows (TMEM lanes of `addr`, a row's values scaled by its lane's inv), rounded to bf16.  A lane holds a row, so a store
// straight from registers is 32 pieces of 16 bytes; through 4 KB of shared memory it is four whole 128-byte lines.
OA_DEVINL void store_o_64(uint8_t* stage, uint32_t addr, float inv, uint16_t* out, size_t pitch, int lane) {
#pragma unroll
    for (int c = 0; c < 64; c += 32) {
        uint32_t o[32];
        tmem_ld_32x32b_x32(addr + (uint32_t)c, o);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i += 8) {
            uint4 w;
            w.x = pack_bf16x2(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
            w.y = pack_bf16x2(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
            w.z = pack_bf16x2(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv);
            w.w = pack_bf16x2(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv);
            *reinterpret_cast<uint4*>(stage + lane * 128 + ((((c + i) >> 3) ^ (lane & 7)) << 4)) = w;
        }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = i * 4 + (lane >> 3), ch = lane & 7;
        const uint4 w = *reinterpret_cast<const uint4*>(stage + r * 128 + ((ch ^ (r & 7)) << 4));
        *reinterpret_cast<uint4*>(out + (size_t)r * pitch + ch * 8) = w;
    }
    __syncwarp();
}

// The same of COLS columns straight from registers, a lane its row: with 64 columns a head a row is one line, and this is the faster way (five prompts of
// 1400 rows, 32 / 8 heads of 64: 74.7 us a layer against 78.9 through shared memory).  So it is for warps with rows missing.
template <int COLS>
OA_DEVINL void store_o_direct(uint32_t addr, float inv, uint16_t* row, bool live) {
#pragma unroll 1
    for (int c = 0; c < COLS; c += 32) {
        uint32_t o[32];
        tmem_ld_32x32b_x32(addr + (uint32_t)c, o);
        tmem_ld_wait();
        if (live) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
                uint4 w;
                w.x = pack_bf16x2(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
                w.y = pack_bf16x2(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
                w.z = pack_bf16x2(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv);
                w.w = pack_bf16x2(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv);
                *reinterpret_cast<uint4*>(row + c + i) = w;
            }
        }
    }
}

// A row's sum, in one order in all three kernels: of each half (64 keys) of a tile the probabilities of even and of odd keys, those two added, and the tiles'
// half sums added up over an item's even and over its odd tiles; each of the four is relative to 2^m of its own last tile until the item ends.
OA_DEVINL float sum_rescale(float m, float m_new) { return m == m_new ? 1.0f : exp2f(m - m_new); }
OA_DEVINL float sum_add(float l, float f, uint64_t pair) { float a, b; unpack_f32x2(pair, a, b); return __fadd_rn(__fmul_rn(l, f), __fadd_rn(a, b)); }

template <int D>
struct PtcCfg {
    static constexpr int HALVES = D / 64;
    static constexpr int HALF_BYTES = 128 * 128;                 // 128 rows x 64 bf16 columns, one swizzle-atom column
    static constexpr int Q_BYTES = HALVES * HALF_BYTES;
    static constexpr int KV_BYTES = HALVES * HALF_BYTES;         // K (or V) of one 128-token tile
    static constexpr int STAGE_BYTES = 2 * KV_BYTES;
    static constexpr int P_BYTES = 2 * HALF_BYTES;               // [128 q, 128 kv] bf16
    static constexpr int XCH_BYTES = 2 * 2 * 128 * 4;            // row-statistic exchange between the two softmax warpgroups: [tile parity][warpgroup][row]
    static constexpr int SMEM_BYTES = Q_BYTES + 2 * STAGE_BYTES + 2 * P_BYTES + 256 + XCH_BYTES;     // D=128: 231,680 B of the 232,448 available — the base is declared 1024-aligned, no slack
    static_assert(SMEM_BYTES <= 232448, "shared memory budget of one CTA");
    static constexpr uint32_t TMEM_COLS = 512;
    static constexpr uint32_t T_COL = 256;                       // S[0] at 0, S[1] at 128, T at 256
};

// NWG = 2 softmax warpgroups: with one, each SM sub-partition holds a single softmax warp and the 128 exp2 + pack + store chain of a tile
// (~1.1 us) is longer than its two MMAs (~0.75 us), and the tensor pipe idles 70 % of the time.  The warps w and w+4
// share the same 32 query rows (same TMEM lanes) and split every S tile by KEY columns — 64 scores, 64 exp2, 8 P stores per thread, two
// warps per sub-partition to hide latencies; the halves' row maxima meet through shared memory once per tile, the row sums once at the end.
static constexpr int NWG = 2;
template <int D>
__global__ void __launch_bounds__(64 + 128 * NWG, 1) prefill_attention_tc_kernel(const __grid_constant__ CUtensorMap tm_q,
                                                                              const __grid_constant__ CUtensorMap tm_kv,
                                                                              const PrefillAttnParams p, const int64_t layer_row0,
                                                                              const int64_t kv_stride_rows) {
    using Cfg = PtcCfg<D>;
    constexpr int HALVES = Cfg::HALVES;
    extern __shared__ __align__(1024) uint8_t smem_raw[];       // 128-byte-swizzled TMA / UMMA tiles need 1024-byte alignment
    uint8_t* smem = smem_raw;
    uint8_t* q_s = smem;
    uint8_t* kv_s = q_s + Cfg::Q_BYTES;                          // [2 stages][K | V]
    uint8_t* p_s = kv_s + 2 * Cfg::STAGE_BYTES;                  // [2][P]
    uint64_t* bars = reinterpret_cast<uint64_t*>(p_s + 2 * Cfg::P_BYTES);
    uint64_t* q_full = bars;                  // 1
    uint64_t* k_full = bars + 1;              // [2]
    uint64_t* k_empty = bars + 3;             // [2]
    uint64_t* v_full = bars + 5;              // [2]
    uint64_t* v_empty = bars + 7;             // [2]
    uint64_t* s_full = bars + 9;              // [2]
    uint64_t* s_empty = bars + 11;            // [2]
    uint64_t* p_full = bars + 13;             // [2]
    uint64_t* t_full = bars + 15;             // 1 (one completion per P·V but the last)
    uint64_t* o_full = bars + 16;             // 1 (the last P·V)
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
    float* xch = reinterpret_cast<float*>(p_s + 2 * Cfg::P_BYTES + 256);       // [2][2][128]

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // warp: uniform, and known to be
    const PrefillTile tile = p.tiles[blockIdx.x];
    const int head = blockIdx.y;
    const int grp = p.n_heads / p.n_kv, kvh = head / grp;
    const int n_kvt = __shfl_sync(0xffffffffu, (tile.pos0 + tile.n_rows + KV_TILE - 1) / KV_TILE, 0);       // KV tiles 0..n_kvt-1 cover every visible key

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_kv);
        mbar_init(q_full, 1);
        for (int i = 0; i < 2; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1);
                                      mbar_init(&s_full[i], 1); mbar_init(&s_empty[i], 4 * NWG); mbar_init(&p_full[i], 4 * NWG); }
        mbar_init(t_full, 1); mbar_init(o_full, 1);
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc<Cfg::TMEM_COLS>(tmem_slot);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    griddep_launch();

    if (warp == 0) {
        griddep_wait();
        if (elect_one()) {
            mbar_expect_tx(q_full, Cfg::Q_BYTES);
#pragma unroll
            for (int h = 0; h < HALVES; ++h) tma_load_2d(q_s + h * Cfg::HALF_BYTES, &tm_q, q_full, head * D + h * 64, tile.q_row0, kEvictFirst);
        }
        __syncwarp();
        const int32_t* bt = p.block_tables + (size_t)tile.seq * p.max_pages_per_seq;
        // K of tile j, then V of the tile before it: K_j's slot is free as soon as S_{j-2} exists, V_{j-1}'s only after P_{j-3}·V
        int32_t page[2] = {0, 0}, prev[2] = {0, 0};
        for (int j = 0; j <= n_kvt; ++j) {
#pragma unroll
            for (int pg = 0; pg < 2; ++pg) {
                prev[pg] = page[pg];
                const int pi = 2 * j + pg;
                if (j < n_kvt) page[pg] = bt[pi < p.max_pages_per_seq ? pi : 2 * j];      // a missing second page is fully masked anyway
            }
#pragma unroll
            for (int v = 0; v < 2; ++v) {
                const int jt = j - v;                                     // tile loaded: K of j, V of j - 1
                if (jt < 0 || jt >= n_kvt) continue;
                const int st = jt & 1;
                uint64_t* full = (v ? v_full : k_full) + st;
                mbar_wait((v ? v_empty : k_empty) + st, (((uint32_t)jt >> 1) & 1) ^ 1);
                if (elect_one()) {
                    uint8_t* dst = kv_s + st * Cfg::STAGE_BYTES + (v ? Cfg::KV_BYTES : 0);
                    mbar_expect_tx(full, Cfg::KV_BYTES);
#pragma unroll
                    for (int pg = 0; pg < 2; ++pg) {
                        const int64_t row = layer_row0 + ((int64_t)(v ? prev[pg] : page[pg]) * p.n_kv + kvh) * 64 + (v ? kv_stride_rows : 0);
#pragma unroll
                        for (int h = 0; h < HALVES; ++h)
                            tma_load_2d(dst + h * Cfg::HALF_BYTES + pg * 8192, &tm_kv, full, h * 64, (int32_t)row, kEvictLast);
                    }
                }
                __syncwarp();
            }
        }
    } else if (warp == 1) {
        // The whole warp walks the loop, an elected lane issues: descriptors stay in uniform registers
        constexpr uint32_t idesc_s = umma_idesc_bf16(128, KV_TILE);
        constexpr uint32_t idesc_t = umma_idesc_bf16_bmn(128, D);
        const uint64_t q_desc = umma_desc_sw128(smem_u32(q_s)), k_desc = umma_desc_sw128(smem_u32(kv_s)), p_desc = umma_desc_sw128(smem_u32(p_s));
        const uint64_t v_desc = umma_desc_sw128_mn(smem_u32(kv_s + Cfg::KV_BYTES), (uint32_t)Cfg::HALF_BYTES, 1024u);
        auto issue_s = [&](int j) {
            const int st = j & 1;
            mbar_wait(&k_full[st], ((uint32_t)j >> 1) & 1);
            mbar_wait(&s_empty[st], (((uint32_t)j >> 1) & 1) ^ 1);
            tcgen05_fence_after();
            if (elect_one()) {
                const uint64_t b = k_desc + (uint64_t)(st * (Cfg::STAGE_BYTES >> 4));
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    const uint64_t off = (uint64_t)(((ks >> 2) * Cfg::HALF_BYTES + (ks & 3) * 32) >> 4);
                    umma_bf16(tmem_base + (uint32_t)(st * 128), q_desc + off, b + off, idesc_s, ks > 0 ? 1u : 0u);
                }
                umma_commit(&s_full[st]);
                umma_commit(&k_empty[st]);                                 // K_j is free once S_j exists
            }
            __syncwarp();
        };
        mbar_wait(q_full, 0);
        issue_s(0);
        for (int j = 0; j < n_kvt; ++j) {
            if (j + 1 < n_kvt) issue_s(j + 1);                         // keep the tensor pipe ahead of the softmax warps
            const int st = j & 1;
            mbar_wait(&p_full[st], ((uint32_t)j >> 1) & 1);            // P_j is in shared memory
            mbar_wait(&v_full[st], ((uint32_t)j >> 1) & 1);
            tcgen05_fence_after();
            if (elect_one()) {
                const uint64_t a = p_desc + (uint64_t)(st * (Cfg::P_BYTES >> 4)), b = v_desc + (uint64_t)(st * (Cfg::STAGE_BYTES >> 4));
#pragma unroll
                for (int ks = 0; ks < KV_TILE / 16; ++ks)              // O accumulates over all KV tiles
                    umma_bf16(tmem_base + Cfg::T_COL, a + (uint64_t)(((ks >> 2) * Cfg::HALF_BYTES + (ks & 3) * 32) >> 4), b + (uint64_t)(ks * (2048 >> 4)), idesc_t, (j > 0 || ks > 0) ? 1u : 0u);
                umma_commit(j + 1 < n_kvt ? t_full : o_full);
                umma_commit(&v_empty[st]);
            }
            __syncwarp();
        }
    } else {
        const int q = warp & 3, wg = (warp - 2) >> 2;               // warps w and w + 4 own the same rows (TMEM lanes 32 * (w % 4) ...)
        const int row = q * 32 + lane;                              // query row of this thread inside the tile
        const int qpos = tile.pos0 + row;
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        constexpr int CH = 4 / NWG;                                 // 32-key chunks of a tile this thread handles
        const int key_base = wg * (KV_TILE / NWG);
        constexpr int OC = D / NWG;                                 // O columns this thread rescales / writes
        const int o_base = wg * OC;
        constexpr float kRescaleThreshold = 8.0f;                   // log2 units: p may reach 2^8 before O is rescaled
        float m_ref = -INFINITY, l_run = 0.f, l_other = 0.f, m_run = -INFINITY, m_other = -INFINITY;      // row sums of this tile's parity and of the other, and what they are relative to
        for (int j = 0; j < n_kvt; ++j) {
            const int sb = j & 1;
            mbar_wait(&s_full[sb], ((uint32_t)j >> 1) & 1);
            tcgen05_fence_after();
            uint32_t v[CH][32];
#pragma unroll
            for (int c = 0; c < CH; ++c) tmem_ld_32x32b_x32(tmem_base + lane_addr + (uint32_t)(sb * 128 + key_base + c * 32), v[c]);
            tmem_ld_wait();
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_empty[sb]);               // S_j is in registers: the tensor core may overwrite the buffer
            const bool diag = (j * KV_TILE + KV_TILE - 1) > tile.pos0;          // some (row, key) pairs of this tile are masked
            if (diag) {                                                         // only the last tile(s) of a row block pay for the mask
#pragma unroll
                for (int c = 0; c < CH; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i)
                        if ((j * KV_TILE + key_base + c * 32 + i) > qpos) v[c][i] = 0xff800000u;   // -inf
            }
            float mraw = -INFINITY;                                             // max of the raw scores; the scale is positive
#pragma unroll
            for (int c = 0; c < CH; ++c)
#pragma unroll
                for (int i = 0; i < 32; ++i) mraw = fmaxf(mraw, __uint_as_float(v[c][i]));
            {                                                                   // the row's other half lives in the partner warpgroup
                xch[(sb * 2 + wg) * 128 + row] = mraw;
                asm volatile("bar.sync 2, 256;" ::: "memory");
                mraw = fmaxf(mraw, xch[(sb * 2 + (wg ^ 1)) * 128 + row]);
            }
            const float mx = mraw * p.scale_log2e;
            // lazy rescaling: raise the reference maximum only when a row would overshoot it by more than 2^8
            const bool raise = mx > m_ref + kRescaleThreshold;      // always true on tile 0 (key 0 is visible to every row)
            if (__any_sync(0xffffffffu, raise)) {                   // both warps of a row pair see the same mx, hence take the same branch
                if (j > 0) {
                    mbar_wait(t_full, (uint32_t)(j - 1) & 1);       // O += P_{j-1}·V_{j-1} has landed; O += P_j·V_j is not issued before p_full
                    tcgen05_fence_after();
                    const float alpha = raise ? exp2f(m_ref - mx) : 1.0f;
#pragma unroll 1
                    for (int c = 0; c < OC; c += 32) {
                        uint32_t o[32];
                        tmem_ld_32x32b_x32(tmem_base + lane_addr + Cfg::T_COL + (uint32_t)(o_base + c), o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st_32x32b_x32(tmem_base + lane_addr + Cfg::T_COL + (uint32_t)(o_base + c), o);
                    }
                    tmem_st_wait();
                    tcgen05_fence_before();
                }
                if (raise) m_ref = mx;
            }
            uint8_t* prow = p_s + sb * Cfg::P_BYTES + row * 128;
            uint64_t psum = 0;
            const float neg_ref = -m_ref;                                       // p = 2^(s*scale - m_ref): one FFMA + one SFU op per score
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                float pr[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) pr[i] = ex2_approx(fmaf(__uint_as_float(v[c][i]), p.scale_log2e, neg_ref));
#pragma unroll
                for (int i = 0; i < 32; i += 2) psum = add_f32x2(psum, pack_f32x2(pr[i], pr[i + 1]));
#pragma unroll
                for (int g8 = 0; g8 < 4; ++g8) {                    // four 16-byte chunks (8 keys each)
                    const int key0 = key_base + c * 32 + g8 * 8, hh = key0 >> 6, chunk = (key0 & 63) >> 3;
                    uint4 w;
                    w.x = pack_bf16x2(pr[g8 * 8 + 0], pr[g8 * 8 + 1]); w.y = pack_bf16x2(pr[g8 * 8 + 2], pr[g8 * 8 + 3]);
                    w.z = pack_bf16x2(pr[g8 * 8 + 4], pr[g8 * 8 + 5]); w.w = pack_bf16x2(pr[g8 * 8 + 6], pr[g8 * 8 + 7]);
                    *reinterpret_cast<uint4*>(prow + hh * Cfg::HALF_BYTES + ((chunk ^ (row & 7)) << 4)) = w;
                }
            }
            fence_proxy_async();                                    // P stores must be visible to the tensor-core (async) proxy
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[sb]);
            const float l_new = sum_add(l_run, sum_rescale(m_run, m_ref), psum);
            l_run = l_other; m_run = m_other; l_other = l_new; m_other = m_ref;
        }
        // A barrier of its own: S of the last tile says that all products up to the third last P·V have landed, no more, and with the second last one still
        // under way a wait for the last one's parity on t_full would find the third last one's phase and pass.  (In the loop S_j says that P_{j-2}·V has
        // landed, so the wait for P_{j-1}·V cannot be taken for an earlier one.)
        mbar_wait(o_full, 0);
        tcgen05_fence_after();
        float l_row;
        {                                                           // the two key halves' sums meet, of either parity (every maximum there has been read: P of the last tile stands)
            xch[wg * 128 + row] = __fmul_rn(l_run, sum_rescale(m_run, m_ref));
            xch[(2 + wg) * 128 + row] = l_other;
            asm volatile("bar.sync 2, 256;" ::: "memory");
            l_row = (xch[row] + xch[128 + row]) + (xch[256 + row] + xch[384 + row]);
        }
        const float inv = 1.0f / l_row;
        uint16_t* orow = reinterpret_cast<uint16_t*>(p.out) + (size_t)(tile.q_row0 + q * 32) * p.n_heads * D + (size_t)head * D;
        const uint32_t o_addr = tmem_base + lane_addr + Cfg::T_COL + (uint32_t)o_base;
        if (OC == 64 && tile.n_rows >= q * 32 + 32) store_o_64(p_s + (warp - 2) * 4096, o_addr, inv, orow + o_base, (size_t)p.n_heads * D, lane);      // P has been read by the last product
        else store_o_direct<OC>(o_addr, inv, orow + (size_t)lane * p.n_heads * D + o_base, row < tile.n_rows);
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) { tcgen05_fence_after(); tmem_dealloc<Cfg::TMEM_COLS>(tmem_base); }
}

// ---------------------------------------------------------------------------------------------
// Two heads of one key/value group per CTA, for batches of short query tiles that fill the chip and for odd groups of heads of 128.
//
// One query tile's chain per KV tile — S, maximum, 128 exponentials a row, P, P·V — keeps either the tensor pipe or the softmax warps waiting
// (30 % of the tensor pipe at prompts of 1.5 thousand tokens).  Here a CTA carries the SAME 128 query rows of TWO heads that read the same keys
// and values, each with a softmax warpgroup of its own: while warpgroup A works on S_A, the tensor core runs P_B·V and the next S_B.  The heads
// see the same keys, so both take the same number of KV tiles, and a K / V tile is fetched once for both.  P goes back into TMEM over its own S
// (bf16, columns 0..63 of the 128) and is the A operand of P·V from there: no shared-memory round trip, and shared memory holds Q of both heads
// and two K and two V tiles.  tcgen05.mma of one thread run in order, so S_X(j+1) may be issued right behind P_X(j)·V: it overwrites P_X(j)
// after that has been read, and its completion says that O_X has landed, which is all that rescaling O_X needs.
// Persistent: one CTA per SM walks (row tile, head pair) items, heaviest first, every second round in reverse; the ring keeps loading across
// items and one warpgroup's output is written under the other's last products.
//   warp 0    : TMA (K, Q, V)        warp 1 : tcgen05.mma        warps 4-7 / 8-11 : softmax and output of head A / B, one query row per thread
// A group with an odd number of heads leaves its last one alone in an item (warpgroup B idles).
// A row's scores, reference maxima, probabilities and sums are those of the kernel above, in its order: which of the two a batch takes moves no bit.
// Measured against the kernel above: 4096 rows behind 12288 cached ones, 64 / 8 heads of 128: 1664 -> 1348 us in a burst; five prompts of 1.4 thousand rows,
// 32 / 8 heads: 147 -> 95 us (40 / 8: 180 -> 129).  Before two probabilities an addition, 1963 -> 1416 and 184 -> 102; of that: the issuing warp stays converged (behind one lane its 32 products a tile pair took longer than the tensor core
// has for them): 1548 -> 1489 and 120 -> 114 us; P is handed over in two parts, so that the first 64 keys are multiplied under the other exponentials:
// -> 1417 and 108 us (three or four parts, or loading S in two halves under the maxima: no difference); O leaves in whole lines and the next item
// is read under the last product: -> 1416 and 102 us.  What bounds it is a head's chain in a tile, 2900 cycles then: 125 to fetch S, 275 for the
// maximum, 1500 for 128 exponentials a row (1024 alone on the special-function units, which the other head's overlap in part), 970 for the rest of P·V
// and the next S.  Tensor and special-function pipes are busy 65 to 70 % of it, and a long loop runs into the 1000 W cap.  Taking exponentials from a reference
// that may still rise, moving an eighth or a quarter of them to the FMA pipe and two threads per row were each 3 to 12 % slower.
// ---------------------------------------------------------------------------------------------
template <int D>
struct PtpCfg {
    static constexpr int HALVES = D / 64;
    static constexpr int HALF_BYTES = 128 * 128;
    static constexpr int TILE_BYTES = HALVES * HALF_BYTES;       // Q of one head, K or V of one 128-token tile
    static constexpr int STAGES = 2;
    static constexpr int OUT_BYTES = D == 128 ? 8 * 4096 : 0;    // what a softmax warp writes its rows of O through
    static constexpr int SMEM_BYTES = (2 + 2 * STAGES) * TILE_BYTES + OUT_BYTES + 256;
    static_assert(SMEM_BYTES <= 232448, "shared memory budget of one CTA");
    static constexpr uint32_t TMEM_COLS = 512;
    static constexpr uint32_t S_COL = 0, O_COL = 256;            // S_A, S_B (P over them), then O_A, O_B: 128 columns each
    static constexpr int THREADS = 3 * 128;
};

struct PtpItem { PrefillTile tile; int head, two, n_kvt; };
// item of this CTA in round r: rounds alternate direction, so that no CTA gets the heaviest item of every round
OA_DEVINL bool ptp_item(const PrefillAttnParams& p, int pairs_per_group, int round, PtpItem& it) {
    const int G = (int)gridDim.x, n_items = p.n_tiles * p.n_kv * pairs_per_group;
    const int idx = round * G + ((round & 1) ? G - 1 - (int)blockIdx.x : (int)blockIdx.x);
    if (idx >= n_items) return false;
    const int per_tile = p.n_kv * pairs_per_group, ti = idx / per_tile, hp = idx - ti * per_tile;
    const int kvh = hp / pairs_per_group, pr = hp - kvh * pairs_per_group, grp = p.n_heads / p.n_kv;
    it.tile = p.tiles[ti];
    it.head = kvh * grp + 2 * pr;
    it.two = 2 * pr + 1 < grp;
    it.n_kvt = (it.tile.pos0 + it.tile.n_rows + KV_TILE - 1) / KV_TILE;
    return true;
}

template <int D>
__global__ void __launch_bounds__(PtpCfg<D>::THREADS, 1) prefill_attention_pair_kernel(const __grid_constant__ CUtensorMap tm_q,
                                                                                       const __grid_constant__ CUtensorMap tm_kv,
                                                                                       const PrefillAttnParams p, const int64_t layer_row0,
                                                                                       const int64_t kv_stride_rows) {
    using Cfg = PtpCfg<D>;
    constexpr int HALVES = Cfg::HALVES, STAGES = Cfg::STAGES;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* q_s = smem_raw;                                     // [2 heads]
    uint8_t* k_s = q_s + 2 * Cfg::TILE_BYTES;                    // [STAGES]
    uint8_t* v_s = k_s + STAGES * Cfg::TILE_BYTES;               // [STAGES]
    uint8_t* out_s = v_s + STAGES * Cfg::TILE_BYTES;             // [8 warps]
    uint64_t* bars = reinterpret_cast<uint64_t*>(out_s + Cfg::OUT_BYTES);
    uint64_t* q_full = bars;                  // 1
    uint64_t* q_empty = bars + 1;             // 1
    uint64_t* k_full = bars + 2;              // [STAGES]
    uint64_t* k_empty = k_full + STAGES;
    uint64_t* v_full = k_empty + STAGES;
    uint64_t* v_empty = v_full + STAGES;
    uint64_t* s_full = v_empty + STAGES;      // [2 heads]
    uint64_t* p_full = s_full + 2;            // [2 heads][lower, upper 64 keys]
    uint64_t* o_full = p_full + 4;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + 2);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // warp: uniform, and known to be
    const int grp = p.n_heads / p.n_kv, ppg = (grp + 1) / 2;
    PtpItem it;

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_kv);
        mbar_init(q_full, 1); mbar_init(q_empty, 1);
        for (int i = 0; i < STAGES; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&p_full[2 * i], 4); mbar_init(&p_full[2 * i + 1], 4); mbar_init(&o_full[i], 1); }
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc<Cfg::TMEM_COLS>(tmem_slot);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    griddep_launch();

    // registers: 384 x 168 at launch = 128 x (88 + 208 + 208)
    if (warp < 4) {
        reg_dec<88>();
        if (warp == 0) {
            griddep_wait();
            uint32_t kc = 0;
            PtpItem next;
            bool more = ptp_item(p, ppg, 0, it);
            for (int r = 0; more; ++r, it = next) {
                const int n_kvt = __shfl_sync(0xffffffffu, it.n_kvt, 0);
                const int32_t* bt = p.block_tables + (size_t)it.tile.seq * p.max_pages_per_seq;
                const int kvh = it.head / grp;
                auto page_row = [&](int pi, int fallback) { return layer_row0 + ((int64_t)bt[pi < p.max_pages_per_seq ? pi : fallback] * p.n_kv + kvh) * 64; };   // a missing second page is fully masked anyway
                auto load = [&](uint8_t* dst, uint64_t* bar, int64_t r0, int64_t r1) {
                    mbar_expect_tx(bar, Cfg::TILE_BYTES);
#pragma unroll
                    for (int h = 0; h < HALVES; ++h) {
                        tma_load_2d(dst + h * Cfg::HALF_BYTES, &tm_kv, bar, h * 64, (int32_t)r0, kEvictLast);
                        tma_load_2d(dst + h * Cfg::HALF_BYTES + 8192, &tm_kv, bar, h * 64, (int32_t)r1, kEvictLast);
                    }
                };
                int64_t r0 = page_row(0, 0), r1 = page_row(1, 0);
                for (int j = 0; j < n_kvt; ++j, ++kc) {
                    const uint32_t st = kc % STAGES, ph = (kc / STAGES) & 1;
                    mbar_wait(&k_empty[st], ph ^ 1);
                    if (elect_one()) load(k_s + st * Cfg::TILE_BYTES, &k_full[st], r0, r1);
                    __syncwarp();
                    if (j == 0) {
                        mbar_wait(q_empty, ((uint32_t)r & 1) ^ 1);
                        if (elect_one()) {
                            mbar_expect_tx(q_full, (it.two ? 2 : 1) * Cfg::TILE_BYTES);
                            for (int x = 0; x <= it.two; ++x)
#pragma unroll
                                for (int h = 0; h < HALVES; ++h)
                                    tma_load_2d(q_s + x * Cfg::TILE_BYTES + h * Cfg::HALF_BYTES, &tm_q, q_full, (it.head + x) * D + h * 64, it.tile.q_row0, kEvictFirst);
                        }
                        __syncwarp();
                        more = ptp_item(p, ppg, r + 1, next);                  // read now, needed an item later
                    }
                    int64_t n0 = r0, n1 = r1;                                  // the next tile's pages are looked up while this one's slot is waited for
                    if (j + 1 < n_kvt) { n0 = page_row(2 * j + 2, 0); n1 = page_row(2 * j + 3, 2 * j + 2); }
                    mbar_wait(&v_empty[st], ph ^ 1);
                    if (elect_one()) load(v_s + st * Cfg::TILE_BYTES, &v_full[st], r0 + kv_stride_rows, r1 + kv_stride_rows);
                    __syncwarp();
                    r0 = n0; r1 = n1;
                }
            }
        } else if (warp == 1) {
            // The whole warp walks the loop, an elected lane issues: descriptors stay in uniform registers
            constexpr uint32_t idesc_s = umma_idesc_bf16(128, KV_TILE), idesc_o = umma_idesc_bf16_bmn(128, D);
            const uint64_t q_desc = umma_desc_sw128(smem_u32(q_s)), k_desc = umma_desc_sw128(smem_u32(k_s)), v_desc = umma_desc_sw128_mn(smem_u32(v_s), (uint32_t)Cfg::HALF_BYTES, 1024u);
            constexpr uint64_t TILE = Cfg::TILE_BYTES >> 4;                    // in a descriptor's address units
            uint32_t kc = 0, vc = 0, pc[2] = {0, 0};                           // K / V tiles taken, P tiles taken per head
            auto issue_s = [&](int x) {                                        // S_x = Q_x K^T with K tile kc
                const uint64_t a = q_desc + x * TILE, b = k_desc + (kc % STAGES) * TILE;
#pragma unroll
                for (int ks = 0; ks < D / 16; ++ks) {
                    const uint64_t off = (uint64_t)(((ks >> 2) * Cfg::HALF_BYTES + (ks & 3) * 32) >> 4);
                    umma_bf16(tmem_base + Cfg::S_COL + x * 128, a + off, b + off, idesc_s, ks > 0 ? 1u : 0u);
                }
                umma_commit(&s_full[x]);
            };
            auto issue_o = [&](int x, int half, bool first) {                  // O_x (+)= P_x V with 64 keys of V tile vc
                const uint64_t b = v_desc + (vc % STAGES) * TILE;
#pragma unroll
                for (int k4 = 0; k4 < KV_TILE / 32; ++k4) {
                    const int ks = half * (KV_TILE / 32) + k4;
                    umma_bf16_ta(tmem_base + Cfg::O_COL + x * 128, tmem_base + Cfg::S_COL + x * 128 + ks * 8, b + (uint64_t)(ks * (2048 >> 4)), idesc_o, (!first || ks > 0) ? 1u : 0u);
                }
            };
            PtpItem next;
            bool more = ptp_item(p, ppg, 0, it);
            for (int r = 0; more; ++r, it = next) {
                const int n_kvt = __shfl_sync(0xffffffffu, it.n_kvt, 0);
                mbar_wait(q_full, (uint32_t)r & 1);
                mbar_wait(&k_full[kc % STAGES], (kc / STAGES) & 1);
                tcgen05_fence_after();
                if (elect_one()) {
                    issue_s(0);
                    if (it.two) issue_s(1);
                    umma_commit(&k_empty[kc % STAGES]);
                    if (n_kvt == 1) umma_commit(q_empty);
                }
                __syncwarp();
                ++kc;
                more = ptp_item(p, ppg, r + 1, next);                          // read now, needed an item later
                for (int j = 0; j < n_kvt; ++j) {
                    const bool last = j + 1 == n_kvt;
                    mbar_wait(&v_full[vc % STAGES], (vc / STAGES) & 1);
                    if (!last) mbar_wait(&k_full[kc % STAGES], (kc / STAGES) & 1);
#pragma unroll
                    for (int x = 0; x < 2; ++x) {
                        if (x > it.two) break;
                        mbar_wait(&p_full[2 * x], pc[x] & 1);
                        tcgen05_fence_after();
                        if (elect_one()) issue_o(x, 0, j == 0);
                        __syncwarp();
                        mbar_wait(&p_full[2 * x + 1], pc[x] & 1); ++pc[x];
                        tcgen05_fence_after();
                        if (elect_one()) {
                            issue_o(x, 1, j == 0);
                            if (last) umma_commit(&o_full[x]); else issue_s(x);
                        }
                        __syncwarp();
                    }
                    if (elect_one()) {
                        umma_commit(&v_empty[vc % STAGES]);
                        if (!last) {
                            umma_commit(&k_empty[kc % STAGES]);
                            if (j + 2 == n_kvt) umma_commit(q_empty);          // the item's last S: the next item's Q may come
                        }
                    }
                    __syncwarp();
                    ++vc;
                    if (!last) ++kc;
                }
            }
        }
    } else {
        reg_inc<208>();
        const int q = warp & 3, x = (warp - 4) >> 2;                // TMEM lanes 32 q ..; head A or B of the item
        const int row = q * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(q * 32) << 16;
        const uint32_t s_addr = tmem_base + lane_addr + Cfg::S_COL + x * 128, o_addr = tmem_base + lane_addr + Cfg::O_COL + x * 128;
        constexpr float kRescaleThreshold = 8.0f;                   // log2 units: p may reach 2^8 before O is rescaled
        const uint64_t scale2 = pack_f32x2(p.scale_log2e, p.scale_log2e);
        griddep_wait();                                             // the output may still be read by a predecessor
        uint32_t sc = 0, oc = 0;                                    // S tiles and items this warpgroup has taken
        bool more = ptp_item(p, ppg, 0, it);
        for (int r = 0; more; ++r) {
            if (x > it.two) { more = ptp_item(p, ppg, r + 1, it); continue; }
            const int qpos = it.tile.pos0 + row;
            float m_ref = -INFINITY, l_lo = 0.f, l_hi = 0.f, m_run = -INFINITY;                   // row sums of the lower and upper 64 keys, tiles of this one's parity
            float o_lo = 0.f, o_hi = 0.f, m_other = -INFINITY;                                    // and of the other
            for (int j = 0; j < it.n_kvt; ++j, ++sc) {
                mbar_wait(&s_full[x], sc & 1);
                tcgen05_fence_after();
                uint32_t v[4][32];
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(s_addr + (uint32_t)(c * 32), v[c]);
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_ld_wait_for(v[c]);
                if (j * KV_TILE + KV_TILE - 1 > it.tile.pos0) {                     // some (row, key) pairs of this tile are masked
#pragma unroll
                    for (int c = 0; c < 4; ++c)
#pragma unroll
                        for (int i = 0; i < 32; ++i) if (j * KV_TILE + c * 32 + i > qpos) v[c][i] = 0xff800000u;
                }
                float m[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    m[k] = __uint_as_float(v[0][k]);
#pragma unroll
                    for (int i = 4; i < 124; i += 8) m[k] = fmax3_nan(m[k], __uint_as_float(v[(i + k) / 32][(i + k) % 32]), __uint_as_float(v[(i + k + 4) / 32][(i + k + 4) % 32]));
                    m[k] = fmax_nan(m[k], __uint_as_float(v[3][28 + k]));
                }
                const float mx = fmax_nan(fmax3_nan(m[0], m[1], m[2]), m[3]) * p.scale_log2e;       // the scale is positive
                // always true on tile 0 (key 0 is visible to every row); also where a score is NaN: then m_ref, every p and the row's result are
                const bool raise = !(mx <= m_ref + kRescaleThreshold);
                if (__any_sync(0xffffffffu, raise)) {
                    if (j > 0) {                                    // S_j has completed, so P_{j-1} V has: O holds every tile before this one
                        const float alpha = raise ? exp2f(m_ref - mx) : 1.0f;
#pragma unroll 1
                        for (int c = 0; c < D; c += 16) {
                            uint32_t o[16];
                            tmem_ld_32x32b_x16(o_addr + (uint32_t)c, o);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                            tmem_st_32x32b_x16(o_addr + (uint32_t)c, o);
                        }
                    }
                    if (raise) m_ref = mx;
                }
                const uint64_t nref2 = pack_f32x2(-m_ref, -m_ref);
                uint64_t sum[2] = {0, 0};                           // the two halves' sums of even and odd keys
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {                    // 64 scores -> 32 columns of P: p = 2^(s * scale - m_ref); handed over as soon as they stand
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        uint32_t pw[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            float p0, p1;
                            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[2 * hf + c][2 * i]), __uint_as_float(v[2 * hf + c][2 * i + 1])), scale2, nref2), p0, p1);
                            p0 = ex2_approx(p0); p1 = ex2_approx(p1);
                            pw[i] = pack_bf16x2(p0, p1);
                            sum[hf] = add_f32x2(sum[hf], pack_f32x2(p0, p1));
                        }
                        tmem_st_32x32b_x16(s_addr + (uint32_t)((2 * hf + c) * 16), pw);
                    }
                    tmem_st_wait();
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&p_full[2 * x + hf]);
                }
                const float f = sum_rescale(m_run, m_ref), n_lo = sum_add(l_lo, f, sum[0]), n_hi = sum_add(l_hi, f, sum[1]);
                l_lo = o_lo; l_hi = o_hi; m_run = m_other; o_lo = n_lo; o_hi = n_hi; m_other = m_ref;
            }
            PtpItem next;
            more = ptp_item(p, ppg, r + 1, next);                   // read under the item's last product, needed after its output
            mbar_wait(&o_full[x], oc & 1); ++oc;
            tcgen05_fence_after();
            const float f = sum_rescale(m_run, m_ref);
            const float inv = 1.0f / ((__fmul_rn(l_lo, f) + __fmul_rn(l_hi, f)) + (o_lo + o_hi));
            uint16_t* orow = reinterpret_cast<uint16_t*>(p.out) + (size_t)(it.tile.q_row0 + q * 32) * p.n_heads * D + (size_t)(it.head + x) * D;
            // a warp with rows missing: their pieces are few (sixteen prompts of 30 rows: 11.1 us against 12.7 through shared memory)
            if (D == 64 || it.tile.n_rows < q * 32 + 32) store_o_direct<D>(o_addr, inv, orow + (size_t)lane * p.n_heads * D, row < it.tile.n_rows);
            else {
#pragma unroll 1
                for (int c = 0; c < D; c += 64) store_o_64(out_s + (warp - 4) * 4096, o_addr + (uint32_t)c, inv, orow + c, (size_t)p.n_heads * D, lane);
            }
            it = next;
            tcgen05_fence_before();                                 // O has been read before this warp's next p_full lets P·V overwrite it
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) { tcgen05_fence_after(); tmem_dealloc<Cfg::TMEM_COLS>(tmem_base); }
}

// ---------------------------------------------------------------------------------------------
// Softmax warpgroups that take a head's key tiles in turn: heads of 128 on a CTA PAIR (two heads of one key/value group), heads of 64 on a CTA.
//
// The kernel above is bound by a head's chain in a tile: its S may only be computed once the P that stands over the last one has been multiplied, and TMEM has
// no room for a second S of two heads.  Here a CTA carries ONE head's 128 rows, so TMEM holds three S tiles and O, and the two softmax
// warpgroups take the tiles in turn: while one takes the exponentials of tile t, the other fetches S and finds the maxima of t + 1, and the tensor core
// runs P V of t - 1 and S of t + 2.  What a head still does in order is one value a row: a tile's reference maximum follows from the last one's, so it goes from
// warpgroup to warpgroup as soon as the maxima stand.  With heads of 128 a CTA alone would fetch 64 KB of keys and values a tile, in 1300 cycles: what the L2 gives
// (32 / 8 heads: five prompts of 1.4 thousand rows 139 us against 97 above, 1400 rows behind 3000 123 against 96).  So two heads' CTAs share them: a product is 256 x 128 x 16
// (cta_group::2) with half of B in each CTA, and each loads one of a tile's two K pages and 64 of V's 128 columns.  Heads of 64 need half the bytes and no pair.
//   warp 0     : TMA: this CTA's Q (two items ahead), its share of K and V       warp 1 (of a pair: the even CTA's): tcgen05.mma
//   warps 4-11 : softmax of even and odd tiles, one query row per thread         warps 12-15: output, while the next item's tiles run
// A row's sums are kept per warpgroup (even and odd tiles of the item) and joined at its end, as in the kernels above: the same bits.
// us, kernels alone, two heads a CTA -> here: 4096 rows behind 12288, 64 / 8 heads of 128 1348 -> 1291; five prompts of 1.4 thousand rows, 32 / 8 heads of 128 95 -> 87;
// 1000 rows behind 6000 100 -> 89; 600 rows 14.7 -> 11.2 (one head a CTA: 14.7); 300 rows behind 6000 57 -> 46 (one head a CTA).  A pair's launch costs 2 us more.
// Heads of 64: the five prompts 87 -> 78, 1400 rows behind 3000 94 -> 73, 600 rows 13.0 -> 8.9, 100 rows behind 3000 29.9 (one head a CTA) -> 22.7.
// What bounds it now (128): a warpgroup takes 2600 cycles a tile, 1650 of them exponentials (1024 alone), 550 fetching S, the maxima and the reference, 120 waiting
// for S; tensor and special-function pipes are busy 79 %, and the clock is down to 1.6 GHz in the long case (1.76 in the short ones).
// What crosses the pair stands in TMEM, ordered by tcgen05.fence, or comes by TMA: arrivals and waits for TMEM are relaxed, of cluster scope; only the loading and the issuing
// warp acquire.  With the softmax warps' arrivals as releases a tile took 2100 cycles instead of 1300: each waits for its thread's stores.  Slower: S of two tiles and P of two in places of their own, S issued as soon as it is fetched (84 -> 90 us),
// P handed over in two halves (85.5); no faster: the first item and its pages looked up ahead of the set-up.
// ---------------------------------------------------------------------------------------------
template <int D, int CTAS>
struct PcpCfg {
    static_assert(CTAS == 1 || D == 128, "a pair's V halves are 64 columns each");
    static constexpr int S_BUFS = 3;
    static constexpr int Q_BYTES = 128 * D * 2, Q_HALF = 128 * 128;
    static constexpr int KV_BYTES = 128 / CTAS * D * 2, K_HALF = 128 / CTAS * 128;      // a CTA's share of a K or V tile of 128 keys (of a pair: 64 keys x 128, 128 keys x 64 columns)
    static constexpr int STAGES = 4;                                     // of 16 KB each
    static constexpr int OUT_WARP_BYTES = 32 * D * 2;
    static constexpr int ROWS_BYTES = 2 * 128 * 4;                       // one value per row and softmax warpgroup
    static constexpr int SMEM_BYTES = 2 * Q_BYTES + 2 * STAGES * KV_BYTES + 4 * OUT_WARP_BYTES + 2 * ROWS_BYTES + 512;
    static_assert(SMEM_BYTES <= 232448, "shared memory budget of one CTA");
    static constexpr uint32_t O_COL = S_BUFS * 128;
    static constexpr int THREADS = 4 * 128;
    static constexpr int REGS_CONTROL = 64, REGS_OUT = 64, REGS_SOFTMAX = 192;
    static_assert(REGS_CONTROL + REGS_OUT + 2 * REGS_SOFTMAX <= 4 * 128, "an increase draws on what the launch gave: 512 threads x 128 registers");
};

// item of this CTA or pair in round r (as above: heaviest first, every second round in reverse)
struct PcpItem { PrefillTile tile; int kvh, head0, n_kvt; };
template <int CTAS>
OA_DEVINL bool pcp_item(const PrefillAttnParams& p, int grp, int round, PcpItem& it) {
    const int G = (int)gridDim.x / CTAS, me = (int)blockIdx.x / CTAS, per_tile = p.n_heads / CTAS;
    const int idx = round * G + ((round & 1) ? G - 1 - me : me);
    if (idx >= p.n_tiles * per_tile) return false;
    const int ti = idx / per_tile;
    it.head0 = (idx - ti * per_tile) * CTAS;
    it.kvh = it.head0 / grp;
    it.tile = p.tiles[ti];
    it.n_kvt = (it.tile.pos0 + it.tile.n_rows + KV_TILE - 1) / KV_TILE;
    return true;
}

template <int D, int CTAS>
__global__ void __launch_bounds__(PcpCfg<D, CTAS>::THREADS, 1) prefill_attention_turns_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_kv,
                                                                                              const PrefillAttnParams p, const int64_t layer_row0, const int64_t kv_stride_rows) {
    using Cfg = PcpCfg<D, CTAS>;
    constexpr int STAGES = Cfg::STAGES, HALVES = D / 64;
    constexpr bool PAIR = CTAS == 2;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* q_s = smem_raw;                                     // [item & 1]
    uint8_t* k_s = q_s + 2 * Cfg::Q_BYTES;                       // [STAGES]
    uint8_t* v_s = k_s + STAGES * Cfg::KV_BYTES;                 // [STAGES]
    uint8_t* out_s = v_s + STAGES * Cfg::KV_BYTES;               // [4 warps]
    float* sum_s = reinterpret_cast<float*>(out_s + 4 * Cfg::OUT_WARP_BYTES);      // [warpgroup][row]: row sums of the item at hand
    float* ref_s = sum_s + 2 * 128;                              // [warpgroup][row]: reference maximum after the warpgroup's last tile
    uint64_t* bars = reinterpret_cast<uint64_t*>(ref_s + 2 * 128);
    uint64_t* q_full = bars;                  // [2]  even CTA
    uint64_t* q_empty = q_full + 2;           // [2]
    uint64_t* k_full = q_empty + 2;           // [STAGES]  even CTA
    uint64_t* k_empty = k_full + STAGES;
    uint64_t* v_full = k_empty + STAGES;      // [STAGES]  even CTA
    uint64_t* v_empty = v_full + STAGES;      // [STAGES]  also: P V of this tile has landed
    uint64_t* s_full = v_empty + STAGES;      // [6]  two per buffer: every one is waited for by one warpgroup alone, phase by phase
    uint64_t* p_full = s_full + 6;            // [S_BUFS]  even CTA
    uint64_t* r_full = p_full + Cfg::S_BUFS;  // [2 warpgroups][4 warps]  a warp's reference maxima stand
    uint64_t* l_full = r_full + 8;            // the item's row sums stand
    uint64_t* l_empty = l_full + 1;           // ... and have been read
    uint64_t* o_full = l_empty + 1;           // the item's last P V has landed
    uint64_t* o_empty = o_full + 1;           // even CTA: O has been read in both
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_empty + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // warp: uniform, and known to be
    const uint32_t rank = PAIR ? gp_rank() : 0;
    const int grp = p.n_heads / p.n_kv;
    // barriers that the pair shares: of loads and freed shared memory, and of what stands in TMEM
    auto wait_smem = [&](uint64_t* bar, uint32_t parity) { if (PAIR) gp_wait(bar, parity); else mbar_wait(bar, parity); };
    auto wait_tmem = [&](uint64_t* bar, uint32_t parity) { if (PAIR) gp_wait_tmem(bar, parity); else mbar_wait(bar, parity); };
    auto arrive_even = [&](uint64_t* bar) { if (PAIR) gp_arrive_tmem(gp_mapa(bar, 0)); else mbar_arrive(bar); };
    PcpItem it;

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tm_q); tma_prefetch_desc(&tm_kv);
        for (int i = 0; i < 2; ++i) { mbar_init(&q_full[i], 1); mbar_init(&q_empty[i], 1); }
        for (int i = 0; i < STAGES; ++i) { mbar_init(&k_full[i], 1); mbar_init(&k_empty[i], 1); mbar_init(&v_full[i], 1); mbar_init(&v_empty[i], 1); }
        for (int i = 0; i < 6; ++i) mbar_init(&s_full[i], 1);
        for (int i = 0; i < Cfg::S_BUFS; ++i) mbar_init(&p_full[i], 4 * CTAS);
        for (int i = 0; i < 8; ++i) mbar_init(&r_full[i], 1);
        mbar_init(l_full, 8); mbar_init(l_empty, 4); mbar_init(o_full, 1); mbar_init(o_empty, 4 * CTAS);
        fence_barrier_init();
    }
    if (warp == 1) {
        if (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else tmem_alloc<512>(tmem_slot);
    }
    tcgen05_fence_before();
    __syncthreads();
    if (PAIR) gp_cluster_sync();                     // the other CTA's barriers are initialised before anything arrives on them
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    griddep_launch();

    if (warp < 4) {
        reg_dec<Cfg::REGS_CONTROL>();
        if (warp == 0) {
            griddep_wait();
            uint32_t kc = 0;
            int r = 0;
            PcpItem next;
            bool more = pcp_item<CTAS>(p, grp, 0, it);
            for (; more; ++r, it = next) {
                const int n_kvt = __shfl_sync(0xffffffffu, it.n_kvt, 0);
                const int32_t* bt = p.block_tables + (size_t)it.tile.seq * p.max_pages_per_seq;
                auto page_row = [&](int pi, int fallback) { return layer_row0 + ((int64_t)bt[pi < p.max_pages_per_seq ? pi : fallback] * p.n_kv + it.kvh) * 64; };   // a missing second page is fully masked anyway
                int64_t r0 = page_row(0, 0), r1 = page_row(1, 0);
                for (int j = 0; j < n_kvt; ++j, ++kc) {
                    const uint32_t st = kc % STAGES, ph = (kc / STAGES) & 1;
                    wait_smem(&k_empty[st], ph ^ 1);
                    if (elect_one()) {
                        uint8_t* dst = k_s + st * Cfg::KV_BYTES;
                        if (rank == 0) mbar_expect_tx(&k_full[st], CTAS * Cfg::KV_BYTES);           // both CTAs' shares
                        if (PAIR) {
                            const uint32_t bar = gp_mapa(&k_full[st], 0);
                            const int32_t row = (int32_t)(rank ? r1 : r0);
                            gp_tma_load(dst, &tm_kv, bar, 0, row, kEvictLast);
                            gp_tma_load(dst + Cfg::K_HALF, &tm_kv, bar, 64, row, kEvictLast);
                        } else
#pragma unroll
                            for (int h = 0; h < HALVES; ++h) {
                                tma_load_2d(dst + h * Cfg::K_HALF, &tm_kv, &k_full[st], h * 64, (int32_t)r0, kEvictLast);
                                tma_load_2d(dst + h * Cfg::K_HALF + 8192, &tm_kv, &k_full[st], h * 64, (int32_t)r1, kEvictLast);
                            }
                    }
                    __syncwarp();
                    if (j == 0) {
                        const int qb = r & 1;
                        wait_smem(&q_empty[qb], (((uint32_t)r >> 1) & 1) ^ 1);
                        if (elect_one()) {
                            uint8_t* dst = q_s + qb * Cfg::Q_BYTES;
                            if (rank == 0) mbar_expect_tx(&q_full[qb], CTAS * Cfg::Q_BYTES);
                            const int32_t col = (it.head0 + (int)rank) * D;
#pragma unroll
                            for (int h = 0; h < HALVES; ++h) {
                                if (PAIR) gp_tma_load(dst + h * Cfg::Q_HALF, &tm_q, gp_mapa(&q_full[qb], 0), col + h * 64, it.tile.q_row0, kEvictFirst);
                                else tma_load_2d(dst + h * Cfg::Q_HALF, &tm_q, &q_full[qb], col + h * 64, it.tile.q_row0, kEvictFirst);
                            }
                        }
                        __syncwarp();
                        more = pcp_item<CTAS>(p, grp, r + 1, next);                  // read now, needed an item later
                    }
                    int64_t n0 = r0, n1 = r1;                                  // the next tile's pages are looked up while this one's slot is waited for
                    if (j + 1 < n_kvt) { n0 = page_row(2 * j + 2, 0); n1 = page_row(2 * j + 3, 2 * j + 2); }
                    wait_smem(&v_empty[st], ph ^ 1);
                    if (elect_one()) {
                        uint8_t* dst = v_s + st * Cfg::KV_BYTES;
                        if (rank == 0) mbar_expect_tx(&v_full[st], CTAS * Cfg::KV_BYTES);
                        if (PAIR) {
                            const uint32_t bar = gp_mapa(&v_full[st], 0);
                            gp_tma_load(dst, &tm_kv, bar, (int)rank * 64, (int32_t)(r0 + kv_stride_rows), kEvictLast);
                            gp_tma_load(dst + 8192, &tm_kv, bar, (int)rank * 64, (int32_t)(r1 + kv_stride_rows), kEvictLast);
                        } else
#pragma unroll
                            for (int h = 0; h < HALVES; ++h) {
                                tma_load_2d(dst + h * 16384, &tm_kv, &v_full[st], h * 64, (int32_t)(r0 + kv_stride_rows), kEvictLast);
                                tma_load_2d(dst + h * 16384 + 8192, &tm_kv, &v_full[st], h * 64, (int32_t)(r1 + kv_stride_rows), kEvictLast);
                            }
                    }
                    __syncwarp();
                    r0 = n0; r1 = n1;
                }
            }
            for (int i = 0; i < STAGES; ++i, ++kc) { wait_smem(&k_empty[kc % STAGES], ((kc / STAGES) & 1) ^ 1); wait_smem(&v_empty[kc % STAGES], ((kc / STAGES) & 1) ^ 1); }   // the last
            for (int i = 0; i < 2; ++i, ++r) wait_smem(&q_empty[r & 1], (((uint32_t)r >> 1) & 1) ^ 1);                  // releases have arrived here before the CTA may go
        } else if (warp == 1 && rank == 0) {
            // The whole warp walks the loop, an elected lane issues: descriptors stay in uniform registers.  S runs two tiles ahead of P V, across items.
            constexpr uint32_t idesc_s = umma_idesc_bf16(128 * CTAS, KV_TILE), idesc_o = umma_idesc_bf16_bmn(128 * CTAS, D);
            auto commit = [&](uint64_t* bar) { if (PAIR) gp_commit(bar); else umma_commit(bar); };
            const uint64_t q_desc = umma_desc_sw128(smem_u32(q_s)), k_desc = umma_desc_sw128(smem_u32(k_s)), v_desc = umma_desc_sw128_mn(smem_u32(v_s), 16384u, 1024u);
            PcpItem s_it, nxt;
            uint32_t sc = 0;                                                   // tiles whose S has been issued
            int s_r = 0, s_j = 0;
            bool s_more = pcp_item<CTAS>(p, grp, 0, s_it);
            int s_n = s_more ? __shfl_sync(0xffffffffu, s_it.n_kvt, 0) : 0;
            auto issue_s = [&] {
                if (!s_more) return;
                if (s_j == 0) wait_smem(&q_full[s_r & 1], ((uint32_t)s_r >> 1) & 1);
                const uint32_t st = sc % STAGES;
                wait_smem(&k_full[st], (sc / STAGES) & 1);
                tcgen05_fence_after();
                if (elect_one()) {
                    const uint64_t a = q_desc + (uint64_t)((s_r & 1) * (Cfg::Q_BYTES >> 4)), b = k_desc + (uint64_t)(st * (Cfg::KV_BYTES >> 4));
                    const uint32_t d = tmem_base + (sc % Cfg::S_BUFS) * 128;
#pragma unroll
                    for (int ks = 0; ks < D / 16; ++ks) {
                        const uint64_t ak = a + (uint64_t)(((ks >> 2) * Cfg::Q_HALF + (ks & 3) * 32) >> 4), bk = b + (uint64_t)(((ks >> 2) * Cfg::K_HALF + (ks & 3) * 32) >> 4);
                        if (PAIR) gp_umma(d, ak, bk, idesc_s, ks > 0 ? 1u : 0u); else umma_bf16(d, ak, bk, idesc_s, ks > 0 ? 1u : 0u);
                    }
                    commit(&s_full[sc % 6]);
                    commit(&k_empty[st]);
                    if (s_j + 1 == s_n) commit(&q_empty[s_r & 1]);
                }
                __syncwarp();
                ++sc;
                if (++s_j == s_n) {
                    s_j = 0; ++s_r;
                    s_more = pcp_item<CTAS>(p, grp, s_r, s_it);
                    s_n = s_more ? __shfl_sync(0xffffffffu, s_it.n_kvt, 0) : 0;
                }
            };
            issue_s(); issue_s();
            uint32_t t = 0;
            bool more = pcp_item<CTAS>(p, grp, 0, it);
            for (int r = 0; more; ++r, it = nxt) {
                const int n_kvt = __shfl_sync(0xffffffffu, it.n_kvt, 0);
                more = pcp_item<CTAS>(p, grp, r + 1, nxt);                           // read now, needed an item later
                for (int j = 0; j < n_kvt; ++j, ++t) {
                    issue_s();                                                 // over the P of tile t - 1, whose product is ahead of it
                    const uint32_t st = t % STAGES;
                    if (j == 0) wait_tmem(o_empty, ((uint32_t)r & 1) ^ 1);       // O of the last item has been read
                    wait_smem(&v_full[st], (t / STAGES) & 1);
                    wait_tmem(&p_full[t % Cfg::S_BUFS], (t / Cfg::S_BUFS) & 1);
                    tcgen05_fence_after();
                    if (elect_one()) {
                        const uint64_t b = v_desc + (uint64_t)(st * (Cfg::KV_BYTES >> 4));
                        const uint32_t a = tmem_base + (t % Cfg::S_BUFS) * 128;
#pragma unroll
                        for (int ks = 0; ks < KV_TILE / 16; ++ks) {
                            if (PAIR) gp_umma_ta(tmem_base + Cfg::O_COL, a + ks * 8, b + (uint64_t)(ks * (2048 >> 4)), idesc_o, (j | ks) != 0 ? 1u : 0u);
                            else umma_bf16_ta(tmem_base + Cfg::O_COL, a + ks * 8, b + (uint64_t)(ks * (2048 >> 4)), idesc_o, (j | ks) != 0 ? 1u : 0u);
                        }
                        commit(&v_empty[st]);
                        if (j + 1 == n_kvt) commit(o_full);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp < 12) {
        reg_inc<Cfg::REGS_SOFTMAX>();
        const int q = warp & 3, w = (warp - 4) >> 2;                // TMEM lanes 32 q ..; this warpgroup takes tiles w, w + 2, .. of all there are
        const int row = q * 32 + lane;
        const uint32_t lane_base = tmem_base + ((uint32_t)(q * 32) << 16), o_addr = lane_base + Cfg::O_COL;
        constexpr float kRescaleThreshold = 8.0f;                   // log2 units: p may reach 2^8 before O is rescaled
        const uint64_t scale2 = pack_f32x2(p.scale_log2e, p.scale_log2e);
        uint32_t t = 0;                                             // tiles so far, of both warpgroups
        auto other_ref = [&] {                                      // the reference maximum after tile t - 1
            mbar_wait(&r_full[(w ^ 1) * 4 + q], ((t - 1) >> 1) & 1);
            return ref_s[(w ^ 1) * 128 + row];
        };
        bool more = pcp_item<CTAS>(p, grp, 0, it);
        for (int r = 0; more; ++r) {
            const int n_kvt = it.n_kvt, pos0 = it.tile.pos0, qpos = pos0 + row;
            more = pcp_item<CTAS>(p, grp, r + 1, it);                     // read now, needed an item later
            float m_own = -INFINITY, l_lo = 0.f, l_hi = 0.f;        // this warpgroup's row sums, relative to 2^m_own
            for (int j = 0; j < n_kvt; ++j, ++t) {
                if ((int)(t & 1) != w) continue;
                const uint32_t s_addr = lane_base + (t % Cfg::S_BUFS) * 128;
                wait_tmem(&s_full[t % 6], (t / 6) & 1);
                tcgen05_fence_after();
                uint32_t v[4][32];
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_ld_32x32b_x32(s_addr + (uint32_t)(c * 32), v[c]);
                const float m_last = j > 0 ? other_ref() : -INFINITY;               // under the loads: it has stood for half a tile's time
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_ld_wait_for(v[c]);
                if (j * KV_TILE + KV_TILE - 1 > pos0 + q * 32) {                    // some (row, key) pairs of this warp are masked
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (j * KV_TILE + c * 32 + 31 > pos0 + q * 32) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) if (j * KV_TILE + c * 32 + i > qpos) v[c][i] = 0xff800000u;
                        }
                }
                float m[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    m[k] = __uint_as_float(v[0][k]);
#pragma unroll
                    for (int i = 4; i < 124; i += 8) m[k] = fmax3_nan(m[k], __uint_as_float(v[(i + k) / 32][(i + k) % 32]), __uint_as_float(v[(i + k + 4) / 32][(i + k + 4) % 32]));
                    m[k] = fmax_nan(m[k], __uint_as_float(v[3][28 + k]));
                }
                const float mx = fmax_nan(fmax3_nan(m[0], m[1], m[2]), m[3]) * p.scale_log2e;       // the scale is positive
                // always true on tile 0 (key 0 is visible to every row); also where a score is NaN: then the reference, every p and the row's result are
                const bool raise = !(mx <= m_last + kRescaleThreshold);
                const float m_ref = raise ? mx : m_last;
                ref_s[w * 128 + row] = m_ref;                       // the other warpgroup has read the last one: it has published since
                __syncwarp();
                if (lane == 0) mbar_arrive(&r_full[w * 4 + q]);
                if (j > 0 && __any_sync(0xffffffffu, raise)) {
                    wait_tmem(&v_empty[(t - 1) % STAGES], ((t - 1) / STAGES) & 1);    // O holds every tile before this one (S_t says that P V of t - 3 has landed: no earlier phase is taken for this)
                    tcgen05_fence_after();
                    const float alpha = raise ? exp2f(m_last - mx) : 1.0f;
#pragma unroll 1
                    for (int c = 0; c < D; c += 16) {
                        uint32_t o[16];
                        tmem_ld_32x32b_x16(o_addr + (uint32_t)c, o);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st_32x32b_x16(o_addr + (uint32_t)c, o);
                    }
                }
                const uint64_t nref2 = pack_f32x2(-m_ref, -m_ref);
                uint64_t sum[2] = {0, 0};                           // the two halves' sums of even and odd keys
#pragma unroll
                for (int c = 0; c < 4; ++c) {                       // 128 scores -> 64 columns of P: p = 2^(s * scale - m_ref)
                    uint32_t pw[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float p0, p1;
                        unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[c][2 * i]), __uint_as_float(v[c][2 * i + 1])), scale2, nref2), p0, p1);
                        p0 = ex2_approx(p0); p1 = ex2_approx(p1);
                        pw[i] = pack_bf16x2(p0, p1);
                        sum[c >> 1] = add_f32x2(sum[c >> 1], pack_f32x2(p0, p1));
                    }
                    tmem_st_32x32b_x16(s_addr + (uint32_t)(c * 16), pw);
                }
                tmem_st_wait();
                tcgen05_fence_before();
                __syncwarp();
                if (lane == 0) arrive_even(&p_full[t % Cfg::S_BUFS]);
                const float f = sum_rescale(m_own, m_ref);
                l_lo = sum_add(l_lo, f, sum[0]); l_hi = sum_add(l_hi, f, sum[1]); m_own = m_ref;
            }
            // the item is over and ended at the reference of its last tile, which either warpgroup may have had
            const float f = sum_rescale(m_own, (int)(t & 1) == w ? other_ref() : m_own);
            mbar_wait(l_empty, ((uint32_t)r & 1) ^ 1);
            sum_s[w * 128 + row] = __fmul_rn(l_lo, f) + __fmul_rn(l_hi, f);
            __syncwarp();
            if (lane == 0) mbar_arrive(l_full);
        }
    } else {
        // Output: O scaled, rounded and written in whole lines while the next item's tiles run.  O is free as soon as it stands in shared memory.
        reg_dec<Cfg::REGS_OUT>();
        constexpr int ROW_BYTES = D * 2, CH = ROW_BYTES / 16, ROWS_AT_ONCE = 32 / CH;      // 16-byte pieces of a row; rows a store instruction covers
        const int q = warp & 3, row = q * 32 + lane;
        uint8_t* stage = out_s + q * Cfg::OUT_WARP_BYTES;
        const uint32_t o_addr = tmem_base + ((uint32_t)(q * 32) << 16) + Cfg::O_COL;
        griddep_wait();                                             // the output may still be read by a predecessor
        bool more = pcp_item<CTAS>(p, grp, 0, it);
        for (int r = 0; more; ++r) {
            const int rows_here = it.tile.n_rows - q * 32;          // of this warp's 32
            uint16_t* orow = reinterpret_cast<uint16_t*>(p.out) + (size_t)(it.tile.q_row0 + q * 32) * p.n_heads * D + (size_t)(it.head0 + (int)rank) * D;
            more = pcp_item<CTAS>(p, grp, r + 1, it);
            mbar_wait(l_full, (uint32_t)r & 1);
            const float inv = 1.0f / (sum_s[row] + sum_s[128 + row]);
            __syncwarp();
            if (lane == 0) mbar_arrive(l_empty);
            wait_tmem(o_full, (uint32_t)r & 1);
            tcgen05_fence_after();
#pragma unroll
            for (int c = 0; c < D; c += 32) {
                uint32_t o[32];
                tmem_ld_32x32b_x32(o_addr + (uint32_t)c, o);
                tmem_ld_wait_for(o);
#pragma unroll
                for (int i = 0; i < 32; i += 8) {
                    uint4 u;
                    u.x = pack_bf16x2(__uint_as_float(o[i]) * inv, __uint_as_float(o[i + 1]) * inv);
                    u.y = pack_bf16x2(__uint_as_float(o[i + 2]) * inv, __uint_as_float(o[i + 3]) * inv);
                    u.z = pack_bf16x2(__uint_as_float(o[i + 4]) * inv, __uint_as_float(o[i + 5]) * inv);
                    u.w = pack_bf16x2(__uint_as_float(o[i + 6]) * inv, __uint_as_float(o[i + 7]) * inv);
                    *reinterpret_cast<uint4*>(stage + lane * ROW_BYTES + ((((c + i) >> 3) ^ (lane & 7)) << 4)) = u;
                }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) arrive_even(o_empty);
#pragma unroll 4
            for (int i = 0; i < 32; i += ROWS_AT_ONCE) {
                const int rr = i + lane / CH, ch = lane % CH;
                if (rr < rows_here)
                    *reinterpret_cast<uint4*>(orow + (size_t)rr * p.n_heads * D + ch * 8) = *reinterpret_cast<const uint4*>(stage + rr * ROW_BYTES + ((ch ^ (rr & 7)) << 4));
            }
            __syncwarp();
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (PAIR) gp_cluster_sync();                     // nothing of the pair may still arrive on, read from or allocate in a CTA that has gone
    if (warp == 1) {
        tcgen05_fence_after();
        if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
        else tmem_dealloc<512>(tmem_base);
    }
}

template <int D, int CTAS>
static cudaError_t launch_pcp(const CUtensorMap* tm_q, const CUtensorMap* tm_kv, const KvLayout& kv, const PrefillAttnParams& p, int sms, cudaStream_t s) {
    using Cfg = PcpCfg<D, CTAS>;
    auto kern = prefill_attention_turns_kernel<D, CTAS>;
    static bool attr_done[16] = {};
    { cudaError_t e = ensure_dynamic_smem(kern, Cfg::SMEM_BYTES, attr_done); if (e != cudaSuccess) return e; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CTAS * std::min(p.n_tiles * (p.n_heads / CTAS), sms / CTAS)); cfg.blockDim = dim3(Cfg::THREADS); cfg.dynamicSmemBytes = Cfg::SMEM_BYTES; cfg.stream = s;
    cudaLaunchAttribute attr[2];
    int n_attr = 0;
    if (CTAS > 1) { attr[n_attr].id = cudaLaunchAttributeClusterDimension; attr[n_attr].val.clusterDim.x = CTAS; attr[n_attr].val.clusterDim.y = 1; attr[n_attr++].val.clusterDim.z = 1; }
    if (pdl_enabled()) { attr[n_attr].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[n_attr++].val.programmaticStreamSerializationAllowed = 1; }
    cfg.attrs = attr; cfg.numAttrs = n_attr;
    count_launch();
    return cudaLaunchKernelEx(&cfg, kern, *tm_q, *tm_kv, p, (int64_t)p.layer * kv.layer_stride_rows, kv.kv_stride_rows);
}

template <int D>
static cudaError_t launch_ptp(const CUtensorMap* tm_q, const CUtensorMap* tm_kv, const KvLayout& kv, const PrefillAttnParams& p, int items, int sms, cudaStream_t s) {
    auto kern = prefill_attention_pair_kernel<D>;
    static bool attr_done[16] = {};
    { cudaError_t e = ensure_dynamic_smem(kern, PtpCfg<D>::SMEM_BYTES, attr_done); if (e != cudaSuccess) return e; }
    return launch_k(kern, dim3(items < sms ? items : sms), dim3(PtpCfg<D>::THREADS), PtpCfg<D>::SMEM_BYTES, s, *tm_q, *tm_kv, p,
                    (int64_t)p.layer * kv.layer_stride_rows, kv.kv_stride_rows);
}

template <int D>
static cudaError_t launch_ptc(const CUtensorMap* tm_q, const CUtensorMap* tm_kv, const KvLayout& kv, const PrefillAttnParams& p, cudaStream_t s) {
    auto kern = prefill_attention_tc_kernel<D>;
    static bool attr_done[16] = {};
    { cudaError_t e = ensure_dynamic_smem(kern, PtcCfg<D>::SMEM_BYTES, attr_done); if (e != cudaSuccess) return e; }
    return launch_k(kern, dim3(p.n_tiles, p.n_heads), dim3(64 + 128 * NWG), PtcCfg<D>::SMEM_BYTES, s, *tm_q, *tm_kv, p,
                    (int64_t)p.layer * kv.layer_stride_rows, kv.kv_stride_rows);
}

static int prefill_sm_count() {
    static const int n = [] { int dev = 0, v = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev); return v > 0 ? v : 148; }();
    return n;
}

// Which of them.  us, kernels alone, 32 to 64 heads over 8, 211 batches of 1 to 32 prompts of 30 to 4000 rows behind 0 to 3000 cached ones, fitted with n tiles of
// 128 keys for the longest item and r rounds over the SMs or pairs: one head a CTA 4.9 + 1.0 n (heads of 64: 4.2 + 1.0 n) while all its CTAs are resident, up to half
// as many items of two heads as SMs; two heads a CTA 6.3 + 2.6 (r - 1) + 1.72 a tile on the longest CTA (5.4 + 1.9 (r - 1) + 1.72); in turns on a pair
// 7.1 + 1.25 (r - 1) + 0.77 a tile, on a CTA 4.9 + 0.7 (r - 1) + 0.77.  Heads of 128, n = 1, 4, 11, 25: one query tile of 100 rows 5.8, 8.9, 15.9, 29.9 one head a CTA,
// 7.5, 9.9, 14.6, 24.7 in turns; nine of them 8.6, 14.3, 26.8, 52.1 two heads a CTA, 10.4, 15.6, 26.5, 49.6.  Heads of 64, n = 1, 6, 25: one tile 5.2, 10.2, 29.9 against
// 5.4, 9.1, 22.7, nine 7.1, 16.0, 48.2 against 7.6, 15.4, 44.5.  Ragged items: the longest CTA has the longest item at least, else the mean one a round.  Rows of a query
// tile that are not there cost nothing where a warp has none, and that is more of an item where its output is not written under the next one: 28 prompts of 23 rows, 64 / 8
// heads of 128, 25.5 two heads a CTA and 27.9 in turns, 20 of 128 rows 26.2 and 23.8; 40 of 20 rows, 32 / 8 heads of 64, 18.5 and 16.8, of 128 rows 22.6 and 17.5.  Over 703
// batches of 1 to 6 key tiles the least estimate's kernel was 0.3 % above the fastest in the mean, and 2 batches (77 without that term) were more than 1.5 % slower
// than they are without the kernels in turns.  A pair takes two heads of a group, so groups of 128 with an odd head stay on the first two (in turns on a CTA alone they meet the L2's limit: five prompts of 1.4 thousand rows, 40 / 8 heads 126 -> 171).
PrefillKernel prefill_attention_kernel_of(int n_tiles, int key_tiles, int max_key_tiles, int rows, int n_heads, int n_kv, int head_dim) {
    const int sms = prefill_sm_count(), grp = n_heads / n_kv, items = n_tiles * n_kv * ((grp + 1) / 2);
    const bool few = items <= sms / 2, small = head_dim == 64, turns_ok = key_tiles > 0 && (small || (head_dim == 128 && grp % 2 == 0 && sms >= 2));
    // (few items of any kind: 400 rows behind 6000, 32 / 8 heads, 64 items: one head a CTA 58 us, two 91)
    const PrefillKernel plain = grp > 1 && !few ? PREFILL_TWO_HEADS : PREFILL_ONE_HEAD, turns = small ? PREFILL_TURNS : PREFILL_TURNS_PAIR;
    if (!turns_ok) return plain;
    if (grp == 1 && !few) return turns;                     // one head a CTA is for items that are all resident
    const double mean = (double)key_tiles / n_tiles, longest = max_key_tiles, empty = 1.0 - rows / (128.0 * n_tiles);      // empty: rows of a query tile that are not there
    const int turn_items = small ? n_tiles * n_heads : items, turn_ctas = small ? sms : sms / 2;
    const int r_plain = (items + sms - 1) / sms, r_turns = (turn_items + turn_ctas - 1) / turn_ctas;
    const double us_plain = few ? (small ? 4.2 : 4.9) + 1.0 * longest - 0.4 * empty
                                : (small ? 5.4 + 1.9 * (r_plain - 1) : 6.3 + 2.6 * (r_plain - 1)) + 1.72 * std::max(longest, mean * r_plain) - (small ? 0.6 : 1.2) * r_plain * empty;
    const double us_turns = (small ? 4.9 + 0.7 * (r_turns - 1) : 7.1 + 1.25 * (r_turns - 1)) + 0.77 * std::max(longest, mean * r_turns) - (small ? 0.05 : 0.4) * r_turns * empty;
    return us_turns < us_plain ? turns : plain;
}

cudaError_t launch_prefill_attention_tc(const CUtensorMap* tm_q, const CUtensorMap* tm_kv, const KvLayout& kv, const PrefillAttnParams& p, cudaStream_t s) {
    if (p.n_tiles <= 0) return cudaSuccess;
    if (kv.page_size != 64 || p.n_heads % p.n_kv != 0) return cudaErrorInvalidValue;
    const int grp = p.n_heads / p.n_kv, items = p.n_tiles * p.n_kv * ((grp + 1) / 2), sms = prefill_sm_count();
    const PrefillKernel k = p.forced ? (PrefillKernel)p.forced : prefill_attention_kernel_of(p.n_tiles, p.key_tiles, p.max_key_tiles, p.rows, p.n_heads, p.n_kv, kv.head_dim);
    if (k == PREFILL_TURNS_PAIR) return kv.head_dim == 128 && grp % 2 == 0 && sms >= 2 ? launch_pcp<128, 2>(tm_q, tm_kv, kv, p, sms, s) : cudaErrorInvalidValue;
    if (k == PREFILL_TURNS) return kv.head_dim == 64 ? launch_pcp<64, 1>(tm_q, tm_kv, kv, p, sms, s) : cudaErrorInvalidValue;
    if (k == PREFILL_TWO_HEADS) {
        if (kv.head_dim == 128) return launch_ptp<128>(tm_q, tm_kv, kv, p, items, sms, s);
        if (kv.head_dim == 64) return launch_ptp<64>(tm_q, tm_kv, kv, p, items, sms, s);
        return cudaErrorInvalidValue;
    }
    if (kv.head_dim == 128) return launch_ptc<128>(tm_q, tm_kv, kv, p, s);
    if (kv.head_dim == 64) return launch_ptc<64>(tm_q, tm_kv, kv, p, s);
    return cudaErrorInvalidValue;
}

}  // namespace oa
