// gemm_tcgen05.cu — C[M,N] = A[M,K] · B[N,K]^T for the QKV / O / gate-up / down / LM-head projections.
//
// sm_100a design (one CTA = one 128 x BLOCK_N output tile):
//   warp 0   : TMA producer — cp.async.bulk.tensor 2D boxes {64 x 128} of A and {64 x BLOCK_N} of B into a
//              STAGES-deep shared-memory ring (128-byte swizzle), completion on `full` mbarriers.
//   warp 1   : allocates TMEM and issues tcgen05.mma (UMMA 128 x BLOCK_N x 16, bf16 -> fp32 in TMEM) from a
//              single thread; tcgen05.commit releases ring slots (`empty`) and finally signals `acc_full`.
//   warps 2-5: epilogue — tcgen05.ld the accumulator (thread = one output row, 32 columns per load), apply the
//              fused epilogue (bias | residual add | SwiGLU | fp32 logits + row arg-max) and store.
// Decode (M <= 128) is weight-streaming and HBM-bound: B tiles are fetched with an evict-first L2 policy, the
// small A operand with evict-last.  K tails and M/N tails rely on TMA zero fill + predicated stores.
//
// The role of this file in the reference's terms: it is the arithmetic that sits behind
// llms.OpenAIClient.Chat (reference pkg/llms/openai.go:69-104) once the `local-cuda` provider replaces the
// remote HTTP server.
#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "kernels.hpp"
#include "sk_consumers.cuh"

namespace oa {

static constexpr int BLOCK_M = 128;
static constexpr int BLOCK_K = 64;     // 64 bf16 = 128 B = one swizzle row
static constexpr int UMMA_K = 16;
static constexpr int GEMM_THREADS = 192;

template <int BN>
struct GemmCfg {
    static constexpr int A_BYTES = BLOCK_M * BLOCK_K * 2;              // 16 KB
    static constexpr int B_BYTES = BN * BLOCK_K * 2;
    static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
    // fill ~200 KB of shared memory.  The narrow tiles serve decoding steps (a few rows, at most one CTA per SM): what bounds them is the
    // weight bytes a CTA has in flight, 4 or 8 KB per stage, so they take as many stages as fit
    static constexpr int STAGES = BN >= 256 ? 4 : (BN >= 128 ? 6 : (BN >= 64 ? 8 : 10));
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 /*align*/ + 256 /*barriers*/;
    static constexpr uint32_t TMEM_COLS = BN < 32 ? 32 : BN;
};

// FEW: a product of up to 64 rows loads only the 16, 32 or 64 of them (the box of tmA) and multiplies 64-row tiles.  Its products, their order and so
// every bit are those of the plain form: a decoding row must not feel how many requests share its step.  (Sharing a tile's k range over a cluster gives
// that up.)  What bounds it is the chain of one tile's k blocks: a barrier's wait, arming and release take 240 cycles in the producer whatever it loads
// (a load only 17 more), and a 128 x 32 x 16 product 40, of which 32 read A.  So a stage holds several k blocks under one barrier (98 cycles a k block
// with four) and the tile has 64 rows (26 a product).  us, a k block a stage and 128-row tiles -> here: 16 x 2048 x 4096 12.7 -> 7.4, 16 x 4096 x 14336
// 42 -> 24, 64 x 6144 x 4096 15.8 -> 13.8, 16 x 8192 x 2048 10.2 -> 7.8.
struct FewRing { int a_rows, stages, kq; };       // kq: k blocks of a stage
static constexpr int FEW_MAX_ROWS = 64, FEW_BAR_BYTES = 512, FEW_M = 64;
static int few_box(int M) { return M <= 16 ? 16 : M <= 32 ? 32 : 64; }
static FewRing few_ring(int M, int N, int bn, int sms) {
    // 160 KB in flight a CTA; with more tiles than SMs 96 KB, so that two CTAs fit one.  A hybrid model's pass with 64, 96, 130, 160 and 200 KB: 4100, 3929,
    // 3871, 3835 and 3829 us; the other figure at 48, 64, 80, 96 and 104 KB: 3879, 3892, 3863, 3846 and 3912.
    const int a_rows = few_box(M), block = (a_rows + bn) * BLOCK_K * 2, room = ((N + bn - 1) / bn > sms ? 96 : 160) * 1024;
    const int kq = block * 4 <= 32 * 1024 ? 4 : block * 2 <= 32 * 1024 ? 2 : 1;
    return FewRing{a_rows, std::max(kq > 1 ? 3 : 4, std::min(28, room / (block * kq))), kq};
}

// 32 columns of one row of the vocabulary head: the row's running arg-max (ties: lowest column) and, where wanted, the logits
OA_DEVINL const uint32_t* logits_mask(const GemmParams& p, int row) {
    const int ms = p.mask_slot ? p.mask_slot[row] : -1;
    return ms >= 0 ? p.mask_table + (size_t)ms * p.mask_words : nullptr;
}
OA_DEVINL void logits_chunk(const GemmParams& p, int row, const uint32_t (&v)[32], int col0, const uint32_t* mask_row, float& best_v, int& best_i, bool store = true) {
    if (mask_row) {
        // grammar-constrained row: only token ids allowed in this sequence's automaton state compete.  The 32 columns of
        // this chunk are 32 consecutive global ids: at most two words of the bitset.
        const uint32_t g0 = (uint32_t)(p.col_offset + col0);
        const uint32_t w0 = (g0 >> 5) < (uint32_t)p.mask_words ? __ldg(mask_row + (g0 >> 5)) : 0u;
        const uint32_t w1 = ((g0 & 31u) && (g0 >> 5) + 1 < (uint32_t)p.mask_words) ? __ldg(mask_row + (g0 >> 5) + 1) : 0u;
        const uint32_t bits = (g0 & 31u) ? __funnelshift_r(w0, w1, g0 & 31u) : w0;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            float f = __uint_as_float(v[j]);
            if (((bits >> j) & 1u) && col0 + j < p.N && f > best_v) { best_v = f; best_i = col0 + j; }
        }
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            float f = __uint_as_float(v[j]);
            if (col0 + j < p.N && f > best_v) { best_v = f; best_i = col0 + j; }
        }
    }
    if (store && p.logits) {
        float* lrow = p.logits + (size_t)row * p.ldl;
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            if (col0 + j < p.N)
                *reinterpret_cast<float4*>(lrow + col0 + j) =
                    make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
        }
    }
}

template <int BN, int EPI, int FEW>      // FEW: 0, or the k blocks of a stage of the few-row form
__global__ void __launch_bounds__(GEMM_THREADS) gemm_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA,
                                                                      const __grid_constant__ CUtensorMap tmB,
                                                                      const GemmParams p, const FewRing few) {
    using Cfg = GemmCfg<BN>;
    // ring: [stage][A | B], a k block a stage; FEW: [stage][k block][A], then [stage][k block][B], A blocks of the rows there are
    constexpr int KQ = FEW ? FEW : 1;
    const int STAGES = FEW ? few.stages : Cfg::STAGES, A_BYTES = FEW ? few.a_rows * BLOCK_K * 2 : Cfg::A_BYTES;
    const int A_STRIDE = FEW ? KQ * A_BYTES : Cfg::STAGE_BYTES, B_STRIDE = FEW ? KQ * Cfg::B_BYTES : Cfg::STAGE_BYTES, B_AT = FEW ? STAGES * A_STRIDE : Cfg::A_BYTES;
    const uint32_t BLOCK_TX = (uint32_t)(A_BYTES + Cfg::B_BYTES);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * KQ * (int)BLOCK_TX);
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* acc_bar = empty_bar + STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);      // warp-uniform, and known to be
    const int lane = threadIdx.x & 31;
    // Grouped rasterisation: CTAs walk bands of RASTER_GROUP_M row tiles, M fastest inside a band, so a band of A
    // (16 x 128 rows) stays L2-resident while each B tile is streamed from HBM once per band instead of once per row tile.
    int n_blk, m_blk;
    {
        const int n_tiles = (p.N + BN - 1) / BN, m_tiles = (p.M + BLOCK_M - 1) / BLOCK_M;
        const int per_band = RASTER_GROUP_M * n_tiles;
        const int band = (int)blockIdx.x / per_band, within = (int)blockIdx.x - band * per_band;
        const int m0 = band * RASTER_GROUP_M;
        const int rows = (m_tiles - m0) < RASTER_GROUP_M ? (m_tiles - m0) : RASTER_GROUP_M;
        m_blk = m0 + within % rows; n_blk = within / rows;
    }
    const int num_kb = (p.K + BLOCK_K - 1) / BLOCK_K;
    int b_row0 = n_blk * BN;
    if (p.m_tile_group) {                 // grouped product: the tile table may come from the preceding kernel, so nothing is prefetched ahead of it
        griddep_wait();
        if (m_blk >= *p.n_m_tiles) return;
        b_row0 += p.m_tile_group[m_blk] * p.group_rows;
    }

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmB);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        mbar_init(acc_bar, 1);
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc<Cfg::TMEM_COLS>(tmem_slot);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    griddep_launch();

    if (warp == 0) {
        // weights (B) are written by no kernel of the chain: fill the ring with them BEFORE waiting for the predecessor
        const int n_st = (num_kb + KQ - 1) / KQ, pre = n_st < STAGES ? n_st : STAGES;      // stages of the whole k range; the last may hold fewer blocks
        for (int st = 0; st < pre; ++st)
            if (elect_one()) {
                const int kb0 = st * KQ, n = num_kb - kb0 < KQ ? num_kb - kb0 : KQ;
                mbar_expect_tx(&full_bar[st], n * BLOCK_TX);
                for (int j = 0; j < KQ; ++j) if (j < n) tma_load_2d(smem + B_AT + st * B_STRIDE + j * Cfg::B_BYTES, &tmB, &full_bar[st], (kb0 + j) * BLOCK_K, b_row0, kEvictFirst);
            }
        griddep_wait();
        for (int st = 0; st < pre; ++st)
            if (elect_one()) {
                const int kb0 = st * KQ, n = num_kb - kb0 < KQ ? num_kb - kb0 : KQ;
                for (int j = 0; j < KQ; ++j) if (j < n) tma_load_2d(smem + st * A_STRIDE + j * A_BYTES, &tmA, &full_bar[st], (kb0 + j) * BLOCK_K, m_blk * BLOCK_M, kEvictLast);
            }
        int s = pre == STAGES ? 0 : pre; uint32_t ph = pre == STAGES ? 1 : 0;
        for (int st = pre; st < n_st; ++st) {
            mbar_wait(&empty_bar[s], ph ^ 1);
            if (elect_one()) {
                const int kb0 = st * KQ, n = num_kb - kb0 < KQ ? num_kb - kb0 : KQ;
                mbar_expect_tx(&full_bar[s], n * BLOCK_TX);
#pragma unroll
                for (int j = 0; j < KQ; ++j) {
                    if (j >= n) break;
                    tma_load_2d(smem + s * A_STRIDE + j * A_BYTES, &tmA, &full_bar[s], (kb0 + j) * BLOCK_K, m_blk * BLOCK_M, kEvictLast);
                    tma_load_2d(smem + B_AT + s * B_STRIDE + j * Cfg::B_BYTES, &tmB, &full_bar[s], (kb0 + j) * BLOCK_K, b_row0, kEvictFirst);
                }
            }
            __syncwarp();
            if (++s == STAGES) { s = 0; ph ^= 1; }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = umma_idesc_bf16(FEW ? FEW_M : BLOCK_M, BN);
        int s = 0; uint32_t ph = 0;
        for (int kb0 = 0; kb0 < num_kb; kb0 += KQ) {
            mbar_wait(&full_bar[s], ph);
            tcgen05_fence_after();
            // FEW: the product reads 64 rows from the start of its A block, the rows beyond those loaded being whatever lies behind it in the ring
            // (inside the block's shared memory: at least two B stages follow, 8 KB and more).  They are rows of the result that nobody looks at.
            const uint64_t a_desc = umma_desc_sw128(smem_u32(smem + s * A_STRIDE));
            const uint64_t b_desc = umma_desc_sw128(smem_u32(smem + B_AT + s * B_STRIDE));
            if (elect_one()) {
#pragma unroll
                for (int j = 0; j < KQ; ++j) {
                    if (j > 0 && kb0 + j >= num_kb) break;
                    const uint64_t aj = a_desc + (uint64_t)(j * (A_BYTES >> 4)), bj = b_desc + (uint64_t)(j * (Cfg::B_BYTES >> 4));
#pragma unroll
                    for (int k = 0; k < BLOCK_K / UMMA_K; ++k)      // 16 bf16 = 32 B further inside the 128 B swizzle row: +2 in the (>>4) address field
                        umma_bf16(tmem_base, aj + (uint64_t)(k * 2), bj + (uint64_t)(k * 2), idesc, (kb0 | j | k) != 0);
                }
                umma_commit(&empty_bar[s]);       // slot reusable once these MMAs have read it
            }
            __syncwarp();
            if (++s == STAGES) { s = 0; ph ^= 1; }
        }
        if (elect_one()) umma_commit(acc_bar);    // accumulator complete
        __syncwarp();
    } else {
        // ---------------- epilogue: warps 2..5, TMEM lane group = warp % 4 ----------------
        const int q = warp & 3;
        // a 64-row tile stands in lanes 0 .. 15 of each warp's 32
        const int row = FEW ? q * 16 + lane : m_blk * BLOCK_M + q * 32 + lane;
        const bool row_ok = row < p.M && (!FEW || lane < 16);
        griddep_wait();                   // bias/residual reads and every store below come after the predecessor grid
        mbar_wait(acc_bar, 0);
        tcgen05_fence_after();
        float best_v = -INFINITY; int best_i = 0x7fffffff;
        const uint32_t* mask_row = nullptr;
        if (EPI == EPI_LOGITS && row_ok) mask_row = logits_mask(p, row);
#pragma unroll 1
        for (int c = 0; c < BN; c += 32) {
            uint32_t v[32];
            tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)c, v);
            tmem_ld_wait();
            const int col0 = n_blk * BN + c;
            if (EPI == EPI_STORE) {
                if (row_ok) {
                    uint16_t* orow = reinterpret_cast<uint16_t*>(p.out) + (size_t)row * p.ldo;
                    const uint16_t* bias = reinterpret_cast<const uint16_t*>(p.bias);
#pragma unroll
                    for (int j = 0; j < 32; j += 8) {
                        if (col0 + j < p.N) {
                            float f[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) f[i] = __uint_as_float(v[j + i]);
                            if (bias) {
                                uint4 bb = *reinterpret_cast<const uint4*>(bias + col0 + j);
                                f[0] += bf16lo(bb.x); f[1] += bf16hi(bb.x); f[2] += bf16lo(bb.y); f[3] += bf16hi(bb.y);
                                f[4] += bf16lo(bb.z); f[5] += bf16hi(bb.z); f[6] += bf16lo(bb.w); f[7] += bf16hi(bb.w);
                            }
                            if (p.store_act == 1) {
#pragma unroll
                                for (int i = 0; i < 8; ++i) { const float r = fmaxf(f[i], 0.f); f[i] = r * r; }
                            } else if (p.store_act == 2) {
#pragma unroll
                                for (int i = 0; i < 8; ++i) f[i] = gelu_tanh_f32(f[i]);
                            } else if (p.store_act == 3 && col0 + j >= p.act_col0 && col0 + j < p.act_col1) {
#pragma unroll
                                for (int i = 0; i < 8; ++i) f[i] = silu_fast_f32(f[i]);
                            }
                            uint4 o;
                            o.x = pack_bf16x2(f[0], f[1]); o.y = pack_bf16x2(f[2], f[3]);
                            o.z = pack_bf16x2(f[4], f[5]); o.w = pack_bf16x2(f[6], f[7]);
                            *reinterpret_cast<uint4*>(orow + col0 + j) = o;
                        }
                    }
                }
            } else if (EPI == EPI_RESID) {
                if (row_ok) {
                    uint16_t* orow = reinterpret_cast<uint16_t*>(p.out) + (size_t)row * p.ldo;
                    const uint16_t* rrow = reinterpret_cast<const uint16_t*>(p.resid) + (size_t)row * p.ldr;
#pragma unroll
                    for (int j = 0; j < 32; j += 8) {
                        if (col0 + j < p.N) {
                            uint4 rr = *reinterpret_cast<const uint4*>(rrow + col0 + j);
                            uint4 o;
                            o.x = pack_bf16x2(__uint_as_float(v[j + 0]) + bf16lo(rr.x), __uint_as_float(v[j + 1]) + bf16hi(rr.x));
                            o.y = pack_bf16x2(__uint_as_float(v[j + 2]) + bf16lo(rr.y), __uint_as_float(v[j + 3]) + bf16hi(rr.y));
                            o.z = pack_bf16x2(__uint_as_float(v[j + 4]) + bf16lo(rr.z), __uint_as_float(v[j + 5]) + bf16hi(rr.z));
                            o.w = pack_bf16x2(__uint_as_float(v[j + 6]) + bf16lo(rr.w), __uint_as_float(v[j + 7]) + bf16hi(rr.w));
                            *reinterpret_cast<uint4*>(orow + col0 + j) = o;
                        }
                    }
                }
            } else if (EPI == EPI_SWIGLU) {
                // columns [c, c+16) = gate, [c+16, c+32) = up for output features (col0/2 .. col0/2+15)
                if (row_ok && col0 < p.N) {
                    uint16_t* orow = reinterpret_cast<uint16_t*>(p.out) + (size_t)row * p.ldo + (col0 >> 1);
                    float f[16];
                    if (p.glu_limit > 0.f) {
                        const float sc = glu_row_scale(p, row);
#pragma unroll
                        for (int i = 0; i < 16; ++i) f[i] = clamped_glu_f32(__uint_as_float(v[i]) * sc, __uint_as_float(v[16 + i]) * sc, p.glu_limit, p.glu_slope);
                    } else if (p.glu_gelu) {
#pragma unroll
                        for (int i = 0; i < 16; ++i) f[i] = gelu_tanh_fast_f32(__uint_as_float(v[i])) * __uint_as_float(v[16 + i]);
                    } else
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float g = __uint_as_float(v[i]), u = __uint_as_float(v[16 + i]);
                        f[i] = __fdividef(g, 1.0f + __expf(-g)) * u;
                    }
                    uint4 o0, o1;
                    o0.x = pack_bf16x2(f[0], f[1]); o0.y = pack_bf16x2(f[2], f[3]); o0.z = pack_bf16x2(f[4], f[5]); o0.w = pack_bf16x2(f[6], f[7]);
                    o1.x = pack_bf16x2(f[8], f[9]); o1.y = pack_bf16x2(f[10], f[11]); o1.z = pack_bf16x2(f[12], f[13]); o1.w = pack_bf16x2(f[14], f[15]);
                    *reinterpret_cast<uint4*>(orow) = o0;
                    *reinterpret_cast<uint4*>(orow + 8) = o1;
                }
            } else if (EPI == EPI_F32) {
                if (row_ok) {
                    float* orow = p.f32_out + (size_t)row * p.ldf;
                    const float al = p.alpha == 0.f ? 1.f : p.alpha;
#pragma unroll
                    for (int j = 0; j < 32; j += 4) {
                        if (col0 + j < p.N) {
                            float4 o = make_float4(__uint_as_float(v[j]) * al, __uint_as_float(v[j + 1]) * al, __uint_as_float(v[j + 2]) * al, __uint_as_float(v[j + 3]) * al);
                            if (p.bias_f32) { const float4 b = *reinterpret_cast<const float4*>(p.bias_f32 + col0 + j); o.x += b.x; o.y += b.y; o.z += b.z; o.w += b.w; }
                            if (p.f32_accumulate) { const float4 r = *reinterpret_cast<const float4*>(orow + col0 + j); o.x += r.x; o.y += r.y; o.z += r.z; o.w += r.w; }
                            *reinterpret_cast<float4*>(orow + col0 + j) = o;
                        }
                    }
                }
            } else {  // EPI_LOGITS
                if (row_ok) logits_chunk(p, row, v, col0, mask_row, best_v, best_i);
            }
        }
        if (EPI == EPI_LOGITS && row_ok) {
            const int n_tiles = (p.N + BN - 1) / BN;
            p.amax_val[(size_t)row * n_tiles + n_blk] = best_v;
            p.amax_idx[(size_t)row * n_tiles + n_blk] = best_i;
        }
        tcgen05_fence_before();
    }
    __syncthreads();
    if (warp == 1) {
        tcgen05_fence_after();
        tmem_dealloc<Cfg::TMEM_COLS>(tmem_base);
    }
}

int gemm_n_tiles(int N, int block_n) { return (N + block_n - 1) / block_n; }

static int sm_count_cached();
// few rows (tmA: a box of few_box(M) rows)
template <int BN, int EPI, int KQ>
static cudaError_t launch_few_kq(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, const FewRing& few, cudaStream_t stream) {
    auto kern = gemm_tcgen05_kernel<BN, EPI, KQ>;
    const int smem = few.stages * few.kq * (few.a_rows + BN) * BLOCK_K * 2 + 1024 + FEW_BAR_BYTES;
    static bool attr_done[16] = {};
    { cudaError_t e = ensure_dynamic_smem(kern, 227 * 1024, attr_done); if (e != cudaSuccess) return e; }
    return launch_k(kern, dim3((p.N + BN - 1) / BN), dim3(GEMM_THREADS), smem, stream, *tmA, *tmB, p, few);
}
template <int BN, int EPI>
static cudaError_t launch_few(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, cudaStream_t stream) {
    const FewRing few = few_ring(p.M, p.N, BN, sm_count_cached());
    // what few_ring gives: 32 columns four k blocks a stage, of 64 rows two; 64 columns two; 128 one
    if constexpr (BN == 32) if (few.kq == 4) return launch_few_kq<BN, EPI, 4>(tmA, tmB, p, few, stream);
    constexpr int KQ = BN <= 64 ? 2 : 1;
    return few.kq == KQ ? launch_few_kq<BN, EPI, KQ>(tmA, tmB, p, few, stream) : cudaErrorInvalidValue;
}
template <int BN>
static cudaError_t launch_few_bn(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, int epi, cudaStream_t s) {
    switch (epi) {
        case EPI_STORE: return launch_few<BN, EPI_STORE>(tmA, tmB, p, s);
        case EPI_RESID: return launch_few<BN, EPI_RESID>(tmA, tmB, p, s);
        case EPI_SWIGLU: return launch_few<BN, EPI_SWIGLU>(tmA, tmB, p, s);
        case EPI_F32: return launch_few<BN, EPI_F32>(tmA, tmB, p, s);
    }
    return cudaErrorInvalidValue;
}

template <int BN, int EPI>
static cudaError_t launch_one(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, cudaStream_t stream) {
    using Cfg = GemmCfg<BN>;
    auto kern = gemm_tcgen05_kernel<BN, EPI, 0>;
    static bool attr_done[16] = {};
    { cudaError_t e = ensure_dynamic_smem(kern, Cfg::SMEM_BYTES, attr_done); if (e != cudaSuccess) return e; }
    dim3 grid(((p.N + BN - 1) / BN) * ((p.M + BLOCK_M - 1) / BLOCK_M), 1, 1);
    return launch_k(kern, grid, dim3(GEMM_THREADS), Cfg::SMEM_BYTES, stream, *tmA, *tmB, p, FewRing{});
}

template <int BN>
static cudaError_t launch_bn(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, int epi, cudaStream_t s) {
    switch (epi) {
        case EPI_STORE: return launch_one<BN, EPI_STORE>(tmA, tmB, p, s);
        case EPI_RESID: return launch_one<BN, EPI_RESID>(tmA, tmB, p, s);
        case EPI_SWIGLU: return launch_one<BN, EPI_SWIGLU>(tmA, tmB, p, s);
        case EPI_LOGITS: return launch_one<BN, EPI_LOGITS>(tmA, tmB, p, s);
        case EPI_F32: return launch_one<BN, EPI_F32>(tmA, tmB, p, s);
    }
    return cudaErrorInvalidValue;
}

static bool persistent_disabled();
static bool head_persistent(int M, int N);
static cudaError_t launch_head(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, int a_rows, cudaStream_t stream);
static constexpr int HEAD_BN = 128;
static int sm_count_cached();
template <int EPI>
static cudaError_t launch_persistent(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, cudaStream_t stream);

// CTA pairs (and how wide a tile) or one of the kernels here: the least estimate of rounds x k blocks x time of a k block plus what a launch costs
// besides.  A k block of a pair's 256 x bn tile takes bn / 256 x (0.28 + 0.14 x busy) + 0.02 us, busy the share of the pairs' rounds that have a tile: the
// more of the chip multiplies, the lower the clock the 1000 W cap leaves.  Fitted to 21 products of 142 .. 7204 rows over the projections of the four model
// sizes, timed in loops at all five widths: the rule takes the fastest of the eight forms timed but for 1 to 2 % (widths in us, 256 224 192 160 128): 372 x 4096 x 14336
// 76 71 67 62 57, 1334 x 5120 x 27648 363 347 401 372 412, 2029 x 7168 x 5120 132 126 128 123 132, 5968 x 28672 x 4096 1070 1077 1094 1110 1161.  A tile of one CTA:
// 128 x 256 0.22 + 0.27 x busy (354 x 57344 x 8192: 353 us, three row tiles instead of two of 256 rows: 384 on pairs), 128 x 128 0.17 + 0.13 x busy, narrower
// 0.15 + 0.07 x busy.  Up to 128 rows half of a pair's rows would be padding.  Every kernel sums k in the same order: the choice moves no bit.
// Either operand's rows may be the 256 of a tile.  With the weights' there, tokens come in steps of 32 instead of 256: 1337 rows are 1344 or 1440, not 1536, 300 are
// 320, not 512, and there are more ways to fill the last round.  The same estimate serves both.  us in loops, on operands that no call before has touched, and alone
// behind a flush of L2, tokens' rows the 256 -> weights': 1337 x 4096 x 14336 127 -> 117, 150 -> 126, 173 -> 153; 300 x 28672 x 4096 83 -> 68, 98 -> 77, 118 -> 96;
// 300 x 7168 x 5120 29 -> 22, 30 -> 24, 48 -> 41; 2366 x 6144 x 4096 91 -> 82, 104 -> 94, 123 -> 114.  It pays where a pair then multiplies fewer columns one after the
// other (chain).  Where only padding goes, the estimate's credit for idle pairs is not there, and an epilogue that turns its chunks is 1 to 2 us longer in a call alone:
// 433 x 4096 x 4096 29.6 -> 31.2, 834 x 8192 x 8192 94 -> 104 in loops, 138 x 10240 x 8192 50 -> 53.  So the chain has to be shorter and the estimate 6 % lower
// (of 50 products short of that, 29 were more than 2 % slower in one of the three kinds of call and one faster in all), 7 % against tiles of one CTA.  Over 70
// products of the four models that take it: 13, 14 and 11 % faster.
struct PairWidth { int bn; double us; bool swapped; long long chain; };      // chain: columns (tokens) a pair multiplies one after the other
static long long ceil_div(long long a, long long b) { return (a + b - 1) / b; }
static PairWidth gemm_pair_width(const GemmParams& p, int sms) {
    const long long pairs = sms / 2, kb = ceil_div(p.K, BLOCK_K);
    auto least = [&](long long rows256, long long rows, bool swapped) {
        PairWidth best{0, 0.0, swapped, 0};
        for (int bn = 256; bn >= 128; bn -= 32) {
            const long long tiles = ceil_div(rows, bn) * ceil_div(rows256, 256), rounds = ceil_div(tiles, pairs);
            const double us = (double)(rounds * kb) * (bn / 256.0 * (0.28 + 0.14 * (double)tiles / (double)(rounds * pairs)) + 0.02) + 8.5;
            if (!best.bn || us < best.us) { best.bn = bn; best.us = us; best.chain = rounds * bn; }
        }
        return best;
    };
    const PairWidth plain = least(p.M, p.N, false);
    if (!p.swap_ok) return plain;
    PairWidth swapped = least(p.N, p.M, true);
    if (swapped.us >= plain.us * 0.94 || swapped.chain >= plain.chain) return plain;
    swapped.us = std::min(swapped.us * 1.07, plain.us);          // what one-CTA tiles have to beat
    return swapped;
}
static GemmKernel kernel_of(const GemmParams& p, int epilogue, int block_n, PairWidth& pair) {
    if (block_n != 32 && block_n != 64 && block_n != 128 && block_n != 256) return GEMM_NONE;
    if (p.M <= 0 || p.N <= 0 || p.K <= 0 || (p.N % 8) != 0 || (p.K % 8) != 0) return GEMM_NONE;
    if (epilogue == EPI_SWIGLU && (p.N % 32) != 0) return GEMM_NONE;
    const int sms = sm_count_cached();
    if (epilogue == EPI_LOGITS) return block_n == HEAD_BN && head_persistent(p.M, p.N) ? GEMM_HEAD : GEMM_TILE;
    // the threshold of the 128 x 256 kernel, where it is set: that kernel and plain tiles are all there is then
    const char* forced = std::getenv("OA_GEMM_PERSISTENT_MIN_TILES");
    if (!forced && p.few_rows_ok && p.M <= FEW_MAX_ROWS && !p.m_tile_group) return GEMM_FEW;
    if (persistent_disabled()) return GEMM_TILE;
    if (!forced && !p.m_tile_group && p.glu_limit <= 0.f && p.M > BLOCK_M && sms >= 2) {
        const long long tiles = ceil_div(p.N, block_n) * ceil_div(p.M, BLOCK_M), rounds = ceil_div(tiles, sms);
        const double busy = (double)tiles / (double)(rounds * sms);
        const double per_kb = block_n >= 256 ? 0.22 + 0.27 * busy : block_n == 128 ? 0.17 + 0.13 * busy : 0.15 + 0.07 * busy;
        pair = gemm_pair_width(p, sms);
        if (pair.us < (double)(rounds * ceil_div(p.K, BLOCK_K)) * per_kb + (block_n >= 256 ? 10.0 : 7.0)) return GEMM_PAIR;
    }
    return block_n == 256 && ceil_div(p.N, 256) * ceil_div(p.M, BLOCK_M) >= (forced ? std::atoll(forced) : 2LL * sms) ? GEMM_PERSISTENT : GEMM_TILE;
}
// The narrowest tiles give the shortest chain a k block; from more than two tiles an SM on, wider ones (each SM then walks several chains in turn).  us at
// 32, 64 and 128 columns, 16 rows: 2048 x 4096 7.4 9.9 13.9, 8192 x 2048 7.8 8.7 10.6, 16384 x 2048 15.6 13.5 15.0, 28672 x 4096 45.0 42.3 40.3.
static int few_width(int N, int sms) {
    for (int bn : {32, 64}) if (ceil_div(N, bn) <= 2 * sms) return bn;
    return 128;
}
GemmChoice gemm_choice(const GemmParams& p, int epilogue, int block_n) {
    PairWidth pair{256, 0.0, false, 0};
    GemmChoice c{kernel_of(p, epilogue, block_n, pair), 128, block_n, block_n};
    if (c.kernel == GEMM_PAIR) { c.width = pair.bn; c.swapped = pair.swapped; (c.swapped ? c.a_box : c.b_box) = pair.bn / 2; if (c.swapped) c.b_box = 128; }
    if (c.kernel == GEMM_FEW) { c.a_box = few_box(p.M); c.width = c.b_box = few_width(p.N, sm_count_cached()); }
    if (c.kernel == GEMM_HEAD && p.few_rows_ok && p.M <= FEW_MAX_ROWS) c.a_box = few_box(p.M);
    return c;
}

cudaError_t launch_gemm(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, int epilogue, int block_n,
                        cudaStream_t stream, const GemmChoice* choice) {
    if (epilogue == EPI_F32 && ((p.ldf % 4) != 0 || !p.f32_out)) return cudaErrorInvalidValue;
    const GemmChoice c = choice ? *choice : gemm_choice(p, epilogue, block_n);
    switch (c.kernel) {
        case GEMM_NONE: return cudaErrorInvalidValue;
        case GEMM_HEAD: return launch_head(tmA, tmB, p, c.a_box, stream);
        case GEMM_PAIR: return launch_gemm_pair(tmA, tmB, p, epilogue, c.width, c.swapped, sm_count_cached(), stream);
        case GEMM_PERSISTENT:      // the widest tile over many rows: the epilogue overlaps the next tile
            switch (epilogue) {
                case EPI_STORE: return launch_persistent<EPI_STORE>(tmA, tmB, p, stream);
                case EPI_RESID: return launch_persistent<EPI_RESID>(tmA, tmB, p, stream);
                case EPI_SWIGLU: return launch_persistent<EPI_SWIGLU>(tmA, tmB, p, stream);
                case EPI_F32: return launch_persistent<EPI_F32>(tmA, tmB, p, stream);
            }
            return cudaErrorInvalidValue;
        case GEMM_FEW:
            switch (c.width) {
                case 32: return launch_few_bn<32>(tmA, tmB, p, epilogue, stream);
                case 64: return launch_few_bn<64>(tmA, tmB, p, epilogue, stream);
                default: return launch_few_bn<128>(tmA, tmB, p, epilogue, stream);
            }
        case GEMM_TILE: break;
    }
    switch (block_n) {
        case 32: return launch_bn<32>(tmA, tmB, p, epilogue, stream);
        case 64: return launch_bn<64>(tmA, tmB, p, epilogue, stream);
        case 128: return launch_bn<128>(tmA, tmB, p, epilogue, stream);
        case 256: return launch_bn<256>(tmA, tmB, p, epilogue, stream);
    }
    return cudaErrorInvalidValue;
}

// =============================================================================================
// persistent tile GEMM (grouped products, and prefill shapes that gemm_choice leaves here): one CTA per SM loops over 128 x 256 tiles in grouped raster order; TMEM holds
// TWO accumulators so the epilogue of tile i (tcgen05.ld -> smem transpose -> coalesced bf16 stores, fused bias /
// residual / SwiGLU) overlaps the tcgen05.mma main loop of tile i+1.
// =============================================================================================
struct PersistCfg {
    static constexpr int BN = 256;
    static constexpr int A_BYTES = BLOCK_M * BLOCK_K * 2, B_BYTES = BN * BLOCK_K * 2, STAGE_BYTES = A_BYTES + B_BYTES;
    static constexpr int STAGES = 4;
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 4 * EPI_WARP_BYTES + 1024 + 256;
    static constexpr uint32_t TMEM_COLS = 512;
};

template <int EPI>
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_persistent_kernel(const __grid_constant__ CUtensorMap tmA,
                                                                            const __grid_constant__ CUtensorMap tmB,
                                                                            const GemmParams p) {
    using Cfg = PersistCfg;
    constexpr int BN = Cfg::BN, STAGES = Cfg::STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float* epi_smem = reinterpret_cast<float*>(smem + STAGES * Cfg::STAGE_BYTES);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES + 4 * EPI_WARP_BYTES);
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* acc_full = empty_bar + STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // warp: uniform, and known to be
    const int n_tiles = (p.N + BN - 1) / BN;
    int m_tiles = (p.M + BLOCK_M - 1) / BLOCK_M;
    if (p.m_tile_group) {                 // grouped product: the number of live row tiles comes from the device (possibly from the preceding kernel)
        griddep_wait();
        const int live = *p.n_m_tiles;
        if (live < m_tiles) m_tiles = live;
    }
    const int total_tiles = n_tiles * m_tiles;
    const int num_kb = (p.K + BLOCK_K - 1) / BLOCK_K;

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 4); }
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
        int s = 0; uint32_t ph = 0;
        for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) {
            int m_blk, n_blk; raster_tile(t, m_tiles, n_tiles, m_blk, n_blk);
            const int b_row0 = n_blk * BN + (p.m_tile_group ? p.m_tile_group[m_blk] * p.group_rows : 0);
            for (int kb = 0; kb < num_kb; ++kb) {
                mbar_wait(&empty_bar[s], ph ^ 1);
                if (elect_one()) {
                    uint8_t* a_dst = smem + s * Cfg::STAGE_BYTES;
                    mbar_expect_tx(&full_bar[s], Cfg::STAGE_BYTES);
                    tma_load_2d(a_dst, &tmA, &full_bar[s], kb * BLOCK_K, m_blk * BLOCK_M, kEvictNormal);
                    tma_load_2d(a_dst + Cfg::A_BYTES, &tmB, &full_bar[s], kb * BLOCK_K, b_row0, kEvictNormal);
                }
                __syncwarp();
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = umma_idesc_bf16(BLOCK_M, BN);
        int s = 0; uint32_t ph = 0; int it = 0;
        for (int t = blockIdx.x; t < total_tiles; t += gridDim.x, ++it) {
            const int as = it & 1;
            mbar_wait(&acc_empty[as], (((uint32_t)it >> 1) & 1) ^ 1);
            tcgen05_fence_after();
            const uint32_t tmem_d = tmem_base + (uint32_t)(as * BN);
            for (int kb = 0; kb < num_kb; ++kb) {
                mbar_wait(&full_bar[s], ph);
                tcgen05_fence_after();
                const uint32_t a_addr = smem_u32(smem + s * Cfg::STAGE_BYTES);
                const uint64_t a_desc = umma_desc_sw128(a_addr), b_desc = umma_desc_sw128(a_addr + Cfg::A_BYTES);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < BLOCK_K / UMMA_K; ++k)
                        umma_bf16(tmem_d, a_desc + (uint64_t)(k * 2), b_desc + (uint64_t)(k * 2), idesc, (kb | k) != 0);
                    umma_commit(&empty_bar[s]);
                }
                __syncwarp();
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
            if (elect_one()) umma_commit(&acc_full[as]);
            __syncwarp();
        }
    } else {
        const int q = warp & 3;
        float* stage = epi_smem + (warp - 2) * (EPI_WARP_BYTES / 4);
        griddep_wait();
        int it = 0;
        for (int t = blockIdx.x; t < total_tiles; t += gridDim.x, ++it) {
            int m_blk, n_blk; raster_tile(t, m_tiles, n_tiles, m_blk, n_blk);
            const int as = it & 1;
            const int row_base = m_blk * BLOCK_M + q * 32;
            float glu_sc[2] = {0.f, 0.f};          // scales of the two rows this lane stores (clamped gated activation), read while the tile is still being multiplied
            if (EPI == EPI_SWIGLU && p.glu_limit > 0.f)
                for (int i2 = 0; i2 < 2; ++i2) if (row_base + i2 * 16 + (lane >> 1) < p.M) glu_sc[i2] = glu_row_scale(p, row_base + i2 * 16 + (lane >> 1));
            mbar_wait(&acc_full[as], ((uint32_t)it >> 1) & 1);
            tcgen05_fence_after();
            persist_epilogue<EPI>(p, stage, tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * BN), row_base, n_blk * BN, BN, lane, glu_sc);
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[as]);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) { tcgen05_fence_after(); tmem_dealloc<Cfg::TMEM_COLS>(tmem_base); }
}

// =============================================================================================
// vocabulary head: persistent 128 x 128 tiles, one CTA per SM, two accumulators.  The head streams its weights once (1 GB for 128 thousand tokens of
// width 4096) and is bound by that.  One CTA per 128 x 256 tile left the last of 3.4 rounds mostly empty and paid each tile's epilogue (logits,
// arg-max) behind its products; here 1002 tiles make 6.8 rounds and the epilogue runs under the next tile's.  128 rows, with logits: 205 -> 183 us.
// Of up to 64 rows only those there are are loaded (boxes of 16, 32 or 64 rows, of which most lie in the tensor: a 128-row box over a handful of rows made
// the head of one conversation slower than that of a hundred), which also leaves room for ten stages instead of six.  us a call with logits at 1, 8, 16, 64 and
// 128 rows, before the boxes, converged warps and whole-line stores of the logits: 256 245 187 200 216; here: 183 182 184 199 210 (200 x 152064 x 5120: 440, 385).
// =============================================================================================
struct HeadCfg {
    static constexpr int BN = HEAD_BN, B_BYTES = BN * BLOCK_K * 2, RING_BYTES = 192 * 1024, MAX_STAGES = 10;
    static constexpr int SMEM_BYTES = RING_BYTES + 4 * EPI_WARP_BYTES + 1024 + 256;
    static constexpr uint32_t TMEM_COLS = 2 * BN;
};
__global__ void __launch_bounds__(GEMM_THREADS, 1) gemm_head_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p, const int a_rows) {
    using Cfg = HeadCfg;
    constexpr int BN = Cfg::BN;
    // ring: [stage][A rows loaded], then [stage][B]; a product reads 128 rows from the start of its A block (see the stream-K kernel)
    const int A_BYTES = a_rows * BLOCK_K * 2, STAGES = min(Cfg::MAX_STAGES, Cfg::RING_BYTES / (A_BYTES + Cfg::B_BYTES));
    const uint32_t STAGE_TX = (uint32_t)(A_BYTES + Cfg::B_BYTES);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* ring_b = smem + STAGES * A_BYTES;
    float* epi_smem = reinterpret_cast<float*>(smem + Cfg::RING_BYTES);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::RING_BYTES + 4 * EPI_WARP_BYTES);
    uint64_t* empty_bar = full_bar + Cfg::MAX_STAGES;
    uint64_t* acc_full = empty_bar + Cfg::MAX_STAGES;
    uint64_t* acc_empty = acc_full + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // warp: uniform, and known to be
    const int n_tiles = (p.N + BN - 1) / BN, m_tiles = (p.M + BLOCK_M - 1) / BLOCK_M, total_tiles = n_tiles * m_tiles;
    const int num_kb = (p.K + BLOCK_K - 1) / BLOCK_K;

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 4); }
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc<Cfg::TMEM_COLS>(tmem_slot);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    griddep_launch();

    if (warp == 0) {
        int s = 0; uint32_t ph = 0;
        const int pre = num_kb < STAGES ? num_kb : STAGES;      // the first tile's weights before the wait: no predecessor writes them
        for (int t = blockIdx.x, first = 1; t < total_tiles; t += gridDim.x, first = 0) {
            int m_blk, n_blk; raster_tile(t, m_tiles, n_tiles, m_blk, n_blk);
            if (first) {
                for (int kb = 0; kb < pre; ++kb)
                    if (elect_one()) {
                        mbar_expect_tx(&full_bar[kb], STAGE_TX);
                        tma_load_2d(ring_b + kb * Cfg::B_BYTES, &tmB, &full_bar[kb], kb * BLOCK_K, n_blk * BN, kEvictFirst);
                    }
                griddep_wait();
            }
            for (int kb = 0; kb < num_kb; ++kb) {
                const bool fresh = !first || kb >= pre;
                if (fresh) mbar_wait(&empty_bar[s], ph ^ 1);
                if (elect_one()) {
                    if (fresh) {
                        mbar_expect_tx(&full_bar[s], STAGE_TX);
                        tma_load_2d(ring_b + s * Cfg::B_BYTES, &tmB, &full_bar[s], kb * BLOCK_K, n_blk * BN, m_tiles > 1 ? kEvictNormal : kEvictFirst);
                    }
                    tma_load_2d(smem + s * A_BYTES, &tmA, &full_bar[s], kb * BLOCK_K, m_blk * BLOCK_M, kEvictLast);
                }
                __syncwarp();
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = umma_idesc_bf16(BLOCK_M, BN);
        int s = 0; uint32_t ph = 0; int it = 0;
        for (int t = blockIdx.x; t < total_tiles; t += gridDim.x, ++it) {
            const int as = it & 1;
            mbar_wait(&acc_empty[as], (((uint32_t)it >> 1) & 1) ^ 1);
            tcgen05_fence_after();
            const uint32_t tmem_d = tmem_base + (uint32_t)(as * BN);
            for (int kb = 0; kb < num_kb; ++kb) {
                mbar_wait(&full_bar[s], ph);
                tcgen05_fence_after();
                const uint64_t a_desc = umma_desc_sw128(smem_u32(smem + s * A_BYTES)), b_desc = umma_desc_sw128(smem_u32(ring_b + s * Cfg::B_BYTES));
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < BLOCK_K / UMMA_K; ++k)
                        umma_bf16(tmem_d, a_desc + (uint64_t)(k * 2), b_desc + (uint64_t)(k * 2), idesc, (kb | k) != 0);
                    umma_commit(&empty_bar[s]);
                }
                __syncwarp();
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
            if (elect_one()) umma_commit(&acc_full[as]);
            __syncwarp();
        }
    } else {
        const int q = warp & 3;
        float* stage = epi_smem + (warp - 2) * (EPI_WARP_BYTES / 4);
        griddep_wait();
        int it = 0;
        for (int t = blockIdx.x; t < total_tiles; t += gridDim.x, ++it) {
            int m_blk, n_blk; raster_tile(t, m_tiles, n_tiles, m_blk, n_blk);
            const int as = it & 1, row = m_blk * BLOCK_M + q * 32 + lane;
            const bool row_ok = row < p.M;
            const uint32_t* mask_row = row_ok ? logits_mask(p, row) : nullptr;
            float best_v = -INFINITY; int best_i = 0x7fffffff;
            mbar_wait(&acc_full[as], ((uint32_t)it >> 1) & 1);
            tcgen05_fence_after();
#pragma unroll 1
            for (int c = 0; c < BN; c += 32) {
                uint32_t v[32];
                tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * BN + c), v);
                tmem_ld_wait();
                if (row_ok) logits_chunk(p, row, v, n_blk * BN + c, mask_row, best_v, best_i, false);
                if (p.logits) {          // through shared memory: four whole 128-byte lines a store instruction
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < 32; j += 4)
                        *reinterpret_cast<float4*>(stage + lane * EPI_ROW_FLOATS + j) =
                            make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                    __syncwarp();
                    const int c4 = (lane & 7) * 4, row0 = m_blk * BLOCK_M + q * 32;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int r = i * 4 + (lane >> 3);
                        if (row0 + r < p.M && n_blk * BN + c + c4 < p.N)
                            *reinterpret_cast<float4*>(p.logits + (size_t)(row0 + r) * p.ldl + n_blk * BN + c + c4) = *reinterpret_cast<const float4*>(stage + r * EPI_ROW_FLOATS + c4);
                    }
                }
            }
            if (row_ok) { p.amax_val[(size_t)row * n_tiles + n_blk] = best_v; p.amax_idx[(size_t)row * n_tiles + n_blk] = best_i; }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[as]);
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) { tcgen05_fence_after(); tmem_dealloc<Cfg::TMEM_COLS>(tmem_base); }
}
static cudaError_t launch_head(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, int a_rows, cudaStream_t stream) {
    static bool attr_done[16] = {};
    { cudaError_t e = ensure_dynamic_smem(gemm_head_kernel, HeadCfg::SMEM_BYTES, attr_done); if (e != cudaSuccess) return e; }
    const int tiles = gemm_n_tiles(p.N, HeadCfg::BN) * ((p.M + BLOCK_M - 1) / BLOCK_M);
    return launch_k(gemm_head_kernel, dim3(std::min(tiles, sm_count_cached())), dim3(GEMM_THREADS), HeadCfg::SMEM_BYTES, stream, *tmA, *tmB, p, a_rows);
}
// the persistent kernel from two rounds of its tiles on; the narrow tiles of a small vocabulary fill the SMs better one CTA each
static bool head_persistent(int M, int N) { return (long long)gemm_n_tiles(N, HeadCfg::BN) * ((M + BLOCK_M - 1) / BLOCK_M) >= 2LL * sm_count_cached(); }
int gemm_logits_bn(int M, int N, int block_n) { return (block_n == 128 || block_n == 256) && head_persistent(M, N) ? HeadCfg::BN : block_n; }

static bool persistent_disabled() { static const bool off = [] { const char* e = std::getenv("OA_GEMM_PERSISTENT"); return e && e[0] == '0'; }(); return off; }
static int sm_count_cached() {
    static int n = 0;
    if (n == 0) { int dev = 0; cudaGetDevice(&dev); cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev); if (n <= 0) n = 148; }
    return n;
}

template <int EPI>
static cudaError_t launch_persistent(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, cudaStream_t stream) {
    auto kern = gemm_persistent_kernel<EPI>;
    static bool attr_done[16] = {};
    { cudaError_t e = ensure_dynamic_smem(kern, PersistCfg::SMEM_BYTES, attr_done); if (e != cudaSuccess) return e; }
    const int tiles = ((p.N + 255) / 256) * ((p.M + BLOCK_M - 1) / BLOCK_M);
    const int grid = tiles < sm_count_cached() ? tiles : sm_count_cached();
    return launch_k(kern, dim3(grid), dim3(GEMM_THREADS), PersistCfg::SMEM_BYTES, stream, *tmA, *tmB, p);
}

// =============================================================================================
// stream-K (decode, M <= 128): persistent CTAs, balanced weight streaming, fp32 partials
// =============================================================================================
template <int BN, int MT, int OCC = 1>     // MT = 128-row tiles of A per unit (1: M <= 128, 2: M <= 256); OCC = CTAs per SM the ring is sized for
struct SkCfg {
    static constexpr int B_BYTES = BN * BLOCK_K * 2;
    static constexpr int RING_BYTES = (OCC == 2 ? 92 : 200) * 1024, MAX_STAGES = 12;
    // A rows a stage holds (MT tiles of those loaded) and stages that fit: 6 of 32 KB (128 rows, BN = 128), 10 of 20 KB (32 rows); halved for 2 CTAs/SM
    __host__ __device__ static constexpr int a_tile_bytes(int a_rows) { return a_rows * BLOCK_K * 2; }
    __host__ __device__ static constexpr int stages(int a_rows) { return RING_BYTES / (MT * a_tile_bytes(a_rows) + B_BYTES) < MAX_STAGES ? RING_BYTES / (MT * a_tile_bytes(a_rows) + B_BYTES) : MAX_STAGES; }
    static constexpr int EPI_ROW_FLOATS = 36;                          // 32 + 4 pad: conflict-free 16-byte smem accesses
    static constexpr int EPI_WARP_BYTES = 32 * EPI_ROW_FLOATS * 4;     // one 32x32 fp32 chunk per epilogue warp
    static constexpr int SMEM_BYTES = RING_BYTES + 4 * EPI_WARP_BYTES + 1024 + 256;
    static constexpr uint32_t TMEM_COLS = 2 * MT * BN;                 // two accumulator stages of MT row tiles
    static_assert(TMEM_COLS * OCC <= 512, "TMEM holds 512 columns per SM");
};

// Epilogues finished INSIDE the stream-K GEMM by the CTA that holds a tile's first k-block (FUSE != 0): it adds the other CTAs' published
// pieces to its TMEM accumulator in CTA order (the stand-alone consumers' order: bit-identical sums) and writes the final bf16 result.
//   FUSE 1  gate/up : act = silu(gate) * up
//   FUSE 2  o / down: x += acc            (residual stream, bf16, in place)
//   FUSE 3  qkv     : (+ bias) -> bf16 -> RoPE -> q_out / paged K rows; V rows copied
struct SkFuse {
    uint16_t* act; int F; unsigned int* tile_flags;
    uint16_t* x; int ldx; int N;        // FUSE 2 (N = logical output columns; also the bound of FUSE 3)
    SkRopeArgs rope;                    // FUSE 3
};

// Loads and products are issued by converged warps that walk (tile, k block) along: behind one lane, with a 64-bit division a unit, a unit took 480 cycles
// and more of the 700 in which HBM delivers it, and a step's start, where the ring is full and only has to be multiplied, ran at that rate.  A stage
// holds the rows of A there are, so a step of 32 rows has ten units in flight instead of six.  us a decoding step of four 8B layers, 32 conversations: 489 ->
// 466; products alone, 64 x 57344 x 8192 175.7 -> 171.2, 64 x 5120 x 27648 67.2 -> 64.4, 32 x 4096 x 14336 42.1 -> 40.6 a call.
template <int BN, int MT, int OCC, int FUSE = 0>
__global__ void __launch_bounds__(GEMM_THREADS, OCC) gemm_streamk_kernel(const __grid_constant__ CUtensorMap tmA,
                                                                         const __grid_constant__ CUtensorMap tmB, const int M,
                                                                         const StreamK sk, const SkFuse fz) {
    using Cfg = SkCfg<BN, MT, OCC>;
    // ring: [stage][MT][A rows loaded], then [stage][B].  A product reads 128 rows from the start of its A block, beyond those loaded whatever lies behind
    // it in the ring (inside it: the B stages follow): rows of the result that nobody looks at.
    const int A_TILE = Cfg::a_tile_bytes(sk.a_rows), A_STRIDE = MT * A_TILE, STAGES = Cfg::stages(sk.a_rows);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* ring_b = smem + STAGES * A_STRIDE;
    float* epi_smem = reinterpret_cast<float*>(smem + Cfg::RING_BYTES);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + Cfg::RING_BYTES + 4 * Cfg::EPI_WARP_BYTES);
    uint64_t* empty_bar = full_bar + Cfg::MAX_STAGES;
    uint64_t* acc_full = empty_bar + Cfg::MAX_STAGES;      // [2]
    uint64_t* acc_empty = acc_full + 2;           // [2]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // warp: uniform, and known to be
    const long long c = blockIdx.x, G = gridDim.x;
    const long long u0 = c * sk.total / G, u1 = (c + 1) * sk.total / G;
    const uint32_t stage_tx = (uint32_t)(MT * A_TILE + Cfg::B_BYTES);

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 4); }
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc<Cfg::TMEM_COLS>(tmem_slot);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    griddep_launch();

    if (warp == 0) {
        // (tile, k block) of the next unit, walked along: one division
        const int n_units = (int)(u1 - u0), tile0 = (int)(u0 / sk.kb), kblk0 = (int)(u0 - (long long)tile0 * sk.kb);
        int tile = tile0, kblk = kblk0;
        auto next = [&]() { if (++kblk == sk.kb) { kblk = 0; ++tile; } };
        // weights first: they depend on no predecessor, so the HBM stream starts while the previous kernel drains
        const int pre = n_units < STAGES ? n_units : STAGES;
        for (int i = 0; i < pre; ++i, next())
            if (elect_one()) {
                mbar_expect_tx(&full_bar[i], stage_tx);
                tma_load_2d(ring_b + i * Cfg::B_BYTES, &tmB, &full_bar[i], kblk * BLOCK_K, tile * BN, kEvictFirst);
            }
        if (sk.l2_prefetch_units > 0) {          // ... and pull the next weight tiles into L2 while the (L2-bound) predecessor still runs and HBM is idle
            const int t1 = tile, k1 = kblk, pf = n_units - pre < sk.l2_prefetch_units ? n_units - pre : sk.l2_prefetch_units;
            for (int i = 0; i < pf; ++i, next())
                if (elect_one()) tma_prefetch_l2_2d(&tmB, kblk * BLOCK_K, tile * BN);
            tile = t1; kblk = k1;
        }
        griddep_wait();
        {
            int k0 = kblk0;
            for (int i = 0; i < pre; ++i) {
                if (elect_one()) {
#pragma unroll
                    for (int m = 0; m < MT; ++m) tma_load_2d(smem + i * A_STRIDE + m * A_TILE, &tmA, &full_bar[i], k0 * BLOCK_K, m * BLOCK_M, kEvictLast);
                }
                if (++k0 == sk.kb) k0 = 0;
            }
        }
        int s = pre == STAGES ? 0 : pre; uint32_t ph = pre == STAGES ? 1 : 0;
        for (int i = pre; i < n_units; ++i, next()) {
            mbar_wait(&empty_bar[s], ph ^ 1);
            if (elect_one()) {
                mbar_expect_tx(&full_bar[s], stage_tx);
                tma_load_2d(ring_b + s * Cfg::B_BYTES, &tmB, &full_bar[s], kblk * BLOCK_K, tile * BN, kEvictFirst);
#pragma unroll
                for (int m = 0; m < MT; ++m) tma_load_2d(smem + s * A_STRIDE + m * A_TILE, &tmA, &full_bar[s], kblk * BLOCK_K, m * BLOCK_M, kEvictLast);
            }
            __syncwarp();
            if (++s == STAGES) { s = 0; ph ^= 1; }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = umma_idesc_bf16(BLOCK_M, BN);
        int s = 0; uint32_t ph = 0; int seg = 0;
        int kblk = (int)(u0 - (long long)(int)(u0 / sk.kb) * sk.kb);
        for (int left = (int)(u1 - u0); left > 0; ++seg) {
            const int n = left < sk.kb - kblk ? left : sk.kb - kblk;      // this CTA's units of one tile
            const int as = seg & 1;
            mbar_wait(&acc_empty[as], (((uint32_t)seg >> 1) & 1) ^ 1);      // epilogue has drained this accumulator
            tcgen05_fence_after();
            const uint32_t tmem_d = tmem_base + (uint32_t)(as * MT * BN);
            for (int i = 0; i < n; ++i) {
                mbar_wait(&full_bar[s], ph);
                tcgen05_fence_after();
                const uint64_t a_desc = umma_desc_sw128(smem_u32(smem + s * A_STRIDE)), b_desc = umma_desc_sw128(smem_u32(ring_b + s * Cfg::B_BYTES));
                if (elect_one()) {
#pragma unroll
                    for (int m = 0; m < MT; ++m)
#pragma unroll
                        for (int k = 0; k < BLOCK_K / UMMA_K; ++k)
                            umma_bf16(tmem_d + (uint32_t)(m * BN), a_desc + (uint64_t)(m * (A_TILE >> 4) + k * 2), b_desc + (uint64_t)(k * 2), idesc, (i > 0 || k > 0) ? 1u : 0u);
                    umma_commit(&empty_bar[s]);
                }
                __syncwarp();
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
            if (elect_one()) umma_commit(&acc_full[as]);
            __syncwarp();
            left -= n; kblk = 0;
        }
    } else {
        const int q = warp & 3;
        int seg = 0;
        griddep_wait();                   // the predecessor may still be reading the partial workspace
        for (long long u = u0; u < u1; ++seg) {
            const int tile = (int)(u / sk.kb);
            const long long uend = min(u1, (long long)(tile + 1) * sk.kb);
            const int as = seg & 1;
            mbar_wait(&acc_full[as], ((uint32_t)seg >> 1) & 1);
            tcgen05_fence_after();
            if constexpr (FUSE == 2 || FUSE == 3) {
                // Same publish / finish protocol as the SwiGLU epilogue below (see there for why the finishing CTA never waits on a
                // waiting CTA); only what the finisher does with the summed 128 x 128 tile differs.
                uint32_t cf, cl;
                sk_tile_ctas(sk, (uint32_t)tile, cf, cl);
                const int c_first = (int)cf, c_last = (int)cl;
                const int row = q * 32 + lane;
                unsigned int* flag = fz.tile_flags + tile;
                if ((int)c == c_first) {
                    const int n_other = c_last - c_first;
                    if (n_other > 0) {
                        if (threadIdx.x == 64) { grid_counter_wait32(flag, (unsigned int)n_other); *flag = 0u; }
                        asm volatile("bar.sync 1, 128;" ::: "memory");
                    }
                    const float* other = sk.ws + (size_t)(c_first + 1 + tile) * (BLOCK_M * BN) + row;
                    const bool live = row < M;
                    // acc[0..32) = this row's sums of columns [mc, mc+32) of the tile: own accumulator, then the other pieces in CTA order
                    auto acc_chunk = [&](int mc, float (&acc)[32]) {
                        uint32_t v[32];
                        tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * BN + mc), v);
                        tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; ++j) acc[j] = 0.f + __uint_as_float(v[j]);      // "0 +" as in sk_sum8
                        for (int o = 0; o < n_other; ++o) {
                            const float* pc = other + (size_t)o * (BLOCK_M * BN) + (size_t)mc * BLOCK_M;
                            float t[32];
#pragma unroll
                            for (int j = 0; j < 32; ++j) t[j] = live ? __ldcg(pc + (size_t)j * BLOCK_M) : 0.f;
#pragma unroll
                            for (int j = 0; j < 32; ++j) acc[j] += t[j];
                        }
                    };
                    if constexpr (FUSE == 2) {
#pragma unroll 1
                        for (int mc = 0; mc < BN; mc += 32) {
                            const int col0 = tile * BN + mc;
                            if (col0 >= fz.N) break;
                            float acc[32];
                            acc_chunk(mc, acc);
                            if (live) {
                                uint4* xr = reinterpret_cast<uint4*>(fz.x + (size_t)row * fz.ldx + col0);
#pragma unroll
                                for (int h = 0; h < 4; ++h) {
                                    const uint4 xo = __ldcg(xr + h);
                                    uint4 xn;
                                    xn.x = pack_bf16x2(bf16lo(xo.x) + acc[8 * h + 0], bf16hi(xo.x) + acc[8 * h + 1]); xn.y = pack_bf16x2(bf16lo(xo.y) + acc[8 * h + 2], bf16hi(xo.y) + acc[8 * h + 3]);
                                    xn.z = pack_bf16x2(bf16lo(xo.z) + acc[8 * h + 4], bf16hi(xo.z) + acc[8 * h + 5]); xn.w = pack_bf16x2(bf16lo(xo.w) + acc[8 * h + 6], bf16hi(xo.w) + acc[8 * h + 7]);
                                    xr[h] = xn;
                                }
                            }
                        }
                    } else {
                        const SkRopeArgs& a = fz.rope;
                        const int D = a.D, half = D >> 1;
                        int pos = 0, page = 0, off = 0;
                        if (live) { pos = a.positions[row]; const int slot = a.slots[row]; page = slot / a.page_size; off = slot - page * a.page_size; }
                        auto finish32 = [&](int col, float (&v)[32]) {          // + bias, round: the projection output is a bf16 tensor (sk_finish8_bf16)
                            if (a.bias) {
#pragma unroll
                                for (int h = 0; h < 4; ++h) {
                                    const uint4 bb = *reinterpret_cast<const uint4*>(a.bias + col + 8 * h);
                                    v[8 * h + 0] += bf16lo(bb.x); v[8 * h + 1] += bf16hi(bb.x); v[8 * h + 2] += bf16lo(bb.y); v[8 * h + 3] += bf16hi(bb.y);
                                    v[8 * h + 4] += bf16lo(bb.z); v[8 * h + 5] += bf16hi(bb.z); v[8 * h + 6] += bf16lo(bb.w); v[8 * h + 7] += bf16hi(bb.w);
                                }
                            }
#pragma unroll
                            for (int k = 0; k < 32; ++k) v[k] = bf16_bits_to_f32(f32_to_bf16_bits(v[k]));
                        };
                        auto store32 = [&](uint16_t* dst, const float (&v)[32]) {
#pragma unroll
                            for (int h = 0; h < 4; ++h) {
                                uint4 o;
                                o.x = pack_bf16x2(v[8 * h + 0], v[8 * h + 1]); o.y = pack_bf16x2(v[8 * h + 2], v[8 * h + 3]);
                                o.z = pack_bf16x2(v[8 * h + 4], v[8 * h + 5]); o.w = pack_bf16x2(v[8 * h + 6], v[8 * h + 7]);
                                reinterpret_cast<uint4*>(dst)[h] = o;
                            }
                        };
#pragma unroll 1
                        for (int mc = 0; mc < BN; mc += 32) {
                            const int col0 = tile * BN + mc;
                            if (col0 >= fz.N) break;
                            const int head = col0 / D, i0 = col0 - head * D;
                            if (head >= a.nh + a.nkv) {                    // V: straight copy into the V plane
                                float vv[32];
                                acc_chunk(mc, vv);
                                finish32(col0, vv);
                                if (live) store32(a.kv_base + (size_t)(a.v_plane_row0 + ((int64_t)page * a.nkv + (head - a.nh - a.nkv)) * a.page_size + off) * D + i0, vv);
                                continue;
                            }
                            if (i0 >= half) continue;                       // the high half is rotated together with its low partner
                            float av[32], bv[32];
                            acc_chunk(mc, av);
                            acc_chunk(mc + half, bv);                       // same tile: BN is a multiple of D
                            finish32(col0, av);
                            finish32(col0 + half, bv);
                            if (live) {
                                const float* cr = a.rope_cos + (size_t)pos * half + i0;
                                const float* sr = a.rope_sin + (size_t)pos * half + i0;
                                float ra[32], rb[32];
#pragma unroll
                                for (int h = 0; h < 8; ++h) {
                                    const float4 c4 = *reinterpret_cast<const float4*>(cr + 4 * h), s4 = *reinterpret_cast<const float4*>(sr + 4 * h);
                                    const float cv[4] = {c4.x, c4.y, c4.z, c4.w}, sv[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                                    for (int k = 0; k < 4; ++k) {
                                        ra[4 * h + k] = av[4 * h + k] * cv[k] - bv[4 * h + k] * sv[k];
                                        rb[4 * h + k] = bv[4 * h + k] * cv[k] + av[4 * h + k] * sv[k];
                                    }
                                }
                                uint16_t* dst;
                                if (head < a.nh) dst = a.q_out + (size_t)row * a.nh * D + (size_t)head * D;
                                else dst = a.kv_base + (size_t)(a.k_plane_row0 + ((int64_t)page * a.nkv + (head - a.nh)) * a.page_size + off) * D;
                                store32(dst + i0, ra);
                                store32(dst + i0 + half, rb);
                            }
                        }
                    }
                } else {
                    float* dst = sk.ws + (size_t)(c + tile) * (BLOCK_M * BN) + row;
#pragma unroll 1
                    for (int mc = 0; mc < BN; mc += 32) {
                        uint32_t v[32];
                        tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * BN + mc), v);
                        tmem_ld_wait();
                        if (row < M) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) dst[(size_t)(mc + j) * BLOCK_M] = __uint_as_float(v[j]);
                        }
                    }
                    __threadfence();
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (threadIdx.x == 64) atomicAdd(flag, 1u);
                }
            } else if constexpr (FUSE == 1) {
                // Pieces of this tile live in CTAs c_first..c_last (same arithmetic as sk_sum8).  The CTA holding the FIRST k-block
                // finishes the tile: it reaches this segment last (it is the tail of its unit range, while the other pieces are the
                // HEAD of their CTAs' ranges), adds the published pieces to its accumulator in CTA order — the stand-alone
                // consumer's order, so results are bit-identical — and writes silu(gate)*up.  Private piece layout: [col][row],
                // so that publisher stores and finisher loads are one full 128-byte line per warp instruction.
                uint32_t cf, cl;
                sk_tile_ctas(sk, (uint32_t)tile, cf, cl);
                const int c_first = (int)cf, c_last = (int)cl;
                const int row = q * 32 + lane;
                unsigned int* flag = fz.tile_flags + tile;
                if ((int)c == c_first) {
                    const int n_other = c_last - c_first;
                    if (n_other > 0) {
                        if (threadIdx.x == 64) { grid_counter_wait32(flag, (unsigned int)n_other); *flag = 0u; }
                        asm volatile("bar.sync 1, 128;" ::: "memory");
                    }
                    const float* other = sk.ws + (size_t)(c_first + 1 + tile) * (BLOCK_M * BN) + row;
                    uint16_t* act_row = fz.act + (size_t)row * fz.F;
                    const bool live = row < M;
                    float t[2][32];
                    auto load_piece = [&](float (&dst)[32], const float* base, int mc) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) dst[j] = live ? __ldcg(base + (size_t)(mc + j) * BLOCK_M) : 0.f;
                    };
                    if (n_other > 0) load_piece(t[0], other, 0);
#pragma unroll
                    for (int k4 = 0; k4 < BN / 32; ++k4) {
                        const int mc = k4 * 32;
                        if (n_other > 0 && k4 + 1 < BN / 32) load_piece(t[(k4 + 1) & 1], other, mc + 32);      // next chunk's piece is in flight during this chunk's math
                        uint32_t v[32];
                        tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * BN + mc), v);
                        tmem_ld_wait();
                        float acc[32];
#pragma unroll
                        for (int j = 0; j < 32; ++j) acc[j] = 0.f + __uint_as_float(v[j]);      // "0 +" as in sk_sum8
                        if (n_other > 0) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) acc[j] += t[k4 & 1][j];
                        }
                        for (int o = 1; o < n_other; ++o) {                                      // tiles cut into more than two pieces (small shapes)
                            float x[32];
                            load_piece(x, other + (size_t)o * (BLOCK_M * BN), mc);
#pragma unroll
                            for (int j = 0; j < 32; ++j) acc[j] += x[j];
                        }
                        const int f0 = (tile * BN + mc) >> 1;          // 32 physical columns = 16 gate + 16 up -> 16 outputs
                        if (live && f0 < fz.F) {
                            float f[16];
#pragma unroll
                            for (int k = 0; k < 16; ++k) f[k] = __fdividef(acc[k], 1.0f + __expf(-acc[k])) * acc[16 + k];
                            uint4 o0, o1;
                            o0.x = pack_bf16x2(f[0], f[1]); o0.y = pack_bf16x2(f[2], f[3]); o0.z = pack_bf16x2(f[4], f[5]); o0.w = pack_bf16x2(f[6], f[7]);
                            o1.x = pack_bf16x2(f[8], f[9]); o1.y = pack_bf16x2(f[10], f[11]); o1.z = pack_bf16x2(f[12], f[13]); o1.w = pack_bf16x2(f[14], f[15]);
                            *reinterpret_cast<uint4*>(act_row + f0) = o0;
                            *reinterpret_cast<uint4*>(act_row + f0 + 8) = o1;
                        }
                    }
                } else {
                    float* dst = sk.ws + (size_t)(c + tile) * (BLOCK_M * BN) + row;
#pragma unroll 1
                    for (int mc = 0; mc < BN; mc += 32) {
                        uint32_t v[32];
                        tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * BN + mc), v);
                        tmem_ld_wait();
                        if (row < M) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) dst[(size_t)(mc + j) * BLOCK_M] = __uint_as_float(v[j]);
                        }
                    }
                    __threadfence();
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                    if (threadIdx.x == 64) atomicAdd(flag, 1u);
                }
            } else {
            // TMEM gives each thread one row x 32 columns; transpose through padded smem so that every global store
            // instruction writes four full 128-byte lines (8 lanes per row) instead of 32 scattered 16-byte pieces.
            float* stage = epi_smem + (warp - 2) * (Cfg::EPI_WARP_BYTES / 4);
            const int r_sub = lane >> 3, c4 = (lane & 7) * 4;
#pragma unroll 1
            for (int mc = 0; mc < MT * BN; mc += 32) {
                const int m = mc / BN, cc = mc - m * BN;
                float* dst = sk.ws + ((size_t)(c + tile) * (MT * BLOCK_M) + m * BLOCK_M + q * 32) * BN;
                uint32_t v[32];
                tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * MT * BN + mc), v);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    *reinterpret_cast<float4*>(stage + lane * Cfg::EPI_ROW_FLOATS + j) =
                        make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
                __syncwarp();
#pragma unroll
                for (int it = 0; it < 8; ++it) {
                    const int r = it * 4 + r_sub;
                    const float4 val = *reinterpret_cast<const float4*>(stage + r * Cfg::EPI_ROW_FLOATS + c4);
                    if (m * BLOCK_M + q * 32 + r < M) *reinterpret_cast<float4*>(dst + (size_t)r * BN + cc + c4) = val;
                }
                __syncwarp();
            }
            }
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[as]);
            u = uend;
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    if (warp == 1) { tcgen05_fence_after(); tmem_dealloc<Cfg::TMEM_COLS>(tmem_base); }
}

StreamK make_streamk(float* ws, int N, int K, int bn, int G, int rows, int a_rows) {
    StreamK sk{}; sk.a_rows = rows > 128 ? 128 : a_rows; sk.ws = ws; sk.bn = bn; sk.rows = rows > 128 ? 256 : 128; sk.kb = (K + BLOCK_K - 1) / BLOCK_K; sk.n_tiles = (N + bn - 1) / bn;
    sk.total = (long long)sk.n_tiles * sk.kb; sk.G = (int)std::min<long long>(G, sk.total);
    sk.l2_prefetch_units = 0;
    return sk;
}
size_t streamk_ws_bytes(int N, int bn, int G, int rows) { return (size_t)(G + (N + bn - 1) / bn) * (rows > 128 ? 256 : 128) * bn * sizeof(float); }

template <int BN, int MT, int OCC = 1, int FUSE = 0>
static cudaError_t launch_sk(const CUtensorMap* tmA, const CUtensorMap* tmB, int M, const StreamK& sk, cudaStream_t stream, SkFuse fz = SkFuse{}) {
    auto kern = gemm_streamk_kernel<BN, MT, OCC, FUSE>;
    static bool attr_done[16] = {};
    { cudaError_t e = ensure_dynamic_smem(kern, SkCfg<BN, MT, OCC>::SMEM_BYTES, attr_done); if (e != cudaSuccess) return e; }
    return launch_k(kern, dim3(sk.G), dim3(GEMM_THREADS), SkCfg<BN, MT, OCC>::SMEM_BYTES, stream, *tmA, *tmB, M, sk, fz);
}
cudaError_t launch_gemm_streamk_swiglu(const CUtensorMap* tmA, const CUtensorMap* tmB, int M, int F, int K, const StreamK& sk, void* act,
                                       unsigned int* tile_flags, cudaStream_t stream) {
    if (M <= 0 || M > BLOCK_M || M > sk.a_rows || sk.rows != 128 || sk.bn != 128 || (F % 16) != 0 || (K % 8) != 0 || !act || !tile_flags) return cudaErrorInvalidValue;
    if (sk.G > sm_count_cached()) return cudaErrorInvalidValue;      // finishing CTAs wait for publishing CTAs: all must be resident
    SkFuse fz{}; fz.act = reinterpret_cast<uint16_t*>(act); fz.F = F; fz.tile_flags = tile_flags;
    return launch_sk<128, 1, 1, 1>(tmA, tmB, M, sk, stream, fz);
}
cudaError_t launch_gemm_streamk_resid(const CUtensorMap* tmA, const CUtensorMap* tmB, int M, int N, int K, const StreamK& sk, void* x, int ldx,
                                      unsigned int* tile_flags, cudaStream_t stream) {
    if (M <= 0 || M > BLOCK_M || M > sk.a_rows || sk.rows != 128 || sk.bn != 128 || (N % 32) != 0 || (K % 8) != 0 || !x || !tile_flags || (ldx % 8) != 0) return cudaErrorInvalidValue;
    if (sk.G > sm_count_cached()) return cudaErrorInvalidValue;      // finishing CTAs wait for publishing CTAs: all must be resident
    SkFuse fz{}; fz.tile_flags = tile_flags; fz.x = reinterpret_cast<uint16_t*>(x); fz.ldx = ldx; fz.N = N;
    return launch_sk<128, 1, 1, 2>(tmA, tmB, M, sk, stream, fz);
}
cudaError_t launch_gemm_streamk_rope(const CUtensorMap* tmA, const CUtensorMap* tmB, int M, int N, int K, const StreamK& sk, const SkRopeArgs& rope,
                                     unsigned int* tile_flags, cudaStream_t stream) {
    if (M <= 0 || M > BLOCK_M || M > sk.a_rows || sk.rows != 128 || sk.bn != 128 || (K % 8) != 0 || !tile_flags) return cudaErrorInvalidValue;
    if ((rope.D != 64 && rope.D != 128) || N != (rope.nh + 2 * rope.nkv) * rope.D) return cudaErrorInvalidValue;      // BN must be a multiple of D; chunks of 32 never straddle a head
    if (sk.G > sm_count_cached()) return cudaErrorInvalidValue;
    SkFuse fz{}; fz.tile_flags = tile_flags; fz.N = N; fz.rope = rope;
    return launch_sk<128, 1, 1, 3>(tmA, tmB, M, sk, stream, fz);
}
cudaError_t launch_gemm_streamk(const CUtensorMap* tmA, const CUtensorMap* tmB, int M, int N, int K, const StreamK& sk, cudaStream_t stream) {
    if (M <= 0 || (sk.rows == 128 && M > sk.a_rows) || M > sk.rows || (N % 8) != 0 || (K % 8) != 0) return cudaErrorInvalidValue;
    if (sk.rows == 256) return sk.bn == 128 ? launch_sk<128, 2>(tmA, tmB, M, sk, stream) : cudaErrorInvalidValue;
    if (sk.bn == 256) return launch_sk<256, 1>(tmA, tmB, M, sk, stream);
    if (sk.bn == 128) return sk.G > sm_count_cached() ? launch_sk<128, 1, 2>(tmA, tmB, M, sk, stream) : launch_sk<128, 1, 1>(tmA, tmB, M, sk, stream);
    if (sk.bn == 64) return launch_sk<64, 1, 1>(tmA, tmB, M, sk, stream);       // half the partial bytes again; per-projection opt-in (sk_bn_o / sk_bn_down / sk_bn_qkv)
    return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------------------------
__global__ void argmax_reduce_kernel(const float* __restrict__ val, const int* __restrict__ idx, int M, int n_tiles,
                                     int32_t* __restrict__ out_ids, float* __restrict__ out_val) {
    const int row = blockIdx.x;
    griddep_launch(); griddep_wait();
    float bv = -INFINITY; int bi = 0x7fffffff;
    for (int t = threadIdx.x; t < n_tiles; t += blockDim.x) {
        float v = val[(size_t)row * n_tiles + t]; int i = idx[(size_t)row * n_tiles + t];
        if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        float ov = __shfl_xor_sync(0xffffffffu, bv, o); int oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > bv || (ov == bv && oi < bi)) { bv = ov; bi = oi; }
    }
    __shared__ float sv[8]; __shared__ int si[8];
    if ((threadIdx.x & 31) == 0) { sv[threadIdx.x >> 5] = bv; si[threadIdx.x >> 5] = bi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
            if (sv[w] > bv || (sv[w] == bv && si[w] < bi)) { bv = sv[w]; bi = si[w]; }
        out_ids[row] = bi == 0x7fffffff ? 0 : bi;
        if (out_val) out_val[row] = bv;
    }
}

cudaError_t launch_argmax_reduce(const float* amax_val, const int* amax_idx, int M, int n_tiles, int32_t* out_ids,
                                 float* out_val, cudaStream_t stream) {
    return launch_k(argmax_reduce_kernel, dim3(M), dim3(256), 0, stream, amax_val, amax_idx, M, n_tiles, out_ids, out_val);
}

}  // namespace oa
