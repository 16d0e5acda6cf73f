// gemm_rows.cu — products of a few rows (decoding steps): C[M,N] = A[M,K] · B[N,K]^T with M <= 128, the WEIGHTS in the tensor core's 128 rows.
//
// A tile of 128 activation rows is mostly padding here, and one CTA per output tile walks all of K by itself: 16 rows x 2048 x 4096 took 64 CTAs
// 64 k blocks each, 21 us for 17 MB.  With the operands swapped a CTA multiplies 128 weight rows by the NR = 16, 32, 64 or 128 activation rows there
// are, so nearly every byte it loads is a weight, and a cluster of S CTAs shares one tile's k range: the partials go through distributed shared
// memory to the CTA that owns their row, which adds them in rank order (a fixed order) and finishes them.
//   warp 0   : TMA producer (weights before griddepcontrol.wait: they depend on no predecessor)
//   warp 1   : tcgen05.mma 128 x NR x 16
//   warps 2-5: one weight row (output column) per thread; partials to the owners, then the epilogue of this CTA's NR / S rows
// us, one CTA per tile -> here: 16 x 2048 x 4096 19.3 -> 8.2, 16 x 4096 x 14336 61 -> 21, 32 x 6144 x 4096 20.6 -> 14.3, 64 x 4096 x 4096 20.4 -> 13.2.
// Shared memory stays under half an SM's (but for NR = 128), so that the next kernel of a step is resident, and its weights on their way, while this one drains.
#include <algorithm>

#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "kernels.hpp"

namespace oa {

static constexpr int GR_BK = 64, GR_THREADS = 192, GR_W_BYTES = 128 * GR_BK * 2;

template <int NR>
struct GrCfg {
    static constexpr int X_BYTES = NR * GR_BK * 2, STAGE_BYTES = GR_W_BYTES + X_BYTES;
    static constexpr int STAGES = NR == 16 ? 5 : NR == 32 ? 4 : 3;
    static constexpr int RECV_BYTES = NR * 128 * 4;              // [S sources][NR / S rows][128 columns]
    static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + RECV_BYTES + 256;
    static constexpr uint32_t TMEM_COLS = NR < 32 ? 32 : NR;
};

OA_DEVINL uint32_t gr_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
OA_DEVINL uint32_t gr_mapa(uint32_t addr, uint32_t rank) { uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank)); return r; }
OA_DEVINL void gr_st_cluster(uint32_t addr, uint32_t v) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }
OA_DEVINL void gr_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int NR, int EPI>
__global__ void __launch_bounds__(GR_THREADS) gemm_rows_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX,
                                                               const GemmParams p, const int S) {
    using Cfg = GrCfg<NR>;
    constexpr int STAGES = Cfg::STAGES;
    extern __shared__ __align__(1024) uint8_t smem[];
    float* recv = reinterpret_cast<float*>(smem + STAGES * Cfg::STAGE_BYTES);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * Cfg::STAGE_BYTES + Cfg::RECV_BYTES);
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* acc_bar = empty_bar + STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_bar + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)gr_rank(), tile = (int)blockIdx.x / S;
    const int kb_total = (p.K + GR_BK - 1) / GR_BK;
    const int kb0 = rank * kb_total / S, n_kb = (rank + 1) * kb_total / S - kb0;      // host: kb_total >= S

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmW); tma_prefetch_desc(&tmX);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        mbar_init(acc_bar, 1);
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc<Cfg::TMEM_COLS>(tmem_slot);
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    griddep_launch();

    if (warp == 0) {
        if (lane == 0) {
            const int pre = n_kb < STAGES ? n_kb : STAGES;
            for (int i = 0; i < pre; ++i) {
                mbar_expect_tx(&full_bar[i], Cfg::STAGE_BYTES);
                tma_load_2d(smem + i * Cfg::STAGE_BYTES, &tmW, &full_bar[i], (kb0 + i) * GR_BK, tile * 128, kEvictFirst);
            }
            griddep_wait();
            for (int i = 0; i < pre; ++i) tma_load_2d(smem + i * Cfg::STAGE_BYTES + GR_W_BYTES, &tmX, &full_bar[i], (kb0 + i) * GR_BK, 0, kEvictLast);
            int s = pre == STAGES ? 0 : pre; uint32_t ph = pre == STAGES ? 1 : 0;
            for (int i = pre; i < n_kb; ++i) {
                mbar_wait(&empty_bar[s], ph ^ 1);
                uint8_t* dst = smem + s * Cfg::STAGE_BYTES;
                mbar_expect_tx(&full_bar[s], Cfg::STAGE_BYTES);
                tma_load_2d(dst, &tmW, &full_bar[s], (kb0 + i) * GR_BK, tile * 128, kEvictFirst);
                tma_load_2d(dst + GR_W_BYTES, &tmX, &full_bar[s], (kb0 + i) * GR_BK, 0, kEvictLast);
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc = umma_idesc_bf16(128, NR);
            int s = 0; uint32_t ph = 0;
            for (int i = 0; i < n_kb; ++i) {
                mbar_wait(&full_bar[s], ph);
                tcgen05_fence_after();
                const uint32_t w_addr = smem_u32(smem + s * Cfg::STAGE_BYTES);
                const uint64_t w_desc = umma_desc_sw128(w_addr), x_desc = umma_desc_sw128(w_addr + GR_W_BYTES);
#pragma unroll
                for (int k = 0; k < GR_BK / 16; ++k) umma_bf16(tmem_base, w_desc + (uint64_t)(k * 2), x_desc + (uint64_t)(k * 2), idesc, (i | k) != 0);
                umma_commit(&empty_bar[s]);
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
            umma_commit(acc_bar);
        }
    }
    __syncwarp();
    gr_cluster_sync();                                            // every CTA of the cluster runs before anybody writes into its shared memory
    const int lg_own = 31 - __clz(NR / S), rows_own = 1 << lg_own;          // rows this CTA finishes
    const int q = warp & 3, c = q * 32 + lane, col = tile * 128 + c;        // epilogue warps: TMEM lane = weight row = column of the tile
    // what a row's result is added to, and the column's bias: read ahead of the exchange, later rows' one group of four ahead
    constexpr bool ADDS = EPI == EPI_RESID || EPI == EPI_F32;
    float add[4] = {0.f, 0.f, 0.f, 0.f}, bias = 0.f;
    auto load_add = [&](int r0) {
        if constexpr (ADDS) {
            if (col >= p.N || (EPI == EPI_F32 && !p.f32_accumulate)) return;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int row = rank * rows_own + r0 + j;
                if (r0 + j < rows_own && row < p.M)
                    add[j] = EPI == EPI_RESID ? bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(p.resid)[(size_t)row * p.ldr + col]) : p.f32_out[(size_t)row * p.ldf + col];
            }
        }
    };
    if (warp >= 2) {
        griddep_wait();
        load_add(0);
        if (EPI == EPI_STORE && p.bias && col < p.N) bias = bf16_bits_to_f32(reinterpret_cast<const uint16_t*>(p.bias)[col]);
        if (EPI == EPI_F32 && p.bias_f32 && col < p.N) bias = p.bias_f32[col];
        mbar_wait(acc_bar, 0);
        tcgen05_fence_after();
        const uint32_t local = smem_u32(recv) + (uint32_t)((rank * rows_own * 128 + c) * 4);
        auto send = [&](int i, uint32_t v) {                      // row i's partial of this column to the row's owner
            if (i < p.M) gr_st_cluster(gr_mapa(local + (uint32_t)((i & (rows_own - 1)) * 512), (uint32_t)(i >> lg_own)), v);
        };
        if constexpr (NR == 16) {
            uint32_t v[16];
            tmem_ld_32x32b_x16(tmem_base + ((uint32_t)(q * 32) << 16), v);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) send(i, v[i]);
        } else {
#pragma unroll 1
            for (int b = 0; b < NR && b < p.M; b += 32) {
                uint32_t v[32];
                tmem_ld_32x32b_x32(tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)b, v);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) send(b + i, v[i]);
            }
        }
        tcgen05_fence_before();
    }
    __syncwarp();
    gr_cluster_sync();                                            // all partials of this CTA's rows have landed
    if (warp >= 2) {
#pragma unroll 1
        for (int r0 = 0; r0 < rows_own && rank * rows_own + r0 < p.M; r0 += 4) {
            float f[4] = {0.f, 0.f, 0.f, 0.f}, now[4];
#pragma unroll
            for (int s = 0; s < 8; ++s)                           // rank order = ascending k
                if (s < S) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) if (r0 + j < rows_own) f[j] += recv[(s * rows_own + r0 + j) * 128 + c];
                }
#pragma unroll
            for (int j = 0; j < 4; ++j) now[j] = add[j];
            load_add(r0 + 4);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int row = rank * rows_own + r0 + j;
                const bool live = r0 + j < rows_own && row < p.M && col < p.N;
                if (EPI == EPI_SWIGLU) {
                    // 32 weight rows = 16 gate then 16 up: the gate's lane finishes output (tile * 128 + 32 q) / 2 + lane
                    const float up = __shfl_down_sync(0xffffffffu, f[j], 16);
                    if (lane < 16 && live) {
                        float o;
                        if (p.glu_limit > 0.f) { const float sc = glu_row_scale(p, row); o = clamped_glu_f32(f[j] * sc, up * sc, p.glu_limit, p.glu_slope); }
                        else if (p.glu_gelu) o = gelu_tanh_fast_f32(f[j]) * up;
                        else o = __fdividef(f[j], 1.0f + __expf(-f[j])) * up;
                        reinterpret_cast<uint16_t*>(p.out)[(size_t)row * p.ldo + ((tile * 128 + q * 32) >> 1) + lane] = f32_to_bf16_bits(o);
                    }
                } else if (live) {
                    if (EPI == EPI_F32) {
                        const float v = f[j] * (p.alpha == 0.f ? 1.f : p.alpha) + bias;
                        p.f32_out[(size_t)row * p.ldf + col] = p.f32_accumulate ? v + now[j] : v;
                    } else {
                        float v = f[j] + (EPI == EPI_RESID ? now[j] : bias);
                        if (EPI == EPI_STORE) {
                            if (p.store_act == 1) { const float r1 = fmaxf(v, 0.f); v = r1 * r1; }
                            else if (p.store_act == 2) v = gelu_tanh_f32(v);
                            else if (p.store_act == 3 && col >= p.act_col0 && col < p.act_col1) v = silu_fast_f32(v);
                        }
                        reinterpret_cast<uint16_t*>(p.out)[(size_t)row * p.ldo + col] = f32_to_bf16_bits(v);
                    }
                }
            }
        }
    }
    __syncthreads();
    if (warp == 1) { tcgen05_fence_after(); tmem_dealloc<Cfg::TMEM_COLS>(tmem_base); }
}

template <int NR, int EPI>
static cudaError_t launch_gr(const CUtensorMap* tmX, const CUtensorMap* tmW, const GemmParams& p, int S, cudaStream_t stream) {
    auto kern = gemm_rows_kernel<NR, EPI>;
    static bool attr_done[16] = {};
    { cudaError_t e = ensure_dynamic_smem(kern, GrCfg<NR>::SMEM_BYTES, attr_done); if (e != cudaSuccess) return e; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((p.N + 127) / 128 * S); cfg.blockDim = dim3(GR_THREADS); cfg.dynamicSmemBytes = GrCfg<NR>::SMEM_BYTES; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension; attr[0].val.clusterDim.x = S; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = pdl_enabled() ? 2 : 1;
    count_launch();
    return cudaLaunchKernelEx(&cfg, kern, *tmW, *tmX, p, S);
}
template <int EPI>
static cudaError_t launch_gr_nr(int nr, const CUtensorMap* tmX, const CUtensorMap* tmW, const GemmParams& p, int S, cudaStream_t st) {
    switch (nr) {
        case 16: return launch_gr<16, EPI>(tmX, tmW, p, S, st);
        case 32: return launch_gr<32, EPI>(tmX, tmW, p, S, st);
        case 64: return launch_gr<64, EPI>(tmX, tmW, p, S, st);
        case 128: return launch_gr<128, EPI>(tmX, tmW, p, S, st);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_gemm_rows(const CUtensorMap* tmX, const CUtensorMap* tmW, const GemmParams& p, int epilogue, int S, cudaStream_t stream) {
    const int nr = gemm_rows_box(p.M);
    if (nr == 0 || p.m_tile_group || (S != 1 && S != 2 && S != 4 && S != 8) || (p.K + GR_BK - 1) / GR_BK < S) return cudaErrorInvalidValue;
    switch (epilogue) {
        case EPI_STORE: return launch_gr_nr<EPI_STORE>(nr, tmX, tmW, p, S, stream);
        case EPI_RESID: return launch_gr_nr<EPI_RESID>(nr, tmX, tmW, p, S, stream);
        case EPI_SWIGLU: return launch_gr_nr<EPI_SWIGLU>(nr, tmX, tmW, p, S, stream);
        case EPI_F32: return launch_gr_nr<EPI_F32>(nr, tmX, tmW, p, S, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace oa
