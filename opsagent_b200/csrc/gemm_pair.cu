// gemm_pair.cu — prefill projections on CTA pairs: C[M,N] = A[M,K] · B[N,K]^T with tcgen05.mma.cta_group::2.
//
// The two CTAs of a cluster (two SMs of one TPC) share one 256 x bn output tile: each holds its own 128 rows of one operand (U) and HALF of the bn rows of the
// other (V) in shared memory, and one thread of the even CTA issues 256 x bn x 16 products that read both halves.  U is A (the tokens) and bn 128, 160, .. 256, or
// U is B (the weights) and bn as many tokens, whichever leaves a pair less to multiply (gemm_pair_width).  Against a 128 x 256 tile per SM that is 2/3
// of the shared-memory reads and of the L2 traffic per product.  Large products run against the 1000 W cap here (85 % of the tensor peak at a clock that is
// down to 1.25 GHz), so what counts there is the energy per product: 8192 x 28672 x 4096 gated 1505 us a call in a loop on 128 x 256 tiles, 1445 on pairs.
// The width is what fills the last round: 1337 x 4096 x 14336 (residual) is 96 tiles of 256 columns, two rounds of 74 pairs of which the second is a third
// full, and 132 tiles of 192: 149 -> 127 us; 1000 x 5120 x 27648 80 tiles of 256, 128 of 160: 288 -> 205; 400 x 2048 x 2048 19.8 -> 12.0 at 128.  Narrow tiles
// take warps that stay converged and issue under elect.sync: behind `if (lane == 0)` a k block cost 0.26 us whatever its width.
//   warp 0   : TMA producer of this CTA's U rows and half of V; both CTAs' bytes are counted on the EVEN CTA's `full` barrier
//   warp 1   : allocates TMEM (both CTAs); in the even CTA it issues the products; commits release the ring slot in both CTAs
//   warps 2-5: epilogue of this CTA's 128 rows while the next tile is multiplied (two accumulators)
// Persistent over tiles in grouped raster order.  Every tile sums its k blocks in ascending order in one accumulator, as the single-CTA kernels do: a
// row's bits depend neither on how many rows share the product nor on its place among them, nor on the width.
#include <algorithm>

#include "common.cuh"
#include "cta_pair.cuh"
#include "gemm_epilogue.cuh"
#include "kernels.hpp"

namespace oa {

static constexpr int GP_BK = 64, GP_THREADS = 192, GP_MAX_STAGES = 8, GP_ACC_COLS = 256, GP_BAR_BYTES = 256;
static constexpr int GP_A_BYTES = 128 * GP_BK * 2;
// a stage: this CTA's 128 rows of U and half of the tile's bn rows of V; as many stages as fit
struct PairRing { int bn, stages; };
static int gp_stage_bytes(int bn) { return GP_A_BYTES + bn / 2 * GP_BK * 2; }
static int gp_smem_bytes(const PairRing& r) { return r.stages * gp_stage_bytes(r.bn) + 4 * EPI_WARP_BYTES + GP_BAR_BYTES; }
static PairRing gp_ring(int bn) { return PairRing{bn, std::min(GP_MAX_STAGES, (232448 - 4 * EPI_WARP_BYTES - GP_BAR_BYTES) / gp_stage_bytes(bn))}; }
static constexpr int GP_GROUP_M = RASTER_GROUP_M / 2;           // a band of tiles whose rows of U stay in L2

// SWAPPED: the weights' rows are the 256 of a tile (operand U) and the tokens its bn (operand V); else the other way round
template <int EPI, bool SWAPPED>
__global__ void __launch_bounds__(GP_THREADS, 1) gemm_pair_kernel(const __grid_constant__ CUtensorMap tmU, const __grid_constant__ CUtensorMap tmV,
                                                                  const GemmParams p, const PairRing ring) {
    const int BN = ring.bn, STAGES = ring.stages, STAGE_BYTES = GP_A_BYTES + BN * GP_BK;
    extern __shared__ __align__(1024) uint8_t smem[];
    float* epi_smem = reinterpret_cast<float*>(smem + STAGES * STAGE_BYTES);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES + 4 * EPI_WARP_BYTES);
    uint64_t* empty_bar = full_bar + STAGES;
    uint64_t* acc_full = empty_bar + STAGES;         // [2]
    uint64_t* acc_empty = acc_full + 2;              // [2], used in the even CTA
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;      // warp: uniform, and known to be
    const uint32_t rank = gp_rank();
    const int v_tiles = ((SWAPPED ? p.M : p.N) + BN - 1) / BN, u_tiles = ((SWAPPED ? p.N : p.M) + 255) / 256, tiles = v_tiles * u_tiles;
    const int num_kb = (p.K + GP_BK - 1) / GP_BK, pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmU); tma_prefetch_desc(&tmV);
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(&acc_full[s], 1); mbar_init(&acc_empty[s], 8); }
        fence_barrier_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(tmem_slot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    __syncthreads();
    gp_cluster_sync();                               // the other CTA's barriers are initialised before anything arrives on them
    tcgen05_fence_after();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
    griddep_launch();

    if (warp == 0) {
        griddep_wait();
        int s = 0; uint32_t ph = 0;
        for (int t = pair; t < tiles; t += pairs) {
            int u_blk, v_blk; raster_tile(t, u_tiles, v_tiles, u_blk, v_blk, GP_GROUP_M);
            const int u_row = u_blk * 256 + (int)rank * 128, v_row = v_blk * BN + (int)rank * (BN / 2);
            for (int kb = 0; kb < num_kb; ++kb) {
                gp_wait(&empty_bar[s], ph ^ 1);
                if (elect_one()) {
                    uint8_t* dst = smem + s * STAGE_BYTES;
                    if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * STAGE_BYTES);      // both CTAs' rows of U and halves of V
                    const uint32_t bar = gp_mapa(&full_bar[s], 0);
                    gp_tma_load(dst, &tmU, bar, kb * GP_BK, u_row, kEvictNormal);
                    gp_tma_load(dst + GP_A_BYTES, &tmV, bar, kb * GP_BK, v_row, kEvictNormal);
                }
                __syncwarp();
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
        }
        for (int i = 0; i < STAGES; ++i) {      // the last products' releases have arrived here before the CTA may go
            gp_wait(&empty_bar[s], ph ^ 1);
            if (++s == STAGES) { s = 0; ph ^= 1; }
        }
    } else if (warp == 1) {
        if (rank == 0) {
            const uint32_t idesc = umma_idesc_bf16(256, (uint32_t)BN);
            int s = 0; uint32_t ph = 0; int it = 0;
            for (int t = pair; t < tiles; t += pairs, ++it) {
                const int as = it & 1;
                gp_wait(&acc_empty[as], (((uint32_t)it >> 1) & 1) ^ 1);
                tcgen05_fence_after();
                const uint32_t tmem_d = tmem_base + (uint32_t)(as * GP_ACC_COLS);
                for (int kb = 0; kb < num_kb; ++kb) {
                    gp_wait(&full_bar[s], ph);
                    tcgen05_fence_after();
                    const uint32_t a_addr = smem_u32(smem + s * STAGE_BYTES);
                    const uint64_t a_desc = umma_desc_sw128(a_addr), b_desc = umma_desc_sw128(a_addr + GP_A_BYTES);
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < GP_BK / 16; ++k) gp_umma(tmem_d, a_desc + (uint64_t)(k * 2), b_desc + (uint64_t)(k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
                        gp_commit(&empty_bar[s]);
                    }
                    __syncwarp();
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
                if (elect_one()) gp_commit(&acc_full[as]);
                __syncwarp();
            }
        }
    } else {
        const int q = warp & 3;
        float* stage = epi_smem + (warp - 2) * (EPI_WARP_BYTES / 4);
        const float no_scale[2] = {0.f, 0.f};
        griddep_wait();
        int it = 0;
        for (int t = pair; t < tiles; t += pairs, ++it) {
            int u_blk, v_blk; raster_tile(t, u_tiles, v_tiles, u_blk, v_blk, GP_GROUP_M);
            const int as = it & 1, u_base = u_blk * 256 + (int)rank * 128 + q * 32;
            const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * GP_ACC_COLS);
            gp_wait(&acc_full[as], ((uint32_t)it >> 1) & 1);
            tcgen05_fence_after();
            if (SWAPPED) { if (u_base < p.N) persist_epilogue<EPI, false, true>(p, stage, acc, v_blk * BN, u_base, BN, lane, no_scale); }
            else if (u_base < p.M) persist_epilogue<EPI, false, false>(p, stage, acc, u_base, v_blk * BN, BN, lane, no_scale);
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) gp_arrive_remote(gp_mapa(&acc_empty[as], 0));
        }
    }
    tcgen05_fence_before();
    __syncthreads();
    gp_cluster_sync();                               // nothing of the pair may still arrive on, read from or allocate in a CTA that has gone
    if (warp == 1) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, 512;" ::"r"(tmem_base) : "memory");
    }
}

template <int EPI, bool SWAPPED>
static cudaError_t launch_gp(const CUtensorMap* tmU, const CUtensorMap* tmV, const GemmParams& p, const PairRing& ring, int sms, cudaStream_t stream) {
    auto kern = gemm_pair_kernel<EPI, SWAPPED>;
    static bool attr_done[16] = {};
    { cudaError_t e = ensure_dynamic_smem(kern, 227 * 1024, attr_done); if (e != cudaSuccess) return e; }
    const int tiles = SWAPPED ? ((p.M + ring.bn - 1) / ring.bn) * ((p.N + 255) / 256) : ((p.N + ring.bn - 1) / ring.bn) * ((p.M + 255) / 256);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * std::min(tiles, sms / 2)); cfg.blockDim = dim3(GP_THREADS); cfg.dynamicSmemBytes = gp_smem_bytes(ring); cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension; attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = pdl_enabled() ? 2 : 1;
    count_launch();
    return cudaLaunchKernelEx(&cfg, kern, *tmU, *tmV, p, ring);
}

cudaError_t launch_gemm_pair(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, int epilogue, int bn, bool swapped, int sms, cudaStream_t stream) {
    if (p.m_tile_group || p.glu_limit > 0.f || sms < 2 || bn < 128 || bn > 256 || bn % 32 != 0) return cudaErrorInvalidValue;
    const PairRing ring = gp_ring(bn);
    switch (epilogue) {
        case EPI_STORE: return swapped ? launch_gp<EPI_STORE, true>(tmB, tmA, p, ring, sms, stream) : launch_gp<EPI_STORE, false>(tmA, tmB, p, ring, sms, stream);
        case EPI_RESID: return swapped ? launch_gp<EPI_RESID, true>(tmB, tmA, p, ring, sms, stream) : launch_gp<EPI_RESID, false>(tmA, tmB, p, ring, sms, stream);
        case EPI_SWIGLU: return swapped ? launch_gp<EPI_SWIGLU, true>(tmB, tmA, p, ring, sms, stream) : launch_gp<EPI_SWIGLU, false>(tmA, tmB, p, ring, sms, stream);
        case EPI_F32: return swapped ? launch_gp<EPI_F32, true>(tmB, tmA, p, ring, sms, stream) : launch_gp<EPI_F32, false>(tmA, tmB, p, ring, sms, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace oa
