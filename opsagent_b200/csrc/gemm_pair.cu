// gemm_pair.cu — prefill projections on CTA pairs: C[M,N] = A[M,K] · B[N,K]^T with tcgen05.mma.cta_group::2.
//
// The two CTAs of a cluster (two SMs of one TPC) share one 256 x 256 output tile: each holds its own 128 rows of A and HALF of the B tile in shared
// memory, and one thread of the even CTA issues 256 x 256 x 16 products that read both halves.  Against a 128 x 256 tile per SM that is 2/3 of the
// shared-memory reads and of the L2 traffic per product, and six k blocks of 32 KB in flight instead of four of 48 KB.  Large products run against the
// 1000 W cap here (85 % of the tensor peak at a clock that is down to 1.25 GHz), so what counts is the energy per product.  Against 128 x 256 tiles,
// us a call in a loop: 8192 x 28672 x 4096 gated 1505 -> 1445, 8192 x 7168 x 5120 499 -> 471; for a single prompt, where the rounds of tiles count: 614 x
// 6144 x 4096 47 -> 32, 1337 x 4096 x 4096 residual 72 -> 53.
//   warp 0   : TMA producer of this CTA's A rows and B half; both CTAs' bytes are counted on the EVEN CTA's `full` barrier
//   warp 1   : allocates TMEM (both CTAs); in the even CTA one thread issues the products; commits release the ring slot in both CTAs
//   warps 2-5: epilogue of this CTA's 128 rows while the next tile is multiplied (two accumulators of 256 columns)
// Persistent over tiles in grouped raster order.  Every tile sums its k blocks in ascending order in one accumulator, as the single-CTA kernels do: a
// row's bits depend neither on how many rows share the product nor on its place among them.  (The last round's tiles cut along k filled idle pairs,
// 16 to 20 us of a product whose tiles fill half a round, and gave that up: 1337 x 4096 x 14336 residual 153 -> 170, against 191 in single-CTA tiles.)
#include <algorithm>

#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "kernels.hpp"

namespace oa {

static constexpr int GP_BN = 256, GP_BK = 64, GP_THREADS = 192, GP_STAGES = 6;
static constexpr int GP_A_BYTES = 128 * GP_BK * 2, GP_B_BYTES = GP_BN / 2 * GP_BK * 2, GP_STAGE_BYTES = GP_A_BYTES + GP_B_BYTES;
static constexpr int GP_SMEM_BYTES = GP_STAGES * GP_STAGE_BYTES + 4 * EPI_WARP_BYTES + 256;
static_assert(GP_SMEM_BYTES <= 232448, "shared memory budget of one CTA");
static constexpr int GP_GROUP_M = RASTER_GROUP_M / 2;           // a band of row tiles whose A rows stay in L2

OA_DEVINL uint32_t gp_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
OA_DEVINL uint32_t gp_mapa(const void* p, uint32_t rank) { uint32_t r; asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank)); return r; }
OA_DEVINL void gp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// TMA load into this CTA's shared memory that completes on a barrier of either CTA of the pair
OA_DEVINL void gp_tma_load(void* dst, const void* tmap, uint32_t bar, int32_t c0, int32_t c1, uint64_t policy) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
        " [%0], [%1, {%3, %4}], [%2], %5;"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(c0), "r"(c1), "l"(policy) : "memory");
}
OA_DEVINL void gp_umma(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
// arrive on the barrier at this offset in BOTH CTAs once every product issued so far has completed
OA_DEVINL void gp_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3) : "memory");
}
OA_DEVINL void gp_arrive_remote(uint32_t bar) { asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory"); }
// as mbar_wait, for barriers the other CTA arrives on
OA_DEVINL void gp_wait(uint64_t* bar, uint32_t parity) {
    uint32_t spins = 0, ok;
    do {
        asm volatile(
            "{\n\t.reg .pred P;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, P;\n\t}"
            : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (!ok && ++spins > OA_MBAR_SPIN_LIMIT) { __trap(); }
    } while (!ok);
}

template <int EPI>
__global__ void __launch_bounds__(GP_THREADS, 1) gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                                                                  const GemmParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    float* epi_smem = reinterpret_cast<float*>(smem + GP_STAGES * GP_STAGE_BYTES);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + GP_STAGES * GP_STAGE_BYTES + 4 * EPI_WARP_BYTES);
    uint64_t* empty_bar = full_bar + GP_STAGES;
    uint64_t* acc_full = empty_bar + GP_STAGES;      // [2]
    uint64_t* acc_empty = acc_full + 2;              // [2], used in the even CTA
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = gp_rank();
    const int n_tiles = (p.N + GP_BN - 1) / GP_BN, m_tiles = (p.M + 255) / 256, tiles = n_tiles * m_tiles;
    const int num_kb = (p.K + GP_BK - 1) / GP_BK, pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;

    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB);
        for (int s = 0; s < GP_STAGES; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
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
    const uint32_t tmem_base = *tmem_slot;
    griddep_launch();

    if (warp == 0) {
        if (lane == 0) {
            griddep_wait();
            int s = 0; uint32_t ph = 0;
            for (int t = pair; t < tiles; t += pairs) {
                int m_blk, n_blk; raster_tile(t, m_tiles, n_tiles, m_blk, n_blk, GP_GROUP_M);
                const int a_row = m_blk * 256 + (int)rank * 128, b_row = n_blk * GP_BN + (int)rank * 128;
                for (int kb = 0; kb < num_kb; ++kb) {
                    gp_wait(&empty_bar[s], ph ^ 1);
                    uint8_t* dst = smem + s * GP_STAGE_BYTES;
                    if (rank == 0) mbar_expect_tx(&full_bar[s], 2 * GP_STAGE_BYTES);      // both CTAs' A rows and B halves
                    const uint32_t bar = gp_mapa(&full_bar[s], 0);
                    gp_tma_load(dst, &tmA, bar, kb * GP_BK, a_row, kEvictNormal);
                    gp_tma_load(dst + GP_A_BYTES, &tmB, bar, kb * GP_BK, b_row, kEvictNormal);
                    if (++s == GP_STAGES) { s = 0; ph ^= 1; }
                }
            }
            for (int i = 0; i < GP_STAGES; ++i) {      // the last products' releases have arrived here before the CTA may go
                gp_wait(&empty_bar[s], ph ^ 1);
                if (++s == GP_STAGES) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && lane == 0) {
            constexpr uint32_t idesc = umma_idesc_bf16(256, GP_BN);
            int s = 0; uint32_t ph = 0; int it = 0;
            for (int t = pair; t < tiles; t += pairs, ++it) {
                const int as = it & 1;
                gp_wait(&acc_empty[as], (((uint32_t)it >> 1) & 1) ^ 1);
                tcgen05_fence_after();
                const uint32_t tmem_d = tmem_base + (uint32_t)(as * GP_BN);
                for (int kb = 0; kb < num_kb; ++kb) {
                    gp_wait(&full_bar[s], ph);
                    tcgen05_fence_after();
                    const uint32_t a_addr = smem_u32(smem + s * GP_STAGE_BYTES);
                    const uint64_t a_desc = umma_desc_sw128(a_addr), b_desc = umma_desc_sw128(a_addr + GP_A_BYTES);
#pragma unroll
                    for (int k = 0; k < GP_BK / 16; ++k) gp_umma(tmem_d, a_desc + (uint64_t)(k * 2), b_desc + (uint64_t)(k * 2), idesc, (kb | k) != 0 ? 1u : 0u);
                    gp_commit(&empty_bar[s]);
                    if (++s == GP_STAGES) { s = 0; ph ^= 1; }
                }
                gp_commit(&acc_full[as]);
            }
        }
    } else {
        const int q = warp & 3;
        float* stage = epi_smem + (warp - 2) * (EPI_WARP_BYTES / 4);
        const float no_scale[2] = {0.f, 0.f};
        griddep_wait();
        int it = 0;
        for (int t = pair; t < tiles; t += pairs, ++it) {
            int m_blk, n_blk; raster_tile(t, m_tiles, n_tiles, m_blk, n_blk, GP_GROUP_M);
            const int as = it & 1, row_base = m_blk * 256 + (int)rank * 128 + q * 32;
            const uint32_t acc = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(as * GP_BN);
            gp_wait(&acc_full[as], ((uint32_t)it >> 1) & 1);
            tcgen05_fence_after();
            if (row_base < p.M) persist_epilogue<EPI, false>(p, stage, acc, row_base, n_blk * GP_BN, GP_BN, lane, no_scale);
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

template <int EPI>
static cudaError_t launch_gp(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, int sms, cudaStream_t stream) {
    auto kern = gemm_pair_kernel<EPI>;
    static bool attr_done[16] = {};
    { cudaError_t e = ensure_dynamic_smem(kern, GP_SMEM_BYTES, attr_done); if (e != cudaSuccess) return e; }
    const int tiles = ((p.N + GP_BN - 1) / GP_BN) * ((p.M + 255) / 256);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * std::min(tiles, sms / 2)); cfg.blockDim = dim3(GP_THREADS); cfg.dynamicSmemBytes = GP_SMEM_BYTES; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension; attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = pdl_enabled() ? 2 : 1;
    count_launch();
    return cudaLaunchKernelEx(&cfg, kern, *tmA, *tmB, p);
}

cudaError_t launch_gemm_pair(const CUtensorMap* tmA, const CUtensorMap* tmB, const GemmParams& p, int epilogue, int sms, cudaStream_t stream) {
    if (p.m_tile_group || p.glu_limit > 0.f || sms < 2) return cudaErrorInvalidValue;
    switch (epilogue) {
        case EPI_STORE: return launch_gp<EPI_STORE>(tmA, tmB, p, sms, stream);
        case EPI_RESID: return launch_gp<EPI_RESID>(tmA, tmB, p, sms, stream);
        case EPI_SWIGLU: return launch_gp<EPI_SWIGLU>(tmA, tmB, p, sms, stream);
        case EPI_F32: return launch_gp<EPI_F32>(tmA, tmB, p, sms, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace oa
