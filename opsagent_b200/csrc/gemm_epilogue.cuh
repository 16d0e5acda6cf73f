// gemm_epilogue.cuh — what the persistent prefill GEMMs share: the order in which they walk their tiles and the fused epilogue of one row block
// (bias and activation, residual, gated activations, fp32), through a padded shared-memory transpose to coalesced stores.
#pragma once
#include "common.cuh"
#include "kernels.hpp"

namespace oa {

static constexpr int RASTER_GROUP_M = 16;
static constexpr int EPI_ROW_FLOATS = 36, EPI_WARP_BYTES = 32 * EPI_ROW_FLOATS * 4;      // 32 + 4 pad: conflict-free 16-byte accesses; one 32 x 32 chunk per warp

OA_DEVINL float glu_row_scale(const GemmParams& p, int row) {
    if (!p.row_scale) return 1.0f;
    const int i = p.row_scale_idx[row];
    return i >= 0 ? p.row_scale[i] : 0.0f;
}

OA_DEVINL void raster_tile(int idx, int m_tiles, int n_tiles, int& m_blk, int& n_blk, int group = RASTER_GROUP_M) {
    const int per_band = group * n_tiles;
    const int band = idx / per_band, within = idx - band * per_band;
    const int m0 = band * group;
    const int rows = (m_tiles - m0) < group ? (m_tiles - m0) : group;
    m_blk = m0 + within % rows; n_blk = within / rows;
}

// One warp: rows row_base .. row_base + 31 (TMEM lanes of `acc`), columns n0 .. n0 + bn - 1 of the product.  glu_sc: scales of the two rows this
// lane stores in a clamped gated activation.  SWAPPED: the lanes are columns n0 .. n0 + 31 and the accumulator's columns rows row_base .. row_base + bn - 1: a
// chunk is turned on its way through shared memory and goes on as the other form's.
template <int EPI, bool CLAMPED = true, bool SWAPPED = false>      // CLAMPED: the product may ask for the clamped gated activation (only grouped ones do)
OA_DEVINL void persist_epilogue(const GemmParams& p, float* stage, uint32_t acc, int row_start, int n0, int bn, int lane, const float (&glu_sc)[2]) {
    // residual of the columns at hand and, on their way meanwhile, of the next ones (each lane reads and writes its own places: out may be resid)
    uint4 res[4], res_next[4];
    auto load_res = [&](int cc, uint4 (&rr)[4]) {
#pragma unroll
        for (int i4 = 0; i4 < 4; ++i4) {
            const int row = row_start + (SWAPPED ? cc : 0) + i4 * 8 + (lane >> 2), col = n0 + (SWAPPED ? 0 : cc) + (lane & 3) * 8;
            if (row < p.M && col < p.N) rr[i4] = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.resid) + (size_t)row * p.ldr + col);
        }
    };
    if (EPI == EPI_RESID) load_res(0, res_next);
#pragma unroll 1
    for (int cc = 0; cc < bn; cc += 32) {
        const int col0 = n0 + (SWAPPED ? 0 : cc), row_base = row_start + (SWAPPED ? cc : 0);
        if (SWAPPED && row_base >= p.M) break;
        uint32_t v[32];
        tmem_ld_32x32b_x32(acc + (uint32_t)cc, v);
        tmem_ld_wait();
        if (EPI == EPI_RESID) {
#pragma unroll
            for (int i4 = 0; i4 < 4; ++i4) res[i4] = res_next[i4];
            if (cc + 32 < bn) load_res(cc + 32, res_next);
        }
        if (SWAPPED) {
#pragma unroll
            for (int j = 0; j < 32; ++j) stage[j * EPI_ROW_FLOATS + lane] = __uint_as_float(v[j]);
        } else {
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<float4*>(stage + lane * EPI_ROW_FLOATS + j) =
                    make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
        }
        __syncwarp();
        if (EPI == EPI_SWIGLU) {
            // chunk = 16 gate + 16 up columns -> 16 output features; lane = (row, 8-feature half)
            const int h = lane & 1;
#pragma unroll
            for (int i2 = 0; i2 < 2; ++i2) {
                const int r = i2 * 16 + (lane >> 1), row = row_base + r;
                const float* sp = stage + r * EPI_ROW_FLOATS + h * 8;
                const float4 g0 = *reinterpret_cast<const float4*>(sp), g1 = *reinterpret_cast<const float4*>(sp + 4);
                const float4 u0 = *reinterpret_cast<const float4*>(sp + 16), u1 = *reinterpret_cast<const float4*>(sp + 20);
                const float gg[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
                const float uu[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
                float f[8];
                if (CLAMPED && p.glu_limit > 0.f) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) f[k] = clamped_glu_f32(gg[k] * glu_sc[i2], uu[k] * glu_sc[i2], p.glu_limit, p.glu_slope);
                } else if (p.glu_gelu) {
#pragma unroll
                    for (int k = 0; k < 8; ++k) f[k] = gelu_tanh_fast_f32(gg[k]) * uu[k];
                } else
#pragma unroll
                for (int k = 0; k < 8; ++k) f[k] = __fdividef(gg[k], 1.0f + __expf(-gg[k])) * uu[k];
                if (row < p.M && col0 < p.N) {
                    uint4 o; o.x = pack_bf16x2(f[0], f[1]); o.y = pack_bf16x2(f[2], f[3]); o.z = pack_bf16x2(f[4], f[5]); o.w = pack_bf16x2(f[6], f[7]);
                    *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out) + (size_t)row * p.ldo + (col0 >> 1) + h * 8) = o;
                }
            }
        } else {
            // lane = (row, 8-column group): 8 rows x 64 B per store instruction
            const int c8 = (lane & 3) * 8, col = col0 + c8;
#pragma unroll
            for (int i4 = 0; i4 < 4; ++i4) {
                const int r = i4 * 8 + (lane >> 2), row = row_base + r;
                const float* sp = stage + r * EPI_ROW_FLOATS + c8;
                const float4 a0 = *reinterpret_cast<const float4*>(sp), a1 = *reinterpret_cast<const float4*>(sp + 4);
                float f[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
                if (EPI == EPI_F32) {
                    if (row < p.M && col < p.N) {
                        const float al = p.alpha == 0.f ? 1.f : p.alpha;
                        float* op = p.f32_out + (size_t)row * p.ldf + col;
                        float4 o0 = make_float4(f[0] * al, f[1] * al, f[2] * al, f[3] * al), o1 = make_float4(f[4] * al, f[5] * al, f[6] * al, f[7] * al);
                        if (p.bias_f32) {
                            const float4 b0 = *reinterpret_cast<const float4*>(p.bias_f32 + col), b1 = *reinterpret_cast<const float4*>(p.bias_f32 + col + 4);
                            o0.x += b0.x; o0.y += b0.y; o0.z += b0.z; o0.w += b0.w; o1.x += b1.x; o1.y += b1.y; o1.z += b1.z; o1.w += b1.w;
                        }
                        if (p.f32_accumulate) {
                            const float4 r0 = *reinterpret_cast<const float4*>(op), r1 = *reinterpret_cast<const float4*>(op + 4);
                            o0.x += r0.x; o0.y += r0.y; o0.z += r0.z; o0.w += r0.w; o1.x += r1.x; o1.y += r1.y; o1.z += r1.z; o1.w += r1.w;
                        }
                        *reinterpret_cast<float4*>(op) = o0; *reinterpret_cast<float4*>(op + 4) = o1;
                    }
                } else if (row < p.M && col < p.N) {
                    if (EPI == EPI_STORE) {
                        if (p.bias) {
                            const uint4 bb = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(p.bias) + col);
                            f[0] += bf16lo(bb.x); f[1] += bf16hi(bb.x); f[2] += bf16lo(bb.y); f[3] += bf16hi(bb.y);
                            f[4] += bf16lo(bb.z); f[5] += bf16hi(bb.z); f[6] += bf16lo(bb.w); f[7] += bf16hi(bb.w);
                        }
                        if (p.store_act == 1) {
#pragma unroll
                            for (int k = 0; k < 8; ++k) { const float r = fmaxf(f[k], 0.f); f[k] = r * r; }
                        } else if (p.store_act == 2) {
#pragma unroll
                            for (int k = 0; k < 8; ++k) f[k] = gelu_tanh_f32(f[k]);
                        } else if (p.store_act == 3 && col >= p.act_col0 && col < p.act_col1) {
#pragma unroll
                            for (int k = 0; k < 8; ++k) f[k] = silu_fast_f32(f[k]);
                        }
                    } else {
                        const uint4 rr = res[i4];
                        f[0] += bf16lo(rr.x); f[1] += bf16hi(rr.x); f[2] += bf16lo(rr.y); f[3] += bf16hi(rr.y);
                        f[4] += bf16lo(rr.z); f[5] += bf16hi(rr.z); f[6] += bf16lo(rr.w); f[7] += bf16hi(rr.w);
                    }
                    uint4 o; o.x = pack_bf16x2(f[0], f[1]); o.y = pack_bf16x2(f[2], f[3]); o.z = pack_bf16x2(f[4], f[5]); o.w = pack_bf16x2(f[6], f[7]);
                    *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.out) + (size_t)row * p.ldo + col) = o;
                }
            }
        }
        __syncwarp();
    }
}

}  // namespace oa
