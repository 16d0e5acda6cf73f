// capi_kernels.cpp — kernel-level C entry points on raw device pointers: the launchers that the models' forwards call, one product or one attention a
// call, for programs that bring their own memory (tests and measurements bring torch's).  The engine calls the launchers, not these entries: what a call
// adds here (scratch, tables, a synchronisation) is not part of a serving step.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <string>
#include <vector>

#include "../../include/opsagent_b200.h"
#include <map>
#include <memory>
#include <mutex>
#include "grammar.hpp"
#include "token_mask.hpp"
#include "tokenizer.hpp"
#include "model.hpp"
#include "hybrid_kernels.hpp"
#include "pinned_pool.hpp"
#include "sk_consumers.cuh"
#include "tokenizer.hpp"

using namespace oa;

namespace {
// Scratch of one call (partials, plans, tables) comes from a stream-ordered pool of this library's own, one per device, made at the first use:
// cudaMalloc and cudaFree stop the whole device and cost 0.1 ms to several ms a call, more than most kernels here (paged attention of 6 x 3000
// tokens: 10 us of kernels in a call of 0.7 ms and more; from the pool 0.05 ms).  An allocation is ordered on the call's stream, so calls on
// several streams and threads never share a block; what the pool keeps between calls is bounded, the rest goes back to the device when a call
// synchronises.
constexpr uint64_t SCRATCH_KEEP_BYTES = 64ull << 20;
cudaMemPool_t scratch_pool() {
    static std::mutex mu;
    static cudaMemPool_t pools[64] = {};         // by device; nothing here may throw through the C boundary
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    std::lock_guard<std::mutex> lk(mu);
    cudaMemPool_t& pool = pools[dev];
    if (!pool) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned; props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice; props.location.id = dev;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) { pool = nullptr; return nullptr; }
        uint64_t keep = SCRATCH_KEEP_BYTES;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    return pool;
}
struct DevBuf {
    void* p = nullptr;
    cudaStream_t s;
    DevBuf(size_t n, cudaStream_t stream) : s(stream) {
        if (n == 0) return;
        cudaMemPool_t pool = scratch_pool();
        if (!pool || cudaMallocFromPoolAsync(&p, n, pool, s) != cudaSuccess) p = nullptr;
    }
    DevBuf(const DevBuf&) = delete;
    ~DevBuf() { if (p) cudaFreeAsync(p, s); }
};
// Pinned host memory for the arrays of one call: a copy from pageable memory is pushed or staged by the calling thread (6 to 10 us for 8 to 16 KB, against 2
// to 3 from pinned memory in a loop of its own; six conversations of 1750 tokens: 40.3 -> 38.3 us a call).  A buffer belongs to one call at a time and goes
// back once the call's stream has passed its copy.  (A kernel that reads the pinned buffer instead of a copy was slower than either for such sizes: it and
// the attention behind it run one after the other, 41.8 us.)
uint8_t* pin_host(size_t bytes) {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;          // pinning touches no stream: another thread's capture goes on
    cudaThreadExchangeStreamCaptureMode(&mode);
    void* p = nullptr;
    if (cudaHostAlloc(&p, bytes, cudaHostAllocPortable) != cudaSuccess) { p = nullptr; cudaGetLastError(); }
    cudaThreadExchangeStreamCaptureMode(&mode);
    return (uint8_t*)p;
}
PinnedPool& pinned_pool() { static PinnedPool* pool = new PinnedPool(pin_host); return *pool; }      // never destroyed: the driver may be gone by then
// Host arrays of one call, packed so that ONE copy brings them to the device (each on a 16-byte boundary)
struct Packed {
    CallMemory mem; size_t used = 0;
    explicit Packed(size_t bytes) : mem(pinned_pool(), bytes) {}
    size_t reserve(size_t bytes) { const size_t at = (used + 15) & ~size_t(15); used = at + bytes; return at; }
    uint8_t* data() const { return mem.get(); }
    size_t add(const void* src, size_t n) {
        const size_t at = reserve(n);
        if (n) std::memcpy(data() + at, src, n);
        return at;
    }
};
size_t packed_bytes(std::initializer_list<size_t> parts) { size_t n = 0; for (size_t p : parts) n += (p + 15) & ~size_t(15); return n; }
int rc_of(cudaError_t e) { return e == cudaSuccess ? OA_OK : OA_ERR_INTERNAL; }
}  // namespace

// materialise the deterministic fixed-order sum of stream-K partials as fp32 [M,N]: 8 columns of a row per thread, every partial's loads in
// flight together (a row per CTA with one column and one load at a time was latency-bound: 23 us for 32 x 6144, more than the product itself)
__global__ void sk_reduce_f32_kernel(const StreamK sk, float* __restrict__ out, int N, int aligned) {
    griddep_launch();
    const int row = blockIdx.y, col = (blockIdx.x * blockDim.x + threadIdx.x) * 8;
    const SkCols at = sk_locate(sk, row, col < N ? col : 0);
    griddep_wait();
    if (col >= N) return;
    float acc[8];
    sk_sum8(sk, at, acc);
    float* o = out + (size_t)row * N + col;
    if (aligned) {
        reinterpret_cast<float4*>(o)[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
        reinterpret_cast<float4*>(o)[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) o[i] = acc[i];
    }
}

extern "C" {

int oa_k_gemm_streamk(const void* A, const void* B, int32_t M, int32_t N, int32_t K, int32_t block_n, int32_t n_ctas, float* out_f32, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    CUtensorMap tmA, tmB;
    if (make_tmap_bf16_2d(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)K, (uint32_t)streamk_a_rows(M), 64) != 0) return OA_ERR_INTERNAL;
    if (make_tmap_bf16_2d(&tmB, B, (uint64_t)N, (uint64_t)K, (uint64_t)K, (uint32_t)block_n, 64) != 0) return OA_ERR_INTERNAL;
    DevBuf ws(streamk_ws_bytes(N, block_n, n_ctas, M), s);
    if (!ws.p) return OA_ERR_INTERNAL;
    StreamK sk = make_streamk((float*)ws.p, N, K, block_n, n_ctas, M, streamk_a_rows(M));
    cudaError_t e = launch_gemm_streamk(&tmA, &tmB, M, N, K, sk, s);
    if (e == cudaSuccess) e = launch_k(sk_reduce_f32_kernel, dim3((N / 8 + 127) / 128, M), dim3(128), 0, s, sk, out_f32, N, (int)(((uintptr_t)out_f32 & 15) == 0));
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return rc_of(e);
}

int oa_k_rmsnorm(const void* x, const void* gain, void* y, int32_t T, int32_t H, float eps, void* stream) {
    return rc_of(launch_rmsnorm(x, gain, y, T, H, eps, (cudaStream_t)stream));
}

int oa_k_init_weight(void* dst, uint64_t seed, uint64_t tensor_id, int64_t tensor_id_b, int64_t rows, int64_t cols, float std,
                     float mean, void* stream) {
    return rc_of(launch_init_weight(dst, seed, tensor_id, tensor_id_b, rows, cols, std, mean, (cudaStream_t)stream));
}

int oa_k_gemm(const void* A, const void* B, int32_t M, int32_t N, int32_t K, int32_t epilogue, int32_t block_n, void* out,
              const void* bias, const void* resid, float* logits, int32_t* argmax_out, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    CUtensorMap tmA, tmB;
    GemmParams p{}; p.M = M; p.N = N; p.K = K; p.out = out; p.ldo = epilogue == EPI_SWIGLU ? N / 2 : N;
    p.bias = bias; p.resid = resid; p.ldr = N; p.logits = logits; p.ldl = N;
    if (epilogue == EPI_LOGITS) block_n = gemm_logits_bn(M, N, block_n);
    p.few_rows_ok = p.swap_ok = 1;
    const GemmChoice choice = gemm_choice(p, epilogue, block_n);
    if (make_tmap_bf16_2d(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)K, (uint32_t)choice.a_box, 64) != 0) return OA_ERR_INTERNAL;
    if (make_tmap_bf16_2d(&tmB, B, (uint64_t)N, (uint64_t)K, (uint64_t)K, (uint32_t)choice.b_box, 64) != 0) return OA_ERR_INTERNAL;
    if (epilogue == EPI_LOGITS) {
        const int nt = gemm_n_tiles(N, block_n);
        DevBuf av((size_t)M * nt * 4, s), ai((size_t)M * nt * 4, s);
        if (!av.p || !ai.p) return OA_ERR_INTERNAL;
        p.amax_val = (float*)av.p; p.amax_idx = (int*)ai.p;
        cudaError_t e = launch_gemm(&tmA, &tmB, p, epilogue, block_n, s, &choice);
        if (e == cudaSuccess) e = launch_argmax_reduce(p.amax_val, p.amax_idx, M, nt, argmax_out, nullptr, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        return rc_of(e);
    }
    return rc_of(launch_gemm(&tmA, &tmB, p, epilogue, block_n, s, &choice));
}

int oa_k_hybrid_gemm(int32_t mode, const void* A, int32_t lda, const void* B, int32_t ldb, void* C, int32_t ldc, int32_t M, int32_t N, int32_t K, float alpha,
                     int32_t batch, int64_t stride_a, int64_t stride_b, int64_t stride_c, void* stream) {
    if (mode != HY_STORE && mode != HY_STORE_F32 && mode != HY_ACC_F32) return OA_ERR_BAD_REQUEST;
    return rc_of(hy_gemm(false, mode, A, lda, B, ldb, C, ldc, M, N, K, nullptr, alpha, batch, stride_a, stride_b, stride_c, (cudaStream_t)stream));
}

int oa_k_gemm_ext(const void* A, const void* B, int32_t M, int32_t N, int32_t K, int32_t epilogue, int32_t block_n, void* out, const void* bias, int32_t act, int32_t act_col0,
                  int32_t act_col1, float alpha, int32_t accumulate, void* stream) {
    if (epilogue != EPI_STORE && epilogue != EPI_SWIGLU && epilogue != EPI_F32) return OA_ERR_BAD_REQUEST;
    if (act < 0 || act > 3 || (epilogue == EPI_F32 && act != 0) || (epilogue == EPI_SWIGLU && act != 0 && act != 2)) return OA_ERR_BAD_REQUEST;
    CUtensorMap tmA, tmB;
    GemmParams p{}; p.M = M; p.N = N; p.K = K; p.few_rows_ok = p.swap_ok = 1;
    if (epilogue == EPI_F32) { p.f32_out = (float*)out; p.ldf = N; p.bias_f32 = (const float*)bias; p.alpha = alpha; p.f32_accumulate = accumulate; }
    else { p.out = out; p.ldo = epilogue == EPI_SWIGLU ? N / 2 : N; p.bias = epilogue == EPI_STORE ? bias : nullptr; }
    if (epilogue == EPI_STORE) { p.store_act = act; p.act_col0 = act_col0; p.act_col1 = act_col1; } else p.glu_gelu = act == 2;
    const GemmChoice choice = gemm_choice(p, epilogue, block_n);
    if (make_tmap_bf16_2d(&tmA, A, (uint64_t)M, (uint64_t)K, (uint64_t)K, (uint32_t)choice.a_box, 64) != 0) return OA_ERR_INTERNAL;
    if (make_tmap_bf16_2d(&tmB, B, (uint64_t)N, (uint64_t)K, (uint64_t)K, (uint32_t)choice.b_box, 64) != 0) return OA_ERR_INTERNAL;
    return rc_of(launch_gemm(&tmA, &tmB, p, epilogue, block_n, (cudaStream_t)stream, &choice));
}

int oa_host_gemm_kernel(int32_t M, int32_t N, int32_t K, int32_t epilogue, int32_t block_n, int32_t few_rows, int32_t grouped) {
    GemmParams p{}; p.M = M; p.N = N; p.K = K; p.few_rows_ok = few_rows; p.swap_ok = !grouped;
    static const int32_t group = 0;
    if (grouped) p.m_tile_group = &group;
    return (int)gemm_choice(p, epilogue, block_n).kernel;
}

int oa_host_gemm_pair_width(int32_t M, int32_t N, int32_t K, int32_t epilogue, int32_t block_n) {
    GemmParams p{}; p.M = M; p.N = N; p.K = K; p.few_rows_ok = p.swap_ok = 1;
    const GemmChoice c = gemm_choice(p, epilogue, block_n);
    return c.kernel == GEMM_PAIR && !c.swapped ? c.width : 0;
}

int oa_host_prefill_attention_kernel(const int32_t* ctx_lens, const int32_t* q_lens, int32_t n_seqs, int32_t n_heads, int32_t n_kv, int32_t head_dim) {
    if (n_seqs < 0 || n_kv <= 0 || n_heads <= 0 || n_heads % n_kv != 0) return OA_ERR_BAD_REQUEST;
    int n_tiles = 0, sum = 0, longest = 0, rows = 0;
    for (int i = 0; i < n_seqs; ++i)
        for (int r = 0; r < q_lens[i]; r += PREFILL_TILE_ROWS) {
            const int k = (ctx_lens[i] - q_lens[i] + std::min(r + PREFILL_TILE_ROWS, q_lens[i]) + 127) / 128;
            ++n_tiles; sum += k; longest = std::max(longest, k); rows += std::min(PREFILL_TILE_ROWS, q_lens[i] - r);
        }
    return (int)prefill_attention_kernel_of(n_tiles, sum, longest, rows, n_heads, n_kv, head_dim);
}

int oa_host_gemm_pair_swapped(int32_t M, int32_t N, int32_t K, int32_t epilogue, int32_t block_n) {
    GemmParams p{}; p.M = M; p.N = N; p.K = K; p.few_rows_ok = p.swap_ok = 1;
    const GemmChoice c = gemm_choice(p, epilogue, block_n);
    return c.kernel == GEMM_PAIR && c.swapped ? c.width : 0;
}

static int paged_attention(const void* q, void* out, const void* kv_cache, int32_t num_pages, const int32_t* block_tables,
                           int32_t max_pages_per_seq, const int32_t* ctx_lens, const int32_t* q_lens, int32_t n_seqs,
                           int32_t n_heads, int32_t n_kv, int32_t head_dim, int32_t force_splits, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    KvLayout kv{}; kv.base = const_cast<void*>(kv_cache); kv.page_size = 64; kv.n_kv = n_kv; kv.head_dim = head_dim; kv.num_pages = num_pages;
    kv.kv_stride_rows = (int64_t)num_pages * n_kv * 64; kv.layer_stride_rows = 2 * kv.kv_stride_rows;
    CUtensorMap tm;
    if (make_tmap_bf16_2d(&tm, kv_cache, (uint64_t)kv.layer_stride_rows, (uint64_t)head_dim, (uint64_t)head_dim, 64, 64) != 0) return OA_ERR_INTERNAL;
    const float scale_log2e = (1.0f / std::sqrt((float)head_dim)) * 1.4426950408889634f;
    const int grp = n_heads / n_kv;
    bool decode = true; int total_q = 0;
    for (int i = 0; i < n_seqs; ++i) { if (q_lens && q_lens[i] != 1) decode = false; total_q += q_lens ? q_lens[i] : 1; }
    const size_t table_bytes = (size_t)n_seqs * max_pages_per_seq * 4, ctx_bytes = (size_t)n_seqs * 4;
    cudaError_t e;
    // every path below that has started the copy waits for the stream before the host memory goes back
    if (decode) {
        static thread_local DecodePlan plan;         // its vectors keep their room from call to call
        plan_decode_attention(ctx_lens, n_seqs, n_kv, 2 * 148, force_splits, plan);
        const size_t seg_bytes = plan.segs.size() * sizeof(DecodeSeg), ptr_bytes = plan.cta_ptr.size() * 4, count_bytes = (size_t)(plan.n_cut + 1) * 4;
        Packed host(packed_bytes({table_bytes, ctx_bytes, seg_bytes, ptr_bytes, count_bytes}));
        const size_t o_bt = host.add(block_tables, table_bytes), o_ctx = host.add(ctx_lens, ctx_bytes);
        const size_t o_segs = host.add(plan.segs.data(), seg_bytes), o_ptr = host.add(plan.cta_ptr.data(), ptr_bytes);
        const size_t o_count = host.reserve(count_bytes);                        // merge counters: the CTA with an item's last piece merges it
        std::memset(host.data() + o_count, 0, count_bytes);
        const size_t o_po = (host.used + 255) & ~size_t(255), o_pml = o_po + (size_t)(plan.n_slots + 1) * grp * head_dim * 4;
        DevBuf d_meta(o_pml + (size_t)(plan.n_slots + 1) * grp * 2 * 4, s);       // [tables, plan, counters | partial outputs | partial maxima and sums]
        if (!d_meta.p) return OA_ERR_INTERNAL;
        e = cudaMemcpyAsync(d_meta.p, host.data(), host.used, cudaMemcpyHostToDevice, s);
        const char* meta = (const char*)d_meta.p;
        DecodeAttnParams a{}; a.q = q; a.out = out; a.block_tables = (const int32_t*)(meta + o_bt); a.ctx_lens = (const int32_t*)(meta + o_ctx);
        a.max_pages_per_seq = max_pages_per_seq; a.segs = (const DecodeSeg*)(meta + o_segs); a.cta_seg_ptr = (const int32_t*)(meta + o_ptr);
        a.n_ctas = (int)plan.cta_ptr.size() - 1; a.part_o = (float*)(meta + o_po); a.part_ml = (float*)(meta + o_pml); a.layer = 0;
        a.n_heads = n_heads; a.n_kv = n_kv; a.scale_log2e = scale_log2e;
        a.merge_counters = (int32_t*)((char*)d_meta.p + o_count);
        if (e == cudaSuccess) e = launch_decode_attention(&tm, kv, a, s);
        const cudaError_t done = cudaStreamSynchronize(s);
        return rc_of(e == cudaSuccess ? done : e);
    }
    static thread_local std::vector<PrefillTile> tiles;
    tiles.clear();
    int row = 0;
    for (int i = 0; i < n_seqs; ++i) {
        const int ql = q_lens[i], p0 = ctx_lens[i] - ql;
        for (int r = 0; r < ql; r += PREFILL_TILE_ROWS) tiles.push_back(PrefillTile{i, row + r, p0 + r, std::min(PREFILL_TILE_ROWS, ql - r)});
        row += ql;
    }
    // the tiles with most keys first, as the engine has them: the causal triangle otherwise ends in a tail of heavy tiles
    std::stable_sort(tiles.begin(), tiles.end(), [](const PrefillTile& x, const PrefillTile& y) { return x.pos0 + x.n_rows > y.pos0 + y.n_rows; });
    const size_t tile_bytes = tiles.size() * sizeof(PrefillTile);
    Packed host(packed_bytes({table_bytes, tile_bytes}));
    const size_t o_bt = host.add(block_tables, table_bytes), o_tiles = host.add(tiles.data(), tile_bytes);
    DevBuf d_meta(host.used, s);
    if (!d_meta.p) return OA_ERR_INTERNAL;
    PrefillAttnParams a{}; a.q = q; a.out = out; a.block_tables = (const int32_t*)((const char*)d_meta.p + o_bt); a.max_pages_per_seq = max_pages_per_seq;
    a.tiles = (const PrefillTile*)((const char*)d_meta.p + o_tiles); a.n_tiles = (int)tiles.size(); a.layer = 0; a.n_heads = n_heads; a.n_kv = n_kv; a.scale_log2e = scale_log2e;
    set_key_tiles(a, tiles.data(), tiles.size());
    const char* env = std::getenv("OA_PREFILL_ATTN");            // for tests: the kernel that runs, where it takes these heads (else the call is refused)
    const std::string which = env ? env : "";
    const bool legacy = which == "legacy";
    a.forced = which == "one_head" ? PREFILL_ONE_HEAD : which == "two_heads" ? PREFILL_TWO_HEADS : which == "turns" ? (head_dim == 64 ? PREFILL_TURNS : PREFILL_TURNS_PAIR) : 0;
    CUtensorMap tmq;
    if (!legacy && make_tmap_bf16_2d(&tmq, q, (uint64_t)total_q, (uint64_t)n_heads * head_dim, (uint64_t)n_heads * head_dim, 128, 64) != 0) return OA_ERR_INTERNAL;
    e = cudaMemcpyAsync(d_meta.p, host.data(), host.used, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = legacy ? launch_prefill_attention(&tm, kv, a, s) : launch_prefill_attention_tc(&tmq, &tm, kv, a, s);
    const cudaError_t done = cudaStreamSynchronize(s);
    return rc_of(e == cudaSuccess ? done : e);
}
int oa_k_paged_attention(const void* q, void* out, const void* kv_cache, int32_t num_pages, const int32_t* block_tables,
                         int32_t max_pages_per_seq, const int32_t* ctx_lens, const int32_t* q_lens, int32_t n_seqs,
                         int32_t n_heads, int32_t n_kv, int32_t head_dim, int32_t force_splits, void* stream) {
    try {      // the host arrays are packed into vectors: no exception may cross the C boundary
        return paged_attention(q, out, kv_cache, num_pages, block_tables, max_pages_per_seq, ctx_lens, q_lens, n_seqs, n_heads, n_kv, head_dim, force_splits, stream);
    } catch (const std::exception&) { return OA_ERR_INTERNAL; }
}


int oa_host_apply_chat_template(const char* config_json, const oa_msg* msgs, int32_t n_msgs, int32_t* out_ids, int32_t cap, int32_t* n_out) {
    try {
        ModelConfig mc; EngineOptions eo; parse_config(config_json ? config_json : "{}", mc, eo);
        Tokenizer tok(mc, eo.tokenizer);
        std::vector<ChatMessage> m;
        for (int i = 0; i < n_msgs; ++i) m.push_back(ChatMessage{msgs[i].role, msgs[i].content});
        auto ids = tok.apply_chat_template(m);
        *n_out = (int32_t)ids.size();
        if (out_ids) std::memcpy(out_ids, ids.data(), (size_t)std::min<int32_t>(cap, (int32_t)ids.size()) * 4);
    } catch (const std::exception&) { return OA_ERR_BAD_REQUEST; }
    return OA_OK;
}

static int export_decode_plan(const DecodePlan& plan, int32_t* segs_out, int32_t cap_segs, int32_t* cta_ptr_out, int32_t cap_ctas, int32_t* n_ctas_out,
                              int32_t* n_segs_out, int32_t* n_slots_out) {
    if ((int)plan.segs.size() > cap_segs || (int)plan.cta_ptr.size() > cap_ctas + 1) return OA_ERR_BAD_REQUEST;
    for (size_t i = 0; i < plan.segs.size(); ++i) {
        const DecodeSeg& g = plan.segs[i];
        int32_t* o = segs_out + i * 5; o[0] = g.seq; o[1] = g.kvh; o[2] = g.chunk_begin; o[3] = g.chunk_end; o[4] = g.partial_slot;
    }
    std::memcpy(cta_ptr_out, plan.cta_ptr.data(), plan.cta_ptr.size() * 4);
    *n_ctas_out = (int32_t)plan.cta_ptr.size() - 1; *n_segs_out = (int32_t)plan.segs.size(); *n_slots_out = plan.n_slots;
    return OA_OK;
}
int oa_host_decode_plan(const int32_t* ctx_lens, int32_t n_seqs, int32_t n_kv, int32_t n_ctas_target, int32_t force_splits,
                        int32_t* segs_out, int32_t cap_segs, int32_t* cta_ptr_out, int32_t cap_ctas, int32_t* n_ctas_out,
                        int32_t* n_segs_out, int32_t* n_slots_out) {
    DecodePlan plan;
    build_decode_plan(ctx_lens, n_seqs, n_kv, n_ctas_target, force_splits, plan);
    return export_decode_plan(plan, segs_out, cap_segs, cta_ptr_out, cap_ctas, n_ctas_out, n_segs_out, n_slots_out);
}
int oa_host_decode_attention_plan(const int32_t* ctx_lens, int32_t n_seqs, int32_t n_kv, int32_t n_ctas_target, int32_t force_splits,
                                  int32_t* segs_out, int32_t cap_segs, int32_t* cta_ptr_out, int32_t cap_ctas, int32_t* n_ctas_out,
                                  int32_t* n_segs_out, int32_t* n_slots_out) {
    DecodePlan plan;
    plan_decode_attention(ctx_lens, n_seqs, n_kv, n_ctas_target, force_splits, plan);
    return export_decode_plan(plan, segs_out, cap_segs, cta_ptr_out, cap_ctas, n_ctas_out, n_segs_out, n_slots_out);
}

int oa_host_streamk_plan(int32_t N, int32_t K, int32_t block_n, int32_t n_ctas, int64_t* cta_unit0_out, int32_t cap_ctas,
                         int32_t* tile_first_out, int32_t* tile_last_out, int32_t cap_tiles, int32_t* n_ctas_out, int32_t* n_tiles_out,
                         int32_t* kb_out) {
    if (N <= 0 || K <= 0 || n_ctas <= 0 || (block_n != 128 && block_n != 256)) return OA_ERR_BAD_REQUEST;
    const StreamK sk = make_streamk(nullptr, N, K, block_n, n_ctas);
    if (sk.G > cap_ctas || sk.n_tiles > cap_tiles) return OA_ERR_BAD_REQUEST;
    for (int c = 0; c <= sk.G; ++c) cta_unit0_out[c] = (long long)c * sk.total / sk.G;            // the kernels' u0/u1
    for (int t = 0; t < sk.n_tiles; ++t) {                                                        // the very function the kernels call
        uint32_t cf, cl;
        sk_tile_ctas(sk, (uint32_t)t, cf, cl);
        tile_first_out[t] = (int32_t)cf; tile_last_out[t] = (int32_t)cl;
    }
    *n_ctas_out = sk.G; *n_tiles_out = sk.n_tiles; *kb_out = sk.kb;
    return OA_OK;
}

int oa_host_grammar_step(int32_t kind, const uint8_t* prefix, int32_t n, uint32_t* mask_out, int32_t* done_out) {
    return oa_host_grammar_step_ex(kind, "", prefix, n, mask_out, done_out);
}
int oa_host_grammar_step_ex(int32_t kind, const char* functions, const uint8_t* prefix, int32_t n, uint32_t* mask_out, int32_t* done_out) {
    if (kind < GRAMMAR_TOOLCALL || kind > GRAMMAR_TEXT) return OA_ERR_BAD_REQUEST;
    ToolPromptGrammar g(kind, functions ? functions : "");
    if (!g.active()) return OA_ERR_BAD_REQUEST;
    for (int i = 0; i < n; ++i) if (!g.advance(prefix[i])) return OA_ERR_BAD_REQUEST;
    g.allowed(mask_out); *done_out = g.done() ? 1 : 0;
    return OA_OK;
}

int oa_host_grammar_token_mask(const char* tokenizer_json_path, int32_t vocab, int32_t kind, const char* functions, const uint8_t* prefix, int32_t n,
                               uint32_t* mask_out, int32_t cap_words, char* key_out, int32_t key_cap) {
    if (kind < GRAMMAR_TOOLCALL || kind > GRAMMAR_TEXT || vocab <= 0 || !mask_out) return OA_ERR_BAD_REQUEST;
    try {
        // one trie per (tokenizer, vocab), built once: the same structure the engine builds at start-up
        static std::mutex mu; static std::map<std::string, std::shared_ptr<TokenTrie>> tries;
        const std::string tk = std::string(tokenizer_json_path ? tokenizer_json_path : "") + "#" + std::to_string(vocab);
        std::shared_ptr<TokenTrie> trie;
        {
            std::lock_guard<std::mutex> lk(mu);
            auto it = tries.find(tk);
            if (it == tries.end()) {
                ModelConfig mc; mc.vocab = vocab; mc.chat_template = "llama3";
                std::vector<std::string> bytes;
                if (tokenizer_json_path && tokenizer_json_path[0]) bytes = BpeTokenizer::load(tokenizer_json_path)->text_token_bytes();
                else { bytes.resize(256); for (int b = 0; b < 256; ++b) bytes[b] = std::string(1, (char)b); }
                trie = std::make_shared<TokenTrie>(); trie->build(bytes, vocab); tries[tk] = trie;
            } else trie = it->second;
        }
        if (trie->words() > cap_words) return OA_ERR_BAD_REQUEST;
        ToolPromptGrammar g(kind, functions ? functions : "");
        if (!g.active()) return OA_ERR_BAD_REQUEST;
        for (int i = 0; i < n; ++i) if (!g.advance(prefix[i])) return OA_ERR_BAD_REQUEST;
        trie->allowed_tokens(g, g.cursor(), mask_out);
        if (key_out && key_cap > 0) std::snprintf(key_out, (size_t)key_cap, "%s", grammar_mask_key(g, g.cursor()).c_str());
    } catch (const std::exception&) { return OA_ERR_BAD_REQUEST; }
    return OA_OK;
}

int oa_host_model_info(const char* config_json, char* buf, size_t n) {
    try {
        ModelConfig c; EngineOptions eo; parse_config(config_json ? config_json : "{}", c, eo);
        std::snprintf(buf, n, "{\"model\": \"%s\", \"hidden\": %d, \"n_layers\": %d, \"n_heads\": %d, \"n_kv_heads\": %d, \"head_dim\": %d, "
                      "\"ffn\": %d, \"vocab\": %d, \"tie_embeddings\": %d, \"qkv_bias\": %d, \"rope_scaling\": %d, \"rope_theta\": %.1f, "
                      "\"rms_eps\": %g, \"template\": \"%s\", \"decode_weight_bytes\": %.0f, \"kv_bytes_per_token\": %zu}",
                      c.name.c_str(), c.hidden, c.n_layers, c.n_heads, c.n_kv_heads, c.head_dim, c.ffn, c.vocab, c.tie_embeddings, c.qkv_bias,
                      c.rope_scaling, c.rope_theta, c.rms_eps, c.chat_template.c_str(), c.decode_weight_bytes(), c.kv_bytes_per_token());
    } catch (const std::exception&) { return OA_ERR_BAD_REQUEST; }
    return OA_OK;
}

}  // extern "C"
