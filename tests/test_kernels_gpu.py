"""Kernel-level parity on the B200 (pytest -m gpu): every hand-written sm_100a kernel through its C-ABI entry
point against (a) the CPU oracle where it has the same function and (b) a plain torch fp32 reference of the op."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from opsagent_b200 import _lib  # noqa: E402
from oracle import oracle as O  # noqa: E402  (checker only)

EPI_STORE, EPI_RESID, EPI_SWIGLU, EPI_LOGITS = 0, 1, 2, 3


@pytest.fixture(scope="module")
def L():
    return _lib.load()


def dev():
    return torch.device("cuda:0")


def ptr(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def bf16_bits(t):
    return t.view(torch.int16).cpu().numpy().view(np.uint16)


# ------------------------------------------------------------------------------------------------
def test_weight_init_bit_exact_vs_oracle(L):
    rows, cols = 96, 320
    dst = torch.empty(rows, cols, dtype=torch.bfloat16, device=dev())
    assert L.oa_k_init_weight(ptr(dst), 1234, 37, -1, rows, cols, 0.02, 0.0, None) == 0
    torch.cuda.synchronize()
    got = bf16_bits(dst)
    lib = O.lib()
    exp = np.array([lib.oa_ref_gen_bf16(1234, 37, i, 0.02, 0.0) for i in range(rows * cols)], dtype=np.uint16).reshape(rows, cols)
    assert (got == exp).all()
    # norm-gain style (mean 1) and the interleaved gate/up layout
    dst2 = torch.empty(1, cols, dtype=torch.bfloat16, device=dev())
    assert L.oa_k_init_weight(ptr(dst2), 99, 7, -1, 1, cols, 0.1, 1.0, None) == 0
    exp2 = np.array([lib.oa_ref_gen_bf16(99, 7, i, 0.1, 1.0) for i in range(cols)], dtype=np.uint16)
    torch.cuda.synchronize()
    assert (bf16_bits(dst2)[0] == exp2).all()
    F, H = 64, 64
    gu = torch.empty(2 * F, H, dtype=torch.bfloat16, device=dev())
    assert L.oa_k_init_weight(ptr(gu), 5, 4, 5, 2 * F, H, 0.02, 0.0, None) == 0
    torch.cuda.synchronize()
    g = np.array([lib.oa_ref_gen_bf16(5, 4, i, 0.02, 0.0) for i in range(F * H)], dtype=np.uint16).reshape(F, H)
    u = np.array([lib.oa_ref_gen_bf16(5, 5, i, 0.02, 0.0) for i in range(F * H)], dtype=np.uint16).reshape(F, H)
    got = bf16_bits(gu)
    for r in range(2 * F):
        blk, w = divmod(r, 32)
        src = g if w < 16 else u
        assert (got[r] == src[blk * 16 + (w & 15)]).all()


@pytest.mark.parametrize("T,H", [(1, 256), (7, 320), (128, 4096), (33, 8192), (5, 2048)])
def test_rmsnorm_vs_oracle(L, T, H):
    g = torch.Generator(device="cpu").manual_seed(T * 1000 + H)
    x = (torch.randn(T, H, generator=g) * 1.7).to(torch.bfloat16)
    gain = (1 + 0.1 * torch.randn(H, generator=g)).to(torch.bfloat16)
    xd, gd = x.to(dev()), gain.to(dev())
    y = torch.empty_like(xd)
    assert L.oa_k_rmsnorm(ptr(xd), ptr(gd), ptr(y), T, H, 1e-5, None) == 0
    torch.cuda.synchronize()
    xf = np.ascontiguousarray(x.float().numpy()); ref = np.empty_like(xf)
    gb = np.ascontiguousarray(bf16_bits(gain))
    O.lib().oa_ref_rmsnorm(xf.ctypes.data, gb.ctypes.data, ref.ctypes.data, T, H, 1e-5, 1)
    got = y.float().cpu().numpy()
    # identical up to the fp32-vs-double sum of squares: at most one bf16 ulp on a handful of elements
    ulp = np.maximum(np.abs(ref), 1e-3) * 2.0 ** -7
    assert (np.abs(got - ref) <= ulp).all()
    assert (got != ref).mean() < 0.02


GEMM_CASES = [  # M, N, K
    (128, 512, 256), (77, 256, 320), (300, 1024, 512), (1, 2304, 256), (128, 4096, 4096), (130, 1000, 192),
]


@pytest.mark.parametrize("bn", [32, 64, 128, 256])
@pytest.mark.parametrize("M,N,K", GEMM_CASES)
def test_gemm_store_and_bias(L, M, N, K, bn):
    g = torch.Generator(device="cpu").manual_seed(M + N + K + bn)
    A = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16).to(dev())
    B = (torch.randn(N, K, generator=g) * 0.5).to(torch.bfloat16).to(dev())
    bias = torch.randn(N, generator=g).to(torch.bfloat16).to(dev())
    ref = A.float() @ B.float().T
    for use_bias in (False, True):
        out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=dev())
        assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_STORE, bn, ptr(out), ptr(bias) if use_bias else None, None, None, None, None) == 0
        torch.cuda.synchronize()
        r = ref + bias.float() if use_bias else ref
        err = (out.float() - r).abs()
        tol = r.abs() * 2.0 ** -8 + 2e-3 * (K ** 0.5) * 0.25 * 2.0 ** -8 + 1e-4
        assert torch.isfinite(out.float()).all()
        assert (err <= tol * 1.01 + 1e-3).all(), float((err - tol).max())


@pytest.mark.parametrize("bn", [32, 128, 256])
def test_gemm_residual_in_place(L, bn):
    M, N, K = 200, 768, 512
    g = torch.Generator(device="cpu").manual_seed(bn)
    A = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16).to(dev())
    B = (torch.randn(N, K, generator=g) * 0.5).to(torch.bfloat16).to(dev())
    x = torch.randn(M, N, generator=g).to(torch.bfloat16).to(dev())
    ref = (A.float() @ B.float().T + x.float()).to(torch.bfloat16)
    assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_RESID, bn, ptr(x), None, ptr(x), None, None, None) == 0
    torch.cuda.synchronize()
    diff = (x.float() - ref.float()).abs()
    assert (diff <= ref.float().abs() * 2.0 ** -7 + 1e-3).all()
    assert (x != ref).float().mean() < 0.01      # only accumulation-order rounding flips


@pytest.mark.parametrize("bn", [32, 64, 128, 256])
def test_gemm_swiglu(L, bn):
    M, F, K = 150, 512, 256
    g = torch.Generator(device="cpu").manual_seed(bn + 1)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16).to(dev())
    Wg = (torch.randn(F, K, generator=g) * 0.1).to(torch.bfloat16)
    Wu = (torch.randn(F, K, generator=g) * 0.1).to(torch.bfloat16)
    # physical layout: 16 gate rows then 16 up rows per 32-row block
    W = torch.stack([Wg.view(F // 16, 16, K), Wu.view(F // 16, 16, K)], dim=1).reshape(2 * F, K).contiguous().to(dev())
    out = torch.empty(M, F, dtype=torch.bfloat16, device=dev())
    assert L.oa_k_gemm(ptr(A), ptr(W), M, 2 * F, K, EPI_SWIGLU, bn, ptr(out), None, None, None, None, None) == 0
    torch.cuda.synchronize()
    gt = A.float() @ Wg.to(dev()).float().T
    up = A.float() @ Wu.to(dev()).float().T
    ref = torch.nn.functional.silu(gt) * up
    assert ((out.float() - ref).abs() <= ref.abs() * 2.0 ** -7 + 2e-3).all()


@pytest.mark.parametrize("bn", [64, 256])
@pytest.mark.parametrize("M,N,K", [(128, 2304, 256), (3, 1280, 320), (200, 128256, 256)])
def test_gemm_logits_argmax(L, M, N, K, bn):
    g = torch.Generator(device="cpu").manual_seed(N + bn)
    A = torch.randn(M, K, generator=g).to(torch.bfloat16).to(dev())
    B = (torch.randn(N, K, generator=g) * 0.1).to(torch.bfloat16).to(dev())
    logits = torch.empty(M, N, dtype=torch.float32, device=dev())
    ids = torch.empty(M, dtype=torch.int32, device=dev())
    assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_LOGITS, bn, None, None, None, ptr(logits), ptr(ids), None) == 0
    torch.cuda.synchronize()
    ref = A.float() @ B.float().T
    assert ((logits - ref).abs() <= 1e-4 * (K ** 0.5) + 1e-5 * ref.abs()).all()
    # fused arg-max is exact on the kernel's own logits, ties -> lowest index
    mx = logits.max(dim=1, keepdim=True).values
    first = torch.where(logits == mx, torch.arange(N, device=dev())[None, :], N).min(dim=1).values
    assert (ids.long() == first).all()
    # ... and without materialising logits
    ids2 = torch.empty(M, dtype=torch.int32, device=dev())
    assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_LOGITS, bn, None, None, None, None, ptr(ids2), None) == 0
    assert (ids2 == ids).all()


@pytest.mark.parametrize("M,N,K", [(5000, 2304, 320), (300, 1024, 512), (8192, 6144, 256)])
def test_gemm_persistent_kernel_all_epilogues(L, M, N, K, monkeypatch):
    """prefill path: persistent 128x256 tiles, double-buffered TMEM, transposed coalesced epilogue (forced for small shapes)"""
    monkeypatch.setenv("OA_GEMM_PERSISTENT_MIN_TILES", "1")
    g = torch.Generator(device="cpu").manual_seed(M + N)
    A = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16).to(dev())
    B = (torch.randn(N, K, generator=g) * 0.5).to(torch.bfloat16).to(dev())
    bias = torch.randn(N, generator=g).to(torch.bfloat16).to(dev())
    ref = A.float() @ B.float().T
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=dev())
    assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_STORE, 256, ptr(out), ptr(bias), None, None, None, None) == 0
    torch.cuda.synchronize()
    r = ref + bias.float()
    assert torch.isfinite(out.float()).all()
    assert ((out.float() - r).abs() <= r.abs() * 2.0 ** -8 * 1.01 + 2e-3).all()
    x = torch.randn(M, N, generator=g).to(torch.bfloat16).to(dev())
    refx = (ref + x.float()).to(torch.bfloat16)
    assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_RESID, 256, ptr(x), None, ptr(x), None, None, None) == 0
    torch.cuda.synchronize()
    assert ((x.float() - refx.float()).abs() <= refx.float().abs() * 2.0 ** -7 + 1e-3).all()
    F = N // 2
    out2 = torch.full((M, F), float("nan"), dtype=torch.bfloat16, device=dev())
    assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_SWIGLU, 256, ptr(out2), None, None, None, None, None) == 0
    torch.cuda.synchronize()
    acc = ref.view(M, N // 32, 2, 16)
    rs = (torch.nn.functional.silu(acc[:, :, 0]) * acc[:, :, 1]).reshape(M, F)
    assert torch.isfinite(out2.float()).all()
    assert ((out2.float() - rs).abs() <= rs.abs() * 2.0 ** -7 + 3e-3).all()


@pytest.mark.parametrize("bn", [128, 256])
@pytest.mark.parametrize("M,N,K,G", [(128, 4096, 4096, 148), (128, 6144, 4096, 148), (77, 1024, 14336, 148), (1, 320, 320, 148),
                                      (128, 28672, 4096, 148), (16, 2304, 256, 5), (128, 512, 512, 3), (100, 1000, 192, 148),
                                      (256, 4096, 4096, 148), (200, 1792, 5120, 148), (129, 320, 320, 7)])
def test_gemm_streamk_partials_sum_to_the_product(L, M, N, K, G, bn):
    if M > 128 and bn != 128:
        pytest.skip("two 128-row tiles need BN=128 (TMEM columns)")
    g = torch.Generator(device="cpu").manual_seed(N + K + bn + G)
    A = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16).to(dev())
    B = (torch.randn(N, K, generator=g) * 0.5).to(torch.bfloat16).to(dev())
    out = torch.full((M, N), float("nan"), dtype=torch.float32, device=dev())
    assert L.oa_k_gemm_streamk(ptr(A), ptr(B), M, N, K, bn, G, ptr(out), None) == 0, _lib.last_error()
    ref = A.float() @ B.float().T
    assert torch.isfinite(out).all()
    assert ((out - ref).abs() <= 2e-4 * (K ** 0.5) + 1e-5 * ref.abs()).all(), float((out - ref).abs().max())
    # fixed summation order => bitwise reproducible run to run
    out2 = torch.empty_like(out)
    assert L.oa_k_gemm_streamk(ptr(A), ptr(B), M, N, K, bn, G, ptr(out2), None) == 0
    assert torch.equal(out, out2)


# ------------------------------------------------------------------------------------------------
def _attn_ref(q, kcache, vcache, bt, ctx, qlens, nh, nkv, D):
    """fp32 reference of paged causal GQA attention.  q: [sum(qlens), nh, D]"""
    grp = nh // nkv
    outs, row = [], 0
    for i, (c, ql) in enumerate(zip(ctx, qlens)):
        pages = bt[i, : (c + 63) // 64]
        K = kcache[pages].permute(0, 2, 1, 3).reshape(-1, nkv, D)[:c].float()    # [c, nkv, D]
        V = vcache[pages].permute(0, 2, 1, 3).reshape(-1, nkv, D)[:c].float()
        qi = q[row:row + ql].float()                                              # [ql, nh, D]
        Kh = K.repeat_interleave(grp, dim=1); Vh = V.repeat_interleave(grp, dim=1)
        s = torch.einsum("qhd,khd->hqk", qi, Kh) / (D ** 0.5)
        qpos = torch.arange(c - ql, c, device=q.device)[:, None]; kpos = torch.arange(c, device=q.device)[None, :]
        s = s.masked_fill((kpos > qpos)[None], float("-inf"))
        p = torch.softmax(s, dim=-1)
        outs.append(torch.einsum("hqk,khd->qhd", p, Vh)); row += ql
    return torch.cat(outs, 0)


def _mk_cache(num_pages, nkv, D, seed):
    g = torch.Generator(device="cpu").manual_seed(seed)
    kv = torch.randn(2, num_pages, nkv, 64, D, generator=g).to(torch.bfloat16).to(dev())
    return kv


@pytest.mark.parametrize("splits", [0, 3])
@pytest.mark.parametrize("nh,nkv,D", [(32, 8, 128), (8, 2, 64), (5, 1, 64), (8, 1, 128), (40, 8, 128)])
def test_paged_decode_attention(L, nh, nkv, D, splits):
    ctx = [1, 63, 64, 65, 200, 1000, 129, 517]
    n = len(ctx); maxp = 20; num_pages = 150
    kv = _mk_cache(num_pages, nkv, D, 11)
    g = torch.Generator(device="cpu").manual_seed(5)
    perm = torch.randperm(num_pages, generator=g)
    bt = torch.zeros(n, maxp, dtype=torch.int32); k = 0
    for i, c in enumerate(ctx):
        npg = (c + 63) // 64; bt[i, :npg] = perm[k:k + npg].to(torch.int32); k += npg
    q = torch.randn(n, nh, D, generator=g).to(torch.bfloat16).to(dev())
    out = torch.full((n, nh, D), float("nan"), dtype=torch.bfloat16, device=dev())
    ctx_a = np.array(ctx, np.int32); ql = np.ones(n, np.int32); bt_np = np.ascontiguousarray(bt.numpy())
    rc = L.oa_k_paged_attention(ptr(q), ptr(out), ptr(kv), num_pages, bt_np.ctypes.data, maxp, ctx_a.ctypes.data, ql.ctypes.data, n,
                                nh, nkv, D, splits, None)
    assert rc == 0, _lib.last_error()
    ref = _attn_ref(q, kv[0], kv[1], bt.to(dev()).long(), ctx, [1] * n, nh, nkv, D)
    err = (out.float() - ref).abs().max().item()
    assert torch.isfinite(out.float()).all()
    assert err < 2e-2, err


@pytest.mark.parametrize("nh,nkv,D", [(8, 2, 128), (4, 2, 64), (5, 1, 64)])
def test_paged_prefill_attention(L, nh, nkv, D):
    # (ctx after the chunk, new rows): fresh prompts, a chunk continuing a cached prefix, ragged tile tails
    cases = [(64, 64), (130, 130), (200, 37), (1, 1), (333, 100), (128, 128)]
    ctx = [c for c, _ in cases]; qlens = [q for _, q in cases]
    n = len(ctx); maxp = 8; num_pages = 40
    kv = _mk_cache(num_pages, nkv, D, 3)
    g = torch.Generator(device="cpu").manual_seed(9)
    perm = torch.randperm(num_pages, generator=g)
    bt = torch.zeros(n, maxp, dtype=torch.int32); k = 0
    for i, c in enumerate(ctx):
        npg = (c + 63) // 64; bt[i, :npg] = perm[k:k + npg].to(torch.int32); k += npg
    T = sum(qlens)
    q = torch.randn(T, nh, D, generator=g).to(torch.bfloat16).to(dev())
    out = torch.full((T, nh, D), float("nan"), dtype=torch.bfloat16, device=dev())
    ctx_a = np.array(ctx, np.int32); ql = np.array(qlens, np.int32); bt_np = np.ascontiguousarray(bt.numpy())
    rc = L.oa_k_paged_attention(ptr(q), ptr(out), ptr(kv), num_pages, bt_np.ctypes.data, maxp, ctx_a.ctypes.data, ql.ctypes.data, n,
                                nh, nkv, D, 0, None)
    assert rc == 0, _lib.last_error()
    ref = _attn_ref(q, kv[0], kv[1], bt.to(dev()).long(), ctx, qlens, nh, nkv, D)
    assert torch.isfinite(out.float()).all()
    err = (out.float() - ref).abs().max().item()
    assert err < 2e-2, err


# prefill attention's kernels that take such heads, by the names that OA_PREFILL_ATTN asks for
def _prefill_kernels(nh, nkv, D):
    return ["one_head", "two_heads"] + (["turns"] if D == 64 or nh // nkv % 2 == 0 else [])


# An output may only be read once its last products have landed, however late their values come: one to six key tiles, keys in L2 and values not, full and ragged last
# tiles; in every kernel, a prompt alone and among copies of itself, with the same bits
@pytest.mark.parametrize("nh,nkv,D", [(8, 2, 128), (16, 4, 64), (10, 2, 128), (15, 3, 64)])
@pytest.mark.parametrize("ctx,rows", [(128, 128), (256, 128), (256, 100), (257, 129), (512, 32), (700, 33), (700, 200)])
def test_prefill_output_waits_for_the_last_values(L, monkeypatch, nh, nkv, D, ctx, rows):
    pages, maxp = (ctx + 63) // 64, (ctx + 63) // 64
    kv = _mk_cache(pages, nkv, D, 41)
    g = torch.Generator(device="cpu").manual_seed(12)
    q1 = torch.randn(rows, nh, D, generator=g).to(torch.bfloat16).to(dev())
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev())

    def attend(copies, kernel):
        monkeypatch.setenv("OA_PREFILL_ATTN", kernel)
        q = q1.repeat(copies, 1, 1).contiguous()
        out = torch.full_like(q, float("nan"))
        bt = np.tile(np.arange(pages, dtype=np.int32)[::-1], (copies, 1)).copy()
        c, n = np.full(copies, ctx, np.int32), np.full(copies, rows, np.int32)
        flush.zero_(); kv[0].float().sum().item()
        assert L.oa_k_paged_attention(ptr(q), ptr(out), ptr(kv), pages, bt.ctypes.data, maxp, c.ctypes.data, n.ctypes.data, copies, nh, nkv, D, 0, None) == 0, _lib.last_error()
        return out

    want = attend(40, "two_heads")
    ref = _attn_ref(q1, kv[0], kv[1], torch.arange(pages - 1, -1, -1, device=dev())[None], [ctx], [rows], nh, nkv, D)
    # probabilities and result are rounded to bf16 (2^-9 relative each); |values| stay below 5
    assert (want[:rows].float() - ref).abs().max().item() < 2 * 5 * 2.0 ** -8
    assert torch.equal(want, want[:rows].repeat(40, 1, 1))
    for kernel in _prefill_kernels(nh, nkv, D):
        for _ in range(5):
            assert torch.equal(attend(1, kernel), want[:rows]), kernel
        assert torch.equal(attend(40, kernel), want), kernel


# Batches that fill the chip, in every kernel: an even and an odd number of heads per group (two heads a CTA leave the last head of an odd group alone), portions behind a
# cached prefix, tiles of one row, key tiles whose second page is missing, and more items than CTAs
@pytest.mark.parametrize("nh,nkv,D,kernel", [(*h, k) for h in [(32, 8, 128), (20, 4, 128), (32, 8, 64), (15, 3, 64), (16, 2, 128)] for k in _prefill_kernels(*h)])
def test_paged_prefill_attention_of_full_batches(L, monkeypatch, nh, nkv, D, kernel):
    monkeypatch.setenv("OA_PREFILL_ATTN", kernel)
    cases = [(64, 64), (130, 130), (200, 37), (1, 1), (700, 513), (128, 128), (65, 65), (449, 1), (333, 300), (1000, 129)] * 2
    ctx = [c for c, _ in cases]; qlens = [q for _, q in cases]
    n = len(ctx); maxp = 16; num_pages = 140
    kv = _mk_cache(num_pages, nkv, D, 3)
    g = torch.Generator(device="cpu").manual_seed(9)
    perm = torch.randperm(num_pages, generator=g)
    bt = torch.zeros(n, maxp, dtype=torch.int32); k = 0
    for i, c in enumerate(ctx):
        npg = (c + 63) // 64; bt[i, :npg] = perm[k:k + npg].to(torch.int32); k += npg
    T = sum(qlens)
    q = torch.randn(T, nh, D, generator=g)
    q[::7] *= 12                                     # scores that raise a row's maximum by more than 2^8 in a later tile
    q[5, 0, 3] = float("nan")                        # a query with a NaN: its own result, and nothing else, is NaN
    q = q.to(torch.bfloat16).to(dev())
    out = torch.full((T, nh, D), 7.0, dtype=torch.bfloat16, device=dev())
    ctx_a = np.array(ctx, np.int32); ql = np.array(qlens, np.int32); bt_np = np.ascontiguousarray(bt.numpy())
    rc = L.oa_k_paged_attention(ptr(q), ptr(out), ptr(kv), num_pages, bt_np.ctypes.data, maxp, ctx_a.ctypes.data, ql.ctypes.data, n,
                                nh, nkv, D, 0, None)
    assert rc == 0, _lib.last_error()
    ref = _attn_ref(q, kv[0], kv[1], bt.to(dev()).long(), ctx, qlens, nh, nkv, D)
    assert torch.equal(torch.isnan(out), torch.isnan(ref)) and torch.isnan(out).sum().item() == D
    # probabilities and result are rounded to bf16 (2^-9 relative each); |values| stay below 5
    err = (out.float() - ref).nan_to_num().abs().max().item()
    assert err < 2 * 5 * 2.0 ** -8, err


# One head a CTA, two heads a CTA, key tiles in turns on a CTA pair (heads of 128, even groups) or a CTA (heads of 64): a batch takes the kernel that the estimate of its time
# names, and a row's bits are the same in all.  Items of one, two, three and many key tiles (in turns two warpgroups take them: odd and even ends, items shorter than what is
# on its way), a last tile without its second page, fewer and more items than CTAs, references raised in later tiles
@pytest.mark.parametrize("nh,nkv,D", [(8, 4, 128), (16, 2, 128), (10, 2, 128), (12, 4, 64), (16, 2, 64), (4, 4, 64)])
@pytest.mark.parametrize("ctx,rows", [(2, 2), (64, 64), (128, 128), (129, 129), (256, 255), (384, 130), (449, 33), (1000, 130), (1280, 65)])
def test_prefill_attention_kernels_agree(L, monkeypatch, nh, nkv, D, ctx, rows):
    pages = (ctx + 63) // 64
    kv = _mk_cache(pages, nkv, D, 5)
    g = torch.Generator(device="cpu").manual_seed(ctx)
    q1 = torch.randn(rows, nh, D, generator=g)
    q1[::5] *= 9
    q1 = q1.to(torch.bfloat16).to(dev())

    def attend(copies, kernel):
        if kernel:
            monkeypatch.setenv("OA_PREFILL_ATTN", kernel)
        else:
            monkeypatch.delenv("OA_PREFILL_ATTN")
        q = q1.repeat(copies, 1, 1).contiguous()
        out = torch.full_like(q, float("nan"))
        c, n, bt = np.full(copies, ctx, np.int32), np.full(copies, rows, np.int32), np.tile(np.arange(pages, dtype=np.int32)[::-1], (copies, 1)).copy()
        rc = L.oa_k_paged_attention(ptr(q), ptr(out), ptr(kv), pages, bt.ctypes.data, pages, c.ctypes.data, n.ctypes.data, copies, nh, nkv, D, 0, None)
        return out if rc == 0 else None

    first = attend(1, "one_head")
    ref = _attn_ref(q1, kv[0], kv[1], torch.arange(pages - 1, -1, -1, device=dev())[None], [ctx], [rows], nh, nkv, D)
    # probabilities and result are rounded to bf16 (2^-9 relative each); |values| stay below 5
    assert (first.float() - ref).abs().max().item() < 2 * 5 * 2.0 ** -8
    kernels = _prefill_kernels(nh, nkv, D)
    for copies in (1, 7, 75):
        for kernel in [*kernels, None]:
            assert torch.equal(attend(copies, kernel), first.repeat(copies, 1, 1)), (copies, kernel)
    if "turns" not in kernels:                       # heads that a kernel does not take are refused, not given to another
        assert attend(1, "turns") is None


def _decode_route(L, ctx, nkv):
    """segments, CTAs and partial slots of the plan that a decoding batch runs on 148 SMs"""
    ctx = np.ascontiguousarray(ctx, np.int32); cap = int(((ctx + 63) // 64).sum()) * nkv + 512
    segs, cta_ptr = np.zeros((cap, 5), np.int32), np.zeros(cap + 1, np.int32)
    n = [C.c_int32() for _ in range(3)]
    assert L.oa_host_decode_attention_plan(ctx.ctypes.data, len(ctx), nkv, 296, 0, segs.ctypes.data, cap, cta_ptr.ctypes.data, cap, *[C.byref(x) for x in n]) == 0
    return n[1].value, n[0].value, n[2].value


# few long contexts: an item is cut over up to 37 CTAs and the last of them merges the pieces (one, two, several, more than four at a time)
@pytest.mark.parametrize("ctx,nh,nkv,D", [([9000], 32, 8, 128), ([9001, 5, 70], 16, 2, 128), ([5000, 64], 32, 8, 64), ([700], 5, 1, 64), ([3333, 3334, 129], 40, 8, 128)])
def test_paged_decode_attention_merges_many_pieces(L, ctx, nh, nkv, D):
    segs, ctas, slots = _decode_route(L, ctx, nkv)
    assert slots > 0 and ctas != len(ctx) * nkv          # items shared by CTAs
    n = len(ctx); maxp = (max(ctx) + 63) // 64; num_pages = sum((c + 63) // 64 for c in ctx)
    kv = _mk_cache(num_pages, nkv, D, 17)
    g = torch.Generator(device="cpu").manual_seed(6)
    perm = torch.randperm(num_pages, generator=g)
    bt = torch.zeros(n, maxp, dtype=torch.int32); k = 0
    for i, c in enumerate(ctx):
        npg = (c + 63) // 64; bt[i, :npg] = perm[k:k + npg].to(torch.int32); k += npg
    q = (torch.randn(n, nh, D, generator=g) * 2).to(torch.bfloat16).to(dev())
    out = torch.full((n, nh, D), float("nan"), dtype=torch.bfloat16, device=dev())
    ctx_a = np.array(ctx, np.int32); bt_np = np.ascontiguousarray(bt.numpy())
    for _ in range(2):
        assert L.oa_k_paged_attention(ptr(q), ptr(out), ptr(kv), num_pages, bt_np.ctypes.data, maxp, ctx_a.ctypes.data, None, n, nh, nkv, D, 0, None) == 0, _lib.last_error()
    ref = _attn_ref(q, kv[0], kv[1], bt.to(dev()).long(), ctx, [1] * n, nh, nkv, D)
    # probabilities and result are rounded to bf16 (2^-9 relative each); |values| stay below 3
    assert (out.float() - ref).abs().max().item() < 2 * 3 * 2.0 ** -8


# a sequence more that is one chunk above the line takes the batch from one CTA an item to shared items, and leaves the pieces of the others where they are
@pytest.mark.parametrize("n,nh,nkv,D,ctx", [(10, 5, 1, 64, 320), (12, 8, 1, 128, 257), (6, 32, 8, 128, 319), (16, 32, 8, 64, 320), (28, 40, 8, 128, 257)])
def test_decode_rows_keep_their_bits_whoever_runs_their_pieces(L, n, nh, nkv, D, ctx):
    per = -(-5 * n * nkv // min(296, 5 * n * nkv // 2))
    last = 64 * (per + 4)
    assert per == -(-(5 * n + per + 4) * nkv // min(296, (5 * n + per + 4) * nkv // 2))
    lens = [ctx] * n + [last]
    num_pages = 5 * n + per + 4
    kv = _mk_cache(num_pages, nkv, D, 23)
    g = torch.Generator(device="cpu").manual_seed(9)
    bt = np.zeros((n + 1, per + 4), np.int32); perm = torch.randperm(num_pages, generator=g).numpy(); k = 0
    for i, c in enumerate(lens):
        npg = (c + 63) // 64; bt[i, :npg] = perm[k:k + npg]; k += npg
    q = (torch.randn(n + 1, nh, D, generator=g) * 2).to(torch.bfloat16).to(dev())
    outs = []
    for m, together in ((n, True), (n + 1, False)):
        segs, ctas, slots = _decode_route(L, lens[:m], nkv)
        assert (ctas == m * nkv) == together and slots > 0
        out = torch.full((m, nh, D), float("nan"), dtype=torch.bfloat16, device=dev())
        a = np.array(lens[:m], np.int32)
        assert L.oa_k_paged_attention(ptr(q), ptr(out), ptr(kv), num_pages, bt.ctypes.data, per + 4, a.ctypes.data, None, m, nh, nkv, D, 0, None) == 0, _lib.last_error()
        outs.append(out)
    assert not torch.isnan(outs[1]).any() and torch.equal(outs[0], outs[1][:n])


# all pieces of an item on one CTA or shared items: batches on both sides of the line (3 chunks above an equal share; one item more than CTAs)
@pytest.mark.parametrize("D", [128, 64])
@pytest.mark.parametrize("nh,nkv,ctx,together", [(8, 1, [320], True), (8, 1, [321], False), (8, 1, [640], False), (8, 1, [641], False), (32, 8, [320] * 2 + [1], True),
                                                 (32, 8, [321] * 2 + [1], False), (32, 8, [640] * 2 + [1], False),
                                                 (32, 8, [1] * 7 + [1152], False), (32, 8, [1] * 7 + [1153], False), (32, 8, [3] * 6 + [320], True),
                                                 (32, 8, [3] * 6 + [321], False), (32, 8, [640] + [3] * 6, False), (32, 8, [641] + [3] * 6, False),
                                                 (32, 8, [70, 300, 5, 129] * 9 + [64], True), (32, 8, [70, 300, 5, 129] * 9 + [64, 65], False), (12, 4, list(range(1, 741, 10)), False),
                                                 (12, 4, list(range(1, 449, 7)), True)])
def test_decode_attention_whole_items_and_cut_ones(L, nh, nkv, D, ctx, together):
    assert (_decode_route(L, ctx, nkv)[1] == len(ctx) * nkv) == together
    n = len(ctx); maxp = (max(ctx) + 63) // 64; num_pages = sum((c + 63) // 64 for c in ctx)
    kv = _mk_cache(num_pages, nkv, D, 19)
    g = torch.Generator(device="cpu").manual_seed(8)
    perm = torch.randperm(num_pages, generator=g)
    bt = torch.zeros(n, maxp, dtype=torch.int32); k = 0
    for i, c in enumerate(ctx):
        npg = (c + 63) // 64; bt[i, :npg] = perm[k:k + npg].to(torch.int32); k += npg
    q = (torch.randn(n, nh, D, generator=g) * 2).to(torch.bfloat16).to(dev())
    out = torch.full((n, nh, D), float("nan"), dtype=torch.bfloat16, device=dev())
    ctx_a = np.array(ctx, np.int32); bt_np = np.ascontiguousarray(bt.numpy())
    for _ in range(2):
        assert L.oa_k_paged_attention(ptr(q), ptr(out), ptr(kv), num_pages, bt_np.ctypes.data, maxp, ctx_a.ctypes.data, None, n, nh, nkv, D, 0, None) == 0, _lib.last_error()
    ref = _attn_ref(q, kv[0], kv[1], bt.to(dev()).long(), ctx, [1] * n, nh, nkv, D)
    # probabilities and result are rounded to bf16 (2^-9 relative each); a mean of unit normals weighted by them stays below 4.5, alone (one token) or not
    assert (out.float() - ref).abs().max().item() < 2 * 4.5 * 2.0 ** -8


def test_attention_calls_of_several_threads(L):
    """calls of different sizes at once, each on a stream of its own: none sees another's tables (one of the tables is larger than what is kept between calls)"""
    import threading
    nh, nkv, D = 32, 8, 128
    jobs = []
    for k, (ctx, qlens, maxp) in enumerate([([70, 300, 5], None, 8), ([1000] * 40, None, 20), ([130, 64], [130, 10], 4), ([400, 90, 33], [33, 90, 1], 150000)]):
        n, pages = len(ctx), sum((c + 63) // 64 for c in ctx)
        kv = _mk_cache(pages, nkv, D, 30 + k)
        bt = np.zeros((n, maxp), np.int32); at = 0
        for i, c in enumerate(ctx):
            npg = (c + 63) // 64; bt[i, :npg] = np.arange(at, at + npg)[::-1]; at += npg
        q = torch.randn(sum(qlens or [1] * n), nh, D, generator=torch.Generator(device="cpu").manual_seed(k)).to(torch.bfloat16).to(dev())
        jobs.append((q, kv, pages, bt, maxp, np.array(ctx, np.int32), np.array(qlens, np.int32) if qlens else None, n))

    def attend(job, out, stream):
        q, kv, pages, bt, maxp, ctx, ql, n = job
        return L.oa_k_paged_attention(ptr(q), ptr(out), ptr(kv), pages, bt.ctypes.data, maxp, ctx.ctypes.data, ql.ctypes.data if ql is not None else None, n, nh, nkv, D, 0, stream)

    want = []
    for job in jobs:
        out = torch.empty_like(job[0]); assert attend(job, out, None) == 0; want.append(out)
    bad = []

    def work(t):
        stream = torch.cuda.Stream()
        for r in range(20):
            k = (t + r) % len(jobs)
            out = torch.full_like(jobs[k][0], float("nan"))
            stream.wait_stream(torch.cuda.current_stream())
            rc = attend(jobs[k], out, C.c_void_p(stream.cuda_stream))
            if rc != 0 or not torch.equal(out, want[k]):
                bad.append((t, r, k, rc))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad, bad[:5]


def test_streamk_result_on_any_float_boundary(L):
    M, N, K = 37, 1000, 320
    g = torch.Generator(device="cpu").manual_seed(1)
    A = (torch.randn(M, K, generator=g) * 0.5).to(torch.bfloat16).to(dev()); B = (torch.randn(N, K, generator=g) * 0.5).to(torch.bfloat16).to(dev())
    whole = torch.empty(M * N + 1, dtype=torch.float32, device=dev())
    out = torch.empty(M, N, dtype=torch.float32, device=dev())
    assert L.oa_k_gemm_streamk(ptr(A), ptr(B), M, N, K, 128, 148, ptr(out), None) == 0
    assert L.oa_k_gemm_streamk(ptr(A), ptr(B), M, N, K, 128, 148, ptr(whole[1:]), None) == 0
    assert torch.equal(whole[1:].view(M, N), out)


TILE, FEW, PERSISTENT, PAIR, HEAD = 0, 1, 2, 3, 4                  # oa_host_gemm_kernel


# CTA-pair kernel: one round of tiles and several, ragged last rows and columns, one CTA's rows all beyond the last, and k ranges shorter than the ring
# over many tiles (ring phases run across tiles, accumulators change hands every block or two); store, residual and gated.  Which kernel a product takes, and
# whose rows are the 256 of its tiles, is asserted: a rule that moves must not empty a case.
PAIR_TOKENS = [(257, 6144, 320), (257, 6152, 192), (700, 6152, 2056), (400, 2048, 8192), (449, 8192, 1032), (1000, 4096, 4096), (1000, 5120, 4160), (384, 296, 27648), (2000, 1000, 8192),
               (7900, 14336, 320), (8192, 24576, 192)]
PAIR_WEIGHTS = [(614, 6144, 4096), (257, 6152, 4096), (614, 4096, 14336), (1337, 4096, 14336)]


@pytest.mark.parametrize("M,N,K,swapped", [(*c, 0) for c in PAIR_TOKENS] + [(*c, 1) for c in PAIR_WEIGHTS])
def test_gemm_cta_pairs(L, M, N, K, swapped):
    assert L.oa_host_gemm_kernel(M, N, K, EPI_STORE, 256, 1, 0) == PAIR
    assert (L.oa_host_gemm_pair_width(M, N, K, EPI_STORE, 256) > 0) == (not swapped) and (L.oa_host_gemm_pair_swapped(M, N, K, EPI_STORE, 256) > 0) == bool(swapped)
    g = torch.Generator(device=dev()).manual_seed(M + N + K)
    A = torch.randn(M, K, generator=g, device=dev()).to(torch.bfloat16)
    B = (torch.randn(N, K, generator=g, device=dev()) * 0.05).to(torch.bfloat16)
    ref = A.double() @ B.double().T
    bias = torch.randn(N, generator=g, device=dev()).to(torch.bfloat16)
    # bf16 result: half an ulp (2^-9 relative) of the rounded value plus what fp32 sums of K products may be off by
    def close(got, want, extra=0.0):
        s = 0.05 * K ** 0.5 * K * 2.0 ** -24
        assert torch.isfinite(got.float()).all()
        assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + s + extra + 1e-6).all(), float((got.double() - want).abs().max())
    outs = []
    for _ in range(2):                               # the order of summation is fixed
        out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=dev())
        assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_STORE, 256, ptr(out), ptr(bias), None, None, None, None) == 0
        torch.cuda.synchronize(); outs.append(out)
    assert torch.equal(outs[0], outs[1])
    close(outs[0], ref + bias.double())
    x = torch.randn(M, N, generator=g, device=dev()).to(torch.bfloat16)
    want = ref + x.double()
    assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_RESID, 256, ptr(x), None, ptr(x), None, None, None) == 0       # in place
    torch.cuda.synchronize()
    close(x, want)
    if N % 32 == 0:
        y = torch.full((M, N // 2), float("nan"), dtype=torch.bfloat16, device=dev())
        assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_SWIGLU, 256, ptr(y), None, None, None, None, None) == 0
        torch.cuda.synchronize()
        v = ref.view(M, N // 32, 2, 16)
        close(y, (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(M, N // 2), 2e-5 * float(v.abs().max()) ** 2)


# products of a few rows: every box of loaded rows and the plain tile behind the last, fewer k blocks than ring stages and more, ragged rows and columns,
# tiles for one CTA per SM and for two; store, residual and gated
ROWS_CASES = [(1, 1024, 1088), (3, 2048, 4096), (16, 28672, 320), (17, 4096, 2056), (16, 9000, 1024), (32, 6144, 4160), (33, 2048, 1024), (64, 1000, 8192), (50, 6208, 4096), (65, 2048, 4096), (128, 4096, 4160), (100, 296, 14336)]


@pytest.mark.parametrize("M,N,K", ROWS_CASES)
def test_gemm_few_rows(L, M, N, K):
    assert L.oa_host_gemm_kernel(M, N, K, EPI_STORE, 128, 1, 0) == (FEW if M <= 64 else TILE)
    g = torch.Generator(device=dev()).manual_seed(M + N + K)
    A = torch.randn(M, K, generator=g, device=dev()).to(torch.bfloat16)
    B = (torch.randn(N, K, generator=g, device=dev()) * 0.05).to(torch.bfloat16)
    ref = A.double() @ B.double().T
    bias = torch.randn(N, generator=g, device=dev()).to(torch.bfloat16)
    # bf16 result: half an ulp (2^-9 relative) of the rounded value plus what fp32 sums of K products may be off by
    def close(got, want, extra=0.0):
        s = 0.05 * K ** 0.5 * K * 2.0 ** -24
        assert torch.isfinite(got.float()).all()
        assert ((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + s + extra + 1e-6).all(), float((got.double() - want).abs().max())
    outs = []
    for use_bias in (True, True, False):
        out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=dev())
        assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_STORE, 128, ptr(out), ptr(bias) if use_bias else None, None, None, None, None) == 0
        torch.cuda.synchronize(); outs.append(out)
    assert torch.equal(outs[0], outs[1])             # a fixed order of summation
    close(outs[0], ref + bias.double()); close(outs[2], ref)
    x = torch.randn(M, N, generator=g, device=dev()).to(torch.bfloat16)
    want = ref + x.double()
    assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_RESID, 128, ptr(x), None, ptr(x), None, None, None) == 0
    torch.cuda.synchronize()
    close(x, want)
    if N % 32 == 0:
        y = torch.full((M, N // 2), float("nan"), dtype=torch.bfloat16, device=dev())
        assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_SWIGLU, 128, ptr(y), None, None, None, None, None) == 0
        torch.cuda.synchronize()
        v = ref.view(M, N // 32, 2, 16)
        close(y, (torch.nn.functional.silu(v[:, :, 0]) * v[:, :, 1]).reshape(M, N // 2), 2e-5 * float(v.abs().max()) ** 2)


# a stage of the few-row form holds four k blocks (32-column tiles of up to 32 rows), two (of 64 rows; 64-column tiles) or one (128): last stages of every
# remainder, fewer stages than the ring and more, tiles of 32, 64 and 128 columns with a ragged last one
@pytest.mark.parametrize("M,N,K", [(16, 520, 64), (2, 2048, 4104), (31, 9472, 192), (32, 2056, 8256), (33, 2056, 4160), (64, 9472, 136), (5, 9480, 1088), (64, 12008, 1096), (17, 18944, 64), (64, 18952, 2112), (1, 57344, 264)])
def test_few_row_stages_of_several_blocks(L, M, N, K):
    test_gemm_few_rows(L, M, N, K)


# persistent vocabulary head: fewer k blocks than ring stages and more, one and several row tiles, a ragged last tile, the largest in the last column
@pytest.mark.parametrize("M,N,K", [(1, 128256, 64), (128, 38016, 200), (3, 128256, 1024), (129, 40008, 512), (64, 152064, 448)])
def test_persistent_vocabulary_head(L, M, N, K):
    assert L.oa_host_gemm_kernel(M, N, K, EPI_LOGITS, 128, 1, 0) == HEAD
    g = torch.Generator(device=dev()).manual_seed(N + K)
    A = torch.randn(M, K, generator=g, device=dev()).to(torch.bfloat16)
    B = (torch.randn(N, K, generator=g, device=dev()) * 0.1).to(torch.bfloat16)
    B[N - 1] = (A[0].float() * 0.5).to(torch.bfloat16)
    logits = torch.full((M, N), float("nan"), dtype=torch.float32, device=dev())
    ids = torch.empty(M, dtype=torch.int32, device=dev()); ids2 = torch.empty_like(ids)
    assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_LOGITS, 256, None, None, None, ptr(logits), ptr(ids), None) == 0
    assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_LOGITS, 128, None, None, None, None, ptr(ids2), None) == 0
    ref = A.double() @ B.double().T
    # fp32 sums of K products of size about 0.1 |a|
    assert ((logits.double() - ref).abs() <= 0.1 * 4 * K * 2.0 ** -23 + 1e-5 * ref.abs()).all()
    mx = logits.max(dim=1, keepdim=True).values
    first = torch.where(logits == mx, torch.arange(N, device=dev())[None, :], N).min(dim=1).values
    assert (ids.long() == first).all() and (ids2 == ids).all() and ids[0].item() == N - 1


# rings of 16, 32, 64 and 128 loaded rows (head and stream-K): rows have the bits they have among 128, more k blocks than stages and fewer
@pytest.mark.parametrize("N,K", [(38016, 1000), (40008, 72), (38400, 136)])
def test_rings_of_few_rows_keep_the_bits(L, N, K):
    g = torch.Generator(device=dev()).manual_seed(N + K)
    A = torch.randn(128, K, generator=g, device=dev()).to(torch.bfloat16)
    B = (torch.randn(N, K, generator=g, device=dev()) * 0.1).to(torch.bfloat16)

    def products(M):
        logits, ids, sk = torch.full((M, N), float("nan"), device=dev()), torch.full((M,), -1, dtype=torch.int32, device=dev()), torch.full((M, N), float("nan"), device=dev())
        assert L.oa_host_gemm_kernel(M, N, K, EPI_LOGITS, 128, 1, 0) == HEAD
        assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_LOGITS, 128, None, None, None, ptr(logits), ptr(ids), None) == 0
        assert L.oa_k_gemm_streamk(ptr(A), ptr(B), M, N, K, 128, 148, ptr(sk), None) == 0
        return logits, ids, sk

    whole = products(128)
    # fp32 sums of K products of size about 0.1 |a| (the bits are compared below)
    assert ((whole[0].double() - A.double() @ B.double().T).abs() <= 0.1 * 4 * K * 2.0 ** -23 + 1e-6).all()
    for M in (1, 7, 15, 16, 17, 32, 33, 64, 65, 127):
        for got, want in zip(products(M), whole):
            assert torch.equal(got, want[:M]), M


@pytest.mark.parametrize("M", [5, 100, 700])
@pytest.mark.parametrize("epi", [EPI_STORE, EPI_SWIGLU, EPI_LOGITS])
@pytest.mark.parametrize("bn", [0, 16, 96, 192, 512, -64])
def test_gemm_refuses_tile_widths_it_has_no_kernel_for(L, M, epi, bn):
    """whatever kernel the shape would take: a width that is refused for one shape is refused for all"""
    N, K = 40960, 64
    A = torch.zeros(M, K, dtype=torch.bfloat16, device=dev()); B = torch.zeros(N, K, dtype=torch.bfloat16, device=dev())
    out = torch.zeros(M, N, dtype=torch.bfloat16, device=dev()); ids = torch.zeros(M, dtype=torch.int32, device=dev())
    assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, epi, bn, ptr(out), None, None, None, ptr(ids), None) != 0
    torch.cuda.synchronize()


def test_gemm_with_a_partial_last_round_under_stream_capture(L):
    """a product on CTA pairs whose tiles do not fill the last round: captured, it replays to the same bits"""
    M, N, K = 614, 4096, 14336
    g = torch.Generator(device=dev()).manual_seed(5)
    A = torch.randn(M, K, generator=g, device=dev()).to(torch.bfloat16); B = (torch.randn(N, K, generator=g, device=dev()) * 0.05).to(torch.bfloat16)
    want = torch.empty(M, N, dtype=torch.bfloat16, device=dev()); got = torch.zeros_like(want)
    assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_STORE, 256, ptr(want), None, None, None, None, None) == 0
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        rc = L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_STORE, 256, ptr(got), None, None, None, None, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    for _ in range(3):
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(got, want)


# A row of a product has the same bits whatever shares the product with it: every kernel and tile width sums k in ascending order in one accumulator.
# Rows alone or among others, at another place of the batch, on both sides of every kernel's and tile width's border.
def _products(L, A, B, x, widths):
    """every epilogue's result over these rows, per tile width"""
    (M, K), N = A.shape, B.shape[0]
    outs = []
    for bn in widths:
        y = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=dev()); r = x[:M].clone(); h = torch.full((M, N // 2), float("nan"), dtype=torch.bfloat16, device=dev())
        assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_STORE, bn, ptr(y), ptr(B[0, :1].expand(N).contiguous()), None, None, None, None) == 0
        assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_RESID, bn, ptr(r), None, ptr(r), None, None, None) == 0
        assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_SWIGLU, bn, ptr(h), None, None, None, None, None) == 0
        torch.cuda.synchronize()
        outs.append((y, r, h))
    return outs


def _bits_follow_the_row(L, N, K, total, spans, widths):
    g = torch.Generator(device=dev()).manual_seed(N + K)
    A = torch.randn(total, K, generator=g, device=dev()).to(torch.bfloat16)
    B = (torch.randn(N, K, generator=g, device=dev()) * 0.05).to(torch.bfloat16)
    x = torch.randn(1, N, generator=g, device=dev()).to(torch.bfloat16).expand(total, N).contiguous()
    whole = _products(L, A, B, x, widths[:1])[0]
    for r0, r1 in spans:
        for bn, got in zip(widths, _products(L, A[r0:r1].contiguous(), B, x, widths)):
            for name, w, v in zip(("store", "residual", "gated"), whole, got):
                assert torch.equal(v, w[r0:r1]), (r0, r1, bn, name, int((v != w[r0:r1]).sum()))


@pytest.mark.parametrize("N,K", [(4096, 14336), (4096, 4096), (6144, 4096), (2048, 2048), (1024, 328)])
def test_prefill_rows_keep_their_bits_beside_others(L, N, K):
    _bits_follow_the_row(L, N, K, 1337, [(0, 1337), (0, 129), (0, 200), (100, 357), (0, 400), (700, 1314), (313, 1337)], (256, 128, 64))


# Every width of a pair's tile: one round and several, ragged last rows and columns (N no multiple of the width, and where the gated form runs, of 64), a k
# range shorter than the ring; the bits of one-CTA tiles.  The width a case is for is asserted.
@pytest.mark.parametrize("M,N,K,width", [(257, 264, 2056, 128), (129, 9000, 1032, 128), (700, 3080, 1032, 160), (1100, 4096, 320, 160), (385, 10240, 4096, 160), (1000, 6152, 2056, 192),
                                         (513, 4096, 320, 192), (321, 6152, 4096, 192), (640, 5120, 4096, 224), (2000, 8192, 320, 224), (1000, 9000, 2056, 256),
                                         (2000, 2048, 320, 256), (900, 4096, 4096, 256)])
def test_pair_tiles_of_every_width(L, M, N, K, width):
    assert L.oa_host_gemm_pair_width(M, N, K, EPI_STORE, 256) == width
    g = torch.Generator(device=dev()).manual_seed(M + N + K)
    A = torch.randn(M, K, generator=g, device=dev()).to(torch.bfloat16)
    B = (torch.randn(N, K, generator=g, device=dev()) * 0.05).to(torch.bfloat16)
    bias, resid = torch.randn(N, generator=g, device=dev()).to(torch.bfloat16), torch.randn(M, N, generator=g, device=dev()).to(torch.bfloat16)
    ref = A.double() @ B.double().T
    room = 0.05 * K ** 1.5 * 2.0 ** -24              # fp32 sums of K products; the rounding to bf16 besides

    def products(a, add, bn):
        rows = a.shape[0]
        outs = [torch.full((rows, N), float("nan"), dtype=torch.bfloat16, device=dev()) for _ in range(2)] + [torch.full((rows, N // 2), float("nan"), dtype=torch.bfloat16, device=dev())]
        assert L.oa_k_gemm(ptr(a), ptr(B), rows, N, K, EPI_STORE, bn, ptr(outs[0]), ptr(bias), None, None, None, None) == 0
        assert L.oa_k_gemm(ptr(a), ptr(B), rows, N, K, EPI_RESID, bn, ptr(outs[1]), None, ptr(add), None, None, None) == 0
        if N % 32 == 0:
            assert L.oa_k_gemm(ptr(a), ptr(B), rows, N, K, EPI_SWIGLU, bn, ptr(outs[2]), None, None, None, None, None) == 0
        torch.cuda.synchronize()
        return outs[:3 if N % 32 == 0 else 2]

    got = products(A, resid, 256)
    for o, want in ((got[0], ref + bias.double()), (got[1], ref + resid.double())):
        assert ((o.double() - want).abs() <= want.abs() * 2.0 ** -8 + room + 1e-6).all(), float((o.double() - want).abs().max())
    for r0 in range(0, M, 128):                      # up to 128 rows take one-CTA tiles
        part = products(A[r0:r0 + 128].contiguous(), resid[r0:r0 + 128].contiguous(), 64)
        for o, q in zip(got, part):
            assert torch.equal(o[r0:r0 + 128], q)


@pytest.mark.parametrize("N,K", [(4096, 14336), (2048, 4096), (6144, 2056), (2048, 2048), (1024, 72), (28672, 1024)])
def test_decoding_rows_keep_their_bits_beside_others(L, N, K):
    _bits_follow_the_row(L, N, K, 300, [(0, 300), (0, 1), (17, 18), (0, 16), (3, 20), (0, 32), (7, 40), (0, 64), (30, 95), (0, 128), (50, 179), (299, 300)], (32, 64, 128, 256))


# Tiles on CTA pairs with the weights' rows as their 256: every width in tokens that the rule takes, one round and several, rows and columns that end inside a tile
# (and inside a warp's 32), a k range shorter than the ring, every epilogue; the bits of one-CTA tiles.  The width a case is for is asserted.
@pytest.mark.parametrize("M,N,K,width", [(257, 5120, 1032, 128), (1337, 3080, 1032, 128), (321, 28672, 192, 128), (258, 9000, 320, 160), (800, 3080, 2056, 160), (130, 28672, 192, 160),
                                         (322, 9000, 1032, 192), (513, 16384, 320, 192), (385, 9000, 2056, 224), (1537, 10240, 320, 224),
                                         (300, 5120, 4096, 128), (513, 8192, 1032, 160), (2000, 2048, 4096, 224)])
def test_pair_tiles_with_the_operands_swapped(L, monkeypatch, M, N, K, width):
    assert L.oa_host_gemm_pair_swapped(M, N, K, EPI_STORE, 256) == width
    g = torch.Generator(device=dev()).manual_seed(M + N + K)
    A = torch.randn(M, K, generator=g, device=dev()).to(torch.bfloat16)
    B = (torch.randn(N, K, generator=g, device=dev()) * 0.05).to(torch.bfloat16)
    bias, resid = torch.randn(N, generator=g, device=dev()).to(torch.bfloat16), torch.randn(M, N, generator=g, device=dev()).to(torch.bfloat16)
    bias32 = torch.randn(N, generator=g, device=dev())
    ref = A.double() @ B.double().T
    room = 0.05 * K ** 1.5 * 2.0 ** -24              # fp32 sums of K products; the rounding to bf16 besides

    def products(bn):
        bf = lambda cols: torch.full((M, cols), float("nan"), dtype=torch.bfloat16, device=dev())
        outs = [bf(N), bf(N), bf(N), torch.full((M, N), 1.0, device=dev()), bf(N // 2)]
        assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_STORE, bn, ptr(outs[0]), ptr(bias), None, None, None, None) == 0
        assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_RESID, bn, ptr(outs[1]), None, ptr(resid), None, None, None) == 0
        assert L.oa_k_gemm_ext(ptr(A), ptr(B), M, N, K, EPI_STORE, bn, ptr(outs[2]), None, 3, 64, 200, 1.0, 0, None) == 0
        assert L.oa_k_gemm_ext(ptr(A), ptr(B), M, N, K, 4, bn, ptr(outs[3]), ptr(bias32), 0, 0, 0, 0.5, 1, None) == 0
        if N % 32 == 0:
            assert L.oa_k_gemm(ptr(A), ptr(B), M, N, K, EPI_SWIGLU, bn, ptr(outs[4]), None, None, None, None, None) == 0
        torch.cuda.synchronize()
        return outs

    got = products(256)
    with monkeypatch.context() as m:                 # with that threshold set, one-CTA tiles are all there is
        m.setenv("OA_GEMM_PERSISTENT_MIN_TILES", "1000000000")
        assert L.oa_host_gemm_kernel(M, N, K, EPI_STORE, 64, 0, 0) == 0
        plain = products(64)
    want = [ref + bias.double(), ref + resid.double(), ref.clone(), 1.0 + 0.5 * ref + bias32.double()]
    want[2][:, 64:200] = torch.nn.functional.silu(want[2][:, 64:200])
    if N % 32 == 0:
        y = ref.view(M, -1, 2, 16)
        want.append((torch.nn.functional.silu(y[:, :, 0]) * y[:, :, 1]).reshape(M, -1))
    for i, w in enumerate(want):
        o = got[i].double()
        assert torch.isfinite(o).all()
        # bf16 outputs round to 2^-9 relative; the fast exponential and divide of the activations another 2^-9; sums as above, through a gate's slope (below 1.1) and factor
        assert ((o - w).abs() <= 2.0 ** -8 * w.abs() + 8 * room * (1 + w.abs())).all(), i
        assert torch.equal(got[i], plain[i]), i
    # rows alone or among others: the bits do not move
    part = slice(37, 37 + 130) if M > 170 else slice(0, M)
    a = A[part].contiguous(); alone = torch.full((a.shape[0], N), float("nan"), dtype=torch.bfloat16, device=dev())
    assert L.oa_k_gemm(ptr(a), ptr(B), a.shape[0], N, K, EPI_STORE, 64, ptr(alone), ptr(bias), None, None, None, None) == 0
    torch.cuda.synchronize()
    assert torch.equal(alone, got[0][part])


# A prompt's attention has the same bits alone (in the one-head kernel) and beside others (in any): all take the same keys per tile, raise a row's reference maximum at the
# same scores and sum its exponentials in the same order.
@pytest.mark.parametrize("nh,nkv,D", [(32, 8, 128), (20, 4, 128), (32, 8, 64), (15, 3, 64), (16, 2, 128)])
def test_prefill_attention_keeps_its_bits_beside_others(L, monkeypatch, nh, nkv, D):
    pairs = nkv * ((nh // nkv + 1) // 2)
    half = torch.cuda.get_device_properties(0).multi_processor_count // 2
    few = half // pairs                                  # row tiles of a lone prompt that are all resident in the one-head kernel
    cases = [(c, min(q, 128 * few)) for c, q in [(64, 64), (130, 130), (700, 200), (513, 513), (1, 1), (999, 385), (2000, 129)]] * 2
    ctx = [c for c, _ in cases]; qlens = [q for _, q in cases]
    assert sum((q + 127) // 128 for q in qlens) * pairs > half and all((q + 127) // 128 * pairs <= half for q in qlens)
    n = len(ctx); maxp = 32; num_pages = sum((c + 63) // 64 for c in ctx)
    kv = _mk_cache(num_pages, nkv, D, 21)
    g = torch.Generator(device="cpu").manual_seed(4)
    perm = torch.randperm(num_pages, generator=g)
    bt = torch.zeros(n, maxp, dtype=torch.int32); k = 0
    for i, c in enumerate(ctx):
        npg = (c + 63) // 64; bt[i, :npg] = perm[k:k + npg].to(torch.int32); k += npg
    T = sum(qlens)
    q = torch.randn(T, nh, D, generator=g)
    q[::5] *= 9                                          # scores that raise a row's reference maximum in later tiles
    q = q.to(torch.bfloat16).to(dev())

    def attend(seqs, rows):
        out = torch.full((len(rows), nh, D), float("nan"), dtype=torch.bfloat16, device=dev())
        qq = q[rows].contiguous()
        ca = np.array([ctx[i] for i in seqs], np.int32); qa = np.array([qlens[i] for i in seqs], np.int32); b = np.ascontiguousarray(bt[seqs].numpy())
        assert L.oa_k_paged_attention(ptr(qq), ptr(out), ptr(kv), num_pages, b.ctypes.data, maxp, ca.ctypes.data, qa.ctypes.data, len(seqs), nh, nkv, D, 0, None) == 0
        return out

    whole = attend(list(range(n)), list(range(T)))
    for kernel in _prefill_kernels(nh, nkv, D):
        monkeypatch.setenv("OA_PREFILL_ATTN", kernel)
        assert torch.equal(attend(list(range(n)), list(range(T))), whole), kernel
    monkeypatch.setenv("OA_PREFILL_ATTN", "one_head")
    row0 = 0
    for i in range(n):
        if qlens[i] > 1:                                 # (a lone row is a decoding row: another kernel)
            rows = list(range(row0, row0 + qlens[i]))
            alone = attend([i], rows)
            assert torch.equal(alone, whole[row0:row0 + qlens[i]]), (i, int((alone != whole[row0:row0 + qlens[i]]).sum()))
        row0 += qlens[i]


# Plain FMA kernel of a few rows (hybrid models: absorbed products of decoding rows; every product of a few rows with hy_tensor_core = 0): the fp32 chain it
# promises, bit for bit.  A lane sums its pieces of eight k in ascending order with one rounding per product, then a butterfly from distance 16 down.
@pytest.mark.parametrize("M,N,K,batch", [(1, 24, 8, 1), (5, 41, 128, 3), (16, 512, 128, 4), (17, 33, 136, 2), (32, 64, 512, 2), (9, 17, 1000, 1), (8, 130, 1024, 2), (3, 7, 120, 5)])
def test_few_row_products_are_an_fp32_chain(L, M, N, K, batch):
    g = torch.Generator(device="cpu").manual_seed(M * N + K)
    A = torch.randn(batch, M, K, generator=g).to(torch.bfloat16); B = torch.randn(batch, N, K, generator=g).to(torch.bfloat16)
    a, b = A.double().numpy(), B.double().numpy()
    lanes = np.zeros((batch, M, N, 32), np.float32)
    for piece in range(0, K, 256):
        for e in range(8):
            k = piece + np.arange(32) * 8 + e
            ok = k < K
            prod = a[:, :, None, k[ok]] * b[:, None, :, k[ok]]                                      # exact in 64 bits
            lanes[..., ok] = (lanes[..., ok].astype(np.float64) + prod).astype(np.float32)          # one rounding, as a fused multiply-add
    for o in (16, 8, 4, 2, 1):
        lanes = lanes + lanes[..., np.arange(32) ^ o]
    want = lanes[..., 0]
    Ad, Bd = A.to(dev()), B.to(dev())
    out = torch.full((batch, M, N), float("nan"), dtype=torch.float32, device=dev()); out16 = out.to(torch.bfloat16)
    for mode, o in ((1, out), (0, out16)):
        assert L.oa_k_hybrid_gemm(mode, ptr(Ad), K, ptr(Bd), K, ptr(o), N, M, N, K, 1.0, batch, M * K, N * K, M * N, None) == 0
    torch.cuda.synchronize()
    assert (out.cpu().numpy() == want).all(), int((out.cpu().numpy() != want).sum())
    assert torch.equal(out16, out.to(torch.bfloat16))


# What the hybrid models ask of the epilogues, on every kernel that has them: fp32 results with alpha, bias and accumulation, activations on a store, the
# gated form of GELU; ragged rows and columns, whole and partial tiles.
EXT_CASES = [(1, 2048, 1024, 32, FEW), (17, 1000, 328, 64, FEW), (64, 4104, 2056, 128, FEW), (40, 512, 64, 256, FEW), (100, 1032, 520, 64, TILE), (200, 1024, 512, 64, TILE),
             (1337, 4096, 4096, 256, PAIR), (1100, 6152, 2056, 256, PAIR), (7900, 14336, 320, 256, PAIR), (9000, 2560, 128, 256, PERSISTENT)]


@pytest.mark.parametrize("M,N,K,bn,kernel", EXT_CASES)
def test_gemm_epilogues_of_the_hybrid_models(L, M, N, K, bn, kernel, monkeypatch):
    if kernel == PERSISTENT:
        monkeypatch.setenv("OA_GEMM_PERSISTENT_MIN_TILES", "1")       # leaves the pairs out
    for epi in (0, 4) + ((2,) if N % 32 == 0 else ()):
        assert L.oa_host_gemm_kernel(M, N, K, epi, bn, 1, 0) == kernel
    g = torch.Generator(device=dev()).manual_seed(M + N + K)
    A = torch.randn(M, K, generator=g, device=dev()).to(torch.bfloat16)
    B = (torch.randn(N, K, generator=g, device=dev()) * K ** -0.5).to(torch.bfloat16)
    ref = A.double() @ B.double().T
    s = 4 * K ** 0.5 * 2.0 ** -23                                     # fp32 sums of K products of unit variance in all
    bias32 = torch.randn(N, generator=g, device=dev())
    for alpha, use_bias, acc in ((1.0, True, 0), (-0.375, True, 1), (0.0, False, 1), (1.7, False, 0)):
        start = torch.randn(M, N, generator=g, device=dev())
        out = start.clone() if acc else torch.full((M, N), float("nan"), device=dev())
        assert L.oa_k_gemm_ext(ptr(A), ptr(B), M, N, K, 4, bn, ptr(out), ptr(bias32) if use_bias else None, 0, 0, 0, alpha, acc, None) == 0
        torch.cuda.synchronize()
        want = ref * (alpha if alpha != 0 else 1.0) + (bias32.double() if use_bias else 0) + (start.double() if acc else 0)
        assert ((out.double() - want).abs() <= 2 * s + want.abs() * 2.0 ** -22).all(), float((out.double() - want).abs().max())
    bias = torch.randn(N, generator=g, device=dev()).to(torch.bfloat16)
    v = ref + bias.double()
    c0, c1 = N // 4 // 8 * 8, N // 2 // 8 * 8
    cols = torch.arange(N, device=dev())
    silu = torch.where((cols >= c0) & (cols < c1), torch.nn.functional.silu(v), v)
    for act, want in ((0, v), (1, torch.relu(v) ** 2), (2, torch.nn.functional.gelu(v, approximate="tanh")), (3, silu)):
        out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=dev())
        assert L.oa_k_gemm_ext(ptr(A), ptr(B), M, N, K, 0, bn, ptr(out), ptr(bias), act, c0, c1, 0.0, 0, None) == 0
        torch.cuda.synchronize()
        # half an ulp of bf16, and fp32 arithmetic of the activation: relative 2^-16 of the arguments it is made of, whose slope stays under 2 |v| + 2
        assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + (2 * v.abs() + 2) * (s + v.abs() * 2.0 ** -16) + 1e-6).all(), (act, float((out.double() - want).abs().max()))
    if N % 32 == 0:
        gate, up = ref.view(M, N // 32, 2, 16)[:, :, 0], ref.view(M, N // 32, 2, 16)[:, :, 1]
        for act, f in ((0, torch.nn.functional.silu(gate)), (2, torch.nn.functional.gelu(gate, approximate="tanh"))):
            out = torch.full((M, N // 2), float("nan"), dtype=torch.bfloat16, device=dev())
            assert L.oa_k_gemm_ext(ptr(A), ptr(B), M, N, K, 2, bn, ptr(out), None, act, 0, 0, 0.0, 0, None) == 0
            torch.cuda.synchronize()
            want = (f * up).reshape(M, N // 2)
            room = ((gate.abs() + 1) * (up.abs() + 1)).reshape(M, N // 2)
            assert ((out.double() - want).abs() <= want.abs() * 2.0 ** -8 + room * (4 * s + 2.0 ** -15) + 1e-6).all(), (act, float((out.double() - want).abs().max()))
