"""Each kernel alone against a plain PyTorch float32/float64 restatement of the same
operation, at sizes other than the engine's tiny models use."""
import math

import numpy as np
import pytest
import torch

import plain_llama as P
from sampler_cases import CASES

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
PAGE = 64


def K():
    from rustyllm_b200 import kernels
    return kernels


def _rand(*shape, dtype=torch.float32, seed=0, scale=1.0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(dtype).to(DEV)


def _tol(dtype):
    return dict(rtol=2e-2, atol=2e-2) if dtype == torch.bfloat16 else dict(rtol=1e-5, atol=1e-5)


# ----------------------------------------------------------------------------- random weights
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("mean", [0.0, 1.0])
def test_random_fill_gives_the_hosts_numbers_bit_for_bit(dtype, mean):
    from rustyllm_b200.weights.random_init import normal_values
    n, seed = 100003, (1 << 62) + 12345
    out = torch.empty(n, dtype=dtype, device=DEV)
    K().random_fill(out, seed, mean, 0.02)
    host = torch.from_numpy(normal_values(seed, n, mean, 0.02)).to(dtype)
    assert torch.equal(out.cpu(), host)


# ----------------------------------------------------------------------------- elementwise
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_embedding_gathers_rows_and_flags_bad_ids(dtype):
    table = _rand(1000, 100, dtype=dtype)
    ids = torch.tensor([0, 999, 5, 5, 123], dtype=torch.int32, device=DEV)
    out = torch.empty(5, 100, device=DEV)
    flag = torch.zeros(1, dtype=torch.int32, device=DEV)
    K().embedding(table, ids, out, flag)
    assert torch.equal(out, table[ids.long()].float()) and flag.item() == 0
    K().embedding(table, torch.tensor([1000], dtype=torch.int32, device=DEV), out[:1], flag)
    assert flag.item() == 1


@pytest.mark.parametrize("d", [7, 100, 4096, 5000])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_rmsnorm(d, out_dtype):
    x = _rand(9, d, seed=1, scale=3.0)
    w = _rand(d, seed=2) + 1.0
    out = torch.empty(9, d, dtype=out_dtype, device=DEV)
    K().rmsnorm(x, w, out, 1e-6)
    ref = P.rms_norm(x.double().cpu(), w.double().cpu(), 1e-6)
    torch.testing.assert_close(out.double().cpu(), ref, **(dict(rtol=1e-2, atol=1e-2) if out_dtype == torch.bfloat16 else dict(rtol=2e-6, atol=2e-6)))
    rows = torch.tensor([8, 0, 3], dtype=torch.int32, device=DEV)
    out2 = torch.empty(3, d, dtype=out_dtype, device=DEV)
    K().rmsnorm(x, w, out2, 1e-6, rows)
    assert torch.equal(out2, out[rows.long()])


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("I", [172, 256, 14336])
def test_swiglu(dtype, I):
    gu = _rand(13, 2 * I, dtype=dtype, seed=3, scale=2.0)
    out = torch.empty(13, I, dtype=dtype, device=DEV)
    K().swiglu(gu, out)
    g, u = gu[:, :I].double().cpu(), gu[:, I:].double().cpu()
    torch.testing.assert_close(out.double().cpu(), P.swiglu(g, u), **_tol(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("I", [100, 50, 51])
def test_swiglu_interleaved(dtype, I):
    gu = _rand(7, 2 * I, dtype=dtype, seed=3, scale=2.0)
    out = torch.empty(7, I, dtype=dtype, device=DEV)
    K().swiglu(gu, out, interleaved=True)
    torch.testing.assert_close(out.double().cpu(), P.swiglu(gu[:, 0::2].double().cpu(), gu[:, 1::2].double().cpu()), **_tol(dtype))


@pytest.mark.parametrize("M,N,K_,parts", [(1, 256, 128, 0), (8, 28672, 512, 0), (8, 1024, 4096, 8), (40, 400, 72, 0), (64, 512, 1024, 4),
                                          (300, 344, 264, 0), (17, 130, 104, 2), (100, 640, 2048, 0), (130, 344, 1024, 4),
                                          (256, 512, 512, 2)])
def test_gemm_tc_swiglu_epilogue(M, N, K_, parts):
    k = K()
    a = _rand(M, K_, dtype=torch.bfloat16, seed=24)
    w = _rand(N, K_, dtype=torch.bfloat16, seed=25, scale=0.1)
    bias = _rand(N, seed=26, scale=0.1)
    out = torch.full((M, N // 2), float("nan"), dtype=torch.bfloat16, device=DEV)
    k.gemm_tc(a, w, out, k.OUT_SWIGLU, bias, force_splits=parts)
    k.check_device_errors()
    y = a.double().cpu() @ w.double().cpu().T + bias.double().cpu()
    torch.testing.assert_close(out.double().cpu(), P.swiglu(y[:, 0::2], y[:, 1::2]), rtol=2e-2, atol=2e-2)


def test_convert_rounds_to_nearest_even():
    # SimonWaldherr/RustyLLM src/simd.rs:88-96 (f32_to_bf16) and its tests at 9203-9225
    x = torch.tensor([1.0, 1.00390625, 1.005859375, 1.01171875, -2.5, 3.0e38, 1e-40], device=DEV)
    out = torch.empty(7, dtype=torch.bfloat16, device=DEV)
    K().convert(x, out)
    assert torch.equal(out, x.to(torch.bfloat16))
    assert out[1].item() == 1.0 and out[3].item() == 1.015625   # ties go to the even mantissa
    back = torch.empty(7, device=DEV)
    K().convert(out, back)
    assert torch.equal(back, out.float())


# ----------------------------------------------------------------------------- GEMM
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("M,N,K_", [(1, 7, 5), (3, 96, 96), (17, 130, 172), (64, 64, 64), (65, 300, 33),
                                    (200, 257, 100), (8, 1000, 256)])
def test_gemm_simt_all_modes(dtype, M, N, K_):
    k = K()
    a = _rand(M, K_, dtype=dtype, seed=4)
    w = _rand(N, K_, dtype=dtype, seed=5)
    bias = _rand(N, seed=6)
    ref = a.double().cpu() @ w.double().cpu().T
    tol = dict(rtol=1e-2, atol=1e-2 * math.sqrt(K_)) if dtype == torch.bfloat16 else dict(rtol=1e-5, atol=2e-5 * math.sqrt(K_))
    out = torch.empty(M, N, dtype=dtype, device=DEV)
    k.gemm_simt(a, w, out, k.OUT_SAME)
    torch.testing.assert_close(out.double().cpu(), ref, **tol)
    out32 = torch.empty(M, N, device=DEV)
    k.gemm_simt(a, w, out32, k.OUT_F32, bias)
    torch.testing.assert_close(out32.double().cpu(), ref + bias.double().cpu(), rtol=1e-5, atol=2e-5 * math.sqrt(K_))
    res = _rand(M, N, seed=7)
    acc = res.clone()
    k.gemm_simt(a, w, acc, k.OUT_ADD_F32)
    torch.testing.assert_close(acc.double().cpu(), ref + res.double().cpu(), rtol=1e-5, atol=2e-5 * math.sqrt(K_))


def test_gemm_simt_rows_do_not_depend_on_the_batch():
    """The sum in the order of k (here for float sums shorter than 256; longer ones with more than 8 rows go by tiles of tokens and differ by
    rounding)."""
    k = K()
    a = _rand(130, 172, seed=8)
    w = _rand(96, 172, seed=9)
    full = torch.empty(130, 96, device=DEV)
    k.gemm_simt(a, w, full, k.OUT_F32)
    for rows in ([5], [0, 64, 129], list(range(20, 60))):
        sub = torch.empty(len(rows), 96, device=DEV)
        k.gemm_simt(a[rows].contiguous(), w, sub, k.OUT_F32)
        assert torch.equal(sub, full[rows]), "bit-equal whatever else is in the batch"
    # strided rows of A (a column block of a wider buffer)
    wide = _rand(10, 300, seed=10)
    sub = torch.empty(10, 96, device=DEV)
    k.gemm_simt(wide[:, 100:272], w, sub, k.OUT_F32)
    ref = torch.empty(10, 96, device=DEV)
    k.gemm_simt(wide[:, 100:272].contiguous(), w, ref, k.OUT_F32)
    assert torch.equal(sub, ref)


# ----------------------------------------------------------------------------- tensor-core GEMM
@pytest.mark.parametrize("M,N,K_", [(1, 128, 64), (1, 4096, 4096), (5, 96, 96), (16, 256, 128), (17, 130, 104),
                                    (33, 1000, 264), (64, 512, 1024), (100, 384, 4096), (129, 300, 72),
                                    (300, 2048, 512), (1000, 768, 320)])
def test_gemm_tc_all_modes(M, N, K_):
    k = K()
    a = _rand(M, K_, dtype=torch.bfloat16, seed=4)
    w = _rand(N, K_, dtype=torch.bfloat16, seed=5)
    bias = _rand(N, seed=6)
    assert k.gemm_tc_supported(a, w, None)
    ref = (a.float() @ w.float().T).double().cpu() if M * N * K_ > 1e8 else a.double().cpu() @ w.double().cpu().T
    scale = math.sqrt(K_)
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    k.gemm_tc(a, w, out, k.OUT_SAME)
    torch.testing.assert_close(out.double().cpu(), ref, rtol=1e-2, atol=1e-2 * scale)
    out32 = torch.empty(M, N, device=DEV)
    k.gemm_tc(a, w, out32, k.OUT_F32, bias)
    torch.testing.assert_close(out32.double().cpu(), ref + bias.double().cpu(), rtol=1e-4, atol=2e-5 * scale * 4)
    res = _rand(M, N, seed=7)
    acc = res.clone()
    k.gemm_tc(a, w, acc, k.OUT_ADD_F32)
    torch.testing.assert_close(acc.double().cpu(), ref + res.double().cpu(), rtol=1e-4, atol=2e-5 * scale * 4)
    k.check_device_errors()
    # the same product on the CUDA cores agrees to float accumulation order
    simt = torch.empty(M, N, device=DEV)
    k.gemm_simt(a, w, simt, k.OUT_F32, bias)
    torch.testing.assert_close(out32, simt, rtol=1e-4, atol=2e-5 * scale * 4)


@pytest.mark.parametrize("M,N,K_", [(1, 4096, 4096), (8, 6144, 4096), (8, 4096, 14336), (8, 512, 512), (64, 1024, 4096),
                                    (33, 300, 1096), (16, 128, 256),
                                    # more than 64 tokens, few tiles: 128- and 256-token tiles in parts as well
                                    (128, 4096, 4096), (100, 520, 2048), (200, 640, 1096), (256, 256, 1024), (300, 1100, 640),
                                    (512, 4096, 4096), (700, 4096, 1024)])
def test_gemm_tc_split_k_is_deterministic_and_matches_the_unsplit_product(M, N, K_):
    k = K()
    a = _rand(M, K_, dtype=torch.bfloat16, seed=14)
    w = _rand(N, K_, dtype=torch.bfloat16, seed=15)
    bias = _rand(N, seed=16)
    res = _rand(M, N, seed=17)
    whole = res.clone()
    k.gemm_tc(a, w, whole, k.OUT_ADD_F32, bias, force_splits=1)
    runs = []
    for parts in (0, 0, 0, 2, 4, 8):
        o = res.clone()
        k.gemm_tc(a, w, o, k.OUT_ADD_F32, bias, force_splits=parts)
        runs.append(o)
    for o in runs[3:]:
        torch.testing.assert_close(o, whole, rtol=1e-4, atol=1e-4 * math.sqrt(K_))
    k.check_device_errors()
    assert torch.equal(runs[0], runs[1]) and torch.equal(runs[0], runs[2])        # fixed order of the parts
    torch.testing.assert_close(runs[0], whole, rtol=1e-4, atol=1e-4 * math.sqrt(K_))
    ref = a.double().cpu() @ w.double().cpu().T + bias.double().cpu() + res.double().cpu()
    torch.testing.assert_close(runs[0].double().cpu(), ref, rtol=1e-4, atol=1e-4 * math.sqrt(K_))
    out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    k.gemm_tc(a, w, out, k.OUT_SAME)
    torch.testing.assert_close(out.double().cpu(), ref - bias.double().cpu() - res.double().cpu(), rtol=1e-2, atol=1e-2 * math.sqrt(K_))
    if (M, N, K_) in [(1, 4096, 4096), (8, 6144, 4096), (8, 4096, 14336), (128, 4096, 4096), (100, 520, 2048), (200, 640, 1096)]:
        assert k.gemm_tc_splits(M, N, K_) > 1
    if (M, N, K_) == (512, 4096, 4096):
        assert k.gemm_tc_splits(M, N, K_) == 2      # 64 tiles of 256 tokens: two parts fill most of the SMs
    if (M, N, K_) == (700, 4096, 1024):
        assert k.gemm_tc_splits(M, N, K_) == 1      # 96 tiles: the persistent kernel takes them whole


@pytest.mark.parametrize("M,N,K_,parts", [(8, 384, 512, 0), (8, 384, 512, 1), (5, 200, 256, 4), (40, 136, 192, 2),
                                          (64, 512, 1024, 8), (33, 264, 320, 0), (64, 520, 128, 1)])
def test_gemm_tc_starts_the_norm_of_the_updated_residual(M, N, K_, parts):
    """Add-into-residual epilogue with the next RMSNorm riding along: the residual times
    the norm weight in bf16, and the rows' sums of squares in pieces."""
    k = K()
    a = _rand(M, K_, dtype=torch.bfloat16, seed=31)
    w = _rand(N, K_, dtype=torch.bfloat16, seed=32, scale=0.2)
    bias = _rand(N, seed=33)
    g = (_rand(N, seed=34) * 0.3 + 1.0)
    res = _rand(M, N, seed=35, scale=3.0)
    out = res.clone()
    xg = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    sumsq = torch.full((M, k.norm_pieces(N)), float("nan"), device=DEV)
    k.gemm_tc(a, w, out, k.OUT_ADD_F32, bias, force_splits=parts, norm_weight=g, norm_out=xg, norm_sumsq=sumsq)
    k.check_device_errors()
    plain = res.clone()
    k.gemm_tc(a, w, plain, k.OUT_ADD_F32, bias, force_splits=parts)
    assert torch.equal(out, plain)                                   # the residual itself is what it was without the norm
    assert torch.equal(xg, (out * g).to(torch.bfloat16))             # float product, rounded once
    want = (out.double() ** 2).sum(1)
    torch.testing.assert_close(sumsq.double().sum(1), want, rtol=1e-5, atol=0)
    assert not torch.isnan(sumsq).any()


@pytest.mark.parametrize("mode", ["same", "f32", "add", "swiglu"])
@pytest.mark.parametrize("M,N,K_,parts", [(8, 384, 512, 0), (8, 384, 512, 1), (5, 200, 256, 4), (40, 136, 192, 2),
                                          (33, 264, 320, 0), (64, 520, 128, 1), (17, 4096, 4096, 0)])
def test_gemm_tc_finishes_a_norm_of_its_input(M, N, K_, parts, mode):
    """The input is x * norm weight; the epilogue multiplies row m by rsqrt(mean(x_m^2) + eps),
    the mean coming as sums of squares in pieces: the result is the product with RMSNorm(x)."""
    k = K()
    eps = 1e-3
    x = _rand(M, K_, seed=41, scale=5.0) * (1 + torch.arange(M, device=DEV).float()[:, None])    # rows of very different size
    g = _rand(K_, seed=42) * 0.3 + 1.0
    xg = (x * g).to(torch.bfloat16)
    w = _rand(N, K_, dtype=torch.bfloat16, seed=43, scale=0.2)
    bias = _rand(N, seed=44)
    pieces = 7
    cut = torch.rand(M, pieces, device=DEV) + 0.1
    sumsq = ((x.double() ** 2).sum(1, keepdim=True) * (cut / cut.sum(1, keepdim=True)).double()).float().contiguous()
    r = 1.0 / torch.sqrt((x.double().cpu() ** 2).mean(1, keepdim=True) + eps)
    y = (xg.double().cpu() @ w.double().cpu().T) * r + bias.double().cpu()
    res = _rand(M, N, seed=45)
    tol = dict(rtol=1e-4, atol=2e-5 * math.sqrt(K_) * 4)
    if mode == "same":
        out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
        k.gemm_tc(xg, w, out, k.OUT_SAME, bias, force_splits=parts, row_sumsq=sumsq, row_eps=eps)
        torch.testing.assert_close(out.double().cpu(), y, rtol=1e-2, atol=1e-2)
    elif mode == "f32":
        out = torch.empty(M, N, device=DEV)
        k.gemm_tc(xg, w, out, k.OUT_F32, bias, force_splits=parts, row_sumsq=sumsq, row_eps=eps)
        torch.testing.assert_close(out.double().cpu(), y, **tol)
    elif mode == "add":
        out = res.clone()
        k.gemm_tc(xg, w, out, k.OUT_ADD_F32, bias, force_splits=parts, row_sumsq=sumsq, row_eps=eps)
        torch.testing.assert_close(out.double().cpu(), y + res.double().cpu(), **tol)
    else:
        if N % 2:
            pytest.skip("the SwiGLU epilogue needs an even number of rows")
        out = torch.empty(M, N // 2, dtype=torch.bfloat16, device=DEV)
        k.gemm_tc(xg, w, out, k.OUT_SWIGLU, bias, force_splits=parts, row_sumsq=sumsq, row_eps=eps)
        torch.testing.assert_close(out.double().cpu(), P.swiglu(y[:, 0::2], y[:, 1::2]), rtol=2e-2, atol=2e-2)
    k.check_device_errors()


def test_gemm_tc_strided_rows_and_refusals():
    k = K()
    # a norm rides along for up to 64 tokens only
    with pytest.raises(k.KernelError, match="up to 64 tokens"):
        k.gemm_tc(_rand(65, 64, dtype=torch.bfloat16), _rand(128, 64, dtype=torch.bfloat16), torch.empty(65, 128, device=DEV),
                  k.OUT_F32, row_sumsq=torch.ones(65, 4, device=DEV), row_eps=1e-5)
    wide = _rand(40, 640, dtype=torch.bfloat16, seed=8)
    w = _rand(200, 256, dtype=torch.bfloat16, seed=9)
    a = wide[:, 128:384]
    assert k.gemm_tc_supported(a, w, None)
    out = torch.empty(40, 200, device=DEV)
    k.gemm_tc(a, w, out, k.OUT_F32)
    torch.testing.assert_close(out.double().cpu(), a.double().cpu() @ w.double().cpu().T, rtol=1e-4, atol=1e-3)
    k.check_device_errors()
    # K = 172: rows of 344 bytes are no multiple of 16 bytes, TMA cannot address them
    assert not k.gemm_tc_supported(_rand(4, 172, dtype=torch.bfloat16), _rand(8, 172, dtype=torch.bfloat16), None)
    assert not k.gemm_tc_supported(wide[:, 4:260], w, None)      # base not 16-byte aligned
    with pytest.raises(k.KernelError, match="not supported"):
        k.gemm_tc(_rand(4, 172, dtype=torch.bfloat16), _rand(8, 172, dtype=torch.bfloat16),
                  torch.empty(4, 8, device=DEV), k.OUT_F32)


# ----------------------------------------------------------------------------- rope + cache write
def _paged(G, hd, n_pages, dtype, seed=0):
    g = torch.Generator().manual_seed(seed)
    k_pool = torch.randn(n_pages, G, PAGE, hd, generator=g).to(dtype).to(DEV)   # stale contents on purpose
    v_pool = torch.randn(n_pages, G, PAGE, hd, generator=g).to(dtype).to(DEV)
    return k_pool, v_pool


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,hd,rot,interleaved", [(4, 2, 16, 16, False), (3, 1, 32, 32, True), (5, 5, 48, 24, False),
                                                    (8, 2, 128, 128, False), (2, 2, 256, 64, True), (6, 3, 80, 0, False)])
def test_rope_kv_write(dtype, H, G, hd, rot, interleaved):
    k = K()
    M = 11
    qkv = _rand(M, (H + 2 * G) * hd + 8, dtype=dtype, seed=11)[:, :(H + 2 * G) * hd + 8]   # padded row stride
    positions = torch.tensor([0, 1, 63, 64, 65, 200, 5, 6, 7, 130, 131], dtype=torch.int32, device=DEV)
    slot_of_token = torch.tensor([0, 0, 0, 0, 0, 0, 2, 2, 2, 2, 2], dtype=torch.int32, device=DEV)
    page_table = torch.tensor([[7, 3, 1, 9], [0, 0, 0, 0], [2, 8, 4, 5]], dtype=torch.int32, device=DEV)
    inv = torch.tensor([1.0 / (10000.0 ** (2 * i / max(rot, 2))) for i in range(max(rot // 2, 1))], device=DEV)
    k_pool, v_pool = _paged(G, hd, 10, dtype)
    k_before, v_before = k_pool.clone(), v_pool.clone()
    src = qkv.clone()
    k.rope_kv_write(qkv, positions, slot_of_token, page_table, inv, H, G, hd, rot, interleaved, k_pool, v_pool)

    x = src[:, :(H + 2 * G) * hd].double().cpu()
    q, kk, v = x[:, :H * hd].view(M, H, hd), x[:, H * hd:(H + G) * hd].view(M, G, hd), x[:, (H + G) * hd:].view(M, G, hd)
    if rot:
        sin, cos = P.rope_angles(positions.cpu(), inv.cpu())
        f = P.apply_rope_interleaved if interleaved else P.apply_rope_half
        q = torch.cat([f(q[..., :rot], sin, cos), q[..., rot:]], -1)
        kk = torch.cat([f(kk[..., :rot], sin, cos), kk[..., rot:]], -1)
    tol = _tol(dtype)
    torch.testing.assert_close(qkv[:, :H * hd].double().cpu().view(M, H, hd), q, **tol)
    touched = torch.zeros(10, PAGE, dtype=torch.bool)
    for m in range(M):
        p = int(positions[m]); page = int(page_table[int(slot_of_token[m]), p // PAGE]); off = p % PAGE
        touched[page, off] = True
        torch.testing.assert_close(k_pool[page, :, off].double().cpu(), kk[m], **tol)
        assert torch.equal(v_pool[page, :, off].double().cpu(), v[m])
    # nothing else in the pools moved
    keep = ~touched.to(DEV)
    assert torch.equal(k_pool.permute(0, 2, 1, 3)[keep], k_before.permute(0, 2, 1, 3)[keep])
    assert torch.equal(v_pool.permute(0, 2, 1, 3)[keep], v_before.permute(0, 2, 1, 3)[keep])


@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("M,H,G,K_,normed,store", [(1, 3, 1, 1024, False, True), (8, 3, 1, 1024, True, True),
                                                  (11, 2, 2, 2048, False, True), (33, 4, 2, 512, True, True),
                                                  (11, 3, 1, 1024, False, False), (64, 32, 8, 2048, True, True)])
def test_gemm_tc_qkv_rope_is_the_product_then_the_rotation_and_the_cache_write(M, H, G, K_, normed, store, interleaved, hd):
    """The QKV product with rotation and cache write in its epilogue, against float64:
    product, (finished norm,) bias, rotation of query and key heads, keys and values at
    their tokens' places of the paged cache, nothing else in the pools touched."""
    k = K()
    N = (H + 2 * G) * hd              # head size 64: two heads a tile of 128 columns; 5 heads leave the last tile half empty
    x = _rand(M, K_, seed=51, scale=2.0)
    g = _rand(K_, seed=52) * 0.3 + 1.0
    a = (x * g).to(torch.bfloat16) if normed else x.to(torch.bfloat16)
    w = _rand(N, K_, dtype=torch.bfloat16, seed=53, scale=0.05)
    bias = _rand(N, seed=54, scale=0.5)
    assert k.gemm_tc_qkv_rope_supported(a, w, H, G, hd, hd)
    assert not k.gemm_tc_qkv_rope_supported(a, w, H, G, hd, hd // 2)     # partial rotation: the separate kernel
    positions = torch.tensor(([0, 1, 63, 64, 65, 200, 5, 6, 7, 130, 131] * 3 + list(range(31)))[:M], dtype=torch.int32, device=DEV)
    slot_of_token = torch.tensor(([0, 0, 0, 0, 0, 0, 2, 2, 2, 2, 2] + [1] * 11 + [3] * 11 + [4] * 31)[:M], dtype=torch.int32, device=DEV)
    page_table = torch.tensor([[7, 3, 1, 9], [10, 11, 12, 13], [2, 8, 4, 5], [14, 15, 16, 17], [0, 6, 6, 6]], dtype=torch.int32, device=DEV)
    inv = torch.tensor([1.0 / (10000.0 ** (2 * i / hd)) for i in range(hd // 2)], device=DEV)
    k_pool, v_pool = _paged(G, hd, 18, torch.bfloat16)
    k_before, v_before = k_pool.clone(), v_pool.clone()
    eps = 1e-5
    kw = {}
    y = a.double().cpu() @ w.double().cpu().T
    if normed:
        sumsq = ((x.double() ** 2).sum(1, keepdim=True) * torch.tensor([[0.25, 0.5, 0.25]], device=DEV).double()).float().contiguous()
        kw = dict(row_sumsq=sumsq, row_eps=eps)
        y = y / torch.sqrt((x.double().cpu() ** 2).mean(1, keepdim=True) + eps)
    y = y + bias.double().cpu()
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    k.gemm_tc_qkv_rope(a, w, out, bias, positions, slot_of_token, page_table, inv, interleaved, H, G,
                       k_pool if store else None, v_pool if store else None, **kw)
    k.check_device_errors()
    q, kk, v = y[:, :H * hd].view(M, H, hd), y[:, H * hd:(H + G) * hd].view(M, G, hd), y[:, (H + G) * hd:].view(M, G, hd)
    sin, cos = P.rope_angles(positions.cpu(), inv.cpu())
    f = P.apply_rope_interleaved if interleaved else P.apply_rope_half
    q, kk = f(q, sin, cos), f(kk, sin, cos)
    tol = dict(rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(out[:, :H * hd].double().cpu().view(M, H, hd), q, **tol)
    if not store:
        assert torch.equal(k_pool, k_before) and torch.equal(v_pool, v_before)
        return
    touched = torch.zeros(18, PAGE, dtype=torch.bool)
    for m in range(M):
        p = int(positions[m]); page = int(page_table[int(slot_of_token[m]), p // PAGE]); off = p % PAGE
        touched[page, off] = True
        torch.testing.assert_close(k_pool[page, :, off].double().cpu(), kk[m], **tol)
        torch.testing.assert_close(v_pool[page, :, off].double().cpu(), v[m], **tol)
    keep = ~touched.to(DEV)
    assert torch.equal(k_pool.permute(0, 2, 1, 3)[keep], k_before.permute(0, 2, 1, 3)[keep])
    assert torch.equal(v_pool.permute(0, 2, 1, 3)[keep], v_before.permute(0, 2, 1, 3)[keep])


def _llama3_inv_freq(hd, factor):
    return P.rope_inv_freq(500000.0, hd, {"rope_type": "llama3", "factor": factor, "low_freq_factor": 1.0,
                                          "high_freq_factor": 4.0, "original_max_position_embeddings": 8192}).to(DEV)


FAR_POSITIONS = [0, 4095, 4096, 4223, 4224, 8191, 8192, 8703]


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,hd,factor,interleaved", [(8, 2, 128, 8.0, False), (8, 2, 64, 32.0, False), (3, 1, 128, 8.0, True)])
def test_rope_kv_write_at_positions_in_the_thousands(dtype, H, G, hd, factor, interleaved):
    """Positions up to 8,703 with the real models' rope constants: the angle is the float product
    pos * inv_freq, whose sine needs an accurate range reduction there, and the slot's page table
    is 137 entries long."""
    k = K()
    M = len(FAR_POSITIONS)
    qkv = _rand(M, (H + 2 * G) * hd, dtype=dtype, seed=21)
    positions = torch.tensor(FAR_POSITIONS, dtype=torch.int32, device=DEV)
    slot_of_token = torch.full((M,), 1, dtype=torch.int32, device=DEV)
    g = torch.Generator().manual_seed(5)
    page_table = torch.stack([torch.zeros(137, dtype=torch.int64), torch.randperm(140, generator=g)[:137]]).to(torch.int32).to(DEV)
    inv = _llama3_inv_freq(hd, factor)
    k_pool, v_pool = _paged(G, hd, 140, dtype)
    src = qkv.clone()
    k.rope_kv_write(qkv, positions, slot_of_token, page_table, inv, H, G, hd, hd, interleaved, k_pool, v_pool)
    x = src.double().cpu()
    q, kk, v = x[:, :H * hd].view(M, H, hd), x[:, H * hd:(H + G) * hd].view(M, G, hd), x[:, (H + G) * hd:].view(M, G, hd)
    sin, cos = P.rope_angles(positions.cpu(), inv.cpu())
    f = P.apply_rope_interleaved if interleaved else P.apply_rope_half
    q, kk = f(q, sin, cos), f(kk, sin, cos)
    tol = _tol(dtype)
    torch.testing.assert_close(qkv[:, :H * hd].double().cpu().view(M, H, hd), q, **tol)
    for m, p in enumerate(FAR_POSITIONS):
        page = int(page_table[1, p // PAGE]); off = p % PAGE
        torch.testing.assert_close(k_pool[page, :, off].double().cpu(), kk[m], **tol)
        assert torch.equal(v_pool[page, :, off].double().cpu(), v[m])


@pytest.mark.parametrize("hd,rot", [(128, 0), (64, 0), (128, 128), (64, 64)])
@pytest.mark.parametrize("M,H,G,K_,beside,store", [(1, 3, 1, 1024, 4, True), (17, 5, 1, 512, 60, True), (48, 16, 4, 2048, 2048, True), (64, 4, 2, 1024, 132, False),
                                                  (5, 2, 2, 1024, 0, True)])
def test_gemm_tc_qkv_with_columns_beside_the_heads_and_without_rotation(M, H, G, K_, beside, store, hd, rot):
    """Against the product and the kernel behind it (rotation, cache write): where nothing is rotated the same bits - queries, what lies beside
    the heads, keys and values in their pages, the rest of the pools as it was - with rotation to bf16's rounding (the separate kernel
    rounds twice)."""
    k = K()
    N = (H + 2 * G) * hd + beside
    a, w, bias = _rand(M, K_, dtype=torch.bfloat16, seed=51), _rand(N, K_, dtype=torch.bfloat16, seed=53, scale=0.05), _rand(N, seed=54, scale=0.5)
    assert k.gemm_tc_qkv_rope_supported(a, w, H, G, hd, rot, beside)
    assert not k.gemm_tc_qkv_rope_supported(a, w, H, G, hd, hd // 2, beside)
    positions = torch.arange(M, dtype=torch.int32, device=DEV) * 3 % 200
    slot_of_token = torch.arange(M, dtype=torch.int32, device=DEV) % 4
    page_table = torch.randperm(16).to(torch.int32).view(4, 4).to(DEV)
    inv = torch.tensor([1.0 / (10000.0 ** (2 * i / hd)) for i in range(hd // 2)], device=DEV)
    k0, v0 = _paged(G, hd, 16, torch.bfloat16)
    pools = [(k0.clone(), v0.clone()) for _ in range(2)]
    ref, out = torch.empty(M, N, dtype=torch.bfloat16, device=DEV), torch.full((M, N), 7.0, dtype=torch.bfloat16, device=DEV)
    k.gemm_tc(a, w, ref, k.OUT_SAME, bias)
    k.rope_kv_write(ref, positions, slot_of_token, page_table, inv, H, G, hd, rot, False, *(pools[0] if store else (None, None)))
    k.gemm_tc_qkv_rope(a, w, out, bias, positions, slot_of_token, page_table, inv if rot else None, False, H, G,
                       *(pools[1] if store else (None, None)), beside=beside)
    k.check_device_errors()
    same = (lambda x, y: torch.testing.assert_close(x.float(), y.float(), rtol=2e-2, atol=2e-2)) if rot else (lambda x, y: torch.testing.assert_close(x, y, rtol=0, atol=0))
    heads = (H + 2 * G) * hd
    same(out[:, :H * hd], ref[:, :H * hd])
    assert torch.equal(out[:, heads:], ref[:, heads:])
    assert (out[:, H * hd:heads] == 7.0).all()
    same(pools[1][0], pools[0][0])
    assert torch.equal(pools[1][1], pools[0][1])


@pytest.mark.parametrize("interleaved", [False, True])
def test_gemm_tc_qkv_rope_at_positions_in_the_thousands(interleaved):
    k = K()
    H, G, hd, K_ = 4, 2, 128, 1024
    M = len(FAR_POSITIONS)
    N = (H + 2 * G) * hd
    a = _rand(M, K_, dtype=torch.bfloat16, seed=61, scale=1.0)
    w = _rand(N, K_, dtype=torch.bfloat16, seed=62, scale=0.05)
    assert k.gemm_tc_qkv_rope_supported(a, w, H, G, hd, hd)
    positions = torch.tensor(FAR_POSITIONS, dtype=torch.int32, device=DEV)
    slot_of_token = torch.full((M,), 1, dtype=torch.int32, device=DEV)
    g = torch.Generator().manual_seed(6)
    page_table = torch.stack([torch.zeros(137, dtype=torch.int64), torch.randperm(140, generator=g)[:137]]).to(torch.int32).to(DEV)
    inv = _llama3_inv_freq(hd, 8.0)
    k_pool, v_pool = _paged(G, hd, 140, torch.bfloat16)
    out = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device=DEV)
    k.gemm_tc_qkv_rope(a, w, out, None, positions, slot_of_token, page_table, inv, interleaved, H, G, k_pool, v_pool)
    k.check_device_errors()
    y = a.double().cpu() @ w.double().cpu().T
    q, kk, v = y[:, :H * hd].view(M, H, hd), y[:, H * hd:(H + G) * hd].view(M, G, hd), y[:, (H + G) * hd:].view(M, G, hd)
    sin, cos = P.rope_angles(positions.cpu(), inv.cpu())
    f = P.apply_rope_interleaved if interleaved else P.apply_rope_half
    q, kk = f(q, sin, cos), f(kk, sin, cos)
    tol = dict(rtol=2e-2, atol=2e-2)
    torch.testing.assert_close(out[:, :H * hd].double().cpu().view(M, H, hd), q, **tol)
    for m, p in enumerate(FAR_POSITIONS):
        page = int(page_table[1, p // PAGE]); off = p % PAGE
        torch.testing.assert_close(k_pool[page, :, off].double().cpu(), kk[m], **tol)
        torch.testing.assert_close(v_pool[page, :, off].double().cpu(), v[m], **tol)


# ----------------------------------------------------------------------------- attention
def _attention_case(dtype, H, G, hd, lens_q, lens_kv, window=0, seed=0, craft=None):
    """Builds a paged cache with scrambled pages for sequences of lens_kv tokens; the
    last lens_q[b] tokens of each are the step's queries.  Returns inputs and the
    plain float64 result."""
    B = len(lens_kv)
    g = torch.Generator().manual_seed(seed)
    n_pages_each = [-(-n // PAGE) for n in lens_kv]
    total_pages = sum(n_pages_each) + 3
    perm = torch.randperm(total_pages, generator=g).tolist()
    max_pages = max(n_pages_each) + 1
    page_table = torch.full((B + 1, max_pages), 0, dtype=torch.int32)
    k_pool = (torch.randn(total_pages, G, PAGE, hd, generator=g) * 3).to(dtype)   # stale values, large
    v_pool = (torch.randn(total_pages, G, PAGE, hd, generator=g) * 3).to(dtype)
    slots = list(range(B, 0, -1))      # slots in reverse order
    ks, vs, qs = [], [], []
    pi = 0
    for b in range(B):
        n = lens_kv[b]
        kb = torch.randn(n, G, hd, generator=g).to(dtype)
        vb = torch.randn(n, G, hd, generator=g).to(dtype)
        qb = torch.randn(lens_q[b], H, hd, generator=g).to(dtype)
        if craft is not None:
            craft(b, qb, kb, vb)
        for p in range(n_pages_each[b]):
            page = perm[pi]; pi += 1
            page_table[slots[b], p] = page
            lo, hi = p * PAGE, min(n, (p + 1) * PAGE)
            k_pool[page, :, :hi - lo] = kb[lo:hi].transpose(0, 1)
            v_pool[page, :, :hi - lo] = vb[lo:hi].transpose(0, 1)
        ks.append(kb); vs.append(vb); qs.append(qb)
    positions, slot_of_token, refs = [], [], []
    for b in range(B):
        n, nq = lens_kv[b], lens_q[b]
        full_q = torch.zeros(n, H, hd, dtype=torch.float64)
        full_q[n - nq:] = qs[b].double()
        out = P.causal_attention(full_q, ks[b].double(), vs[b].double(), window=window or None)
        refs.append(out[n - nq:].reshape(nq, H * hd))
        positions += list(range(n - nq, n))
        slot_of_token += [slots[b]] * nq
    q = torch.cat([x.reshape(x.shape[0], H * hd) for x in qs]).to(DEV)
    return (q, k_pool.to(DEV), v_pool.to(DEV), page_table.to(DEV),
            torch.tensor(slot_of_token, dtype=torch.int32, device=DEV),
            torch.tensor(positions, dtype=torch.int32, device=DEV), torch.cat(refs))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,hd", [(4, 2, 16), (3, 1, 32), (5, 5, 48), (8, 2, 64), (6, 2, 80), (8, 1, 128), (2, 2, 256), (7, 7, 112)])
def test_attention_simt_prefill_and_decode_shapes(dtype, H, G, hd):
    k = K()
    for lens_q, lens_kv in (([1, 1, 1], [1, 64, 200]), ([5, 70, 1, 33], [5, 70, 129, 97]), ([130], [130])):
        q, kp, vp, pt, sot, pos, ref = _attention_case(dtype, H, G, hd, lens_q, lens_kv, seed=hd + len(lens_q))
        out = torch.empty(q.shape[0], H * hd, dtype=dtype, device=DEV)
        k.attention_simt(q, kp, vp, pt, sot, pos, out, H, G, hd, 1.0 / math.sqrt(hd))
        torch.testing.assert_close(out.double().cpu(), ref, **(_tol(dtype) if dtype == torch.bfloat16 else dict(rtol=2e-5, atol=2e-5)))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_attention_simt_window(dtype):
    k = K()
    H, G, hd, W = 4, 2, 32, 70
    q, kp, vp, pt, sot, pos, ref = _attention_case(dtype, H, G, hd, [40, 1, 150], [40, 300, 150], window=W, seed=3)
    out = torch.empty(q.shape[0], H * hd, dtype=dtype, device=DEV)
    k.attention_simt(q, kp, vp, pt, sot, pos, out, H, G, hd, 1.0 / math.sqrt(hd), W)
    torch.testing.assert_close(out.double().cpu(), ref, **(_tol(dtype) if dtype == torch.bfloat16 else dict(rtol=2e-5, atol=2e-5)))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("far", [0, 63, 64, 449, 450])
def test_attention_finds_one_far_key_among_hundreds(dtype, far):
    """One key is made to stand out (query and key scaled so that its score dominates):
    the output must be that key's value, wherever in the pages it lies."""
    H, G, hd, n = 4, 2, 64, 451

    def craft(b, qb, kb, vb):
        direction = torch.ones(hd) / math.sqrt(hd)
        qb[:] = (direction * 12.0).to(qb.dtype)          # every head asks for the same direction
        kb[:] = (kb.float() * 0.05).to(kb.dtype)
        kb[far] = (direction * 12.0).to(kb.dtype)        # score 144/8 = 18 against ~0 elsewhere
    q, kp, vp, pt, sot, pos, ref = _attention_case(dtype, H, G, hd, [1], [n], seed=5, craft=craft)
    out = torch.empty(1, H * hd, dtype=dtype, device=DEV)
    K().attention_simt(q, kp, vp, pt, sot, pos, out, H, G, hd, 1.0 / math.sqrt(hd))
    torch.testing.assert_close(out.double().cpu(), ref, **(_tol(dtype) if dtype == torch.bfloat16 else dict(rtol=2e-5, atol=2e-5)))
    # and the plain result is, to 1e-4, the far key's value: the test would notice a missed key
    page = int(pt[1, far // PAGE]); v_far = vp[page, :, far % PAGE].double().cpu()   # [G, hd]
    want = v_far.repeat_interleave(H // G, dim=0).reshape(1, H * hd)
    assert (ref - want).abs().max() < 1e-3


# ----------------------------------------------------------------------------- decode attention (tensor cores)
def _decode_inputs(case):
    q, kp, vp, pt, sot, pos, ref = case
    return q, kp, vp, pt, sot.clone(), (pos + 1).to(torch.int32), ref


@pytest.mark.parametrize("H,G,hd", [(32, 8, 128), (8, 8, 128), (6, 2, 64), (16, 1, 64), (5, 5, 128), (24, 8, 64)])
@pytest.mark.parametrize("splits", [1, 2, 7, 32])
@pytest.mark.parametrize("planned", [False, True])
def test_attention_decode_matches_plain(H, G, hd, splits, planned):
    """``planned``: the chunks are dealt to the sequences by length (as the engine does
    for a batch); otherwise every sequence is cut into ``splits`` equal chunks."""
    k = K()
    assert k.attention_decode_supported(torch.bfloat16, H, G, hd)
    lens = [1, 15, 16, 17, 64, 65, 200, 513]
    case = _attention_case(torch.bfloat16, H, G, hd, [1] * len(lens), lens, seed=hd + H + splits)
    q, kp, vp, pt, slots, kv_lens, ref = _decode_inputs(case)
    out = torch.empty(len(lens), H * hd, dtype=torch.bfloat16, device=DEV)
    plan = k.decode_plan(slots, kv_lens, 0, splits) if planned else None
    assert (plan is not None) == (planned and splits > 1)
    k.attention_decode(q, kp, vp, pt, slots, kv_lens, out, H, G, hd, 1.0 / math.sqrt(hd), num_splits=splits, plan=plan)
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))
    # and the any-shape kernel gives the same to bf16 rounding
    simt = torch.empty_like(out)
    k.attention_simt(q, kp, vp, pt, slots, (kv_lens - 1).to(torch.int32), simt, H, G, hd, 1.0 / math.sqrt(hd))
    torch.testing.assert_close(out.float(), simt.float(), rtol=2e-2, atol=2e-2)


@pytest.mark.parametrize("H,G,hd", [(32, 8, 128), (6, 2, 64), (16, 1, 128)])
@pytest.mark.parametrize("splits", [2, 4, 8])
def test_attention_decode_chunks_of_a_sequence_as_a_cluster(H, G, hd, splits):
    """No scratch, one kernel: the chunks' CTAs combine through distributed shared memory."""
    k = K()
    lens = [1, 15, 64, 65, 200, 513, 1100]
    for window in (0, 90):
        case = _attention_case(torch.bfloat16, H, G, hd, [1] * len(lens), lens, window=window, seed=hd + splits)
        q, kp, vp, pt, slots, kv_lens, ref = _decode_inputs(case)
        out = torch.full((len(lens), H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
        before = k.launch_count
        k.attention_decode(q, kp, vp, pt, slots, kv_lens, out, H, G, hd, 1.0 / math.sqrt(hd), window, num_splits=splits, cluster=True)
        assert k.launch_count - before == 1
        torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))


@pytest.mark.parametrize("H,G,hd", [(32, 8, 128), (6, 2, 64)])
def test_attention_decode_whole_sequences_longest_first(H, G, hd):
    """Every sequence whole in one CTA a KV head, started in the order of their lengths (inside the
    window): the order plan lists the sequences longest first, ties in the order of the batch, and
    the answers are those of the batch's own order."""
    k = K()
    lens = [1 + (i * 131) % 700 for i in range(70)] + [1500, 64, 64, 1]
    for window in (0, 90):
        case = _attention_case(torch.bfloat16, H, G, hd, [1] * len(lens), lens, window=window, seed=hd + window)
        q, kp, vp, pt, slots, kv_lens, ref = _decode_inputs(case)
        order = k.decode_order(slots, kv_lens, window)
        n = len(lens)
        entries = order[:4 * n].view(n, 4).cpu().tolist()
        inside = [min(v, window) if window else v for v in lens]
        assert [e[0] for e in entries] == sorted(range(n), key=lambda b: (-inside[b], b))
        assert all(e[1] == 1 << 16 and e[2] == lens[e[0]] and e[3] == int(slots[e[0]]) for e in entries)
        out = torch.full((n, H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
        before = k.launch_count
        k.attention_decode(q, kp, vp, pt, slots, kv_lens, out, H, G, hd, 1.0 / math.sqrt(hd), window, num_splits=1, plan=order)
        assert k.launch_count - before == 1
        torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))
        plain = torch.empty_like(out)
        k.attention_decode(q, kp, vp, pt, slots, kv_lens, plain, H, G, hd, 1.0 / math.sqrt(hd), window, num_splits=1)
        assert torch.equal(out, plain)


@pytest.mark.parametrize("splits,window", [(2, 0), (7, 0), (3, 100)])
def test_attention_decode_deals_chunks_by_length(splits, window):
    """More sequences than a warp has lanes, one of them far longer than the rest: the
    long one gets most of the chunks, and every sequence is still answered whole."""
    k = K()
    H, G, hd = 4, 2, 64
    lens = [1] * 14 + [1500] + [64, 65, 129] * 6 + [700, 3]
    assert len(lens) > 32
    case = _attention_case(torch.bfloat16, H, G, hd, [1] * len(lens), lens, window=window, seed=splits)
    q, kp, vp, pt, slots, kv_lens, ref = _decode_inputs(case)
    out = torch.full((len(lens), H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    plan = k.decode_plan(slots, kv_lens, window, splits)
    # the plan itself: every sequence has at least one chunk, together no more than the grid,
    # neighbours in the grid, and the longer a sequence the more it gets
    B = len(lens)
    entries = plan[:4 * B * splits].view(-1, 4).cpu()
    seqs = plan[4 * B * splits:].view(-1, 2).cpu()
    assert int(seqs[:, 1].min()) >= 1 and int(seqs[:, 1].sum()) <= B * splits
    assert seqs[:, 0].tolist() == [int(x) for x in (torch.cumsum(seqs[:, 1], 0) - seqs[:, 1])]
    assert int(seqs[14, 1]) == int(seqs[:, 1].max()) and int(seqs[0, 1]) == 1
    if window == 0:
        assert int(seqs[14, 1]) > int(seqs[33, 1]) > int(seqs[34, 1])      # 1500, 700 and 3 keys
    for b in range(B):
        for j in range(int(seqs[b, 1])):
            e = entries[int(seqs[b, 0]) + j].tolist()
            assert e == [b, j | (int(seqs[b, 1]) << 16), lens[b], int(slots[b])]
    assert (entries[int(seqs[:, 1].sum()):, 0] == -1).all()
    k.attention_decode(q, kp, vp, pt, slots, kv_lens, out, H, G, hd, 1.0 / math.sqrt(hd), window, num_splits=splits, plan=plan)
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))


def test_attention_decode_window_and_strided_queries():
    k = K()
    H, G, hd, W = 8, 2, 128, 70
    lens = [10, 70, 71, 300]
    case = _attention_case(torch.bfloat16, H, G, hd, [1] * 4, lens, window=W, seed=9)
    q, kp, vp, pt, slots, kv_lens, ref = _decode_inputs(case)
    wide = torch.zeros(4, (H + 2 * G) * hd, dtype=torch.bfloat16, device=DEV)     # q as a view into a qkv buffer
    wide[:, :H * hd] = q
    out = torch.empty(4, H * hd, dtype=torch.bfloat16, device=DEV)
    k.attention_decode(wide[:, :H * hd], kp, vp, pt, slots, kv_lens, out, H, G, hd, 1.0 / math.sqrt(hd), W, num_splits=3)
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))


@pytest.mark.parametrize("far", [0, 15, 16, 63, 64, 449, 450])
@pytest.mark.parametrize("splits", [1, 5])
def test_attention_decode_finds_one_far_key_among_hundreds(far, splits):
    H, G, hd, n = 8, 2, 128, 451

    def craft(b, qb, kb, vb):
        direction = torch.ones(hd) / math.sqrt(hd)
        qb[:] = (direction * 14.0).to(qb.dtype)
        kb[:] = (kb.float() * 0.05).to(kb.dtype)
        kb[far] = (direction * 14.0).to(kb.dtype)
    case = _attention_case(torch.bfloat16, H, G, hd, [1], [n], seed=5, craft=craft)
    q, kp, vp, pt, slots, kv_lens, ref = _decode_inputs(case)
    out = torch.empty(1, H * hd, dtype=torch.bfloat16, device=DEV)
    K().attention_decode(q, kp, vp, pt, slots, kv_lens, out, H, G, hd, 1.0 / math.sqrt(hd), num_splits=splits)
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))
    page = int(pt[1, far // PAGE]); v_far = vp[page, :, far % PAGE].double().cpu()
    assert (ref - v_far.repeat_interleave(H // G, dim=0).reshape(1, H * hd)).abs().max() < 1e-3


def test_attention_decode_ignores_garbage_beyond_the_sequence():
    """Rows of a page beyond the sequence's length may hold anything, NaN included."""
    k = K()
    H, G, hd = 4, 1, 64
    case = _attention_case(torch.bfloat16, H, G, hd, [1, 1], [5, 70], seed=2)
    q, kp, vp, pt, slots, kv_lens, ref = _decode_inputs(case)
    for b, n in enumerate([5, 70]):
        page = int(pt[int(slots[b]), (n - 1) // PAGE])
        kp[page, :, n % PAGE:] = float("nan"); vp[page, :, n % PAGE:] = float("nan")
    out = torch.empty(2, H * hd, dtype=torch.bfloat16, device=DEV)
    k.attention_decode(q, kp, vp, pt, slots, kv_lens, out, H, G, hd, 1.0 / math.sqrt(hd), num_splits=2)
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))


# ----------------------------------------------------------------------------- prefill attention (tensor cores)
def _prefill_inputs(case, lens_q, lens_kv):
    q, kp, vp, pt, sot, pos, ref = case
    B = len(lens_q)
    cu = [0]
    for n in lens_q:
        cu.append(cu[-1] + n)
    slots = list(range(B, 0, -1))        # as _attention_case assigns them
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)
    return q, kp, vp, pt, i32(cu), i32(slots), i32(lens_kv), ref


@pytest.mark.parametrize("H,G,hd", [(32, 8, 128), (4, 4, 128), (6, 2, 64), (3, 1, 64)])
@pytest.mark.parametrize("lens_q,lens_kv", [([1, 5, 64, 65, 200], [1, 5, 64, 65, 200]),      # whole prompts
                                            ([130, 1, 33, 64], [130, 300, 97, 128]),            # chunks after a cached prefix
                                            ([700], [700])])
def test_attention_prefill_matches_plain(H, G, hd, lens_q, lens_kv):
    k = K()
    assert k.attention_prefill_supported(torch.bfloat16, H, G, hd)
    case = _attention_case(torch.bfloat16, H, G, hd, lens_q, lens_kv, seed=hd + H + len(lens_q))
    q, kp, vp, pt, cu, slots, kv_lens, ref = _prefill_inputs(case, lens_q, lens_kv)
    out = torch.full((q.shape[0], H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    k.attention_prefill(q, kp, vp, pt, cu, slots, kv_lens, lens_q, out, H, G, hd, 1.0 / math.sqrt(hd))
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))
    simt = torch.empty_like(out)
    k.attention_simt(q, kp, vp, pt, case[4], case[5], simt, H, G, hd, 1.0 / math.sqrt(hd))
    torch.testing.assert_close(out.float(), simt.float(), rtol=2e-2, atol=2e-2)


def test_attention_prefill_window_and_garbage_beyond_the_sequence():
    k = K()
    H, G, hd, W = 4, 2, 64, 70
    lens_q, lens_kv = [40, 150, 3], [40, 300, 200]
    case = _attention_case(torch.bfloat16, H, G, hd, lens_q, lens_kv, window=W, seed=4)
    q, kp, vp, pt, cu, slots, kv_lens, ref = _prefill_inputs(case, lens_q, lens_kv)
    for b, n in enumerate(lens_kv):       # rows of the last page beyond the sequence: NaN
        if n % PAGE:
            page = int(pt[int(slots[b]), (n - 1) // PAGE])
            kp[page, :, n % PAGE:] = float("nan"); vp[page, :, n % PAGE:] = float("nan")
    out = torch.empty(q.shape[0], H * hd, dtype=torch.bfloat16, device=DEV)
    k.attention_prefill(q, kp, vp, pt, cu, slots, kv_lens, lens_q, out, H, G, hd, 1.0 / math.sqrt(hd), W)
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))


@pytest.mark.parametrize("far", [0, 63, 64, 300])
def test_attention_prefill_finds_one_far_key(far):
    """Every query from position `far` on must return the value of key `far` (its score dominates)."""
    H, G, hd, n = 4, 2, 128, 451

    def craft(b, qb, kb, vb):
        direction = torch.ones(hd) / math.sqrt(hd)
        qb[:] = (direction * 14.0).to(qb.dtype)
        kb[:] = (kb.float() * 0.05).to(kb.dtype)
        kb[far] = (direction * 14.0).to(kb.dtype)
    case = _attention_case(torch.bfloat16, H, G, hd, [n], [n], seed=6, craft=craft)
    q, kp, vp, pt, cu, slots, kv_lens, ref = _prefill_inputs(case, [n], [n])
    out = torch.empty(n, H * hd, dtype=torch.bfloat16, device=DEV)
    K().attention_prefill(q, kp, vp, pt, cu, slots, kv_lens, [n], out, H, G, hd, 1.0 / math.sqrt(hd))
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))
    page = int(pt[1, far // PAGE]); v_far = vp[page, :, far % PAGE].double().cpu()
    want = v_far.repeat_interleave(H // G, dim=0).reshape(1, H * hd)
    assert (ref[far + 1:] - want).abs().max() < 1e-3


# ----------------------------------------------------------------------------- prefill attention (tcgen05)
@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("H,G", [(32, 8), (4, 4), (3, 1)])
@pytest.mark.parametrize("lens_q,lens_kv", [([1, 5, 64, 65, 200], [1, 5, 64, 65, 200]),
                                            ([130, 1, 33, 64], [130, 300, 97, 128]),
                                            ([129], [129]), ([128, 256], [128, 256]), ([700], [700]), ([40], [1000]),
                                            # 18 key tiles, the query tiles not aligned with them: both of a query tile's
                                            # last two key tiles are masked in part, and every ring and barrier wraps
                                            ([1700], [2304])])
def test_attention_prefill_tc_matches_plain(H, G, lens_q, lens_kv, hd):
    k = K()
    assert k.attention_prefill_tc_supported(torch.bfloat16, H, G, hd)
    case = _attention_case(torch.bfloat16, H, G, hd, lens_q, lens_kv, seed=H + len(lens_q) + lens_kv[0])
    q, kp, vp, pt, cu, slots, kv_lens, ref = _prefill_inputs(case, lens_q, lens_kv)
    out = torch.full((q.shape[0], H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    k.attention_prefill_tc(q, kp, vp, pt, cu, slots, kv_lens, lens_q, out, H, G, hd, 1.0 / math.sqrt(hd))
    k.check_device_errors()
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))


@pytest.mark.parametrize("hd", [64, 128])
def test_attention_prefill_tc_window_and_strided_queries(hd):
    k = K()
    H, G, W = 4, 2, 200
    lens_q, lens_kv = [40, 350, 3], [40, 500, 300]
    case = _attention_case(torch.bfloat16, H, G, hd, lens_q, lens_kv, window=W, seed=4)
    q, kp, vp, pt, cu, slots, kv_lens, ref = _prefill_inputs(case, lens_q, lens_kv)
    wide = torch.zeros(q.shape[0], (H + 2 * G) * hd, dtype=torch.bfloat16, device=DEV)
    wide[:, :H * hd] = q
    out = torch.empty(q.shape[0], H * hd, dtype=torch.bfloat16, device=DEV)
    k.attention_prefill_tc(wide[:, :H * hd], kp, vp, pt, cu, slots, kv_lens, lens_q, out, H, G, hd, 1.0 / math.sqrt(hd), W)
    k.check_device_errors()
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("far", [0, 63, 64, 127, 128, 300])
def test_attention_prefill_tc_finds_one_far_key_and_rescales(far, hd):
    """Every query from position `far` on must return the value of key `far`: its score is far
    above the running maximum of the tiles before it, so the lazily kept maximum has to move
    and the accumulator has to be rescaled."""
    H, G, n = 4, 2, 451

    def craft(b, qb, kb, vb):
        direction = torch.ones(hd) / math.sqrt(hd)
        qb[:] = (direction * 14.0).to(qb.dtype)
        kb[:] = (kb.float() * 0.05).to(kb.dtype)
        kb[far] = (direction * 14.0).to(kb.dtype)
    case = _attention_case(torch.bfloat16, H, G, hd, [n], [n], seed=6, craft=craft)
    q, kp, vp, pt, cu, slots, kv_lens, ref = _prefill_inputs(case, [n], [n])
    out = torch.empty(n, H * hd, dtype=torch.bfloat16, device=DEV)
    K().attention_prefill_tc(q, kp, vp, pt, cu, slots, kv_lens, [n], out, H, G, hd, 1.0 / math.sqrt(hd))
    K().check_device_errors()
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))
    page = int(pt[1, far // PAGE]); v_far = vp[page, :, far % PAGE].double().cpu()
    want = v_far.repeat_interleave(H // G, dim=0).reshape(1, H * hd)
    assert (ref[far + 1:] - want).abs().max() < 1e-3


# ----------------------------------------------------------------------------- prefill attention (tcgen05), two CTAs an SM
def _plain_attention_f64(q, kp, vp, pt, slots, lens_q, lens_kv, H, G, hd, scale, window=0, keep_first=0, chunk=0, softcap=0.0, sink=False, sinks=None,
                         gate=None, gate_per_head=False):
    """Float64 attention of a prompt step over the paged cache, with every option of the tensor-core prompt kernel."""
    outs, at = [], 0
    for b, (nq, n) in enumerate(zip(lens_q, lens_kv)):
        pages = pt[int(slots[b]), :-(-n // PAGE)].long()
        kb, vb = ((x[pages].transpose(1, 2).reshape(-1, G, hd)[:n].double().repeat_interleave(H // G, dim=1)) for x in (kp, vp))
        s = torch.einsum("ihd,jhd->hij", q[at:at + nq].view(nq, H, hd).double(), kb) * scale
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        i, j = torch.arange(n - nq, n, device=q.device)[:, None], torch.arange(n, device=q.device)[None]
        seen = j <= i
        if window:
            seen &= (i - j < window) | (j < keep_first)
        if chunk:
            seen &= j >= i - i % chunk
        s = s.masked_fill(~seen, -math.inf)
        if sink:
            extra = torch.zeros(H, dtype=torch.float64, device=q.device) if sinks is None else sinks.double()
            s = torch.cat([s, extra[:, None, None].expand(H, nq, 1)], dim=-1)
        p = torch.softmax(s, dim=-1)[..., :n]
        outs.append(torch.einsum("hij,jhd->ihd", p, vb))
        at += nq
    out = torch.cat(outs)
    if gate is not None:
        out = out * torch.sigmoid(gate.double()).view(out.shape[0], H, -1)
    return out.reshape(out.shape[0], H * hd)


def test_attention_prefill_tc_two_an_sm_where_it_pays():
    """By the CTAs, masks, caps and the rows of a tile."""
    two = K().attention_prefill_tc_two_an_sm
    assert [two([n], 32) for n in (1000, 1152, 1153, 4096)] == [False, False, True, True]
    assert [two([n], 32, softcap=30.0) for n in (1400, 1920, 1921)] == [False, False, True] and two([100] * 12, 32, softcap=30.0)
    for mask in ({"window": 512}, {"chunk": 256}, {"window": 9, "softcap": 5.0}):
        assert not two([8192], 32, **mask) and not two([100] * 12, 32, **mask) and two([40] * 64, 32, **mask) and not two([40] * 9, 32, **mask)


@pytest.mark.parametrize("opts", [{}, {"softcap": 1000.0}], ids=["plain", "cap"])
@pytest.mark.parametrize("far", [0, 63, 64, 127, 128, 191, 192, 300, "stairs"])
def test_attention_prefill_tc_by_halves_of_a_row_rescales(far, opts):
    """Heads of 64 in more CTAs than fit the GPU two an SM at once: the form with two threads a row.  A key in either half of a 128-key tile far
    above the running maximum of all before it, so that both halves' threads must learn of it and rescale their part of the accumulator; "stairs":
    a higher one in every half tile.  With and without the code for masks and caps (a cap that moves a score of 35 by 1.4e-2)."""
    k = K()
    H, G, hd, n = 128, 8, 64, 451

    def craft(b, qb, kb, vb):
        direction = torch.ones(hd) / math.sqrt(hd)
        qb[:] = (direction * 20.0).to(qb.dtype)
        kb[:] = (kb.float() * 0.05).to(kb.dtype)
        for i, pos in enumerate(range(5, n, 64) if far == "stairs" else [far]):
            kb[pos] = (direction * (3.0 * (i + 1) if far == "stairs" else 14.0)).to(kb.dtype)       # a step: 60 / 8 in the score, 2^10.8
    case = _attention_case(torch.bfloat16, H, G, hd, [n], [n], seed=6, craft=craft)
    q, kp, vp, pt, cu, slots, kv_lens, ref = _prefill_inputs(case, [n], [n])
    assert k.attention_prefill_tc_two_an_sm([n], H, **opts)
    out = torch.full((n, H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    k.attention_prefill_tc(q, kp, vp, pt, cu, slots, kv_lens, [n], out, H, G, hd, 1.0 / math.sqrt(hd), **opts)
    k.check_device_errors()
    if opts:
        ref = _plain_attention_f64(q, kp, vp, pt, slots, [n], [n], H, G, hd, 1.0 / math.sqrt(hd), **opts).cpu()
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))
    if far != "stairs":
        page = int(pt[1, far // PAGE]); v_far = vp[page, :, far % PAGE].double().cpu()
        assert (ref[far + 1:] - v_far.repeat_interleave(H // G, dim=0).reshape(1, H * hd)).abs().max() < 1e-3


_SHORT_Q = [1, 64, 33, 17, 2, 48, 63, 50, 128, 1, 40, 5]


@pytest.mark.parametrize("opts", [{}, {"window": 100}, {"window": 200, "keep_first": 70}, {"window": 65, "keep_first": 3, "sink": True}, {"chunk": 96}, {"chunk": 256},
                                  {"softcap": 5.0}, {"softcap": 20.0, "window": 150, "sink": True}, {"sink": True, "gate": "element"},
                                  {"sinks": True, "sink": True, "gate": "head"}, {"gate": "head", "window": 129}, {"chunk": 200, "gate": "element"}],
                         ids=lambda o: "-".join(f"{a}{b}" for a, b in o.items()) or "plain")
@pytest.mark.parametrize("lens_q,lens_kv", [([200, 37, 300, 1], [200, 130, 700, 260]), ([1400], [1400]),
                                            (_SHORT_Q, [n + p for n, p in zip(_SHORT_Q, (700, 0, 95, 300, 128, 64, 1, 500, 260, 63, 127, 191))])],
                         ids=["portions", "prompt", "short"])
def test_attention_prefill_tc_by_halves_of_a_row_with_every_option(lens_q, lens_kv, opts):
    """The same form with caps, sinks and gates, and, where its tiles have few rows, with masks and kept first tokens (longer ones: the form with a thread a
    row, in as many CTAs), against float64: sequences behind what is cached, query tiles that are not whole, rows whose window begins inside a
    tile's first or second half."""
    k = K()
    H, G, hd = 72, 6, 64

    def craft(b, qb, kb, vb):
        qb *= 2                              # scores of standard deviation 2: the running maximum moves
    case = _attention_case(torch.bfloat16, H, G, hd, lens_q, lens_kv, seed=len(lens_q), craft=craft)
    q, kp, vp, pt, cu, slots, kv_lens, _ = _prefill_inputs(case, lens_q, lens_kv)
    kw = dict(opts)
    masked = "window" in kw or "chunk" in kw
    assert k.attention_prefill_tc_two_an_sm(lens_q, H, **{a: v for a, v in kw.items() if a in ("window", "chunk", "softcap")}) == (not masked or len(lens_q) > 4)
    if kw.get("sinks"):
        kw["sinks"] = _rand(H, seed=8, scale=2.0)
    if kw.get("gate"):
        kw["gate_per_head"] = kw["gate"] == "head"
        kw["gate"] = _rand(q.shape[0], H if kw["gate_per_head"] else H * hd, dtype=torch.bfloat16, seed=9)
    out = torch.full((q.shape[0], H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    k.attention_prefill_tc(q, kp, vp, pt, cu, slots, kv_lens, lens_q, out, H, G, hd, 1.0 / math.sqrt(hd), **kw)
    k.check_device_errors()
    ref = _plain_attention_f64(q, kp, vp, pt, slots, lens_q, lens_kv, H, G, hd, 1.0 / math.sqrt(hd), **kw)
    torch.testing.assert_close(out.double(), ref, **_tol(torch.bfloat16))


# ----------------------------------------------------------------------------- attention over thousands of keys
def _far_key_craft(far, hd, gain=16.0):
    def craft(b, qb, kb, vb):
        direction = torch.ones(hd) / math.sqrt(hd)
        qb[:] = (direction * gain).to(qb.dtype)
        kb[:] = (kb.float() * 0.05).to(kb.dtype)
        kb[far] = (direction * gain).to(kb.dtype)      # its score stands far above the thousands of others
    return craft


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("n,far", [(4096, 0), (4096, 4095), (8704, 77), (8704, 8640)])
def test_attention_decode_over_thousands_of_keys(n, far, hd):
    """The contexts the benchmarks decode at: one key among 4,096 or 8,704 made to stand out, a
    short sequence beside it; every way the engine runs it (one chunk, dealt chunks, a cluster)."""
    k = K()
    H, G = 8, 2
    lens = [n, 33]
    craft = _far_key_craft(far, hd)
    case = _attention_case(torch.bfloat16, H, G, hd, [1, 1], lens, seed=n + far,
                           craft=lambda b, qb, kb, vb: craft(b, qb, kb, vb) if b == 0 else None)
    q, kp, vp, pt, slots, kv_lens, ref = _decode_inputs(case)
    page = int(pt[int(slots[0]), far // PAGE]); v_far = vp[page, :, far % PAGE].double().cpu()
    assert (ref[0:1] - v_far.repeat_interleave(H // G, dim=0).reshape(1, H * hd)).abs().max() < 2e-3
    for splits, planned, cluster in ((1, False, False), (8, False, False), (8, True, False), (8, False, True)):
        out = torch.full((2, H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
        plan = k.decode_plan(slots, kv_lens, 0, splits) if planned else None
        k.attention_decode(q, kp, vp, pt, slots, kv_lens, out, H, G, hd, 1.0 / math.sqrt(hd), num_splits=splits,
                           plan=plan, cluster=cluster)
        torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))
    simt = torch.empty(2, H * hd, dtype=torch.bfloat16, device=DEV)
    k.attention_simt(q, kp, vp, pt, slots, (kv_lens - 1).to(torch.int32), simt, H, G, hd, 1.0 / math.sqrt(hd))
    torch.testing.assert_close(simt.double().cpu(), ref, **_tol(torch.bfloat16))


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("lens_q,lens_kv,far", [([4096], [4096], 1), ([4096], [4096], 3900), ([600, 70], [8704, 70], 8100),
                                                ([600, 70], [8704, 70], 5)])
def test_attention_prefill_tc_over_thousands_of_keys(lens_q, lens_kv, far, hd):
    """A whole prompt of 4,096 tokens, and a 600-token portion behind 8,104 cached positions."""
    k = K()
    H, G = 4, 2
    craft = _far_key_craft(far, hd)
    case = _attention_case(torch.bfloat16, H, G, hd, lens_q, lens_kv, seed=far + lens_kv[0],
                           craft=lambda b, qb, kb, vb: craft(b, qb, kb, vb) if b == 0 else None)
    q, kp, vp, pt, cu, slots, kv_lens, ref = _prefill_inputs(case, lens_q, lens_kv)
    out = torch.full((q.shape[0], H * hd), float("nan"), dtype=torch.bfloat16, device=DEV)
    k.attention_prefill_tc(q, kp, vp, pt, cu, slots, kv_lens, lens_q, out, H, G, hd, 1.0 / math.sqrt(hd))
    k.check_device_errors()
    torch.testing.assert_close(out.double().cpu(), ref, **_tol(torch.bfloat16))
    # queries behind the far key return its value
    first_q = lens_kv[0] - lens_q[0]
    page = int(pt[int(slots[0]), far // PAGE]); v_far = vp[page, :, far % PAGE].double().cpu()
    want = v_far.repeat_interleave(H // G, dim=0).reshape(1, H * hd)
    lo = max(far + 1 - first_q, 0)
    assert (ref[lo:lens_q[0]] - want).abs().max() < 2e-3
    other = torch.empty_like(out)
    k.attention_prefill(q, kp, vp, pt, cu, slots, kv_lens, lens_q, other, H, G, hd, 1.0 / math.sqrt(hd))
    torch.testing.assert_close(other.double().cpu(), ref, **_tol(torch.bfloat16))


# ----------------------------------------------------------------------------- sampling
def test_argmax_first_maximum_wins_and_non_finite_is_skipped():
    k = K()
    V = 5000
    logits = _rand(6, V, seed=12)
    logits[0, 4000] = 50.0; logits[0, 17] = 50.0             # tie: the first wins
    logits[1, :] = float("-inf"); logits[1, 4999] = -3.0
    logits[2, 100] = float("nan"); logits[2, 7] = 99.0
    logits[3, :] = float("nan")                              # nothing finite: token 0
    logits[4, 0] = float("inf"); logits[4, 9] = 60.0         # +inf is not finite either
    out = torch.empty(6, dtype=torch.int32, device=DEV)
    k.argmax(logits, out)
    want = [P.argmax_finite(logits[i].cpu().numpy()) for i in range(6)]
    assert out.tolist() == want and want[:5] == [17, 4999, 7, 0, 9]


@pytest.mark.parametrize("V", [7, 384, 5000, 128256])
def test_temperature_sampling_follows_the_plain_sampler(V):
    k = K()
    rows = 24
    logits = _rand(rows, V, seed=13, scale=2.0)
    logits[3, 5 % V] = float("-inf"); logits[4, 2 % V] = float("nan")
    temps = torch.tensor([0.8, 1.0, 0.3, 1.5] * 6)
    rngs = [P.Rng(100 + i) for i in range(rows)]
    for trial in range(6):
        u = torch.tensor([r.next_f32() for r in rngs])
        out = torch.empty(rows, dtype=torch.int32, device=DEV)
        k.sample_temperature(logits, temps.to(DEV), u.to(DEV), out)
        for i in range(rows):
            class Fixed:                      # hands the plain sampler the same uniform
                def next_f32(self, v=float(u[i])): return v
            want = P.sample(logits[i].cpu().numpy(), float(temps[i]), Fixed())
            got = out[i].item()
            if got == want:
                continue
            # The plain sampler sums V weights one after another in float32 (as the
            # reference does); its running sum carries a relative error of up to
            # ~V * 2^-24.  A different answer is right if the exact (float64) running
            # sum around it brackets u * total within that uncertainty.
            l = np.where(np.isfinite(logits[i].cpu().numpy()), logits[i].cpu().numpy(), -np.inf).astype(np.float64)
            w = np.exp((l - l.max()) / float(temps[i]))
            pre = np.cumsum(w) / w.sum()
            slack = max(V * 2.0 ** -24, 1e-6)
            lo = pre[got - 1] if got > 0 else 0.0
            assert lo <= float(u[i]) + slack and pre[got] >= float(u[i]) - slack and w[got] > 0, \
                f"row {i} trial {trial}: {got} vs {want}"
            assert abs(got - want) < 64


def _kept_candidates(logits, temperature, top_k, top_p, min_p):
    """The reference's candidate set in float64: tokens by descending logit (ties: lower index),
    the top-k head of it, min-p's head of that, top-p's head of that; with their weights."""
    n = logits.shape[0]
    v = np.where(np.isfinite(logits), logits, -np.inf).astype(np.float64)
    order = np.lexsort((np.arange(n), -v))
    if 0 < top_k < n:
        order = order[:top_k]
    w = np.exp((v[order] - v[order[0]]) / temperature)
    total, limit = w.sum(), len(order)
    if min_p > 0:
        below = np.nonzero(w < min_p * w[0])[0]
        limit = max(int(below[0]) if below.size else len(order), 1)
    cutoff = limit
    if top_p < 1.0:
        over = np.nonzero(np.cumsum(w[:limit]) > top_p * total)[0]
        cutoff = int(over[0]) + 1 if over.size else limit
    return order[:cutoff], w[:cutoff]


@pytest.mark.parametrize("V", [5000, 128256])
def test_candidate_sampling_at_real_vocabularies_follows_the_plain_sampler(V):
    """Top-k, top-p and min-p in every combination the options allow, at vocabularies far larger
    than a thread block: the same generator seeds as the plain sampler, the same tokens.  Where
    they differ, the uniform number must lie within float rounding of the boundary between the
    two tokens' shares (the kernels add in another order than the reference's float32 loop)."""
    from rustyllm_b200.sampling.config import SamplerConfig
    from rustyllm_b200.sampling.sampler import Sampler, SequenceSamplingState
    options = [dict(top_k=2), dict(top_k=40), dict(top_k=1024), dict(top_k=40, top_p=0.9), dict(top_k=40, min_p=0.05),
               dict(top_k=1024, top_p=0.95, min_p=0.001), dict(top_p=0.9), dict(top_p=0.5, min_p=0.02), dict(top_p=0.99),
               dict(top_p=0.9, top_k=40, repeat_penalty=1.1), dict(top_p=0.3), dict(top_p=0.999, min_p=0.0001)]
    temps = [0.8, 1.3, 0.7]
    rows = len(options)
    g = torch.Generator().manual_seed(V)
    base = torch.randn(rows, V, generator=g) * 3.0
    base[1, 7] = float("-inf"); base[6, 11] = float("nan"); base[2, 100] = base[2, 200] = base[2].max() + 1.0   # a tie at the top
    recent = torch.randint(0, V, (30,), generator=g).tolist()
    configs = [SamplerConfig(temperature=temps[i % 3], **o) for i, o in enumerate(options)]
    sampler = Sampler(torch.device(DEV))
    states = [SequenceSamplingState(c, 500 + i, recent) for i, c in enumerate(configs)]
    twins = [P.Rng(500 + i) for i in range(rows)]
    differed = 0
    for trial in range(8):
        got = sampler.sample(base.clone().to(DEV), states)
        for i, c in enumerate(configs):
            u = twins[i].next_f32()

            class Fixed:
                def next_f32(self, v=u): return v
            lg = base[i].numpy().copy()
            want = P.sample(lg, c.temperature, Fixed(), c.top_k, c.top_p, c.min_p, c.repeat_penalty, recent=recent[-64:])
            if got[i] == want:
                continue
            differed += 1
            P.apply_repeat_penalty(lg, recent[-64:], c.repeat_penalty)
            kept, w = _kept_candidates(lg, c.temperature, c.top_k, c.top_p, c.min_p)
            where = np.nonzero(kept == got[i])[0]
            assert where.size == 1, f"options {options[i]} trial {trial}: token {got[i]} is not among the {len(kept)} kept (plain: {want})"
            j = int(where[0])
            pre = np.cumsum(w) / w.sum()
            slack = max(len(kept) * 2.0 ** -24, 1e-6)
            assert (pre[j - 1] if j else 0.0) <= u + slack and pre[j] >= u - slack, \
                f"options {options[i]} trial {trial}: {got[i]} (place {j}) vs {want}, u = {u}"
    assert differed <= 4, f"{differed} of {8 * rows} draws differ from the plain sampler"



@pytest.mark.parametrize("V", [5000, 128256])
def test_candidate_sampling_with_thousands_of_equal_logits(V):
    """Rows whose boundary classes are large: all logits equal, logits rounded to halves (classes of
    thousands of identical keys), two values in turn, a few thousand equal finite logits among
    -inf.  The selection then refines a class down to all 32 bits and tells its tokens apart by
    index; the answers follow the plain sampler as in the test above."""
    from rustyllm_b200.sampling.config import SamplerConfig
    from rustyllm_b200.sampling.sampler import Sampler, SequenceSamplingState
    g = torch.Generator().manual_seed(V + 1)
    flat = torch.zeros(V)
    halves = (torch.randn(V, generator=g) * 3.0 * 2).round() / 2
    two = torch.where(torch.arange(V) % 2 == 0, torch.tensor(1.0), torch.tensor(0.5))
    few = torch.full((V,), float("-inf")); few[torch.randperm(V, generator=g)[:3000]] = 2.0
    dists = [flat, halves, two, few]
    options = [dict(top_k=40), dict(top_k=1024, top_p=0.9), dict(top_p=0.9), dict(top_p=0.5, min_p=0.5), dict(top_k=2)]
    rows = [(d, o) for d in dists for o in options]
    base = torch.stack([d for d, _ in rows])
    configs = [SamplerConfig(temperature=0.9, **o) for _, o in rows]
    sampler = Sampler(torch.device(DEV))
    states = [SequenceSamplingState(c, 900 + i, []) for i, c in enumerate(configs)]
    twins = [P.Rng(900 + i) for i in range(len(rows))]
    for trial in range(6):
        got = sampler.sample(base.clone().to(DEV), states)
        for i, c in enumerate(configs):
            u = twins[i].next_f32()

            class Fixed:
                def next_f32(self, v=u): return v
            lg = base[i].numpy().copy()
            want = P.sample(lg, c.temperature, Fixed(), c.top_k, c.top_p, c.min_p, c.repeat_penalty, recent=[])
            if got[i] == want:
                continue
            kept, w = _kept_candidates(lg, c.temperature, c.top_k, c.top_p, c.min_p)
            where = np.nonzero(kept == got[i])[0]
            assert where.size == 1, f"row {i} {rows[i][1]} trial {trial}: token {got[i]} is not among the {len(kept)} kept (plain: {want})"
            j = int(where[0])
            pre = np.cumsum(w) / w.sum()
            slack = max(len(kept) * 2.0 ** -24, 1e-6)
            assert (pre[j - 1] if j else 0.0) <= u + slack and pre[j] >= u - slack, \
                f"row {i} {rows[i][1]} trial {trial}: {got[i]} (place {j}) vs {want}, u = {u}"


@pytest.mark.parametrize("rows", [5, 30, 60, 90])
def test_top_k_rows_in_clusters_of_every_size(rows):
    """The top-k kernel gives a row of a large vocabulary to a cluster of 8, 4 or 2 CTAs or to one
    CTA, by the number of rows of the call; the temperature and argmax kernels likewise.  Every
    row of every such call against the plain sampler."""
    from rustyllm_b200.sampling.config import SamplerConfig
    from rustyllm_b200.sampling.sampler import Sampler, SequenceSamplingState
    V = 20000
    g = torch.Generator().manual_seed(rows)
    base = torch.randn(rows, V, generator=g) * 3.0
    kinds = [dict(top_k=40, top_p=0.9), dict(), dict(temperature=0.0), dict(top_k=7, min_p=0.05)]
    configs = [SamplerConfig(**{"temperature": 0.8, **kinds[i % 4]}) for i in range(rows)]
    sampler = Sampler(torch.device(DEV))
    states = [SequenceSamplingState(c, 70 + i, []) for i, c in enumerate(configs)]
    twins = [P.Rng(70 + i) for i in range(rows)]
    differed = 0
    for trial in range(2):
        got = sampler.sample(base.clone().to(DEV), states)
        for i, c in enumerate(configs):
            if c.is_greedy:
                assert got[i] == int(base[i].argmax())
                continue
            u = twins[i].next_f32()

            class Fixed:
                def next_f32(self, v=u): return v
            lg = base[i].numpy().copy()
            want = P.sample(lg, c.temperature, Fixed(), c.top_k, c.top_p, c.min_p, c.repeat_penalty, recent=[])
            if got[i] == want:
                continue
            differed += 1
            if c.top_k > 0:
                kept, w = _kept_candidates(lg, c.temperature, c.top_k, c.top_p, c.min_p)
            else:                     # the whole vocabulary in index order, as the reference walks it
                kept = np.arange(V)
                w = np.exp((lg.astype(np.float64) - lg.max()) / c.temperature)
            where = np.nonzero(kept == got[i])[0]
            assert where.size == 1, f"row {i} {kinds[i % 4]}: token {got[i]} is not among the {len(kept)} kept (plain: {want})"
            j = int(where[0])
            pre = np.cumsum(w) / w.sum()
            slack = max(len(kept) * 2.0 ** -24, 1e-6)
            assert (pre[j - 1] if j else 0.0) <= u + slack and pre[j] >= u - slack, f"row {i}: {got[i]} vs {want}, u = {u}"
    assert differed <= max(2, rows // 10)


def test_a_rows_draw_does_not_depend_on_how_many_rows_the_call_has():
    """The temperature kernel gives a row 8, 4, 2 or 1 CTAs by the number of rows of the call and
    sums the row in the same eight parts either way: the same logits and the same uniform number
    give the same token in calls of 1, 12, 40 and 80 rows, bit for bit the same sums."""
    k = K()
    V = 128256
    g = torch.Generator().manual_seed(11)
    row = (torch.randn(V, generator=g) * 3.0).to(DEV)
    answers = []
    for u in (0.013, 0.37, 0.5, 0.93, 0.999999):
        per_call = []
        for rows in (1, 12, 40, 80):
            logits = row.repeat(rows, 1).contiguous()
            out = torch.empty(rows, dtype=torch.int32, device=DEV)
            k.sample_temperature(logits, torch.full((rows,), 0.8, device=DEV), torch.full((rows,), u, device=DEV), out)
            assert (out == out[0]).all()
            per_call.append(int(out[0]))
        assert len(set(per_call)) == 1, f"u = {u}: {per_call}"
        answers.append(per_call[0])
    assert len(set(answers)) > 2


def test_temperature_zero_rows_are_greedy_and_min_p_cuts():
    k = K()
    logits = torch.tensor([[1.0, 5.0, 2.0, 4.9], [10.0, 9.5, 3.0, 1.0]], device=DEV)
    out = torch.empty(2, dtype=torch.int32, device=DEV)
    for u in (0.0, 0.5, 0.999):
        k.sample_temperature(logits, torch.tensor([0.0, 1.0], device=DEV), torch.tensor([u, u], device=DEV), out,
                             torch.tensor([0.0, 0.3], device=DEV))
        assert out[0].item() == 1 and out[1].item() in (0, 1)
    k.sample_temperature(logits, torch.tensor([1.0, 1.0], device=DEV), torch.tensor([0.999999, 0.999999], device=DEV), out,
                         torch.tensor([0.0, 0.3], device=DEV))
    assert out[1].item() == 1      # the tail (tokens 2, 3) is cut: the last kept candidate


def test_repeat_penalty_kernel():
    k = K()
    logits = torch.tensor([[4.0, -4.0, 2.0, float("nan")], [1.0, 2.0, 3.0, 4.0]], device=DEV)
    recent = torch.zeros(2, 64, dtype=torch.int32, device=DEV)
    recent[0, :4] = torch.tensor([0, 1, 3, 99]); recent[1, :3] = torch.tensor([2, 2, 0])
    k.repeat_penalty(logits, recent, torch.tensor([4, 3], dtype=torch.int32, device=DEV), 2.0)
    assert logits[0, :3].tolist() == [2.0, -8.0, 2.0] and logits[0, 3].item() == float("-inf")
    assert logits[1].tolist() == [0.5, 2.0, 0.75, 4.0]      # token 2 twice: divided twice


def test_sampler_object_runs_the_reference_cases():
    from rustyllm_b200.sampling.config import SamplerConfig
    from rustyllm_b200.sampling.sampler import Sampler, SequenceSamplingState
    s = Sampler(torch.device(DEV))
    for name, opt, seed, draws, logits, recent, allowed, must in CASES:
        st = SequenceSamplingState(SamplerConfig(**opt), seed, recent)
        seen = set()
        for _ in range(draws):
            t = s.sample(torch.tensor([logits], device=DEV), [st])[0]
            assert t in allowed, name
            seen.add(t)
        assert must <= seen, name


def test_kernels_refuse_what_they_cannot_do():
    k = K()
    with pytest.raises(k.KernelError, match="CUDA tensors only"):
        k.swiglu(torch.zeros(2, 4), torch.zeros(2, 2))
    q = torch.zeros(1, 2 * 1100, device=DEV)      # the any-shape kernel takes heads of up to 1,024
    with pytest.raises(k.KernelError, match="head_dim"):
        k.attention_simt(q, torch.zeros(1, 2, PAGE, 1100, device=DEV), torch.zeros(1, 2, PAGE, 1100, device=DEV),
                         torch.zeros(1, 1, dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV),
                         torch.zeros(1, dtype=torch.int32, device=DEV), torch.zeros(1, 2200, device=DEV), 2, 2, 1100, 1.0)
    with pytest.raises(k.KernelError, match="not handled"):
        k.swiglu(torch.zeros(2, 4, dtype=torch.float16, device=DEV), torch.zeros(2, 2, dtype=torch.float16, device=DEV))


@pytest.mark.parametrize("H,G,hd", [(32, 8, 64), (70, 5, 64), (24, 6, 32), (32, 8, 128)])
def test_rope_of_many_tokens_gives_the_bits_of_few(H, G, hd):
    """As many tokens as make a CTA take up to 64 heads (head sizes up to 64; 80 heads are two such CTAs), against the same tokens a
    hundred at a time, whose CTAs take sixteen heads each: rows, keys and values bit for bit."""
    k = K()
    M, P_ = 1300, 1300 // 64 + 1
    qkv = _rand(M, (H + 2 * G) * hd, dtype=torch.bfloat16, seed=1)
    inv = torch.tensor([500000.0 ** (-2.0 * i / hd) for i in range(hd // 2)], dtype=torch.float32, device=DEV)
    pos = torch.arange(M, dtype=torch.int32, device=DEV)
    slot = torch.zeros(M, dtype=torch.int32, device=DEV)
    table = torch.randperm(P_, generator=torch.Generator().manual_seed(2)).to(torch.int32).to(DEV).view(1, P_)
    got = []
    for step in (M, 100):
        x, kp = qkv.clone(), torch.zeros(P_, G, 64, hd, dtype=torch.bfloat16, device=DEV)
        vp = torch.zeros_like(kp)
        for m in range(0, M, step):
            s = slice(m, min(M, m + step))
            k.rope_kv_write(x[s], pos[s], slot[s], table, inv, H, G, hd, hd, False, kp, vp)
        got.append((x, kp, vp))
    for a, b in zip(*got):
        assert torch.equal(a, b)
    assert got[0][1].abs().sum() > 0 and not torch.equal(got[0][0], qkv)


# ----------------------------------------------------------------------------- token tiles of equal height
@pytest.mark.parametrize("M", [65, 79, 81, 129, 143, 145, 256, 257, 271, 289, 293, 513, 530, 769])
@pytest.mark.parametrize("splits", [1, 2, 4])
def test_gemm_tc_token_tiles_of_every_height(M, splits):
    """Numbers of tokens whose equal tiles are and are not multiples of 16 and of 32 (the epilogue's halves), as clusters, and in one part
    (the persistent kernel, which cuts fewer tiles than SMs into narrow ones of 64 tokens; its tiles of full height: the next test), in
    every form of output; rows behind the last stay as they are.  Tolerances as above: K = 520 float sums,
    one rounding to bf16."""
    k = K()
    N, K_ = 390, 520
    a, w, bias = _rand(M, K_, dtype=torch.bfloat16, seed=1), _rand(N, K_, dtype=torch.bfloat16, seed=2), _rand(N, seed=3)
    ref = a.double() @ w.double().T
    f32 = dict(rtol=1e-4, atol=8e-5 * math.sqrt(K_))
    res = _rand(M + 5, N, seed=4)
    out = res.clone()
    k.gemm_tc(a, w, out[:M], k.OUT_ADD_F32, bias, force_splits=splits)
    torch.testing.assert_close(out[:M].double(), ref + bias.double() + res[:M].double(), **f32)
    assert torch.equal(out[M:], res[M:])
    out = res.clone()
    k.gemm_tc(a, w, out[:M], k.OUT_F32, force_splits=splits)
    torch.testing.assert_close(out[:M].double(), ref, **f32)
    assert torch.equal(out[M:], res[M:])
    same = res.to(torch.bfloat16)
    k.gemm_tc(a, w, same[:M], k.OUT_SAME, force_splits=splits)
    torch.testing.assert_close(same[:M].double(), ref, rtol=1e-2, atol=1e-2 * math.sqrt(K_))
    assert torch.equal(same[M:], res[M:].to(torch.bfloat16))
    act = res[:, :N // 2].to(torch.bfloat16).contiguous()
    k.gemm_tc(a, w * 0.05, act[:M], k.OUT_SWIGLU, force_splits=splits)
    small = a.double() @ (w * 0.05).double().T
    torch.testing.assert_close(act[:M].double(), torch.nn.functional.silu(small[:, 0::2]) * small[:, 1::2], rtol=2e-2, atol=2e-2)
    assert torch.equal(act[M:], res[M:, :N // 2].to(torch.bfloat16))
    k.check_device_errors()


@pytest.mark.parametrize("M", [65, 79, 100, 128, 129, 145, 257, 271, 293, 320, 530, 769, 1000])
def test_gemm_tc_persistent_tiles_of_full_height(M):
    """149 weight tiles, so that on 148 SMs every token tile has a wave of its full height (80 to 256 tokens: the epilogue's halves are 64 + 16,
    96 + 48, 96 + 64, 96 + 96, 128 + 80, 128 + 128; the last token tile and the last weight tile are ragged) and narrow tiles follow it: every form
    of output; rows behind the last stay as they are.  K = 72 float sums, one rounding to bf16."""
    k = K()
    N, K_ = 148 * 128 + 66, 72
    a, w, bias = _rand(M, K_, dtype=torch.bfloat16, seed=1), _rand(N, K_, dtype=torch.bfloat16, seed=2), _rand(N, seed=3)
    ref = a.double() @ w.double().T
    f32 = dict(rtol=1e-4, atol=8e-5 * math.sqrt(K_))
    res = _rand(M + 5, N, seed=4)
    out = res.clone()
    k.gemm_tc(a, w, out[:M], k.OUT_ADD_F32, bias)
    torch.testing.assert_close(out[:M].double(), ref + bias.double() + res[:M].double(), **f32)
    assert torch.equal(out[M:], res[M:])
    out = res.clone()
    k.gemm_tc(a, w, out[:M], k.OUT_F32)
    torch.testing.assert_close(out[:M].double(), ref, **f32)
    assert torch.equal(out[M:], res[M:])
    same = res.to(torch.bfloat16)
    k.gemm_tc(a, w, same[:M], k.OUT_SAME, bias)
    torch.testing.assert_close(same[:M].double(), ref + bias.double(), rtol=1e-2, atol=1e-2 * math.sqrt(K_))
    assert torch.equal(same[M:], res[M:].to(torch.bfloat16))
    act = res[:, :N // 2].to(torch.bfloat16).contiguous()
    k.gemm_tc(a, w * 0.15, act[:M], k.OUT_SWIGLU)
    small = a.double() @ (w * 0.15).double().T
    torch.testing.assert_close(act[:M].double(), torch.nn.functional.silu(small[:, 0::2]) * small[:, 1::2], rtol=2e-2, atol=2e-2)
    assert torch.equal(act[M:], res[M:, :N // 2].to(torch.bfloat16))
    k.check_device_errors()


@pytest.mark.parametrize("M,N,K_,by_pairs", [(129, 150 * 128 + 2, 8, ""), (300, 75 * 256 - 130, 1032, ""), (301, 75 * 256 - 136, 264, "as"), (256, 75 * 256, 640, "as"),
                                             (777, 26 * 256 + 8, 2056, "afsg"), (1025, 2303, 8200, "afs"), (300, 75 * 256 - 130, 2056, "afsg"),
                                             (301, 74 * 256 + 64, 1024, "afs"), (301, 74 * 256 + 72, 2184, "afsg"), (129, 75 * 256, 8, "as"), (2000, 2048, 520, ""),
                                             (20000, 248, 520, "as"), (20000, 128, 2048, ""), (20000, 128, 520, "as"), (5200, 640, 2048, "")])
def test_gemm_tc_pairs_rings_and_edges(M, N, K_, by_pairs):
    """More tiles of 256 x 256 than pairs of SMs, or more than three fifths and a long K, so pairs of CTAs take them (``by_pairs``: additions into the
    residual, float, bf16 and gated outputs; the others and those of short K or of more waves by pairs than by CTAs alone go there): a K shorter
    than a block, rings that go round several times with a ragged last block, weight tiles whose second CTA has no rows or some, narrow tiles of the last wave;
    outputs stored by the copy engine (rows of whole 16-byte pieces) that end inside its pieces of 32 x 32, and by the warps.  Float sums of K
    products; rows behind the last stay as they are."""
    k = K()
    assert k.gemm_tc_splits(M, N, K_) == 1
    a, w, bias = _rand(M, K_, dtype=torch.bfloat16, seed=1), _rand(N, K_, dtype=torch.bfloat16, seed=2), _rand(N, seed=3)
    ref = a.double() @ w.double().T
    res = _rand(M + 3, N, seed=4)
    f32 = dict(rtol=1e-4, atol=8e-5 * math.sqrt(K_))
    act = _rand(M + 3, N // 2, dtype=torch.bfloat16, seed=5)
    outs = {"a": (k.OUT_ADD_F32, res), "f": (k.OUT_F32, res), "s": (k.OUT_SAME, res.to(torch.bfloat16)), "g": (k.OUT_SWIGLU, act)}
    assert "".join(c for c, (mode, o) in outs.items() if (c != "g" or N % 2 == 0) and k.gemm_tc_by_pairs(o, mode, M, N, K_)) == by_pairs
    for b in (None, bias):
        full = ref + (b.double() if b is not None else 0.0)
        out, again, flt, same = res.clone(), res.clone(), res.clone(), res.to(torch.bfloat16)
        k.gemm_tc(a, w, out[:M], k.OUT_ADD_F32, b)
        torch.testing.assert_close(out[:M].double(), full + res[:M].double(), **f32)
        k.gemm_tc(a, w, again[:M], k.OUT_ADD_F32, b)
        assert torch.equal(out, again)
        k.gemm_tc(a, w, flt[:M], k.OUT_F32, b)
        torch.testing.assert_close(flt[:M].double(), full, **f32)
        k.gemm_tc(a, w, same[:M], k.OUT_SAME, b)
        torch.testing.assert_close(same[:M].double(), full, rtol=1e-2, atol=1e-2 * math.sqrt(K_))
        assert torch.equal(out[M:], res[M:]) and torch.equal(flt[M:], res[M:]) and torch.equal(same[M:], res[M:].to(torch.bfloat16))
    if N % 2 == 0:
        scale = 2.0 ** -round(math.log2(math.sqrt(K_)))            # gates of about 1; a power of two: the weights stay bf16
        gated = act.clone()
        k.gemm_tc(a, w * scale, gated[:M], k.OUT_SWIGLU)
        small = ref * scale
        torch.testing.assert_close(gated[:M].double(), torch.nn.functional.silu(small[:, 0::2]) * small[:, 1::2], rtol=2e-2, atol=2e-2)
        assert torch.equal(gated[M:], act[M:])
    k.check_device_errors()


@pytest.mark.parametrize("M,N,K_,pad", [(300, 75 * 256 - 130, 520, 2), (300, 75 * 256 - 130, 2056, 1), (1025, 2303, 8200, 1), (129, 2048, 64, 0)])
def test_gemm_tc_additions_into_the_residual_keep_subnormal_numbers(M, N, K_, pad):
    """By pairs (added by the copy engine, and by the warps where rows are no whole 16-byte pieces) and by CTAs alone: residuals below the smallest
    normal float, products that are, and normal ones whose sum is.  A product is one number, so each sum rounds once: the float nearest to
    it, bit for bit."""
    k = K()
    tiny = torch.finfo(torch.float32).tiny
    a, w = torch.zeros(M, K_, device=DEV, dtype=torch.bfloat16), torch.zeros(N, K_, device=DEV, dtype=torch.bfloat16)
    w[:, 0] = (-16.0 * tiny * (1 + torch.arange(N) % 4)).to(DEV)
    a[:, 0] = torch.tensor([0.0, 2.0 ** -4, 2.0 ** -9])[torch.arange(M) % 3].to(DEV)         # nothing, a normal and a subnormal number to add
    small = torch.randint(1, 1 << 22, (M, N + pad), dtype=torch.int32).view(torch.float32)    # bit patterns of subnormal numbers
    res = torch.where(torch.rand(M, N + pad) < 0.5, small, 2.5 * tiny * torch.rand(M, N + pad)).to(DEV)
    out = res.clone()
    assert k.gemm_tc_by_pairs(out[:, :N], k.OUT_ADD_F32, M, N, K_) == (M != 129)
    k.gemm_tc(a, w, out[:, :N], k.OUT_ADD_F32)
    ref = (res[:, :N].double() + a[:, :1].double() * w[:, 0].double()).float()
    k.check_device_errors()
    assert ((ref != 0) & (ref.abs() < tiny)).any()
    assert torch.equal(out[:, :N], ref) and torch.equal(out[:, N:], res[:, N:])


@pytest.mark.parametrize("M,H,N,K_,gap", [(65, 3, 40, 64, 8), (129, 16, 512, 128, 64), (300, 5, 130, 192, 0), (1000, 2, 128, 512, 24)])
def test_gemm_tc_heads_is_a_product_a_head(M, H, N, K_, gap):
    """Heads that lie apart in wider rows on both sides; what lies between them stays as it is.  Float sums, one rounding to bf16."""
    k = K()
    x = _rand(M, H * (K_ + gap), dtype=torch.bfloat16, seed=1)
    w = _rand(H, N, K_, dtype=torch.bfloat16, seed=2)
    old = _rand(M, H * (N + 6), dtype=torch.bfloat16, seed=3)
    out = old.clone()
    assert k.gemm_tc_heads_supported(x, w, K_ + gap)
    k.gemm_tc_heads(x, K_ + gap, w, out, N + 6)
    got, was = out.view(M, H, N + 6), old.view(M, H, N + 6)
    ref = torch.einsum("mhk,hnk->mhn", x.view(M, H, K_ + gap)[:, :, :K_].double(), w.double())
    torch.testing.assert_close(got[:, :, :N].double(), ref, rtol=1e-2, atol=1e-3 * math.sqrt(K_))
    assert torch.equal(got[:, :, N:], was[:, :, N:])
    assert not k.gemm_tc_heads_supported(x, w[:, :, :K_ - 8].contiguous(), K_ + gap)      # a block of K would reach into the next head
    k.check_device_errors()


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("window", [0, 100])
@pytest.mark.parametrize("lens", [[1], [16, 17], [64], [128], [129], [192], [193], [1, 128, 129, 700], [191, 5, 257, 193]])
def test_attention_decode_clusters_with_short_sequences(hd, window, lens):
    """Sequences about the length up to which the first CTA of a cluster takes a sequence whole, alone and beside long ones, against chunks
    combined through global memory (the softmax's sums in another order: bf16 rounding)."""
    k = K()
    H, G, B = 8, 2, len(lens)
    pools = torch.randn(2, 16 * B, G, 64, hd, device=DEV).to(torch.bfloat16)
    pt = torch.randperm(16 * B).to(torch.int32).view(B, 16).to(DEV)
    q = torch.randn(B, (H + 2 * G) * hd, device=DEV).to(torch.bfloat16)
    slots, kv = torch.arange(B, dtype=torch.int32, device=DEV), torch.tensor(lens, dtype=torch.int32, device=DEV)
    for splits in (2, 4, 8):
        out, ref = (torch.zeros(B, H * hd, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        args = (q, pools[0], pools[1], pt, slots, kv)
        k.attention_decode(*args, out, H, G, hd, hd ** -0.5, window, num_splits=splits, cluster=True)
        k.attention_decode(*args, ref, H, G, hd, hd ** -0.5, window, num_splits=splits)
        torch.testing.assert_close(out.float(), ref.float(), rtol=1e-2, atol=2e-3)


# ----------------------------------------------------------------------------- 32-bit attention by tiles of rows
@pytest.mark.parametrize("H,G,hd", [(4, 4, 64), (8, 2, 64), (15, 3, 64), (16, 1, 64), (3, 3, 128), (6, 1, 128), (28, 2, 128)])
def test_attention_f32_tiles_are_exact_and_do_not_depend_on_the_cut(H, G, hd):
    """Sequences whose ends fall beside the edges of 32-key chunks and 64-key pages, tiles of rows that several sequences share,
    and the same rows as single tokens: the float64 result, and bit for bit the same rows whatever shares their tile."""
    k = K()
    lens = [1, 31, 32, 33, 3, 64, 65, 300]
    q, kp, vp, pt, sot, pos, ref = _attention_case(torch.float32, H, G, hd, lens, lens, seed=H + hd)
    scale = 1.0 / math.sqrt(hd)
    wide = torch.zeros(q.shape[0], H * hd + 4, device=DEV)          # rows of a wider buffer
    wide[:, :H * hd] = q
    out = torch.empty_like(q)
    k.attention_simt(wide[:, :H * hd], kp, vp, pt, sot, pos, out, H, G, hd, scale)
    torch.testing.assert_close(out.double().cpu(), ref, rtol=2e-5, atol=2e-5)
    ends = [sum(lens[:b + 1]) - 1 for b in range(len(lens))]
    for rows in (ends, [ends[-1] - 7], list(range(ends[-2] + 5, ends[-1] - 50))):
        some = torch.empty(len(rows), H * hd, device=DEV)
        k.attention_simt(q[rows].contiguous(), kp, vp, pt, sot[rows].contiguous(), pos[rows].contiguous(), some, H, G, hd, scale,
                         single_tokens=len(rows) < 20)
        assert torch.equal(some, out[rows])
    # what a row may not see cannot reach it: infinities behind position 290 of the longest sequence
    slot = int(sot[-1])
    page, at = int(pt[slot, 290 // PAGE]), 290 % PAGE
    kp[page, :, at:], vp[page, :, at:] = math.inf, math.nan
    again = torch.empty_like(q)
    k.attention_simt(q, kp, vp, pt, sot, pos, again, H, G, hd, scale)
    keep = ends[-1] - (299 - 290)
    assert torch.equal(again[:keep], out[:keep]) and not torch.isfinite(again[keep:]).any()


@pytest.mark.parametrize("H,G,hd", [(8, 8, 64), (48, 8, 64), (72, 8, 64), (8, 8, 128), (48, 8, 128), (72, 8, 128)])
def test_attention_f32_single_tokens_do_not_depend_on_how_many_there_are(H, G, hd):
    """18 sequences of 8 KV heads are fewer CTAs than a B200 has SMs, 19 are more (values then take the place of the keys), three
    times as many put two CTAs on an SM: the float64 result, and the same bits as alone."""
    k = K()
    lens = [1 + 37 * i % 610 for i in range(57)]
    q, kp, vp, pt, sot, pos, ref = _attention_case(torch.float32, H, G, hd, [1] * len(lens), lens, seed=H + hd)
    outs = {}
    for n in (1, 18, 19, 57):
        outs[n] = torch.full((n, H * hd), math.nan, device=DEV)
        k.attention_simt(q[-n:].contiguous(), kp, vp, pt, sot[-n:].contiguous(), pos[-n:].contiguous(), outs[n], H, G, hd,
                         1.0 / math.sqrt(hd), single_tokens=True)
    torch.testing.assert_close(outs[57].double().cpu(), ref, rtol=2e-5, atol=2e-5)
    for n in (1, 18, 19):
        assert torch.equal(outs[n], outs[57][-n:])


@pytest.mark.parametrize("H,G,hd", [(8, 2, 64), (6, 1, 128)])
@pytest.mark.parametrize("options", ["sink", "sinks", "gate", "head gate", "softcap"])
def test_attention_f32_options_follow_the_any_shape_kernel(H, G, hd, options):
    """The same call through the any-shape kernel (a chunked mask longer than every sequence is no mask): both are sums of
    float products, a few units in the last place of values of size 1 apart."""
    k = K()
    lens = [40, 1, 130]
    q, kp, vp, pt, sot, pos, _ = _attention_case(torch.float32, H, G, hd, lens, lens, seed=5)
    M = q.shape[0]
    kw = {"sink": dict(sink=True), "sinks": dict(sinks=_rand(H, seed=1)), "gate": dict(gate=_rand(M, H * hd + 3, seed=2)[:, :H * hd]),
          "head gate": dict(gate=_rand(M, H, seed=3), gate_per_head=True), "softcap": dict(softcap=2.0)}[options]
    out, plain = torch.empty_like(q), torch.empty_like(q)
    k.attention_simt(q, kp, vp, pt, sot, pos, out, H, G, hd, 1.0 / math.sqrt(hd), **kw)
    k.attention_simt(q, kp, vp, pt, sot, pos, plain, H, G, hd, 1.0 / math.sqrt(hd), chunk=1 << 20, **kw)
    torch.testing.assert_close(out, plain, rtol=1e-5, atol=4e-6)


@pytest.mark.parametrize("shifted", [(0, 1), (1, 0), (1, 1)])
def test_attention_f32_pools_that_16_byte_pieces_cannot_fetch(shifted):
    """Contiguous pools that begin 4 bytes behind a 16-byte boundary go to the any-shape kernel, whose loads are single elements."""
    k = K()
    H, G, hd, lens = 8, 2, 64, [40, 1, 130]
    q, kp, vp, pt, sot, pos, ref = _attention_case(torch.float32, H, G, hd, lens, lens, seed=9)
    pools = []
    for x, s in zip((kp, vp), shifted):
        room = torch.zeros(x.numel() + 4, device=DEV)
        pools.append(room[s:s + x.numel()].view(x.shape).copy_(x))
    args = (H, G, hd, q.stride(0), H * hd, q.data_ptr())
    assert k.library().rl_attention_f32_supported(*args, kp.data_ptr(), vp.data_ptr(), q.data_ptr()) == 1
    assert k.library().rl_attention_f32_supported(*args, pools[0].data_ptr(), pools[1].data_ptr(), q.data_ptr()) == 0
    out = torch.empty_like(q)
    k.attention_simt(q, *pools, pt, sot, pos, out, H, G, hd, 1.0 / math.sqrt(hd))
    torch.testing.assert_close(out.double().cpu(), ref, rtol=2e-5, atol=2e-5)


# ----------------------------------------------------------------------------- 32-bit products from bf16 cuts
def _f32_split(k, a, w, bias=None, parts=0):
    out = torch.empty(a.shape[0], w.shape[0], device=DEV)
    k.gemm_f32_split(a, w, out, False, bias, parts)
    return out


def _f32_ordered(k, a, w, bias=None):
    """The sum in the order of k, on the CUDA cores."""
    out = torch.empty(a.shape[0], w.shape[0], device=DEV)
    k._check(k.library().rl_gemm_simt(a.data_ptr(), w.data_ptr(), k._ptr(bias), out.data_ptr(), k.F32, k.OUT_F32, a.shape[0], w.shape[0],
                                      a.shape[1], a.stride(0), w.shape[0], k._stream()), "rl_gemm_simt")
    return out


@pytest.mark.parametrize("M,N,K_", [(1, 1, 4), (17, 256, 256), (33, 384, 516), (65, 256, 256), (127, 300, 260), (128, 128, 64), (129, 129, 1028), (200, 500, 2048),
                                    (300, 257, 8192)])
@pytest.mark.parametrize("parts", [0, 1, 2, 4, 8])
def test_gemm_f32_split_is_as_exact_as_the_ordered_sum(M, N, K_, parts):
    """Error against 64 bits, relative to the result's rms, no larger than that of the sum in the order of k from K = 256 on, where
    the product is taken (both are seen to be 1e-7 to 1e-6; 3e-8 is a rounding of the result itself); bias, strided rows and
    addition into the output.  Shorter sums have fewer roundings to save: up to four units in the last place of a sum of 64 values
    that the tensor core cuts off (4 x 2^-24) against the ordered sum's 64 roundings to nearest (8 x 2^-25 in the mean)."""
    k = K()
    a, w, bias = _rand(M, K_ + 4, seed=1)[:, :K_], _rand(N, K_, seed=2), _rand(N, seed=3)
    a = a * torch.exp(2.0 * _rand(M, K_, seed=6))          # values of very different sizes
    wide = torch.zeros(M, K_ + 4, device=DEV)
    wide[:, :K_] = a
    a = wide[:, :K_]
    ref = a.double() @ w.double().T + bias.double()
    out = _f32_split(k, a, w, bias, parts)
    plain = _f32_ordered(k, a, w, bias)
    rms = ref.square().mean().sqrt()
    err = lambda x: ((x.double() - ref).square().mean().sqrt() / rms).item()
    print(f"split {err(out):.3g}, ordered {err(plain):.3g}")
    assert err(out) <= err(plain) * (1.0 if K_ >= 256 else 1.5) + 3e-8
    res = _rand(M, N + 4, seed=4)[:, :N]
    into = res.clone()
    k.gemm_f32_split(a, w, into, True, bias, parts)
    assert torch.equal(into, res + out)
    again = _f32_split(k, a, w, bias, parts)
    assert torch.equal(again, out)


@pytest.mark.parametrize("M", [20, 40, 64, 65, 200])
def test_gemm_f32_split_of_single_products_and_of_one_sign(M):
    """Sums of one product (a row's only value meets a row's only value), significands of every kind beside those whose cuts are worst, M in
    every token tile.  Bound: 2^-24 left out and one rounding to nearest of 2^-24, where the small terms join h h' (their own sums are cut off
    at 2^-8 of a unit); one percent for the terms' own sizes.  And sums of values of one sign, where errors cannot average out."""
    k = K()
    N, K_ = 300, 256
    hard = torch.tensor([1 + 2.0 ** -7 - 2.0 ** -23, 1 + 2.0 ** -8 - 2.0 ** -23, 1 + 2.0 ** -8, 2 - 2.0 ** -23, 1 + 2.0 ** -16 - 2.0 ** -23,
                         1 + 2.0 ** -8 - 2.0 ** -16 - 2.0 ** -23, 1 + 2.0 ** -9 + 2.0 ** -17 + 2.0 ** -23, -(1 + 2.0 ** -7 - 2.0 ** -23)], device=DEV)
    a, w = torch.zeros(M, K_, device=DEV), torch.zeros(N, K_, device=DEV)
    a[:, 77], w[:, 77] = 1.0 + torch.rand(M, device=DEV, generator=torch.Generator(DEV).manual_seed(1)), _rand(N, seed=2)
    a[:8, 77], w[:8, 77] = hard, hard
    got, ref = _f32_split(k, a, w).double(), torch.outer(a[:, 77].double(), w[:, 77].double())
    worst = ((got - ref) / ref).abs().max().item() * 2.0 ** 23
    print(f"worst {worst:.2f} units of 2^-23, mean {((got - ref) / ref).mean().item() * 2.0 ** 23:.3f}")
    assert worst <= 1.01
    a, w = _rand(M, 2048, seed=3).abs(), _rand(N, 2048, seed=4).abs()
    ref = a.double() @ w.double().T
    err = lambda x: ((x.double() - ref) / ref).square().mean().sqrt().item()
    out, plain = _f32_split(k, a, w), _f32_ordered(k, a, w)
    print(f"one sign: split {err(out):.3g}, ordered {err(plain):.3g}")
    assert err(out) <= err(plain)


def test_gemm_f32_split_keeps_what_is_no_finite_number_and_the_largest_floats():
    k = K()
    M, N, K_ = 70, 256, 256
    a, w = _rand(M, K_, seed=1), _rand(N, K_, seed=2)
    a[3, 5], a[4, 7], a[5, 9] = math.inf, math.nan, 3.4e38
    w[6] *= 0.0
    w[6, 9] = 1.0
    w[8, 5] = 0.0
    out = _f32_split(k, a, w)
    plain = _f32_ordered(k, a, w)
    assert torch.equal(torch.isnan(out), torch.isnan(plain)) and torch.equal(torch.isinf(out), torch.isinf(plain))
    assert out[5, 6] == plain[5, 6] == a[5, 9]
    fine = torch.isfinite(plain)
    torch.testing.assert_close(out[fine], plain[fine], rtol=1e-5, atol=1e-4)


@pytest.mark.parametrize("M", [1, 2, 3, 4, 7, 8])
@pytest.mark.parametrize("I,K_", [(1, 256), (131, 260), (2048, 512), (2401, 1028)])
def test_gemm_f32_few_with_swiglu_has_the_bits_of_product_and_activation(M, I, K_):
    """Two and four weight rows a warp (half of them gates), ends of both, rows of a wider output."""
    k = K()
    a, w, bias = _rand(M, K_, seed=1), _rand(2 * I, K_, seed=2), _rand(2 * I, seed=3)
    for b in (None, bias):
        gu, ref = torch.empty(M, 2 * I, device=DEV), torch.empty(M, I, device=DEV)
        k.gemm_simt(a, w, gu, k.OUT_SAME, b, is_weight=True)
        k.swiglu(gu, ref, interleaved=False)
        wide = _rand(M, I + 3, seed=4)
        out = wide.clone()
        assert k.gemm_f32_few_swiglu_supported(a, w)
        k.gemm_f32_few_swiglu(a, w, out[:, :I], b)
        assert torch.equal(out[:, :I], ref) and torch.equal(out[:, I:], wide[:, I:])
    assert not k.gemm_f32_few_swiglu_supported(_rand(9, K_, seed=5), w)


def test_products_of_many_float_rows_take_the_split_kernel():
    k = K()
    lib = k.library()
    a, w = _rand(100, 512, seed=1), _rand(256, 512, seed=2)
    out = torch.empty(100, 256, device=DEV)
    k.gemm_simt(a, w, out, k.OUT_SAME)
    assert torch.equal(out, _f32_split(k, a, w))
    p = a.data_ptr()
    for bad in ((8, 256, 512, 512), (100, 127, 512, 512), (100, 256, 252, 252), (100, 256, 510, 510), (100, 256, 512, 514)):
        assert not lib.rl_gemm_f32_split_supported(p, w.data_ptr(), *bad)
    assert not lib.rl_gemm_f32_split_supported(p + 4, w.data_ptr(), 100, 256, 512, 512)


@pytest.mark.parametrize("N,K_", [(1, 256), (5, 260), (130, 2048), (4736, 512), (4737, 1028), (257, 8192)])
def test_gemm_f32_few_is_more_exact_than_the_ordered_sum_and_rows_do_not_depend_on_the_batch(N, K_):
    """Every number of rows of the kernel's shapes, rows of a wider buffer, bias, addition into the output; a row's bits are the same in
    every one of them.  Error against 64 bits no larger than that of the sum in the order of k (3e-8: the result's own rounding)."""
    k = K()
    wide = _rand(8, K_ + 8, seed=1)
    w, bias = _rand(N, K_, seed=2), _rand(N, seed=3)
    a = wide[:, 4:4 + K_]
    full = torch.empty(8, N, device=DEV)
    k.gemm_simt(a, w, full, k.OUT_F32, bias)
    ref = a.double() @ w.double().T + bias.double()
    err = lambda x: (x.double() - ref).square().mean().sqrt() / ref.square().mean().sqrt()
    plain = _f32_ordered(k, a, w, bias)
    print(f"few {err(full):.3g}, ordered {err(plain):.3g}")
    assert err(full) <= err(plain) + 3e-8
    for rows in ([7], [0, 6], [3, 4, 5], list(range(5)), list(range(1, 8))):
        some = torch.empty(len(rows), N + 3, device=DEV)[:, :N]
        k.gemm_simt(a[rows].contiguous(), w, some, k.OUT_SAME, bias)
        assert torch.equal(some, full[rows])
    res = _rand(8, N, seed=4)
    into = res.clone()
    k.gemm_simt(a, w, into, k.OUT_ADD_F32, bias)
    assert torch.equal(into, res + full)
    lib = k.library()
    for M, kk, lda in ((0, 256, 256), (9, 256, 256), (4, 252, 256), (4, 258, 260), (4, 256, 258)):
        assert not lib.rl_gemm_f32_few_supported(w.data_ptr(), w.data_ptr(), M, N, kk, lda)


def test_gemm_f32_few_waits_for_a_second_operand_that_was_just_written():
    """An operand that a kernel in front has only begun to write (it lets the next kernel start early) is no weight: the product by the
    default call is the one of what was written.  Operands of 64 MB, so that the writing takes longer than the product's start."""
    k = K()
    N, K_ = 8192, 2048
    a, x, ones = _rand(2, K_, seed=1), _rand(N, K_, seed=2), torch.ones(K_, device=DEV)
    w, out = torch.zeros(N, K_, device=DEV), torch.empty(2, N, device=DEV)
    for i in range(8):
        x.add_(1.0)
        k.rmsnorm(x, ones, w, 1e-5)
        k.gemm_simt(a, w, out, k.OUT_F32)
        torch.cuda.synchronize()
        for is_weight in (False, True):
            again = torch.empty_like(out)
            k.gemm_simt(a, w, again, k.OUT_F32, is_weight=is_weight)
            assert torch.equal(again, out)
        w.zero_()


# ----------------------------------------------------------------------------- linear recurrences by chunks
def _scan_case(dtype, mode, H, hpg, dk, dv, lens, seed, decays=(0.9, 0.5, 0.999, 1.0, 0.0)):
    """Inputs as views of one wide buffer, states that are not zero, and the recurrence in float64 on what the kernel reads."""
    M, G = sum(lens), H // hpg
    g = torch.Generator(device=DEV).manual_seed(seed)
    rand = lambda *s: torch.randn(*s, generator=g, device=DEV)
    buf = rand(M, 2 * G * dk + H * dv + H + 4 - H % 4).to(dtype)
    k, q, v = buf[:, :G * dk], buf[:, G * dk:2 * G * dk], buf[:, 2 * G * dk:2 * G * dk + H * dv]
    dt = buf[:, 2 * G * dk + H * dv:2 * G * dk + H * dv + H]
    dt_bias, skip = rand(H), rand(H)
    rate = torch.tensor(list(decays)[:H] * H, device=DEV)[:H].contiguous() if mode == 0 else rand(H) * 2.0
    slots = list(range(len(lens) - 1, -1, -1))
    state = torch.zeros(len(lens) + 1, 4 * H * dk * dv + 256, dtype=torch.uint8, device=DEV)
    state.view(torch.float32).copy_(rand(len(lens) + 1, H * dk * dv + 64))
    act = mode == 0
    f = lambda x: (torch.nn.functional.silu(x.double()) if act else x.double())
    Q, K_, V = (f(x).view(M, -1, w).repeat_interleave(r, dim=1) for x, w, r in ((q, dk, hpg), (k, dk, hpg), (v, dv, 1)))
    if mode:
        b = torch.nn.functional.softplus(dt.double() + dt_bias.double(), threshold=40.0)
        a = torch.exp(-torch.exp(rate.double()) * b)
    else:
        b, a = torch.ones(M, H, dtype=torch.float64, device=DEV), rate.double().expand(M, H)
    ref, last, at = torch.empty(M, H, dv, dtype=torch.float64, device=DEV), {}, 0
    for s, n in zip(slots, lens):
        S = state[s, :4 * H * dk * dv].view(torch.float32).view(H, dv, dk).transpose(1, 2).double()
        for t in range(at, at + n):
            S = a[t][:, None, None] * S + (b[t][:, None] * K_[t])[:, :, None] * V[t][:, None, :]
            ref[t] = (Q[t][:, None, :] @ S)[:, 0] + (skip.double()[:, None] * V[t] if mode else 0.0)
        last[s] = S.transpose(1, 2)
        at += n
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    kw = dict(dt_raw=dt, dt_bias=dt_bias, skip=skip) if mode else dict(silu=True)
    return (q, k, v), state, cu, torch.tensor(slots, dtype=torch.int32, device=DEV), rate, kw, ref.flatten(1), last


def _scan_walk(k, qkv, state, cu, slots, rate, kw, H, hpg, dk, dv):
    """The walk from token to token, whatever the number of tokens."""
    q, kk, v = qkv
    out = torch.empty(q.shape[0], H * dv, device=DEV)
    sp, ss = k._state_args(state)
    dt = kw.get("dt_raw")
    k._check(k.library().rl_linear_scan(q.data_ptr(), q.stride(0), kk.data_ptr(), kk.stride(0), v.data_ptr(), v.stride(0), k._ptr(dt),
                                        dt.stride(0) if dt is not None else 0, k._dt(q), k._ptr(kw.get("dt_bias")), rate.data_ptr(),
                                        k._ptr(kw.get("skip")), int(dt is not None), int(kw.get("silu", False)), cu.data_ptr(),
                                        slots.data_ptr(), slots.numel(), sp, ss, out.data_ptr(), out.stride(0), H, hpg, dk, dv, 1,
                                        k._stream()), "rl_linear_scan")
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("H,hpg,dk,dv", [(5, 1, 128, 128), (4, 2, 64, 128), (4, 4, 128, 64), (3, 1, 64, 64)])
def test_linear_scan_by_chunks_is_as_exact_as_the_walk(dtype, mode, H, hpg, dk, dv):
    """Sequences that end beside the edges of chunks of 64, from states that are not zero, decays from 1 to 0: outputs and states
    against float64, as exact as the walk's (1e-7 of the rms: sums of up to 128 values in float)."""
    k = K()
    lens = [130, 1, 64, 65, 63, 128, 200]
    qkv, state, cu, slots, rate, kw, ref, last = _scan_case(dtype, mode, H, hpg, dk, dv, lens, seed=dk + dv + mode)
    before = state.clone()
    walked_state = state.clone()
    walk = _scan_walk(k, qkv, walked_state, cu, slots, rate, kw, H, hpg, dk, dv)
    out = torch.empty_like(walk)
    launches = k.launch_count
    k.linear_scan(*qkv, out, state, cu, slots, H, hpg, dk, dv, rate, **kw)
    assert k.launch_count - launches == 3, "the chunked form"
    rel = lambda x, y: ((x.double() - y).square().mean().sqrt() / y.square().mean().sqrt()).item()
    print(f"chunks {rel(out, ref):.3g}, walk {rel(walk, ref):.3g}")
    assert rel(out, ref) <= rel(walk, ref) + 1e-7
    n = 4 * H * dk * dv
    for s, S in last.items():
        got, other = (x[s, :n].view(torch.float32).view(H, dv, dk) for x in (state, walked_state))
        assert rel(got, S) <= rel(other, S) + 1e-7
    assert torch.equal(state[:, n:], before[:, n:]) and torch.equal(state[len(lens)], before[len(lens)])


def test_linear_scan_by_chunks_keeps_later_tokens_out_of_earlier_outputs_and_takes_what_it_can():
    k = K()
    H, dk, dv = 2, 128, 64
    qkv, state, cu, slots, rate, kw, ref, _ = _scan_case(torch.float32, 1, H, 1, dk, dv, [260], seed=3)
    out = torch.empty(260, H * dv, device=DEV)
    first = state.clone()
    k.linear_scan(*qkv, out, first, cu, slots, H, 1, dk, dv, rate, **kw)
    qkv[2][85], qkv[1][100] = math.inf, math.nan
    again = torch.empty_like(out)
    k.linear_scan(*qkv, again, state, cu, slots, H, 1, dk, dv, rate, **kw)
    assert torch.equal(again[:85], out[:85]) and not torch.isfinite(again[85:]).any()
    lib, q = k.library(), qkv[0]
    ask = lambda ptr=q.data_ptr(), ld=128, dt=0, st=0, M=256, B=1, a=128, b=128: lib.rl_linear_scan_chunks(
        ptr, ld, q.data_ptr() & ~15, 128, q.data_ptr() & ~15, 128, dt, st, 128, M, B, 16, a, b)
    ok = q.data_ptr() & ~15
    assert ask(ok) == 5
    for bad in (dict(ptr=ok + 4), dict(ld=126), dict(st=4), dict(M=255), dict(M=319, B=10), dict(a=96), dict(b=32), dict(M=100_000)):
        assert ask(**{"ptr": ok, **bad}) == 0, bad


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 128), (128, 64), (64, 64)])
def test_linear_scan_decays_that_do_not_fade(dtype, dk, dv):
    """Decays below zero and beyond one (and no number) in steps of many tokens, beside heads whose decays fade: the walk's bits, and
    float64 where the recurrence stays small."""
    k = K()
    decays = (-0.5, 0.9, -1.0, 1.01, 40.0, -3.0, math.nan, math.inf)
    H, lens = len(decays), [70, 5, 1, 64, 260, 33]
    qkv, state, cu, slots, rate, kw, ref, last = _scan_case(dtype, 0, H, 1, dk, dv, lens, seed=dk + dv, decays=decays)
    state[2] = 0                     # a fresh sequence: zeros stay zeros whatever the growth in front of its first token
    walked_state, before = state.clone(), state.clone()
    walk = _scan_walk(k, qkv, walked_state, cu, slots, rate, kw, H, 1, dk, dv)
    out = torch.empty_like(walk)
    launches = k.launch_count
    k.linear_scan(*qkv, out, state, cu, slots, H, 1, dk, dv, rate, longest=260, **kw)
    assert k.launch_count - launches == 3, "the chunked form"
    n = 4 * H * dk * dv
    heads = lambda x: x.view(-1, H, dv)
    states = lambda x: x[:, :n].contiguous().view(torch.float32).view(-1, H, dv, dk)
    for h, a in enumerate(decays):
        if a != 0.9:
            for x, y in ((heads(out)[:, h], heads(walk)[:, h]), (states(state)[:, h], states(walked_state)[:, h])):
                assert torch.equal(torch.nan_to_num(x, nan=7e33), torch.nan_to_num(y, nan=7e33)), a
        if abs(a) <= 1.01:
            rows = torch.ones(sum(lens), dtype=torch.bool, device=DEV)
            rows[sum(lens[:3]):sum(lens[:4])] = False        # (the sequence whose state was set to zero: slot 2)
            x, y = heads(out)[rows, h].double(), heads(ref)[rows, h]
            assert ((x - y).square().mean().sqrt() / y.square().mean().sqrt()).item() < 1e-6, a
    assert torch.isfinite(heads(out)[:, :4]).all()
    assert torch.equal(state[:, n:], before[:, n:]) and torch.equal(state[len(lens)], before[len(lens)])


@pytest.mark.parametrize("dtype,H,dk,dv,lens,longest,chunked", [
    (torch.bfloat16, 4, 128, 128, [64] * 4, 64, False), (torch.bfloat16, 2, 128, 128, [100] * 3, 100, False),
    (torch.bfloat16, 4, 128, 128, [33] * 16, 33, False), (torch.bfloat16, 4, 128, 128, [32] * 32, 32, True),
    (torch.bfloat16, 2, 128, 128, [256], 256, True), (torch.bfloat16, 8, 64, 64, [64] * 8, 64, False),
    (torch.bfloat16, 2, 64, 64, [100] * 3, 100, True), (torch.bfloat16, 4, 64, 128, [200, 33, 33, 33], 200, True),
    (torch.bfloat16, 4, 64, 128, [75] * 4, 75, False), (torch.float32, 4, 128, 64, [40] * 8, 40, False),
    (torch.bfloat16, 2, 64, 64, [200, 33, 33], 0, True), (torch.bfloat16, 2, 128, 128, [1] * 300, 1, False)])
def test_linear_scan_takes_chunks_where_there_is_enough_to_do(dtype, H, dk, dv, lens, longest, chunked):
    """Few heads and short sequences keep the walk, whose chain is shorter than three kernels; the result is the same to rounding."""
    k = K()
    qkv, state, cu, slots, rate, kw, ref, _ = _scan_case(dtype, 0, H, 1, dk, dv, lens, seed=11)
    walk = _scan_walk(k, qkv, state.clone(), cu, slots, rate, kw, H, 1, dk, dv)
    out, launches = torch.empty_like(walk), k.launch_count
    k.linear_scan(*qkv, out, state, cu, slots, H, 1, dk, dv, rate, longest=longest, **kw)
    assert k.launch_count - launches == (3 if chunked else 1)
    rel = lambda x: ((x.double() - ref).square().mean().sqrt() / ref.square().mean().sqrt()).item()
    assert rel(out) <= rel(walk) + 1e-7
    if not chunked and len(lens) * 4 <= sum(lens):
        assert torch.equal(out, walk)


def test_linear_scan_walks_where_memory_is_short(monkeypatch):
    """A cache that has left no room for the chunked form's states: the step is walked, as it is below 256 tokens."""
    k = K()
    H, dk, dv = 2, 128, 128
    qkv, state, cu, slots, rate, kw, _, _ = _scan_case(torch.bfloat16, 0, H, 1, dk, dv, [300], seed=12)
    walk = _scan_walk(k, qkv, state.clone(), cu, slots, rate, kw, H, 1, dk, dv)
    out, launches, plain = torch.empty_like(walk), k.launch_count, torch.empty

    def no_room(*size, **options):
        if size and isinstance(size[0], int) and size[0] >= 5 * H * dk * dv:
            raise torch.cuda.OutOfMemoryError("no room")
        return plain(*size, **options)
    monkeypatch.setattr(torch, "empty", no_room)
    k.linear_scan(*qkv, out, state, cu, slots, H, 1, dk, dv, rate, longest=300, **kw)
    monkeypatch.undo()
    assert k.launch_count - launches == 1 and torch.equal(out, walk)
