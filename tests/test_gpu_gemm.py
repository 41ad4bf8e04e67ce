"""GPU tier: tcgen05 GEMM in all operand layouts against fp32 PyTorch, and its invariance."""
import pytest
import torch

from kernel_align_b200.ops import gemm

pytestmark = pytest.mark.gpu


def _rand(dev, *shape, seed=0, scale=1.0):
    g = torch.Generator(device=dev).manual_seed(seed)
    return (torch.randn(*shape, device=dev, generator=g) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("m,n,k", [(256, 256, 64), (300, 520, 136), (1000, 4096, 4096), (4096, 6144, 512)])
def test_gemm_nt(cuda_device, m, n, k):
    a, b = _rand(cuda_device, m, k, seed=1), _rand(cuda_device, n, k, seed=2, scale=0.05)
    c = gemm.gemm_bi(a, b)
    gemm.check_status(cuda_device)
    ref = a.float() @ b.float().t()
    assert (c.float() - ref).abs().max().item() <= 0.02 * ref.abs().max().item() + 1e-3
    c32 = gemm.gemm_bi(a, b, out_dtype=torch.float32)
    assert (c32 - ref).abs().max().item() <= 2e-3 * max(1.0, ref.abs().max().item())
    assert torch.equal(c, c32.to(torch.bfloat16))


@pytest.mark.parametrize("m,n,k", [(256, 256, 128), (520, 264, 1000), (2048, 4096, 4096)])
def test_gemm_transposed_operands(cuda_device, m, n, k):
    a, b = _rand(cuda_device, m, k, seed=3), _rand(cuda_device, n, k, seed=4, scale=0.05)
    ref = gemm.gemm_bi(a, b, out_dtype=torch.float32)
    bt = b.t().contiguous()  # stored [K, N]
    at = a.t().contiguous()  # stored [K, M]
    for kw, (aa, bb) in {"nn": (a, bt), "tn": (at, bt), "tt": (at, b)}.items():
        out = gemm.gemm_bi(aa, bb, trans_a=kw[0] == "t", trans_b=(kw == "nn" or kw == "tn"), out_dtype=torch.float32)
        gemm.check_status(cuda_device)
        assert (out - ref).abs().max().item() <= 2e-3 * max(1.0, ref.abs().max().item()), kw


def test_gemm_bitwise_batch_invariant(cuda_device):
    a, b = _rand(cuda_device, 3000, 1024, seed=5), _rand(cuda_device, 2048, 1024, seed=6, scale=0.05)
    full = gemm.gemm_bi(a, b)
    assert torch.equal(full, gemm.gemm_bi(a, b))
    for lo, hi in ((0, 1), (17, 300), (2048, 3000)):
        assert torch.equal(gemm.gemm_bi(a[lo:hi], b), full[lo:hi])


def test_linear_autograd(cuda_device):
    x = _rand(cuda_device, 4, 96, 512, seed=7).requires_grad_()
    w = _rand(cuda_device, 768, 512, seed=8, scale=0.05).requires_grad_()
    y = gemm.linear(x, w)
    dy = _rand(cuda_device, 4, 96, 768, seed=9)
    y.backward(dy)
    xr, wr = x.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    (xr @ wr.t()).backward(dy.float())
    assert (x.grad.float() - xr.grad).abs().max().item() <= 0.02 * xr.grad.abs().max().item()
    assert (w.grad.float() - wr.grad).abs().max().item() <= 0.02 * wr.grad.abs().max().item()


@pytest.mark.parametrize("m", [1, 8, 16, 17, 33, 64])
@pytest.mark.parametrize("n,k", [(4096, 4096), (1000, 520), (28672, 4096), (4096, 14336), (8, 64), (6144, 200),
                                 (19008, 192), (128256, 256)])
def test_skinny_gemm_equals_tiled_kernel_bitwise(cuda_device, m, n, k, monkeypatch):
    """The weight-streaming kernel for decode-sized batches must give the bits of the tiled
    kernel: otherwise a row's result would depend on the batch size it is computed in."""
    g = torch.Generator(device=cuda_device).manual_seed(m * 7 + n)
    a = torch.randn(80, k, device=cuda_device, generator=g).to(torch.bfloat16)
    w = (torch.randn(n, k, device=cuda_device, generator=g) * 0.05).to(torch.bfloat16)
    tiled = gemm.gemm_bi(a, w)                      # 80 rows: the tiled kernel
    skinny = gemm.gemm_skinny(a[:m], w)
    gemm.check_status(cuda_device)
    assert torch.equal(skinny, tiled[:m])
    ref = a[:m].float() @ w.float().t()
    assert (skinny.float() - ref).abs().max().item() <= 0.02 * ref.abs().max().item() + 1e-3
    # and gemm_bi routes small batches to it
    assert torch.equal(gemm.gemm_bi(a[:m], w), tiled[:m])
    monkeypatch.setenv("KA_GEMM_SKINNY", "0")
    assert torch.equal(gemm.gemm_bi(a[:m], w), tiled[:m])


@pytest.mark.parametrize("m", [3, 30, 64])
@pytest.mark.parametrize("n,k", [(40, 64), (4104, 320), (6144, 576), (19000, 448), (1184, 4160), (40, 72)])
def test_skinny_gemm_boxes_behind_the_last_one(cuda_device, m, n, k):
    """K that is no multiple of a stage, in operands whose rows go on behind K: what lies there (NaN) is not
    multiplied, also where one copy brings several boxes."""
    g = torch.Generator(device=cuda_device).manual_seed(k)
    a = torch.full((80, k + 640), float("nan"), device=cuda_device, dtype=torch.bfloat16)
    w = torch.full((n + 130, k + 640), float("nan"), device=cuda_device, dtype=torch.bfloat16)
    a[:, :k] = torch.randn(80, k, device=cuda_device, generator=g).to(torch.bfloat16)
    w[:n, :k] = (torch.randn(n, k, device=cuda_device, generator=g) * 0.05).to(torch.bfloat16)
    got = gemm.gemm_skinny(a[:m, :k], w[:n, :k])
    gemm.check_status(cuda_device)
    assert torch.equal(got, gemm.gemm_bi(a[:, :k].contiguous(), w[:n, :k].contiguous())[:m])


@pytest.mark.parametrize("n,k", [(8, 64), (136, 200), (1032, 512), (4096, 1024)])
@pytest.mark.parametrize("trans_a,trans_b,dtype", [(False, False, torch.bfloat16), (False, True, torch.bfloat16),
                                                   (True, True, torch.float32)])
def test_narrow_tiles_equal_wide_ones_bitwise(cuda_device, n, k, trans_a, trans_b, dtype):
    """Small products take tiles of 128 columns: a row must not tell which tiles it was computed in.
    The tall product has more tiles than the narrow form accepts."""
    g = torch.Generator(device=cuda_device).manual_seed(n + k)
    tall = 256 * 80
    a = torch.randn(tall, k, device=cuda_device, generator=g).to(torch.bfloat16)
    b = (torch.randn(*((k, n) if trans_b else (n, k)), device=cuda_device, generator=g) * 0.05).to(torch.bfloat16)
    op = (lambda t: t.t().contiguous()) if trans_a else (lambda t: t)
    wide = gemm.gemm_bi(op(a), b, trans_a=trans_a, trans_b=trans_b, out_dtype=dtype)
    for m in (72, 256, 264, 512):
        narrow = gemm.gemm_bi(op(a[:m]), b, trans_a=trans_a, trans_b=trans_b, out_dtype=dtype)
        assert torch.equal(narrow, wide[:m]), m
    gemm.check_status(cuda_device)
