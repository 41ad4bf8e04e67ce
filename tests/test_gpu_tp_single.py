"""GPU tier, one GPU: the tensor-parallel kernels with world = 1 (local buffers)."""
import pytest
import torch

from kernel_align_b200.ops import gemm
from kernel_align_b200.parallel.tp_gemm import TPContext, all_gather_gemm, gemm_reduce_scatter

pytestmark = pytest.mark.gpu


def test_reduce_scatter_and_all_gather_world1(cuda_device):
    ctx = TPContext(device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(0)
    x = torch.randn(1000, 1024, device=cuda_device, generator=g).to(torch.bfloat16)
    w = (torch.randn(768, 1024, device=cuda_device, generator=g) * 0.03).to(torch.bfloat16)
    r = torch.randn(1000, 768, device=cuda_device, generator=g).to(torch.bfloat16)
    out = gemm_reduce_scatter(x, w, ctx, residual=r)
    out2 = gemm_reduce_scatter(x, w, ctx, residual=r)
    gemm.check_status(cuda_device)
    assert out.shape == (1000, 768) and torch.equal(out, out2)
    ref = (x.float() @ w.float().t()).bfloat16().float() + r.float()
    assert (out.float() - ref).abs().max().item() <= 0.02 * ref.abs().max().item()
    # batch invariance of the sliced reduction
    part = gemm_reduce_scatter(x[100:356], w, ctx, residual=r[100:356])
    assert torch.equal(part, out[100:356])
    xa = x[:896]
    y = all_gather_gemm(xa, w, ctx)
    gemm.check_status(cuda_device)
    assert torch.equal(y, gemm.gemm_bi(xa, w))


def test_reduce_scatter_matches_cpu_rank_emulator(cuda_device):
    from kernel_align_b200.ops import cpu_ops

    ctx = TPContext(device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(4)
    x = torch.randn(200, 512, device=cuda_device, generator=g).to(torch.bfloat16)
    w = (torch.randn(128, 512, device=cuda_device, generator=g) * 0.05).to(torch.bfloat16)
    r = torch.randn(200, 128, device=cuda_device, generator=g).to(torch.bfloat16)
    out = gemm_reduce_scatter(x, w, ctx, residual=r)
    emu = cpu_ops.gemm_sliced_cpu(x.cpu(), w.cpu(), residual=r.cpu(), world=8)
    # same slices, same roundings, same tree; only the order inside a slice's dot product differs
    diff = (out.cpu().float() - emu).abs()
    assert diff.max().item() <= 0.02 * emu.abs().max().item()
    assert (diff > 0).float().mean().item() < 0.2


@pytest.mark.parametrize("m,n,k,trans_b", [(1, 8, 512, False), (300, 264, 512, False), (1000, 768, 1536, True),
                                           (2049, 1032, 1024, False), (1000, 2056, 512, False), (19000, 256, 512, True)])
def test_slices_summed_in_the_kernel_equal_the_staged_ones_bitwise(cuda_device, m, n, k, trans_b, monkeypatch):
    """One rank may sum the eight K slices of a tile where they are computed (in narrow tiles and in wide
    ones); the staged path, which the multi-rank kernels share, defines the bits."""
    from kernel_align_b200.parallel import tp_gemm

    monkeypatch.setattr(tp_gemm, "_split_pays", lambda *a: False)
    ctx = TPContext(device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(m + n)
    x = torch.randn(m, k, device=cuda_device, generator=g).to(torch.bfloat16)
    w = (torch.randn(*((k, n) if trans_b else (n, k)), device=cuda_device, generator=g) * 0.05).to(torch.bfloat16)
    r = torch.randn(m, n, device=cuda_device, generator=g).to(torch.bfloat16)
    outs = []
    for tree in (False, True):
        monkeypatch.setattr(tp_gemm, "_tree_pays", lambda *a, t=tree: t)
        outs += [[gemm_reduce_scatter(x, w, ctx, residual=res, trans_b=trans_b) for res in (None, r)]]
    gemm.check_status(cuda_device)
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])


@pytest.mark.parametrize("m,n,k,trans_b", [(1, 8, 512, False), (127, 264, 1024, True), (300, 1032, 512, False),
                                           (1000, 2056, 512, False), (1000, 4096, 1536, True), (1100, 4104, 512, False)])
def test_slices_as_units_of_their_own_equal_the_kept_and_the_staged_ones_bitwise(cuda_device, m, n, k, trans_b, monkeypatch):
    """The eight K slices as separate units (one round and several) and a sum over their partials: the bits
    of a tile that keeps its slices, and of the staged path, which defines them."""
    from kernel_align_b200.parallel import tp_gemm

    ctx = TPContext(device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(m + n)
    x = torch.randn(m, k, device=cuda_device, generator=g).to(torch.bfloat16)
    w = (torch.randn(*((k, n) if trans_b else (n, k)), device=cuda_device, generator=g) * 0.05).to(torch.bfloat16)
    r = torch.randn(m, n, device=cuda_device, generator=g).to(torch.bfloat16)
    outs = []
    for own, split in ((False, False), (True, False), (True, True)):
        monkeypatch.setattr(tp_gemm, "_tree_pays", lambda *a, o=own: o)
        monkeypatch.setattr(tp_gemm, "_split_pays", lambda *a, s=split: s)
        outs += [[gemm_reduce_scatter(x, w, ctx, residual=res, trans_b=trans_b) for res in (None, r)]]
    gemm.check_status(cuda_device)
    for other in outs[1:]:
        assert torch.equal(outs[0][0], other[0]) and torch.equal(outs[0][1], other[1])
