"""GRPO objective: CPU library and CUDA kernels against an autograd PyTorch reference."""
import os
import shutil
import subprocess
import sys

import pytest
import torch

from kernel_align_b200 import _native
from kernel_align_b200.ops.grpo_loss import group_advantages, grpo_loss


def _ref(ln, lo, adv, mask, lr, eps, beta, reduction):
    ratio = (ln - lo).exp()
    a = adv[:, None]
    obj = torch.minimum(ratio * a, ratio.clamp(1 - eps, 1 + eps) * a)
    loss = -obj
    if beta > 0:
        d = lr - ln
        loss = loss + beta * (d.exp() - d - 1)
    m = mask.float()
    if reduction == "token_mean":
        return (loss * m).sum() / m.sum()
    per = (loss * m).sum(1) / m.sum(1).clamp(min=1)
    valid = (m.sum(1) > 0).float()
    return (per * valid).sum() / valid.sum()


def _case(dev, seed=0, g=12, l=70):
    gen = torch.Generator().manual_seed(seed)
    lo = -torch.rand(g, l, generator=gen) * 3
    ln = lo + torch.randn(g, l, generator=gen) * 0.3
    lr = lo + torch.randn(g, l, generator=gen) * 0.2
    rewards = torch.randn(g, generator=gen)
    mask = torch.rand(g, l, generator=gen) > 0.2
    mask[3] = False
    return [t.to(dev) for t in (ln, lo, lr, rewards, mask)]


def _check(dev):
    ln, lo, lr, rewards, mask = _case(dev)
    adv = group_advantages(rewards, 4)
    r = rewards.view(-1, 4)
    want = ((r - r.mean(1, keepdim=True)) / (r.std(1, keepdim=True) + 1e-4)).view(-1)
    assert (adv - want).abs().max().item() < 1e-5
    for reduction in ("token_mean", "seq_mean"):
        for beta in (0.0, 0.04):
            x = ln.clone().requires_grad_()
            loss, stats = grpo_loss(x, lo, adv, mask=mask, logp_ref=lr, eps_low=0.2, beta=beta, reduction=reduction,
                                    return_stats=True)
            (loss * 2.0).backward()
            xr = ln.clone().requires_grad_()
            ref = _ref(xr, lo, adv, mask, lr, 0.2, beta, reduction)
            (ref * 2.0).backward()
            assert abs(loss.item() - ref.item()) < 1e-5, (reduction, beta)
            assert (x.grad - xr.grad).abs().max().item() < 1e-6
            assert stats[2].item() == mask.sum().item()
            again = grpo_loss(ln, lo, adv, mask=mask, logp_ref=lr, beta=beta, reduction=reduction)
            assert again.item() == loss.item()  # bitwise repeatable
            floats = grpo_loss(ln, lo, adv, mask=mask.float(), logp_ref=lr, beta=beta, reduction=reduction)
            assert floats.item() == loss.item()


def test_grpo_loss_cpu():
    _check(torch.device("cpu"))


def test_grpo_loss_follows_its_inputs_and_not_the_default_device():
    ln, lo = torch.randn(4, 8, requires_grad=True), torch.randn(4, 8)
    adv = torch.randn(4)
    want, want_stats = grpo_loss(ln, lo, adv, return_stats=True)
    with torch.device("meta"):
        got, stats = grpo_loss(ln, lo, adv, return_stats=True)
        assert torch.equal(grpo_loss(ln, lo, adv), want)
    assert torch.equal(got, want) and torch.equal(stats, want_stats)


def test_an_installed_package_without_the_module_has_the_loss(tmp_path):
    """A package built without torch carries the two plain libraries and no sources: the operators take them."""
    package = os.path.dirname(_native.__file__)
    shutil.copytree(package, tmp_path / "kernel_align_b200", ignore=shutil.ignore_patterns("__pycache__", "_ka_torch*", "*.hash"))
    code = ("import torch; from kernel_align_b200 import _native; from kernel_align_b200.ops import grpo_loss as g\n"
            "assert _native.torch_ops() is None and _native.cuda().ka_grpo_loss_fwd.argtypes\n"
            "x = torch.randn(2, 3, requires_grad=True); g.grpo_loss(x, x.detach(), torch.ones(2)).backward(); print(x.grad.shape)")
    r = subprocess.run([sys.executable, "-c", code], cwd=tmp_path, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "PYTHONPATH": str(tmp_path)})
    assert r.returncode == 0 and "torch.Size([2, 3])" in r.stdout, r.stderr


@pytest.mark.gpu
def test_grpo_loss_gpu_without_the_module(cuda_device, monkeypatch):
    """The Python node reaches the same kernels: the same bits, and what is refused stays refused."""
    ln, lo, lr, rewards, mask = _case(cuda_device)
    got = []
    for gone in (False, True):
        if gone:
            monkeypatch.setattr(_native, "torch_ops", lambda: None)
        assert (_native.torch_ops() is None) == gone
        x = ln.clone().requires_grad_()
        adv = group_advantages(rewards, 4)
        loss, stats = grpo_loss(x, lo, adv, mask=mask, logp_ref=lr, beta=0.04, return_stats=True)
        got.append([adv, loss.detach(), stats, *torch.autograd.grad(loss, x)])
        for bad in ((x, lo.cpu(), adv), (x[0], lo[0], adv)):
            with pytest.raises((RuntimeError, ValueError)):
                grpo_loss(*bad)
    assert all(torch.equal(a, b) for a, b in zip(*got))
    _check(cuda_device)


@pytest.mark.gpu
def test_grpo_loss_gpu(cuda_device):
    _check(cuda_device)
    # Llama-sized: G=64 sequences of 512 tokens
    gen = torch.Generator(device=cuda_device).manual_seed(1)
    lo = -torch.rand(64, 512, device=cuda_device, generator=gen)
    ln = (lo + torch.randn(64, 512, device=cuda_device, generator=gen) * 0.1).requires_grad_()
    adv = group_advantages(torch.randn(64, device=cuda_device, generator=gen), 64)
    a = grpo_loss(ln, lo, adv)
    b = grpo_loss(ln, lo, adv)
    assert a.item() == b.item()
    a.backward()
    assert torch.isfinite(ln.grad).all()


@pytest.mark.gpu
@pytest.mark.parametrize("dtype,strided,mask_dtype", [(torch.float32, False, torch.bool), (torch.bfloat16, True, torch.int64),
                                                      (torch.float64, True, torch.float32), (torch.float32, True, None)])
def test_grpo_loss_gpu_takes_what_the_cpu_takes(cuda_device, dtype, strided, mask_dtype):
    """Types and strides are brought to fp32 rows on both devices; the gradient has the input's type and shape."""
    ln, lo, lr, rewards, mask = (t.to(dtype) if t.is_floating_point() else t for t in _case(torch.device("cpu")))
    grids = [t.t().contiguous().t() if strided else t for t in (ln, lo, lr)]
    m = None if mask_dtype is None else mask.to(mask_dtype)
    got = []
    for dev in (torch.device("cpu"), cuda_device):
        x, o, r = (t.to(dev) for t in grids)
        x = x.detach().requires_grad_()
        adv = group_advantages(rewards.to(dev).view(3, 4), 4)
        assert adv.shape == (3, 4) and adv.dtype == torch.float32
        loss, stats = grpo_loss(x, o, adv.view(-1), mask=None if m is None else m.to(dev), logp_ref=r, beta=0.04, return_stats=True)
        (g,) = torch.autograd.grad(loss, x, torch.tensor(3.0, device=dev, dtype=torch.float64).to(loss.dtype))
        assert g.dtype == dtype and g.shape == x.shape and not stats.requires_grad
        got.append([loss.detach().cpu(), stats.cpu(), g.float().cpu()])
    for a, b in zip(*got):      # sums of 840 fp32 terms in two orders, exponentials of 2 ulp; gradients rounded to 8 bits
        assert (a - b).abs().max().item() <= (1e-5 if dtype != torch.bfloat16 else 1e-2) * max(1.0, a.abs().max().item())


@pytest.mark.gpu
def test_grpo_loss_gpu_as_an_autograd_node(cuda_device):
    """Hooks on saved tensors see them, transforms that read no memory are refused, nothing is recorded without
    gradients, a second derivative is none, another stream and thread work."""
    import threading

    ln, lo, lr, rewards, mask = _case(cuda_device)
    adv = group_advantages(rewards, 4)
    x = ln.clone().requires_grad_()
    (want,) = torch.autograd.grad(grpo_loss(x, lo, adv, mask=mask), x)
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (packed.append(t.shape), t.cpu())[1], lambda t: t.to(cuda_device)):
        loss = grpo_loss(x, lo, adv, mask=mask)
    assert len(packed) == 2 and torch.equal(torch.autograd.grad(loss, x)[0], want)
    for refused in (lambda: torch.func.vmap(lambda a: grpo_loss(ln, lo, a, mask=mask))(torch.stack([adv, adv])),
                    lambda: torch.func.grad(lambda a: grpo_loss(a, lo, adv, mask=mask))(ln),
                    lambda: torch.func.jvp(lambda a: grpo_loss(a, lo, adv, mask=mask), (ln,), (ln,)),
                    lambda: grpo_loss(x, lo.cpu(), adv), lambda: grpo_loss(x[0], lo[0], adv)):
        with pytest.raises((RuntimeError, ValueError, NotImplementedError)):
            refused()
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(ln.clone(), torch.ones_like(ln))
        with pytest.raises((RuntimeError, NotImplementedError)):
            grpo_loss(dual, lo, adv, mask=mask)
    for mode in (torch.no_grad, torch.inference_mode):
        with mode():
            assert grpo_loss(x, lo, adv, mask=mask).item() == loss.item() and not grpo_loss(x, lo, adv).requires_grad
    (g,) = torch.autograd.grad(grpo_loss(x, lo, adv, mask=mask), x, create_graph=True)
    assert torch.equal(g, want) and not g.requires_grad
    out = {}

    def work():
        s = torch.cuda.Stream(cuda_device)
        with torch.cuda.stream(s):
            y = ln.clone().requires_grad_()
            out["g"] = torch.autograd.grad(grpo_loss(y, lo, adv, mask=mask), y)[0]
        s.synchronize()

    torch.cuda.synchronize(cuda_device)
    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert torch.equal(out["g"], want)
    graph_in = ln.clone()
    grpo_loss(graph_in, lo, adv, mask=mask)
    torch.cuda.synchronize(cuda_device)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = grpo_loss(graph_in, lo, adv, mask=mask)
    graph.replay()
    assert captured.item() == loss.item()
