"""RMSNorm / RoPE / SwiGLU: CPU library vs PyTorch, CUDA kernels vs the CPU library."""
import pytest
import torch
import torch.nn.functional as F

from kernel_align_b200.ops.layer_ops import rmsnorm, rope_, rope_tables, swiglu


def _rms_ref(x, w, eps, res=None):
    xr = x.float() if res is None else (x.float() + res.float()).bfloat16().float()
    n = (xr * torch.rsqrt(xr.pow(2).mean(-1, keepdim=True) + eps)).bfloat16().float()
    return (n * w.float()).bfloat16(), xr.bfloat16()


def _rope_ref(x, pos, cos, sin):
    h = x.shape[-1] // 2
    c, s = cos[pos][:, None, :], sin[pos][:, None, :]
    xf = x.float()
    return torch.cat([xf[..., :h] * c - xf[..., h:] * s, xf[..., h:] * c + xf[..., :h] * s], -1).bfloat16()


def test_cpu_layer_ops_match_pytorch():
    g = torch.Generator().manual_seed(0)
    x = torch.randn(9, 256, generator=g).bfloat16()
    w = torch.randn(256, generator=g).bfloat16()
    r = torch.randn(9, 256, generator=g).bfloat16()
    y = rmsnorm(x, w, 1e-5)
    assert (y.float() - _rms_ref(x, w, 1e-5)[0].float()).abs().max() <= 0.04
    y2, ro = rmsnorm(x, w, 1e-5, r)
    ref, ref_ro = _rms_ref(x, w, 1e-5, r)
    assert torch.equal(ro, ref_ro) and (y2.float() - ref.float()).abs().max() <= 0.04
    assert torch.equal(rmsnorm(x[3:4], w, 1e-5), y[3:4])  # batch invariance
    q = torch.randn(11, 4, 128, generator=g).bfloat16()
    cos, sin = rope_tables(64, 128)
    pos = torch.randint(0, 64, (11,), generator=g)
    want = _rope_ref(q, pos, cos, sin)
    got = rope_(q.clone(), pos, cos, sin)
    assert (got.float() - want.float()).abs().max() <= 0.04
    gu = torch.randn(6, 512, generator=g).bfloat16()
    want = (F.silu(gu[:, :256].float()).bfloat16().float() * gu[:, 256:].float()).bfloat16()
    assert (swiglu(gu).float() - want.float()).abs().max() <= 0.04


@pytest.mark.gpu
def test_gpu_layer_ops_match_cpu_library(cuda_device):
    g = torch.Generator().manual_seed(1)
    x = torch.randn(300, 4096, generator=g).bfloat16()
    w = (torch.randn(4096, generator=g) * 0.1 + 1).bfloat16()
    r = torch.randn(300, 4096, generator=g).bfloat16()
    y_cpu, ro_cpu = rmsnorm(x, w, 1e-5, r)
    y_gpu, ro_gpu = rmsnorm(x.to(cuda_device), w.to(cuda_device), 1e-5, r.to(cuda_device))
    assert torch.equal(ro_gpu.cpu(), ro_cpu)
    assert torch.equal(y_gpu.cpu(), y_cpu)  # same summation order, same rounding points
    y1 = rmsnorm(x.to(cuda_device), w.to(cuda_device), 1e-5)
    assert torch.equal(y1[17:18], rmsnorm(x[17:18].to(cuda_device), w.to(cuda_device), 1e-5))
    assert (y1.cpu().float() - _rms_ref(x, w, 1e-5)[0].float()).abs().max() <= 0.07

    q = torch.randn(512, 32, 128, generator=g).bfloat16()
    cos, sin = rope_tables(512, 128)
    pos = torch.arange(512)
    got = rope_(q.clone().to(cuda_device), pos.to(cuda_device), cos.to(cuda_device), sin.to(cuda_device))
    assert torch.equal(got.cpu(), rope_(q.clone(), pos, cos, sin))
    # strided view: q part of a fused qkv projection
    qkv = torch.randn(64, 48, 128, generator=g).bfloat16().to(cuda_device)
    view = qkv[:, :32]
    want = rope_(view.clone().contiguous(), pos[:64].to(cuda_device), cos.to(cuda_device), sin.to(cuda_device))
    rope_(view, pos[:64].to(cuda_device), cos.to(cuda_device), sin.to(cuda_device))
    assert torch.equal(view, want)

    gu = torch.randn(200, 2 * 14336, generator=g).bfloat16()
    out = swiglu(gu.to(cuda_device)).cpu()
    want = (F.silu(gu[:, :14336].float()).bfloat16().float() * gu[:, 14336:].float()).bfloat16()
    assert (out.float() - want.float()).abs().max() <= 0.07
    sep = swiglu(gu[:, :14336].contiguous().to(cuda_device), gu[:, 14336:].contiguous().to(cuda_device)).cpu()
    assert torch.equal(sep, out)


@pytest.mark.parametrize("dev", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
@pytest.mark.parametrize("tokens,rows,hq,hkv", [(1, 128, 4, 2), (130, 256, 32, 8), (257, 257, 3, 1)])
def test_qkv_rope_equals_slices_and_rope_bitwise(dev, tokens, rows, hq, hkv):
    from kernel_align_b200.ops.layer_ops import qkv_rope_fn, rope_fn, rope_tables

    g = torch.Generator(device=dev).manual_seed(tokens)
    width = (hq + 2 * hkv) * 128
    x = torch.randn(rows, width, device=dev, generator=g).to(torch.bfloat16)
    cos, sin = rope_tables(64, 128, device=dev)
    pos = torch.randint(0, 64, (tokens,), device=dev, generator=g)
    a, b = x.clone().requires_grad_(), x.clone().requires_grad_()
    got = qkv_rope_fn(a, pos, cos, sin, hq, hkv, 128)
    cut = [b[:tokens, lo * 128:hi * 128].reshape(tokens, hi - lo, 128)
           for lo, hi in ((0, hq), (hq, hq + hkv), (hq + hkv, hq + 2 * hkv))]
    want = rope_fn(cut[0], pos, cos, sin), rope_fn(cut[1], pos, cos, sin), cut[2]
    d = [torch.randn(t.shape, device=dev, generator=g).to(torch.bfloat16) for t in want]
    torch.autograd.backward(got, d)
    torch.autograd.backward(want, d)
    assert all(torch.equal(p, q) for p, q in zip(got, want)) and torch.equal(a.grad, b.grad)


@pytest.mark.parametrize("dev", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
@pytest.mark.parametrize("rows,d", [(1, 128), (17, 1024), (300, 4096), (64, 8192)])
def test_rmsnorm_fork_adds_the_two_gradients(dev, rows, d):
    from kernel_align_b200.ops.layer_ops import rmsnorm_fn, rmsnorm_fork_fn

    g = torch.Generator(device=dev).manual_seed(rows)
    x = torch.randn(rows, d, device=dev, generator=g).to(torch.bfloat16)
    w = (torch.randn(d, device=dev, generator=g) * 0.1 + 1).to(torch.bfloat16)
    dy, dr = (torch.randn(rows, d, device=dev, generator=g).to(torch.bfloat16) for _ in range(2))
    grads = []
    for fork in (True, False):
        xi, wi = x.clone().requires_grad_(), w.clone().requires_grad_()
        y, r = rmsnorm_fork_fn(xi, wi) if fork else (rmsnorm_fn(xi, wi), xi.clone())
        assert torch.equal(r, x)
        torch.autograd.backward((y, r), (dy, dr))
        grads.append((y, xi.grad, wi.grad))
    assert all(torch.equal(p, q) for p, q in zip(*grads))
    # only one of the two outputs used
    xi = x.clone().requires_grad_()
    rmsnorm_fork_fn(xi, w)[1].backward(dr)
    assert torch.equal(xi.grad, dr)


@pytest.mark.parametrize("dev", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_decoder_layer_takes_positions_of_the_padded_rows_too(dev):
    from kernel_align_b200.models.llama import DecoderLayer, LlamaConfig
    from kernel_align_b200.parallel.tp_gemm import TPContext

    cfg = LlamaConfig(vocab_size=512, hidden=256, n_layers=1, n_heads=4, n_kv_heads=2, head_dim=128, ffn=512, max_pos=256)
    layer = DecoderLayer(cfg, TPContext(device=torch.device(dev)), 1, torch.device(dev))
    cos, sin = rope_tables(cfg.max_pos, cfg.head_dim, cfg.rope_theta, device=dev)
    x = torch.randn(128, cfg.hidden, generator=torch.Generator().manual_seed(4)).bfloat16().to(dev)
    pos = torch.arange(100, device=dev)
    outs = []
    for p in (pos, torch.cat([pos, pos.new_zeros(28)]), torch.cat([pos, pos.new_zeros(28)]).view(1, 128)):
        xi = x.clone().requires_grad_()
        y = layer(xi, 1, 100, p, cos, sin)
        outs.append((y, torch.autograd.grad(y.float().square().sum(), xi)[0]))
    assert all(torch.equal(a, b) for o in outs[1:] for a, b in zip(o, outs[0]))
    with pytest.raises(ValueError):
        layer(x, 1, 100, pos[:99], cos, sin)


class _OnGpu:
    """A CPU tensor that says it is on a GPU: for rules that only look at shapes, strides and addresses."""

    def __init__(self, t, device="cuda:0"):
        self.t, self.device = t, torch.device(device)

    def __getattr__(self, name):
        return getattr(self.t, name)


def test_qkv_rope_takes_only_what_its_kernel_can_read():
    from kernel_align_b200.ops.layer_ops import _qkv_rope_takes

    width, pos = 8 * 128, torch.arange(6)
    x = torch.zeros(9, width, dtype=torch.bfloat16)
    cos, sin = rope_tables(16, 128)
    odd = torch.zeros(16 * 64 + 1)[1:].view(16, 64)          # contiguous, but at an odd offset

    def takes(x=x, pos=pos, cos=cos, sin=sin, tokens=6, head_dim=128, where=(None,) * 4):
        x, pos, cos, sin = (_OnGpu(t, at or "cuda:0") for t, at in zip((x, pos, cos, sin), where))
        return _qkv_rope_takes(x, pos, cos, sin, tokens, head_dim)

    assert takes()
    assert takes(x=torch.zeros(9, 2 * width, dtype=torch.bfloat16)[:, width:])          # rows of a wider matrix
    assert takes(x=x[2:])
    refused = [dict(x=x.half()), dict(x=torch.zeros(width, 9, dtype=torch.bfloat16).t()), dict(tokens=0),
               dict(x=torch.zeros(9, width + 4, dtype=torch.bfloat16)[:, :width]),      # rows 8-byte aligned
               dict(x=torch.zeros(9 * width + 1, dtype=torch.bfloat16)[1:].view(9, width)),
               dict(x=torch.zeros(1, width, dtype=torch.bfloat16).expand(9, width)), dict(where=("cpu", None, None, None)),
               dict(cos=cos.double()), dict(sin=sin.bfloat16()), dict(cos=torch.zeros(64, 16).t()), dict(cos=odd),
               dict(sin=odd), dict(cos=cos[:, :32].contiguous()), dict(cos=cos.view(-1)), dict(head_dim=64),
               dict(where=(None, None, None, "cpu")), dict(where=(None, None, "cuda:1", None)),
               dict(where=(None, "cpu", None, None))]
    for form in refused:
        assert not takes(**form), form


@pytest.mark.parametrize("dev", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_qkv_rope_refuses_a_projection_of_another_width(dev):
    from kernel_align_b200.ops.layer_ops import qkv_rope_fn

    cos, sin = rope_tables(16, 128, device=dev)
    pos = torch.arange(6, device=dev)
    for rows, heads in ((6, 7), (6, 9), (5, 8)):             # too narrow, too wide, too few rows
        with pytest.raises(ValueError):
            qkv_rope_fn(torch.zeros(rows, heads * 128, dtype=torch.bfloat16, device=dev), pos, cos, sin, 4, 2, 128)
    # tables the fused kernel does not read take the other route
    x = torch.randn(6, 8 * 128, generator=torch.Generator().manual_seed(0)).bfloat16().to(dev)
    odd = torch.cat([cos.new_zeros(2), cos.reshape(-1)])[2:].view(16, 64)
    assert all(torch.equal(a, b) for a, b in zip(qkv_rope_fn(x, pos, cos, sin, 4, 2, 128),
                                                 qkv_rope_fn(x, pos, odd, sin, 4, 2, 128)))


def test_qkv_rope_entry_checks_its_arguments(monkeypatch):
    """The native entry refuses before it launches anything, so this needs no GPU."""
    from kernel_align_b200.ops import layer_ops

    monkeypatch.setattr(layer_ops, "_stream", lambda t: None)
    x = torch.zeros(6 * 8 * 128 + 8, dtype=torch.bfloat16)[:6 * 8 * 128].view(6, 8 * 128)
    cos, sin = rope_tables(16, 128)
    q, k, v = (torch.zeros(6, h, 128, dtype=torch.bfloat16) for h in (4, 2, 2))
    pos = torch.arange(6)
    odd = torch.zeros(6 * 2 * 128 + 1, dtype=torch.bfloat16)[1:].view(6, 2, 128)
    for bad in (dict(qkv=x[:, :7 * 128]), dict(qkv=x[:5]), dict(cos=cos.view(-1)[1:]), dict(sin=sin.view(-1)[1:]),
                dict(q=q[:, :3]), dict(v=odd), dict(k=odd)):
        args = dict(dict(qkv=x, positions=pos, cos=cos, sin=sin, q=q, k=k, v=v, tokens=6), **bad)
        for backward in (False, True):
            with pytest.raises(RuntimeError, match=r"ka_qkv_rope failed \(-[12]\)"):
                layer_ops._qkv_rope_launch(**args, backward=backward)


def _odd(t):
    """The same values, contiguous, but not 16-byte aligned: a piece of a packed buffer."""
    flat = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    flat[1:] = t.reshape(-1)
    return flat[1:].view(t.shape)


def test_gradients_reach_the_kernels_aligned(monkeypatch):
    from kernel_align_b200.ops import layer_ops

    seen = []

    class Lib:
        class _Fn:
            def __call__(self, *args):
                seen.extend(a % 16 for a in args if isinstance(a, int) and a > 1 << 20)
                return 0
        ka_qkv_rope, ka_rmsnorm_bwd = _Fn(), _Fn()

        @staticmethod
        def ka_rmsnorm_bwd_chunk():
            return 16

    monkeypatch.setattr(layer_ops._native, "cuda", lambda: Lib)
    monkeypatch.setattr(layer_ops, "_stream", lambda t: None)
    g = torch.zeros(4, 2, 128, dtype=torch.bfloat16)
    cos, sin = rope_tables(16, 128)

    class Ctx:
        saved_tensors, shape = (torch.arange(4), _odd(cos), _odd(sin)), (6, 6 * 128)

    layer_ops._QkvRopeFn.backward(Ctx, _odd(g), _odd(g), _odd(g))
    x = torch.zeros(5, 64, dtype=torch.bfloat16)
    layer_ops._rmsnorm_backward(_OnGpu(_odd(x)), _odd(x[0]), 1e-5, _odd(x), _odd(x))
    assert len(seen) >= 12 and not any(seen)


@pytest.mark.gpu
def test_gpu_gradients_may_start_anywhere(cuda_device):
    from kernel_align_b200.ops.attention import attention, attention_backward
    from kernel_align_b200.ops.layer_ops import qkv_rope_fn, rmsnorm_fork_fn
    from kernel_align_b200.parallel.tp_gemm import TPContext, gemm_reduce_scatter

    g = torch.Generator(device=cuda_device).manual_seed(2)

    def rand(*shape):
        return torch.randn(*shape, device=cuda_device, generator=g).to(torch.bfloat16)

    cos, sin = rope_tables(16, 128, device=cuda_device)
    qkv, pos = rand(9, 8 * 128).requires_grad_(), torch.arange(7, device=cuda_device)
    grads = [rand(7, h, 128) for h in (4, 2, 2)]
    parts = qkv_rope_fn(qkv, pos, cos, sin, 4, 2, 128)
    a, b = (torch.autograd.grad(parts, qkv, [f(t) for t in grads], retain_graph=True)[0] for f in (_odd, torch.clone))
    assert torch.equal(a, b)
    x, w, dy, dr = rand(20, 256).requires_grad_(), rand(256).requires_grad_(), rand(20, 256), rand(20, 256)
    out = rmsnorm_fork_fn(x, w)
    a, b = (torch.autograd.grad(out, (x, w), (f(dy), f(dr)), retain_graph=True) for f in (_odd, torch.clone))
    assert all(torch.equal(p, q) for p, q in zip(a, b))
    q, k, v, do = rand(2, 70, 4, 128), rand(2, 70, 2, 128), rand(2, 70, 2, 128), rand(2, 70, 4, 128)
    o, lse = attention(q, k, v, return_lse=True)
    assert all(torch.equal(p, r) for p, r in zip(attention_backward(q, k, v, _odd(o), do, lse),
                                                 attention_backward(q, k, v, o, do, lse)))
    tp, m, n, res = TPContext(device=cuda_device), rand(128, 512), rand(64, 512), rand(128, 64)
    assert torch.equal(gemm_reduce_scatter(m, n, tp, residual=_odd(res)), gemm_reduce_scatter(m, n, tp, residual=res))


def test_the_fused_rotation_is_profiled_as_rope(monkeypatch):
    from kernel_align_b200.ops import layer_ops
    from kernel_align_b200.utils import profiler as prof

    class Lib:
        class ka_qkv_rope:
            restype = argtypes = None

            def __new__(cls, *args):
                return 0

    monkeypatch.setattr(layer_ops._native, "cuda", lambda: Lib)
    monkeypatch.setattr(layer_ops, "_stream", lambda t: None)
    x, pos = torch.zeros(6, 4 * 128, dtype=torch.bfloat16), torch.arange(6)
    parts = [torch.zeros(6, h, 128, dtype=torch.bfloat16) for h in (2, 1, 1)]
    prof.set_mode("basic")
    prof.profiler.reset()
    try:
        layer_ops._qkv_rope_launch(x, pos, *rope_tables(16, 128), *parts, 6, False)
        assert prof.profiler.summary()["rope"]["calls"] == 1
    finally:
        prof.set_mode("off")
        prof.profiler.reset()


@pytest.mark.gpu
@pytest.mark.parametrize("d", [128, 2048, 2056, 4096, 4104, 8192, 8200])
def test_gpu_rmsnorm_bits_do_not_depend_on_the_number_of_rows(cuda_device, d):
    """Few rows are kept in registers, many are read twice: the same sums in the same order."""
    g = torch.Generator(device=cuda_device).manual_seed(d)
    x, r = (torch.randn(1300, d, device=cuda_device, generator=g).to(torch.bfloat16) for _ in range(2))
    w = (torch.randn(d, device=cuda_device, generator=g) * 0.1 + 1).to(torch.bfloat16)
    y = rmsnorm(x, w)
    yr, ro = rmsnorm(x, w, residual=r)
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    for rows in (1, 17, 2 * sms, 2 * sms + 1, 4 * sms, 4 * sms + 1):
        for lo in (0, 1300 - rows):
            part = slice(lo, lo + rows)
            assert torch.equal(rmsnorm(x[part], w), y[part]), rows
            a, b = rmsnorm(x[part], w, residual=r[part])
            assert torch.equal(a, yr[part]) and torch.equal(b, ro[part]), rows
    want, want_ro = _rms_ref(x.cpu(), w.cpu(), 1e-5, r.cpu())
    # both round the normalised value and the product to bf16: two units in the last place of the largest
    assert torch.equal(ro.cpu(), want_ro)
    assert (yr.cpu().float() - want.float()).abs().max() <= 2 ** -7 * want.float().abs().max()
