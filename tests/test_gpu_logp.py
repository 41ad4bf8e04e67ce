"""GPU tier: fused LM-head log-prob and log-prob from logits against fp32 PyTorch."""
import pytest
import torch

from kernel_align_b200.ops import cpu_ops, fused_logp
from kernel_align_b200.ops.logits_logp import logits_logp

pytestmark = pytest.mark.gpu


def _ref(h, w, ids, scale=1.0):
    out = torch.empty(h.shape[0], dtype=torch.float32, device=h.device)
    lse = torch.empty_like(out)
    for i in range(0, h.shape[0], 1024):
        lg = (h[i:i + 1024].float() @ w.float().T) * scale
        lse[i:i + 1024] = torch.logsumexp(lg, -1)
        out[i:i + 1024] = lg.gather(-1, ids[i:i + 1024, None]).squeeze(-1) - lse[i:i + 1024]
    return out, lse


def _inputs(dev, m, k, v, seed=0):
    g = torch.Generator(device=dev).manual_seed(seed)
    h = torch.randn(m, k, device=dev, generator=g).to(torch.bfloat16)
    w = (torch.randn(v, k, device=dev, generator=g) * 0.02).to(torch.bfloat16)
    ids = torch.randint(0, v, (m,), device=dev, generator=g)
    return h, w, ids


@pytest.mark.parametrize("cta_group", [1, 2])
@pytest.mark.parametrize("m,k,v,scale", [(256, 256, 1024, 1.0), (300, 512, 5000, 1 / 0.7), (1000, 1024, 20000, 1.0),
                                         (130, 4096, 128256, 1.0)])
def test_fused_logp_matches_fp32_reference(cuda_device, cta_group, m, k, v, scale):
    h, w, ids = _inputs(cuda_device, m, k, v)
    out, lse = fused_logp.lmhead_logp(h, w, ids, scale=scale, cta_group=cta_group, return_lse=True, check=True)
    ref, ref_lse = _ref(h, w, ids, scale)
    assert (out - ref).abs().max().item() < 2e-3
    assert (lse - ref_lse).abs().max().item() < 2e-3


def test_fused_logp_vs_cpu_library(cuda_device):
    h, w, ids = _inputs(cuda_device, 256, 256, 1024, seed=3)
    out = fused_logp.lmhead_logp(h, w, ids, check=True)
    ref = cpu_ops.lmhead_logp_cpu(h.cpu(), w.cpu(), ids.cpu())
    assert (out.cpu() - ref).abs().max().item() < 2e-3


def test_fused_logp_bitwise_batch_invariant_and_repeatable(cuda_device):
    h, w, ids = _inputs(cuda_device, 1536, 512, 9000, seed=1)
    full = fused_logp.lmhead_logp(h, w, ids, check=True)
    assert torch.equal(full, fused_logp.lmhead_logp(h, w, ids, check=True))
    for lo, hi in ((0, 1), (5, 133), (700, 1536)):
        part = fused_logp.lmhead_logp(h[lo:hi], w, ids[lo:hi], check=True)
        assert torch.equal(part, full[lo:hi])
    # the row panel size only bounds scratch
    small = fused_logp.lmhead_logp(h, w, ids, panel_rows=512, check=True)
    assert torch.equal(small, full)
    # 1-CTA and 2-CTA tiles issue the same per-row arithmetic
    assert torch.equal(fused_logp.lmhead_logp(h, w, ids, cta_group=1, check=True), full)


def test_fused_logp_every_schedule_gives_the_same_bits_and_autotune_picks_one(cuda_device, monkeypatch):
    """The tile variant and the work order change cycles and power, never a result. The first
    large call of a shape times the candidates; here the size limit is lowered so that a small
    case goes through the same code."""
    h, w, ids = _inputs(cuda_device, 3000, 512, 30000, seed=4)
    want, want_lse = fused_logp.lmhead_logp(h, w, ids, cta_group=2, return_lse=True, check=True)
    for sched in ("2,8", "2,3", "1,4", "1,2", "1,3", "1,1", "1,2,1", "2,4,1", "1,5,1", "1,4,0,1", "2,8,0,2", "1,2,0,3", "2,4,2", "1,3,3,1", "2,5,2,3"):
        monkeypatch.setenv("KA_LOGP_SCHEDULE", sched)
        out, lse = fused_logp.lmhead_logp(h, w, ids, return_lse=True, check=True)
        assert torch.equal(out, want) and torch.equal(lse, want_lse), sched
    monkeypatch.delenv("KA_LOGP_SCHEDULE")
    monkeypatch.setattr(fused_logp, "_AUTOTUNE_MIN_MACS", 0.0)
    monkeypatch.setattr(fused_logp, "_TUNE_MIN_MS", 1.0)
    fused_logp._tuned.clear()
    out = fused_logp.lmhead_logp(h, w, ids, check=True)
    assert torch.equal(out, want)
    assert len(fused_logp._tuned) == 1 and next(iter(fused_logp._tuned.values())) in fused_logp._SCHEDULES
    assert torch.equal(fused_logp.lmhead_logp(h, w, ids, check=True), want)      # the tuned schedule, reused
    fused_logp._tuned.clear()


def test_fused_logp_ignored_ids_and_3d(cuda_device):
    h, w, ids = _inputs(cuda_device, 4 * 64, 256, 1024, seed=2)
    ids = ids.clone()
    ids[3] = -100
    out = fused_logp.lmhead_logp(h.view(4, 64, 256), w, ids.view(4, 64), check=True)
    assert out.shape == (4, 64) and out.view(-1)[3].item() == 0.0


def test_fused_logp_scratch_is_constant_in_rows(cuda_device):
    assert fused_logp.workspace_bytes(128256) < 32 * 2**20
    h, w, ids = _inputs(cuda_device, 2048, 256, 4096)
    fused_logp.lmhead_logp(h, w, ids)
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    fused_logp.lmhead_logp(h, w, ids)
    torch.cuda.synchronize()
    assert torch.cuda.max_memory_allocated() - base < 1 * 2**20  # output + int64 ids only


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_logits_logp(cuda_device, dtype):
    g = torch.Generator(device=cuda_device).manual_seed(4)
    logits = (torch.randn(6, 33, 5003, device=cuda_device, generator=g) * 3).to(dtype)
    ids = torch.randint(0, 5003, (6, 33), device=cuda_device, generator=g)
    out, lse = logits_logp(logits, ids, scale=1 / 0.7, return_lse=True)
    ref = torch.log_softmax(logits.float() / 0.7, -1).gather(-1, ids[..., None]).squeeze(-1)
    assert out.shape == (6, 33)
    assert (out - ref).abs().max().item() < 1e-4
    assert (lse - torch.logsumexp(logits.float() / 0.7, -1)).abs().max().item() < 1e-4
    one = logits_logp(logits[2:3], ids[2:3], scale=1 / 0.7)
    assert torch.equal(one, out[2:3])


def test_logits_logp_llama_vocab(cuda_device):
    g = torch.Generator(device=cuda_device).manual_seed(5)
    logits = (torch.randn(64, 128256, device=cuda_device, generator=g) * 2).to(torch.bfloat16)
    ids = torch.randint(0, 128256, (64,), device=cuda_device, generator=g)
    out = logits_logp(logits, ids)
    ref = torch.log_softmax(logits.float(), -1).gather(-1, ids[:, None]).squeeze(-1)
    assert (out - ref).abs().max().item() < 1e-4


def test_fused_logp_backward_matches_autograd(cuda_device):
    from kernel_align_b200.ops import gemm

    m, k, v = 600, 512, 9000
    h, w, ids = _inputs(cuda_device, m, k, v, seed=11)
    ids = ids.clone()
    ids[5] = -100
    g = torch.randn(m, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(12))
    hq, wq = h.clone().requires_grad_(), w.clone().requires_grad_()
    out = fused_logp.lmhead_logp(hq, wq, ids, scale=1 / 0.7)
    out.backward(g)
    gemm.check_status(cuda_device)
    hr, wr = h.float().requires_grad_(), w.float().requires_grad_()
    lg = (hr @ wr.t()) / 0.7
    ref = torch.log_softmax(lg, -1).gather(-1, ids.clamp(min=0)[:, None]).squeeze(-1)
    ref = ref * (ids >= 0)
    ref.backward(g)
    assert (out - ref.detach()).abs().max().item() < 2e-3
    assert (hq.grad.float() - hr.grad).abs().max().item() <= 0.02 * hr.grad.abs().max().item()
    assert (wq.grad.float() - wr.grad).abs().max().item() <= 0.02 * wr.grad.abs().max().item()
    assert hq.grad[5].abs().max().item() == 0
    # repeatable bit for bit
    h2, w2 = h.clone().requires_grad_(), w.clone().requires_grad_()
    fused_logp.lmhead_logp(h2, w2, ids, scale=1 / 0.7).backward(g)
    assert torch.equal(h2.grad, hq.grad) and torch.equal(w2.grad, wq.grad)


@pytest.mark.parametrize("cta_group,panel_rows", [(None, fused_logp.DEFAULT_PANEL_ROWS), (1, 256), (2, 256)])
@pytest.mark.parametrize("m,k,v,scale", [(1, 64, 64, 1.0), (37, 128, 1920, 0.7), (300, 256, 16448, 1.0), (129, 64, 50304, 1.3),
                                         (700, 64, 1920, 1.0)])
def test_kept_logits_give_the_gradients_of_recomputed_ones(cuda_device, m, k, v, scale, cta_group, panel_rows, monkeypatch):
    """Bit for bit, for one sub-slice of the vocabulary and several, both tile variants, several panels of
    rows, ignored ids, a second pass through the graph, and a graph that finds the allowance used up."""
    g = torch.Generator(device=cuda_device).manual_seed(v)
    h = torch.randn(m, k, device=cuda_device, generator=g).to(torch.bfloat16).requires_grad_()
    w = (torch.randn(v, k, device=cuda_device, generator=g) * 0.2).to(torch.bfloat16).requires_grad_()
    ids = torch.randint(-1, v + 1, (m,), device=cuda_device, generator=g)
    up = torch.randn(m, device=cuda_device, generator=g)
    before = dict(fused_logp._kept_bytes)
    monkeypatch.setattr(fused_logp, "_KEEP_BYTES", sum(before.values()) + 4 * m * v)

    def call():
        return fused_logp.lmhead_logp(h, w, ids, scale=scale, cta_group=cta_group, panel_rows=panel_rows)

    kept, other = call(), call()          # the second one recomputes
    holders = [x.grad_fn.saved_tensors[2]._ka_kept for x in (kept, other)]
    assert holders[0].logits.shape == (m, v) and holders[1] is None
    del holders
    want = torch.autograd.grad(other, (h, w), up)
    for _ in range(2):
        got = torch.autograd.grad(kept, (h, w), up, retain_graph=True)
        assert torch.equal(kept, other) and all(torch.equal(a, b) for a, b in zip(got, want))
    with torch.no_grad():
        assert torch.equal(call(), other)
    del kept, other
    assert {i: n for i, n in fused_logp._kept_bytes.items() if n} == {i: n for i, n in before.items() if n}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("vocab", [1, 7, 8, 17, 33, 4095, 16385, 50257])
@pytest.mark.parametrize("times", [1, 200])
def test_logits_logp_does_not_depend_on_where_a_row_starts(cuda_device, dtype, vocab, times):
    """The same bits for a row on a 16-byte boundary and at every offset from one, in few rows and in many."""
    from kernel_align_b200.ops.logits_logp import logits_logp

    g = torch.Generator(device=cuda_device).manual_seed(vocab)
    width = (vocab + 15) // 8 * 8
    x = torch.full((3, width), float("nan"), device=cuda_device, dtype=dtype)
    x[:, :vocab] = (torch.randn(3, vocab, device=cuda_device, generator=g) * 2).to(dtype)
    ids = torch.tensor([0, vocab - 1, vocab // 2], device=cuda_device)
    want, want_lse = logits_logp(x[:, :vocab], ids, return_lse=True)
    exact = torch.log_softmax(x[:, :vocab].double(), -1).gather(1, ids[:, None])[:, 0]
    # 32-bit sums of at most 50257 terms and two approximate functions of 2^-22 relative error
    assert torch.allclose(want.double(), exact, rtol=1e-6, atol=4e-6)
    rows = 3 * times
    x, ids, want, want_lse = x.repeat(times, 1), ids.repeat(times), want.repeat(times), want_lse.repeat(times)
    for off in range(16 // x.element_size()):
        buf = torch.full((rows * (width + 1) + 8,), float("nan"), device=cuda_device, dtype=dtype)
        for stride in (width, width + 1):
            part = buf[off:off + rows * stride].view(rows, stride)[:, :vocab]
            part.copy_(x[:, :vocab])
            got, got_lse = logits_logp(part, ids, return_lse=True)
            assert torch.equal(got, want) and torch.equal(got_lse, want_lse), (off, stride)


def test_kept_logits_under_checkpoint(cuda_device, monkeypatch):
    """Checkpointed calls of more than half the allowance, and chunks that use it up: the repetition of a
    call may find another part of the allowance free than the call itself."""
    from torch.utils.checkpoint import checkpoint

    g = torch.Generator(device=cuda_device).manual_seed(5)
    m, k, v = 256, 128, 1920
    h = torch.randn(m, k, device=cuda_device, generator=g).to(torch.bfloat16).requires_grad_()
    w = (torch.randn(v, k, device=cuda_device, generator=g) * 0.2).to(torch.bfloat16).requires_grad_()
    ids = torch.randint(0, v, (m,), device=cuda_device, generator=g)
    for chunks, allowance in ((1, m * 6), (4, m * 4), (4, m)):       # bytes per column, 4 * m in all
        monkeypatch.setattr(fused_logp, "_KEEP_BYTES", sum(fused_logp._kept_bytes.values()) + allowance * v)
        grads = []
        for use in (False, True):
            parts = [checkpoint(fused_logp.lmhead_logp, a, w, b, use_reentrant=False) if use
                     else fused_logp.lmhead_logp(a, w, b) for a, b in zip(h.chunk(chunks), ids.chunk(chunks))]
            grads.append(torch.autograd.grad(torch.cat(parts).sum(), (h, w)))
            del parts
        assert all(torch.equal(a, b) for a, b in zip(*grads))


def test_kept_logits_are_gone_after_the_backward_pass(cuda_device):
    """Their share of the allowance as well, whoever holds the result; and with a hook that moves what is
    saved to the host."""
    h, w, ids = _inputs(cuda_device, 64, 128, 1920, seed=3)
    h.requires_grad_()
    before = dict(fused_logp._kept_bytes).get(cuda_device.index or 0, 0)
    nbytes = 4 * 64 * 1920
    results, grads = [], []
    for _ in range(3):
        results.append(fused_logp.lmhead_logp(h, w, ids))
        assert fused_logp._kept_bytes[cuda_device.index or 0] == before + nbytes
        grads += torch.autograd.grad(results[-1].sum(), h)
        assert fused_logp._kept_bytes[cuda_device.index or 0] == before
    with torch.autograd.graph.save_on_cpu():
        results.append(fused_logp.lmhead_logp(h, w, ids))
        assert fused_logp._kept_bytes[cuda_device.index or 0] == before
        grads += torch.autograd.grad(results[-1].sum(), h)
    assert all(torch.equal(a, grads[0]) for a in grads)


def test_kept_logits_need_memory_to_spare(cuda_device, monkeypatch):
    """Neither with the limit at 0 nor while memory is short are logits kept, an allocation that failed is not
    tried again, and the gradients are the same."""
    h, w, ids = _inputs(cuda_device, 64, 128, 1920, seed=4)
    h.requires_grad_()
    monkeypatch.setattr(fused_logp, "_KEEP_UNASKED_BYTES", 0)
    monkeypatch.setattr(fused_logp, "_capacity", {})
    grads, tries, empty = [], [], torch.empty

    def full(*args, **kwargs):
        if args == (64, 1920) and kwargs["dtype"] == torch.float32:
            tries.append(args)
            raise torch.OutOfMemoryError("no room")
        return empty(*args, **kwargs)

    for env, capacity, alloc, kept in (("", {}, empty, True), ("0", {}, empty, False), ("", {0: 1 << 20}, empty, False),
                                       ("", {}, full, False), ("", None, full, False)):
        monkeypatch.setenv("KA_LOGP_KEEP_BYTES", env)
        monkeypatch.setattr(torch, "empty", alloc)
        if capacity is not None:
            monkeypatch.setattr(fused_logp, "_capacity", capacity)
        logp = fused_logp.lmhead_logp(h, w, ids)
        assert (logp.grad_fn.saved_tensors[2]._ka_kept is not None) == kept
        grads += torch.autograd.grad(logp.sum(), h)
    assert len(tries) == 1 and all(torch.equal(g, grads[0]) for g in grads)


def test_schedule_of_a_call_that_keeps_its_logits_is_its_own(cuda_device, monkeypatch):
    """Scoring and training calls of one shape are tuned apart, in whichever order they come."""
    monkeypatch.setattr(fused_logp, "_tuned", {})
    monkeypatch.setattr(fused_logp, "_AUTOTUNE_MIN_MACS", 0.0)
    monkeypatch.setattr(fused_logp, "_TUNE_MIN_MS", 0.1)
    h, w, ids = _inputs(cuda_device, 300, 64, 1920, seed=6)
    want = fused_logp.lmhead_logp(h, w, ids)
    h.requires_grad_()
    for _ in range(2):
        assert torch.equal(fused_logp.lmhead_logp(h, w, ids), want)
    assert sorted(key[-1] for key in fused_logp._tuned) == [False, True]
