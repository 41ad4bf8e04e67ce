"""The allowance for logits that calls with gradients keep (host side; the kernels are in test_gpu_logp.py)."""
import subprocess
import sys
import textwrap

import pytest
import torch
from torch.utils.checkpoint import checkpoint

from kernel_align_b200.ops import fused_logp

_SHARES_IN_CYCLES = """
import gc, threading
from kernel_align_b200.ops import fused_logp as f

def run(n):
    for _ in range(n):
        share = f._Kept.take(0, 8)
        cell = [share]
        cell.append(cell)            # a cycle: only a collection frees it, whenever one runs

gc.set_threshold(5)
threads = [threading.Thread(target=run, args=(20000,)) for _ in range(3)]
for t in threads: t.start()
for t in threads: t.join()
gc.collect()
share = f._Kept.take(0, 8)           # whatever finalizers left behind is counted by now
assert f._kept_bytes[0] == 8, f._kept_bytes
del share
assert f._kept_bytes[0] == 0, f._kept_bytes
"""


def test_share_collected_while_another_is_taken():
    """A collection may run inside take() and free shares that sit in reference cycles: their finalizer
    must not wait for what its own thread holds, and nothing may be lost."""
    r = subprocess.run([sys.executable, "-c", textwrap.dedent(_SHARES_IN_CYCLES)], timeout=120, capture_output=True,
                       text=True)
    assert r.returncode == 0, r.stderr[-2000:]


def _keep_on_cpu(monkeypatch, allowance):
    """Calls on the CPU take shares and keep (unused) logits as calls on a GPU do."""
    def kept_logits(hidden, weight, vocab, group):
        m, v = hidden.numel() // hidden.shape[-1], weight.shape[0]
        kept = fused_logp._Kept.take(99, 4 * m * v)
        if kept is not None:
            kept.logits = torch.empty(m, v)
        return kept

    monkeypatch.setattr(fused_logp, "_kept_logits", kept_logits)
    monkeypatch.setattr(fused_logp, "_KEEP_BYTES", fused_logp._kept_bytes.get(99, 0) + allowance)


def _inputs(m=8, k=16, v=64):
    g = torch.Generator().manual_seed(m)
    h = torch.randn(m, k, generator=g).to(torch.bfloat16).requires_grad_()
    w = torch.randn(v, k, generator=g).to(torch.bfloat16).requires_grad_()
    return h, w, torch.randint(0, v, (m,), generator=g)


@pytest.mark.parametrize("chunks,allowance", [(1, 6 * 8 * 64), (4, 4 * 8 * 64), (4, 8 * 64)])
def test_checkpoint_with_an_allowance_that_is_used_up(monkeypatch, chunks, allowance):
    """The repetition of a checkpointed call may find another part of the allowance free than the call."""
    _keep_on_cpu(monkeypatch, allowance)
    h, w, ids = _inputs()
    grads = []
    for use in (False, True):
        parts = [checkpoint(fused_logp.lmhead_logp, a, w, b, use_reentrant=False) if use
                 else fused_logp.lmhead_logp(a, w, b) for a, b in zip(h.chunk(chunks), ids.chunk(chunks))]
        grads.append(torch.autograd.grad(torch.cat(parts).sum(), (h, w)))
        del parts
    assert all(torch.equal(a, b) for a, b in zip(*grads))


def test_saved_tensors_do_not_depend_on_what_is_kept(monkeypatch):
    h, w, ids = _inputs()
    _keep_on_cpu(monkeypatch, 4 * 8 * 64)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append((tuple(t.shape), t.dtype)) or t, lambda t: t):
        first = fused_logp.lmhead_logp(h, w, ids)
        second = fused_logp.lmhead_logp(h, w, ids)     # finds the allowance used up
    assert seen[:len(seen) // 2] == seen[len(seen) // 2:] and len(seen) == 8
    assert torch.equal(first, second)


def _kept_now():
    return fused_logp._kept_bytes.get(99, 0)


def test_allowance_follows_the_logits_and_not_the_node(monkeypatch):
    """After a backward pass, behind a checkpoint and with a hook that copies, the logits are gone and so is
    their share, whoever still holds the result; a retained graph keeps both."""
    nbytes = 4 * 8 * 64
    _keep_on_cpu(monkeypatch, nbytes)
    before = _kept_now()
    h, w, ids = _inputs()
    results = []
    for _ in range(2):
        logp = fused_logp.lmhead_logp(h, w, ids)
        assert _kept_now() == before + nbytes
        logp.sum().backward(retain_graph=True)
        assert _kept_now() == before + nbytes
        logp.sum().backward()
        assert _kept_now() == before
        results.append(logp)
    results.append(checkpoint(fused_logp.lmhead_logp, h, w, ids, use_reentrant=False))
    assert _kept_now() == before
    with torch.autograd.graph.saved_tensors_hooks(lambda t: t.clone(), lambda t: t):
        results.append(fused_logp.lmhead_logp(h, w, ids))
        assert _kept_now() == before
        want = torch.autograd.grad(results[-1].sum(), (h, w))
    logp = fused_logp.lmhead_logp(h, w, ids)
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(logp.sum(), (h, w)), want))
    fused_logp.lmhead_logp(h, w, ids)          # dropped without a backward pass
    assert _kept_now() == before


def test_limit_from_the_environment(monkeypatch):
    _keep_on_cpu(monkeypatch, 4 * 8 * 64)
    before = _kept_now()
    h, w, ids = _inputs()
    for env, kept in (("0", 0), (str(before + 4 * 8 * 64), 4 * 8 * 64), (str(before + 4 * 8 * 64 - 1), 0)):
        monkeypatch.setenv("KA_LOGP_KEEP_BYTES", env)
        logp = fused_logp.lmhead_logp(h, w, ids)
        assert _kept_now() == before + kept
        del logp
    monkeypatch.setenv("KA_LOGP_KEEP_BYTES", "2G")
    with pytest.raises(ValueError, match="KA_LOGP_KEEP_BYTES"):
        fused_logp.lmhead_logp(h, w, ids)


@pytest.mark.parametrize("capacity,allocated,nbytes,spare", [
    (None, 100 << 30, 1 << 30, True), (None, 179 << 30, 1 << 30, True), (None, (179 << 30) + 1, 1 << 30, False),
    (None, 192 << 30, 1 << 20, True), (None, 192 << 30, 256 << 20, False), (32 << 30, 29 << 30, 1 << 30, True),
    (32 << 30, 30 << 30, 1 << 30, False), (32 << 30, 31 << 30, 1 << 20, False)])
def test_nothing_is_kept_when_memory_is_short(monkeypatch, capacity, allocated, nbytes, spare):
    """192 GiB in all, or 32 as a failed allocation showed, of which a sixteenth has to stay unallocated."""
    class Props:
        total_memory = 192 << 30

    def never(*args):
        raise AssertionError("the driver is not asked: that takes milliseconds on a busy host")

    monkeypatch.setattr(torch.cuda, "get_device_properties", lambda d: Props)
    monkeypatch.setattr(torch.cuda, "mem_get_info", never)
    monkeypatch.setattr(torch.cuda, "memory_stats_as_nested_dict",
                        lambda d: {"allocated_bytes": {"all": {"current": allocated}}})
    monkeypatch.setattr(fused_logp, "_capacity", {} if capacity is None else {0: capacity})
    assert fused_logp._memory_to_spare(0, nbytes) is spare
