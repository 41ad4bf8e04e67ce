"""GPU tier: generation, the GRPO step and checkpoint / resume on one GPU (tiny model)."""
import pytest
import torch

from kernel_align_b200.executors.generation import generate
from kernel_align_b200.executors.rollout import RolloutExecutor
from kernel_align_b200.executors.trainer import GRPOTrainer
from kernel_align_b200.kernels.sampling import SamplerBackend
from kernel_align_b200.models.llama import LlamaConfig, LlamaModel
from kernel_align_b200.ops import gemm
from kernel_align_b200.ops.decode import attention_decode

pytestmark = pytest.mark.gpu


def _model(dev, seed=1):
    return LlamaModel(LlamaConfig.tiny(n_layers=2), seed=seed, device=dev)


def test_decode_attention_matches_math(cuda_device):
    g = torch.Generator(device=cuda_device).manual_seed(0)
    q = torch.randn(3, 8, 128, device=cuda_device, generator=g).to(torch.bfloat16)
    ck = torch.randn(3, 200, 2, 128, device=cuda_device, generator=g).to(torch.bfloat16)
    cv = torch.randn(3, 200, 2, 128, device=cuda_device, generator=g).to(torch.bfloat16)
    lens = torch.tensor([1, 77, 200], dtype=torch.int32, device=cuda_device)
    out = attention_decode(q, ck, cv, lens)
    ref = attention_decode(q.cpu(), ck.cpu(), cv.cpu(), lens.cpu())
    assert (out.cpu().float() - ref.float()).abs().max().item() < 0.03
    assert torch.equal(attention_decode(q[1:2], ck[1:2], cv[1:2], lens[1:2]), out[1:2])


def test_decode_qkv_rope_cache_equals_the_separate_steps_bitwise(cuda_device):
    from kernel_align_b200.ops.decode import decode_qkv_rope_cache
    from kernel_align_b200.ops.layer_ops import rope_, rope_tables

    b, hq, hkv, d, t = 5, 8, 2, 128, 40
    g = torch.Generator(device=cuda_device).manual_seed(1)
    qkv = torch.randn(b, (hq + 2 * hkv) * d, device=cuda_device, generator=g).to(torch.bfloat16)
    pos = torch.tensor([3, 17, 0, 39, 8], device=cuda_device)
    slot = torch.tensor([21], device=cuda_device)
    cos, sin = rope_tables(64, d, 500000.0, device=cuda_device)
    ck = torch.randn(b, t, hkv, d, device=cuda_device, generator=g).to(torch.bfloat16)
    cv = torch.randn(b, t, hkv, d, device=cuda_device, generator=g).to(torch.bfloat16)
    ck2, cv2 = ck.clone(), cv.clone()
    q = decode_qkv_rope_cache(qkv, pos, slot, cos, sin, ck, cv, hq, hkv)
    q_ref = qkv[:, : hq * d].reshape(b, hq, d).contiguous()
    k_ref = qkv[:, hq * d:(hq + hkv) * d].reshape(b, hkv, d).contiguous()
    rope_(q_ref, pos, cos, sin)
    rope_(k_ref, pos, cos, sin)
    ck2.index_copy_(1, slot, k_ref.view(b, 1, hkv, d))
    cv2.index_copy_(1, slot, qkv[:, (hq + hkv) * d:].reshape(b, 1, hkv, d))
    assert torch.equal(q, q_ref) and torch.equal(ck, ck2) and torch.equal(cv, cv2)


def test_fused_logp_backward_with_a_row_count_that_is_not_a_multiple_of_eight(cuda_device):
    from kernel_align_b200.ops.fused_logp import lmhead_logp

    g = torch.Generator(device=cuda_device).manual_seed(2)
    h = torch.randn(380, 256, device=cuda_device, generator=g).to(torch.bfloat16).requires_grad_()
    w = (torch.randn(1000, 256, device=cuda_device, generator=g) * 0.05).to(torch.bfloat16).requires_grad_()
    ids = torch.randint(0, 1000, (380,), device=cuda_device, generator=g)
    lmhead_logp(h, w, ids).sum().backward()
    hr, wr = h.detach().float().requires_grad_(), w.detach().float().requires_grad_()
    torch.log_softmax(hr @ wr.t(), -1).gather(-1, ids[:, None]).sum().backward()
    assert h.grad.shape == h.shape
    assert (h.grad.float() - hr.grad).abs().max().item() < 0.03 * hr.grad.abs().max().item() + 1e-3
    assert (w.grad.float() - wr.grad).abs().max().item() < 0.03 * wr.grad.abs().max().item() + 1e-3


def test_generation_is_seeded_batch_invariant_and_consistent_with_prefill(cuda_device):
    model = _model(cuda_device)
    prompts = torch.randint(0, model.cfg.vocab_size, (3, 16), device=cuda_device,
                            generator=torch.Generator(device=cuda_device).manual_seed(3))
    out = generate(model, prompts, sampler=SamplerBackend(seed=5), max_new_tokens=8, temperature=0.8, top_k=50,
                   top_p=0.95, group_size=2)
    again = generate(model, prompts, sampler=SamplerBackend(seed=5), max_new_tokens=8, temperature=0.8, top_k=50,
                     top_p=0.95, group_size=2)
    gemm.check_status(cuda_device)
    assert out["sequences"].shape == (6, 24)
    assert torch.equal(out["sequences"], again["sequences"]) and torch.equal(out["logp"], again["logp"])
    other = generate(model, prompts, sampler=SamplerBackend(seed=6), max_new_tokens=8, temperature=0.8, top_k=50,
                     top_p=0.95, group_size=2)
    assert not torch.equal(out["sequences"], other["sequences"])
    # the captured decode graph replays exactly the launches of the eager loop
    eager = generate(model, prompts, sampler=SamplerBackend(seed=5), max_new_tokens=8, temperature=0.8, top_k=50,
                     top_p=0.95, group_size=2, cuda_graph=False)
    assert torch.equal(out["sequences"], eager["sequences"]) and torch.equal(out["logp"], eager["logp"])
    # the log-prob recorded during decoding agrees with a fresh full forward over the sequence
    from kernel_align_b200.ops.fused_logp import lmhead_logp

    seq = out["sequences"]
    with torch.no_grad():
        hidden = model.hidden_states(seq[:, :-1])
        lp = lmhead_logp(hidden[: seq[:, :-1].numel()], model.lm_head, seq[:, 1:].reshape(-1), scale=1 / 0.8)
    lp = lp.view(6, -1)[:, 15:]
    assert (lp - out["logp"]).abs().max().item() < 0.08
    # executor entry point with a model attached
    res = RolloutExecutor({"max_new_tokens": 4, "top_k": 20}, model=model, sampler=SamplerBackend(seed=1)) \
        .execute_rollout(prompts)
    assert res["status"] == "success" and res["sequences"].shape == (3, 20)


def _reward(prompts, new_tokens):
    return (new_tokens % 7 == 0).float().mean(1) + 0.1 * (new_tokens[:, 0] % 3).float()


def test_grpo_step_is_bitwise_repeatable_and_resumable(cuda_device, tmp_path):
    prompts = torch.randint(0, 2048, (4, 16), device=cuda_device,
                            generator=torch.Generator(device=cuda_device).manual_seed(9))

    def fresh():
        return GRPOTrainer(_model(cuda_device, seed=2), _reward, group_size=4, max_new_tokens=8, temperature=1.0,
                           top_k=50, lr=1e-4, seed=3)

    a, b = fresh(), fresh()
    la = [a.train_step(prompts)["loss"].item() for _ in range(3)]
    lb0 = b.train_step(prompts)["loss"].item()
    ckpt = b.save(str(tmp_path / "ckpt.pt"))
    c = fresh()
    c.load(ckpt)
    lc = [c.train_step(prompts)["loss"].item() for _ in range(2)]
    gemm.check_status(cuda_device)
    assert all(torch.isfinite(torch.tensor(la)))
    assert lb0 == la[0]                       # run-to-run bitwise equal loss
    assert lc == la[1:]                       # resume reproduces the uninterrupted run
    assert la[0] != la[1] or la[1] != la[2]   # the policy actually moved


@pytest.mark.parametrize("hq,hkv", [(4, 4), (4, 2), (8, 2), (8, 1), (6, 2)])
def test_decode_attention_bits_do_not_depend_on_how_many_ctas_share_a_sequence(cuda_device, hq, hkv):
    """A cluster of up to eight CTAs works on a (sequence, KV head), fewer in a large batch; the
    decomposition of the keys is the same. Lengths around the block and stripe boundaries."""
    lens = torch.tensor([1, 2, 15, 16, 31, 32, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1025],
                        dtype=torch.int32, device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(3)
    n = lens.numel()
    q = torch.randn(n, hq, 128, device=cuda_device, generator=g).to(torch.bfloat16)
    ck = torch.randn(n, 1030, hkv, 128, device=cuda_device, generator=g).to(torch.bfloat16)
    cv = torch.randn(n, 1030, hkv, 128, device=cuda_device, generator=g).to(torch.bfloat16)
    out = attention_decode(q, ck, cv, lens)
    ref = attention_decode(q.cpu().float(), ck.cpu().float(), cv.cpu().float(), lens.cpu())
    # fp32 arithmetic, rounded once to bf16: half a unit in the last place of the largest value
    assert (out.cpu().float() - ref).abs().max().item() <= 2 ** -8 * ref.abs().max().item()
    for reps in (4, 30):
        wide = attention_decode(q.repeat(reps, 1, 1), ck.repeat(reps, 1, 1, 1), cv.repeat(reps, 1, 1, 1), lens.repeat(reps))
        assert torch.equal(wide.view(reps, n, hq, 128), out.expand(reps, n, hq, 128))
    one = [attention_decode(q[i:i + 1], ck[i:i + 1], cv[i:i + 1], lens[i:i + 1]) for i in range(n)]
    assert torch.equal(torch.cat(one), out)
    # a cache that is not 16-byte aligned takes the general kernel
    flat = torch.empty(ck.numel() + 1, dtype=torch.bfloat16, device=cuda_device)
    flat[1:] = ck.reshape(-1)
    off = attention_decode(q, flat[1:].view_as(ck), cv, lens)
    assert (off.float() - out.float()).abs().max().item() <= 2 ** -7 * ref.abs().max().item()


@pytest.mark.parametrize("hq,hkv", [(4, 4), (4, 2), (8, 2), (8, 1), (6, 2)])
def test_decode_attention_special_values(cuda_device, hq, hkv):
    """Whatever lies behind a sequence's length is not looked at; NaN and infinities inside it come
    out where plain softmax attention has them; an empty sequence has no result (0 / 0)."""
    lens = torch.tensor([300, 300, 300, 300, 300, 70, 0], dtype=torch.int32, device=cuda_device)
    g = torch.Generator(device=cuda_device).manual_seed(hq)
    n = lens.numel()
    q = torch.randn(n, hq, 128, device=cuda_device, generator=g).to(torch.bfloat16)
    ck = torch.randn(n, 320, hkv, 128, device=cuda_device, generator=g).to(torch.bfloat16)
    cv = torch.randn(n, 320, hkv, 128, device=cuda_device, generator=g).to(torch.bfloat16)
    for i, l in enumerate(lens.tolist()):
        ck[i, l:], cv[i, l:] = float("nan"), float("nan")
    clean = attention_decode(q, ck, cv, lens)
    assert torch.isfinite(clean[:6]).all() and torch.isnan(clean[6]).all()
    ck[0, 200, 0, 5] = float("nan")              # a score is NaN: the heads of that group are
    ck[1, 17, hkv - 1, 3] = float("inf")         # a score is +inf (NaN probabilities) or -inf (no weight)
    cv[2, 299, 0, 7] = float("inf")              # one element of the result
    cv[3, 64, 0, 9] = float("nan")
    ck[4, :300, 0, 0] = float("-inf")            # every score of the group infinite
    out = attention_decode(q, ck, cv, lens).cpu().float()
    ref = attention_decode(q.cpu().float(), ck.cpu().float(), cv.cpu().float(), lens.cpu())
    ref[6] = float("nan")
    assert torch.equal(torch.isnan(out), torch.isnan(ref)) and torch.equal(torch.isinf(out), torch.isinf(ref))
    ok = torch.isfinite(ref)
    assert (out[ok] - ref[ok]).abs().max() <= 2 ** -8 * ref[ok].abs().max()
    assert torch.equal(out[5], clean[5].cpu().float())


@pytest.mark.parametrize("hq,hkv,per_sm", [(8, 8, 3), (16, 8, 3), (32, 8, 3), (64, 8, 2), (8, 1, 2)])
def test_decode_attention_ctas_are_resident_at_once(cuda_device, hq, hkv, per_sm):
    """More than two CTAs per (sequence, KV head) only while all of them run at the same time (`per_sm`:
    what the registers of the kernel allow), and never more than the cache has blocks."""
    from kernel_align_b200 import _native

    splits = _native.cuda().ka_attention_decode_splits
    sms = torch.cuda.get_device_properties(cuda_device).multi_processor_count
    chosen = [splits(b, hq, hkv, 4096) for b in range(1, 600)]
    assert chosen[0] == 8 and chosen[-1] == 2 and chosen == sorted(chosen, reverse=True)
    assert all(s == 2 or (b + 1) * hkv * s <= per_sm * sms for b, s in enumerate(chosen))
    assert [splits(1, hq, hkv, n) for n in (1, 64, 128, 129, 256, 257)] == [2, 2, 2, 4, 4, 8]
