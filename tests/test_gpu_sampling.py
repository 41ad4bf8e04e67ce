"""GPU tier: the fused sampler returns exactly the tokens of the CPU definition."""
import pytest
import torch

from kernel_align_b200.kernels.sampling import SamplerBackend
from kernel_align_b200.ops import cpu_ops
from kernel_align_b200.ops.sampling import sample

pytestmark = pytest.mark.gpu


def _cpu(logits, top_k, top_p, temperature, seed, step, row_ids=None):
    return cpu_ops.sample_cpu(logits.cpu(), inv_temperature=1.0 / temperature, top_k=top_k or 0,
                              top_p=1.0 if top_p is None else top_p, seed=seed, step=step, row_ids=row_ids)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("top_k,top_p", [(50, 0.9), (1, None), (1024, 0.95), (7, None), (None, 0.9), (None, None),
                                         (3000, 0.8)])
def test_sampler_equals_cpu_definition(cuda_device, dtype, top_k, top_p):
    g = torch.Generator(device=cuda_device).manual_seed(0)
    logits = (torch.randn(24, 8000, device=cuda_device, generator=g) * 2).to(dtype)
    for step in (0, 1):
        tok = sample(logits, top_k=top_k, top_p=top_p, temperature=0.7, seed=9, step=step)
        ref = _cpu(logits, top_k, top_p, 0.7, 9, step)
        assert tok.dtype == torch.int32
        assert torch.equal(tok.cpu(), ref), (top_k, top_p, step)


def test_sampler_llama_vocab_headline_config(cuda_device):
    g = torch.Generator(device=cuda_device).manual_seed(1)
    logits = (torch.randn(256, 128256, device=cuda_device, generator=g) * 2).to(torch.bfloat16)
    tok = sample(logits, top_k=50, top_p=0.9, temperature=0.7, seed=1, step=3)
    assert torch.equal(tok[:32].cpu(), _cpu(logits[:32], 50, 0.9, 0.7, 1, 3))
    # batch invariance: rows 64..128 sampled alone, named by their row ids
    part = sample(logits[64:128], top_k=50, top_p=0.9, temperature=0.7, seed=1, step=3,
                  row_ids=torch.arange(64, 128))
    assert torch.equal(part, tok[64:128])
    assert torch.equal(tok, sample(logits, top_k=50, top_p=0.9, temperature=0.7, seed=1, step=3))


@pytest.mark.parametrize("cluster", ["1", "2", "4"])
def test_sampler_cluster_variants_equal_cpu_definition(cuda_device, cluster, monkeypatch):
    """Few rows of 16-bit logits are sampled by a cluster of CTAs per row; every variant must
    return the tokens of the CPU definition: a vocabulary with a scalar tail, heavy ties that
    overflow the candidate list, k from 1 to 1024."""
    monkeypatch.setenv("KA_SAMPLE_CLUSTER", cluster)
    g = torch.Generator(device=cuda_device).manual_seed(7)
    wide = (torch.randn(12, 50016, device=cuda_device, generator=g) * 2).to(torch.bfloat16)[:, :50011]
    for top_k, top_p in ((50, 0.9), (1, None), (1024, 0.95)):
        tok = sample(wide, top_k=top_k, top_p=top_p, temperature=0.7, seed=3, step=2)
        assert torch.equal(tok.cpu(), _cpu(wide, top_k, top_p, 0.7, 3, 2)), (cluster, top_k, top_p)
    ties = torch.zeros(4, 20000, device=cuda_device, dtype=torch.float16)
    ties[2, 19999] = 1.0
    tok = sample(ties, top_k=50, top_p=0.5, seed=2, step=0)
    assert torch.equal(tok.cpu(), _cpu(ties, 50, 0.5, 1.0, 2, 0))
    llama = (torch.randn(64, 128256, device=cuda_device, generator=g) * 2).to(torch.bfloat16)
    tok = sample(llama, top_k=50, top_p=0.9, temperature=0.7, seed=1, step=5)
    assert torch.equal(tok[:16].cpu(), _cpu(llama[:16], 50, 0.9, 0.7, 1, 5))
    monkeypatch.setenv("KA_SAMPLE_CLUSTER", "1")
    assert torch.equal(tok, sample(llama, top_k=50, top_p=0.9, temperature=0.7, seed=1, step=5))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("vocab,rows", [(5, 3), (1023, 3), (65537, 3), (131081, 2), (33001, 200)])
def test_sampler_top_k_bounds_and_row_starts(cuda_device, dtype, vocab, rows):
    """Both sides of the small-k bound, candidates by the thousand, rows that start off a 16-byte
    boundary, one to four CTAs per row and more rows than are resident; values: plain, heavy ties,
    mostly -inf or the type's lowest, sorted (the largest all in one part of the row), NaN and +inf."""
    g = torch.Generator(device=cuda_device).manual_seed(vocab)
    x = torch.randn(rows, vocab, device=cuda_device, generator=g) * 2
    u = torch.rand(x.shape, device=cuda_device, generator=g)
    values = {"plain": x, "ties": x.round(), "masked": torch.where(u < 0.999, float("-inf"), x),
              "lowest": torch.where(u < 0.9, torch.finfo(dtype).min, x), "sorted": x.sort(1, descending=True).values,
              "special": torch.where(u < 0.01, float("nan"), torch.where(u > 0.9999, float("inf"), x))}
    buf = torch.empty(rows * (vocab + 1) + 3, dtype=dtype, device=cuda_device)
    for name, val in values.items():
        for off, width in ((0, vocab), (3, vocab + 1)):
            logits = buf[off:off + rows * width].view(rows, width)[:, :vocab]
            logits.copy_(val)
            for top_k, top_p in ((1, None), (64, 0.9), (65, 0.5), (1000, 0.95), (1024, None)):
                if top_k >= vocab:
                    continue
                tok = sample(logits, top_k=top_k, top_p=top_p, temperature=0.7, seed=4, step=off)
                ref = _cpu(logits[:4], top_k, top_p, 0.7, 4, off)
                assert torch.equal(tok[:4].cpu(), ref), (name, off, top_k, top_p)


def test_sampler_heavy_ties(cuda_device):
    # constant rows overflow the candidate list: the exact-select path cuts ties by token id
    logits = torch.zeros(4, 20000, device=cuda_device, dtype=torch.bfloat16)
    logits[1, 777] = 1.0
    for top_k, top_p in ((50, None), (50, 0.5), (None, 0.001), (5000, None)):
        tok = sample(logits, top_k=top_k, top_p=top_p, seed=2, step=0)
        assert torch.equal(tok.cpu(), _cpu(logits, top_k, top_p, 1.0, 2, 0)), (top_k, top_p)
    # quantised logits: many exact duplicates around the k-th value
    g = torch.Generator(device=cuda_device).manual_seed(3)
    q = (torch.randn(8, 50000, device=cuda_device, generator=g) * 4).round().to(torch.bfloat16)
    for top_k, top_p in ((50, 0.9), (1000, None), (None, 0.7)):
        tok = sample(q, top_k=top_k, top_p=top_p, seed=4, step=1)
        assert torch.equal(tok.cpu(), _cpu(q, top_k, top_p, 1.0, 4, 1)), (top_k, top_p)


def test_sampler_backend_module(cuda_device):
    s = SamplerBackend(seed=5)
    g = torch.Generator(device=cuda_device).manual_seed(6)
    logits = (torch.randn(8, 4096, device=cuda_device, generator=g)).to(torch.bfloat16)
    a = s.sample(logits, top_k=20, top_p=0.9, temperature=0.8)
    b = s.sample(logits, top_k=20, top_p=0.9, temperature=0.8)
    assert s.step == 2 and a.shape == (8,)
    s.set_rng_state({"seed": 5, "step": 0})
    assert torch.equal(s.sample(logits, top_k=20, top_p=0.9, temperature=0.8), a)
    assert torch.equal(s.sample(logits, top_k=20, top_p=0.9, temperature=0.8), b)
    assert torch.equal(s.sample(logits, top_k=1).long(), logits.float().argmax(-1))


def test_sampler_bf16_without_top_k_threshold_among_negative_values_and_nan(cuda_device):
    """bf16 rows without a (small) top-k search their threshold in a per-key count histogram,
    non-negative keys first; rows whose threshold lies among negative values, rows with NaN / inf
    entries and a Llama-sized vocabulary must give the CPU library's token."""
    g = torch.Generator(device=cuda_device).manual_seed(11)
    neg = (-torch.randn(6, 128256, device=cuda_device, generator=g).abs() * 2 - 1).to(torch.bfloat16)
    mixed = (torch.randn(6, 128256, device=cuda_device, generator=g) * 2).to(torch.bfloat16)
    odd = mixed.clone()
    odd[0, 5] = float("nan")
    odd[1, 77] = float("-inf")
    odd[2, :100] = float("nan")
    odd[3, 9] = 0.0
    odd[3, 10] = -0.0
    for name, logits in (("neg", neg), ("mixed", mixed), ("odd", odd)):
        for top_k, top_p, temp in ((None, 0.9, 0.7), (None, 0.999, 1.0), (None, 0.3, 1.5), (5000, 0.95, 0.7),
                                   (100000, None, 1.0), (None, None, 1.0)):
            tok = sample(logits, top_k=top_k, top_p=top_p, temperature=temp, seed=21, step=4)
            assert torch.equal(tok.cpu(), _cpu(logits, top_k, top_p, temp, 21, 4)), (name, top_k, top_p, temp)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("vocab", [7, 1000, 50257, 140001])
def test_sampler_16_bit_rows_without_top_k(cuda_device, dtype, vocab):
    """One histogram of counts per key serves the search and the draw. Odd vocabularies (rows that
    are not 16-byte aligned), one value in more than 65535 places (a counter overflows), values in
    every corner of the format (more groups than the table holds), and nothing but -inf."""
    g = torch.Generator(device=cuda_device).manual_seed(vocab)
    logits = torch.randn(6, vocab, device=cuda_device, generator=g) * 2
    logits[1] = 1.5
    logits[2] = -logits[2].abs()
    logits[3, : vocab // 2] = 0.25
    logits = logits.to(dtype)
    bits = torch.randint(-2 ** 15, 2 ** 15, (vocab,), device=cuda_device, generator=g).to(torch.int16)
    wild = bits.view(dtype)
    logits[4] = torch.where(torch.isinf(wild), torch.zeros_like(wild), wild)
    logits[5] = float("-inf")
    for top_k, top_p, temp in ((None, 0.9, 0.7), (None, None, 1.0), (None, 0.05, 1.0), (3000, 0.95, 0.7)):
        for step in (0, 1):
            tok = sample(logits, top_k=top_k, top_p=top_p, temperature=temp, seed=5, step=step)
            assert torch.equal(tok.cpu(), _cpu(logits, top_k, top_p, temp, 5, step)), (top_k, top_p, temp)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32, torch.float16])
@pytest.mark.parametrize("vocab", [3, 1025, 33001])
def test_sampler_without_small_top_k_special_values(cuda_device, dtype, vocab):
    """Draws over all elements, and over what a top-p or a large top-k keeps: thresholds close to the
    maximum and far below it (masses from the table, and computed), rows that start off a 16-byte
    boundary, masses of 2^32 by rounding, nothing that has a mass."""
    g = torch.Generator(device=cuda_device).manual_seed(vocab)
    x = torch.randn(4, vocab, device=cuda_device, generator=g) * 2
    u = torch.rand(x.shape, device=cuda_device, generator=g)
    values = {"plain": x, "wide": x * 10, "below_zero": -x.abs() - 1, "masked": torch.where(u < 0.99, float("-inf"), x),
              "lowest": torch.where(u < 0.9, torch.finfo(dtype).min, x), "tiny": x * 1e-6, "zeros": (x * 0).where(u < 0.7, -1.0),
              "inf": torch.where(u > 0.999, float("inf"), x), "nan": torch.where(u < 0.01, float("nan"), x),
              "all_masked": torch.full_like(x, float("-inf"))}
    buf = torch.empty(4 * (vocab + 1) + 3, dtype=dtype, device=cuda_device)
    for name, val in values.items():
        for off, width in ((0, vocab), (3, vocab + 1)):
            logits = buf[off:off + 4 * width].view(4, width)[:, :vocab]
            logits.copy_(val)
            for top_k, top_p, temperature in ((None, None, 0.7), (None, 0.9, 1.0), (None, 0.9999, 2.0), (1500, 0.8, 1.0),
                                              (1500, None, 0.3)):
                k = None if top_k is not None and top_k >= vocab else top_k
                tok = sample(logits, top_k=k, top_p=top_p, temperature=temperature, seed=8, step=off)
                ref = _cpu(logits, k, top_p, temperature, 8, off)
                assert torch.equal(tok.cpu(), ref), (name, off, k, top_p)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("vocab", [1025, 33001, 140001])
def test_sampler_nan_patterns(cuda_device, dtype, vocab):
    """NaNs of every bit pattern and both signs are one key, the lowest: among plain values, as most of a
    row (more of them than a 16-bit counter holds, too), below a maximum next to their own patterns, alone."""
    g = torch.Generator(device=cuda_device).manual_seed(vocab)
    x = torch.randn(4, vocab, device=cuda_device, generator=g) * 2
    u = torch.rand(x.shape, device=cuda_device, generator=g)
    inf = torch.tensor(float("inf"), dtype=dtype).view(torch.int16).item()
    nan = (torch.randint(inf + 1, 0x8000, x.shape, device=cuda_device, generator=g) -
           0x8000 * torch.randint(0, 2, x.shape, device=cuda_device, generator=g)).to(torch.int16).view(dtype)
    assert nan.isnan().all()
    low = torch.full_like(x, torch.finfo(dtype).min).to(dtype)
    low.view(torch.int16)[:, ::3] -= 40               # 40 steps above the lowest value
    x = x.to(dtype)
    for name, val in {"few": torch.where(u < 0.01, nan, x), "most": torch.where(u < 0.9, nan, x),
                      "masked": torch.where(u < 0.3, nan, torch.where(u < 0.9, float("-inf"), x)),
                      "lowest": torch.where(u < 0.5, nan, low), "one_left": torch.where(u < u.max(), nan, x),
                      "all": nan}.items():
        for top_k, top_p, temperature in ((None, 0.9, 1.0), (None, 0.9999, 2.0), (1024, 0.8, 1.0), (1100, None, 0.3),
                                          (20000, 0.99, 1.0), (None, 0.5, 1e30)):
            k = None if top_k is not None and top_k >= vocab else top_k
            tok = sample(val, top_k=k, top_p=top_p, temperature=temperature, seed=6, step=3)
            assert torch.equal(tok.cpu(), _cpu(val, k, top_p, temperature, 6, 3)), (name, k, top_p, temperature)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("vocab,rows", [(1000, 3), (4088, 3), (4104, 3), (50257, 2), (128256, 2), (200064, 2), (128256, 80)])
def test_sampler_candidates_in_few_places(cuda_device, dtype, vocab, rows):
    """Bounds from the warps' keys that are far too low for a part of a row (few finite elements in it, its
    largest in a few warps, none at all) and more candidates than fit: by the hundred and by the thousand."""
    g = torch.Generator(device=cuda_device).manual_seed(vocab)
    x = torch.randn(rows, vocab, device=cuda_device, generator=g) * 2
    u = torch.rand(x.shape, device=cuda_device, generator=g)
    at = torch.arange(vocab, device=cuda_device)
    few = torch.where(u < 1 - 130 / vocab, float("-inf"), x)
    values = {"few_finite": few, "fewer": torch.where(u < 1 - 30 / vocab, float("-inf"), x),
              "one": torch.where(at == vocab // 3, 1.0, torch.full_like(x, float("-inf"))),
              "first_half": torch.where(at < vocab // 2, x, float("-inf")), "last": torch.where(at < vocab - 300, float("-inf"), x),
              "sorted": x.sort(1, descending=True).values, "rising": x.sort(1).values, "equal": torch.ones_like(x),
              "two_values": (u < 0.3).float(), "nan": torch.where(few.isinf(), float("nan"), few)}
    for name, val in values.items():
        val = val.to(dtype)
        for top_k, top_p in ((1, None), (20, 0.9), (50, None), (64, 0.8), (65, 0.9), (200, None), (257, 0.9), (600, 0.95)):
            tok = sample(val, top_k=top_k, top_p=top_p, temperature=0.7, seed=2, step=top_k)
            assert torch.equal(tok[:3].cpu(), _cpu(val[:3], top_k, top_p, 0.7, 2, top_k)), (name, top_k, top_p)


@pytest.mark.parametrize("top_k,top_p,temperature", [(None, 0.9, 1.0), (None, None, 0.7), (2000, 0.95, 1.0), (None, 0.9, 40.0),
                                                     (3000, None, 1e-3), (None, 0.6, 1e30)])
@pytest.mark.parametrize("vocab,rows", [(31, 150), (49155, 3), (33001, 30), (50003, 74), (8193, 300), (131075, 2), (65541, 180),
                                        (50003, 60), (131000, 230), (131201, 230)])
def test_sampler_bf16_parts_of_a_row(cuda_device, vocab, rows, top_k, top_p, temperature):
    """bf16 rows without a small top-k: one to eight CTAs per row (on 148 SMs (50003, 74) stays with the one that takes whole
    rows), rows that start off a 16-byte boundary, counters close to their limit (one value, 131000 columns) and rows that take
    more CTAs because of it, and values inside and outside the magnitudes that are counted at first: plain, far above and
    below them, next to zero, zeros of both signs, one value throughout, masked three ways, thresholds among negative values
    and among values next to zero."""
    g = torch.Generator(device=cuda_device).manual_seed(vocab + rows)
    x = torch.randn(rows, vocab, device=cuda_device, generator=g) * 2
    u = torch.rand(x.shape, device=cuda_device, generator=g)
    at = torch.arange(vocab, device=cuda_device)
    values = {"plain": x, "negative": x - 20, "above": x * 8 + 3000, "below": x * 8 - 5000, "wide": x * 2000, "tiny": x * 1e-18,
              "few_tiny": torch.where(u < 0.01, x * 1e-18, x), "zeros": torch.where(u < 0.5, 0.0, -0.0),
              "half_zero": torch.where(u < 0.5, 0.0, x), "one_value": torch.full_like(x, 3.0),
              "inf_mask": torch.where(u < 0.99, float("-inf"), x), "lowest": torch.where(u < 0.9, torch.finfo(torch.bfloat16).min, x),
              "mask_1e4": torch.where(u < 0.9, -1e4, x), "nan": torch.where(u < 0.1, float("nan"), x),
              "all_nan": torch.full_like(x, float("nan")), "all_inf": torch.full_like(x, float("-inf")),
              "plus_inf": torch.where(u > 0.999, float("inf"), x), "one_tiny": torch.where(at == vocab // 2, 1e-18, x),
              "half_tiny": torch.where(u < 0.5, x * 1e-18, x), "tiny_above": torch.where(u < 0.5, x.abs() * 1e-18, -x.abs()),
              "tiny_below": torch.where(u < 0.9, -x.abs() * 1e-12, x), "subnormal": x * 1e-39,
              "next_to_zero": torch.where(u < 0.3, 0.0, torch.where(u < 0.6, -0.0, x * 10 ** (-40 * u))),
              "small": x * 1e-6, "late": torch.where(at == vocab - 2, 3e12, x), "minus": -x.abs() - 3e9,
              "inf_and_nan": torch.where(u < 0.5, float("nan"), torch.where(u < 0.9, float("-inf"), float("inf")))}
    buf = torch.empty(rows * (vocab + 1) + 3, dtype=torch.bfloat16, device=cuda_device)
    some = torch.arange(0, rows, max(1, rows // 3))[:4]
    for name, val in values.items():
        for off, width in ((0, vocab), (3, vocab + 1)):
            logits = buf[off:off + rows * width].view(rows, width)[:, :vocab]
            logits.copy_(val)
            tok = sample(logits, top_k=top_k, top_p=top_p, temperature=temperature, seed=5, step=1).cpu()
            ref = _cpu(logits[some.to(cuda_device)], top_k, top_p, temperature, 5, 1, row_ids=some)
            assert torch.equal(tok[some], ref), (name, off)
            alone = sample(logits[:2], top_k=top_k, top_p=top_p, temperature=temperature, seed=5, step=1)
            assert torch.equal(alone.cpu(), tok[:2]), (name, off)
