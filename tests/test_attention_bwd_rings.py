"""The barrier protocol of the attention backward kernels with a ring of its own for every streamed operand
(dQ: K and V; dK / dV: Q and dO), run through every interleaving on the CPU by the explorer of
``test_attention_bwd_barriers``."""
import pytest

import test_attention_bwd_barriers as model


def _parties(kernel, n, bars):
    tma, mma, warp = [], [], []

    def load(kind, j):
        if kind.replace("full", "empty") in bars and j >= bars[kind]:
            tma.append(("wait", kind.replace("full", "empty"), j - bars[kind]))
        tma.append(("load", [(kind, j)]))

    if kernel == "CtlDq":
        for kind in ("qdo_full", "kv_full", "do_full"):
            load(kind, 0)
        for j in range(n):
            load("v_full", j)
            if j + 1 < n:
                load("kv_full", j + 1)
        mma += [("wait", "qdo_full", 0), ("wait", "kv_full", 0), ("mma", [("s_full", 0)]), ("wait", "do_full", 0),
                ("wait", "v_full", 0), ("mma", [("dp_full", 0), ("v_empty", 0)])]
    else:
        for kind in ("kv_full", "qdo_full", "v_full", "do_full"):
            load(kind, 0)
        for j in range(1, n):
            load("do_full", j)
            load("qdo_full", j)
        mma += [("wait", "kv_full", 0), ("wait", "qdo_full", 0), ("mma", [("st_full", 0)]), ("wait", "v_full", 0),
                ("wait", "do_full", 0), ("mma", [("dp_full", 0)])]
    for j in range(n):
        last = [("acc_full", 0)] if j + 1 == n else []
        if kernel == "CtlDq":
            if j + 1 < n:
                mma += [("wait", "kv_full", j + 1), ("mma", [("s_full", j + 1)]), ("wait", "v_full", j + 1),
                        ("wait", "dp_read", j), ("mma", [("dp_full", j + 1), ("v_empty", j + 1)])]
            mma += [("wait", "ds_full", j), ("mma", [("kv_empty", j)] + last)]
            warp += [("wait", "s_full", j), ("wait", "dp_full", j), ("arrive", "dp_read", j), ("arrive", "ds_full", j)]
        else:
            mma += [("wait", "p_full", j), ("mma", [("do_empty", j)])]
            if j + 1 < n:
                mma += [("wait", "qdo_full", j + 1), ("mma", [("st_full", j + 1)]), ("wait", "do_full", j + 1),
                        ("wait", "dp_read", j), ("mma", [("dp_full", j + 1)])]
            mma += [("wait", "ds_full", j), ("mma", [("ds_empty", j), ("qdo_empty", j)] + last)]
            warp += [("arrive", "join", j), ("wait", "join", j), ("wait", "st_full", j), ("arrive", "p_full", j),
                     ("wait", "dp_full", j), ("arrive", "dp_read", j)]
            warp += [("wait", "ds_empty", j - 1)] if j else []
            warp.append(("arrive", "ds_full", j))
    warp.append(("wait", "acc_full", 0))
    return tma, mma, warp


@pytest.mark.parametrize("kernel", ["CtlDq", "CtlDkv"])
@pytest.mark.parametrize("tiles", [1, 2, 3, 4, 7])
def test_every_interleaving_comes_to_its_end(kernel, tiles, monkeypatch):
    monkeypatch.setattr(model, "_parties", _parties)
    assert model._explore(kernel, tiles, model._barriers(kernel)) is None


def test_the_model_sees_a_stage_that_is_handed_back_by_nobody(monkeypatch):
    def forgets(kernel, n, bars):
        tma, mma, warp = _parties(kernel, n, bars)
        return tma, [(op, [e for e in ev if e[0] != "v_empty"]) if op == "mma" else (op, ev, *j) for op, ev, *j in mma], warp

    monkeypatch.setattr(model, "_parties", forgets)
    assert "stuck" in model._explore("CtlDq", 4, model._barriers("CtlDq"))
