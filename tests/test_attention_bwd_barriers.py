"""The barrier protocol of the attention backward kernels, run through every interleaving on the CPU.

An mbarrier is waited for by the parity of a phase, so a waiter that is overtaken by two phases sees
the parity it started from and waits on. The model holds what each party of a CTA waits for and
arrives at, per tile; how many barriers of a kind there are is read from the kernel's source (barrier
``j % n`` serves tile ``j``, with parity ``j / n``). Every reachable state must let somebody move, and
no wait may end before the phase it is meant for.
"""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "csrc", "sm100", "attention_bwd.cu")
WARPS = 2       # element-wise warps: two are enough for one to be ahead of the other


def _barriers(struct):
    with open(SRC) as f:
        body = re.search(r"struct %s \{(.*?)\n\};" % struct, f.read(), re.S).group(1)
    out = {}
    for decl in re.findall(r"uint64_t ([^;]+);", body):
        for name, n in re.findall(r"(\w+)(?:\[(\d)\])?", decl):
            out[name] = int(n or 1)
    return out


def _parties(kernel, n, bars):
    """Programs of the TMA thread, the MMA thread and a warp. ('wait', kind, j): the phase of tile j;
    ('load' / 'mma', [(kind, j)...]): asynchronous, arrives when done; ('arrive', kind, j)."""
    tma, mma, warp = [], [], []
    stage, kept = ("kv", "qdo") if kernel == "CtlDq" else ("qdo", "kv")
    s_full = "s_full" if kernel == "CtlDq" else "st_full"
    tma.append(("load", [(kept + "_full", 0)]))
    for j in range(n):
        if j >= bars[stage + "_empty"]:
            tma.append(("wait", stage + "_empty", j - bars[stage + "_empty"]))
        tma.append(("load", [(stage + "_full", j)]))
    mma += [("wait", kept + "_full", 0), ("wait", stage + "_full", 0), ("mma", [(s_full, 0)]), ("mma", [("dp_full", 0)])]
    for j in range(n):
        if kernel == "CtlDkv":
            mma += [("wait", "p_full", j), ("mma", [])]
        if j + 1 < n:
            mma += [("wait", stage + "_full", j + 1), ("mma", [(s_full, j + 1)]), ("wait", "dp_read", j),
                    ("mma", [("dp_full", j + 1)])]
        done = [("ds_empty", j)] if kernel == "CtlDkv" else []
        mma += [("wait", "ds_full", j), ("mma", done + [(stage + "_empty", j)] + ([("acc_full", 0)] if j + 1 == n else []))]
        if kernel == "CtlDkv":
            warp += [("arrive", "join", j), ("wait", "join", j)]
        warp.append(("wait", s_full, j))
        if kernel == "CtlDkv":
            warp.append(("arrive", "p_full", j))
        warp += [("wait", "dp_full", j), ("arrive", "dp_read", j)]
        if kernel == "CtlDkv" and j > 0:
            warp.append(("wait", "ds_empty", j - 1))
        warp.append(("arrive", "ds_full", j))
    warp.append(("wait", "acc_full", 0))
    return tma, mma, warp


def _explore(kernel, n, bars):
    """None, or what goes wrong in some interleaving."""
    tma, mma, warp = _parties(kernel, n, bars)
    bars = dict(bars, join=1 << 20)        # the named barrier counts, it has no parity to miss
    loads = [op[1] for op in tma if op[0] == "load"]
    mmas = [op[1] for op in mma if op[0] == "mma"]
    per_warp = {k for op, k, *_ in warp if op == "arrive"}

    def prefix(events):                    # arrivals per barrier after the first i events
        out = [{}]
        for arrivals in events:
            cur = dict(out[-1])
            for kind, j in arrivals:
                cur[kind, j % bars[kind]] = cur.get((kind, j % bars[kind]), 0) + 1
            out.append(cur)
        return out

    load_arr, mma_arr = prefix(loads), prefix(mmas)
    warp_arr = prefix([[op[1:]] if op[0] == "arrive" else [] for op in warp])
    load_cnt, mma_cnt = ([sum(op[0] == k for op in prog[:i]) for i in range(len(prog) + 1)]
                         for k, prog in (("load", tma), ("mma", mma)))
    progs = [tma, mma] + [warp] * WARPS
    start = (0,) * (2 + len(progs))        # loads done, products done, program counters
    seen, todo = {start}, [start]
    while todo:
        state = todo.pop()
        ld, mm, pcs = state[0], state[1], state[2:]

        def phases(kind, j):
            key = (kind, j % bars[kind])
            total = load_arr[ld].get(key, 0) + mma_arr[mm].get(key, 0) + sum(warp_arr[pc].get(key, 0) for pc in pcs[2:])
            return total // (WARPS if kind in per_warp else 1)

        nxt = []
        if ld < load_cnt[pcs[0]]:
            nxt.append((ld + 1, mm) + pcs)
        if mm < mma_cnt[pcs[1]]:
            nxt.append((ld, mm + 1) + pcs)
        for a, prog in enumerate(progs):
            if pcs[a] == len(prog):
                continue
            op = prog[pcs[a]]
            if op[0] == "wait":
                phase, done = op[2] // bars[op[1]], phases(*op[1:])
                if done % 2 == phase % 2:  # the barrier is in a phase of the awaited parity: not over yet
                    continue
                if done <= phase:
                    return f"{kernel}: the wait for {op[1]} of tile {op[2]} ends early"
            nxt.append((ld, mm) + pcs[:a] + (pcs[a] + 1,) + pcs[a + 1:])
        if not nxt and any(pc < len(p) for pc, p in zip(pcs, progs)):
            return f"{kernel}: stuck at " + ", ".join(str(p[pc]) for pc, p in zip(pcs, progs) if pc < len(p))
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


@pytest.mark.parametrize("kernel", ["CtlDq", "CtlDkv"])
@pytest.mark.parametrize("tiles", [1, 2, 3, 6])
def test_every_interleaving_of_a_cta_comes_to_its_end(kernel, tiles):
    assert _explore(kernel, tiles, _barriers(kernel)) is None


def test_the_model_sees_a_phase_that_is_overtaken():
    """One barrier for dS of dQ's tiles is not enough: its writers may finish the next tile before
    the thread that issues the products has looked."""
    bars = dict(_barriers("CtlDq"), ds_full=1)
    assert "stuck" in _explore("CtlDq", 3, bars)
