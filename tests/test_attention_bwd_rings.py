"""The barrier protocol of the attention backward kernel, a persistent CTA that takes one tile after the other with a ring
for every streamed operand, run through every interleaving on the CPU. A CTA of its own per tile is the case of one tile.

An mbarrier is waited for by the parity of a phase, so a waiter that is overtaken by two phases sees the parity it started
from and waits on. The model holds what each party of a CTA waits for and arrives at; how many barriers of a kind there are is
read from the kernel's source (barrier ``j % n`` serves number ``j``, with parity ``j / n``). Every reachable state must let
somebody move, and no wait may end before the phase it is meant for.
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


def _bars(kernel):
    return dict(_barriers(kernel), item_full=2, item_empty=2, join=1 << 20)   # the named barrier has no parity to miss


def _programs(kernel, sizes, bars):
    """Programs of the loading thread, the issuing thread and the element-wise warps for tiles of the given numbers of
    streamed tiles. ('async', [(kind, j)...]): arrives some time later, in the thread's order."""
    tma, mma, warp = [], [], []

    def load(kind, j):
        empty = kind.replace("full", "empty")
        if empty in bars and j >= bars[kind]:
            tma.append(("wait", empty, j - bars[kind]))
        tma.append(("async", [(kind, j)]))

    def stationary(full, free, i):
        if i:
            tma.append(("wait", free, i - 1))
        tma.append(("async", [(full, i)]))

    def item(i):
        if i > 1:
            tma.append(("wait", "item_empty", i - 2))
        tma.append(("arrive", "item_full", i))
        for p in (mma, warp):
            p.extend([("wait", "item_full", i), ("arrive", "item_empty", i)])
        if kernel == "CtlDkv":
            warp.extend([("arrive", "join", len(warp)), ("wait", "join", len(warp))])

    g = 0
    for i, n in enumerate(sizes):
        item(i)
        last = lambda j, kind: [(kind, i)] if j + 1 == n else []   # noqa: E731, B023
        if kernel == "CtlDq":
            stationary("qdo_full", "q_free", i)
            load("kv_full", g)
            stationary("do_full", "do_free", i)
            s = lambda j: [("wait", "kv_full", g + j), ("async", [("s_full", g + j)] + last(j, "q_free"))]   # noqa: E731, B023
            dp = lambda j: ("async", [("dp_full", g + j), ("v_empty", g + j)] + last(j, "do_free"))   # noqa: E731, B023
            mma += [("wait", "qdo_full", i)] + s(0) + [("wait", "do_full", i), ("wait", "v_full", g), dp(0)]
            for j in range(n):
                load("v_full", g + j)
                if j + 1 < n:
                    load("kv_full", g + j + 1)
                    mma += s(j + 1) + [("wait", "v_full", g + j + 1), ("wait", "dp_read", g + j), dp(j + 1)]
                mma += [("wait", "ds_full", g + j), ("async", [("kv_empty", g + j)] + last(j, "acc_full"))]
                warp += [("wait", "s_full", g + j), ("wait", "dp_full", g + j), ("arrive", "dp_read", g + j),
                         ("arrive", "ds_full", g + j)]
        else:
            stationary("kv_full", "k_free", i)
            load("qdo_full", g)
            stationary("v_full", "v_free", i)
            load("do_full", g)
            for j in range(1, n):
                load("do_full", g + j)
                load("qdo_full", g + j)
            s = lambda j: [("wait", "qdo_full", g + j), ("async", [("st_full", g + j)] + last(j, "k_free"))]   # noqa: E731, B023
            dp = lambda j: ("async", [("dp_full", g + j)] + last(j, "v_free"))   # noqa: E731, B023
            mma += [("wait", "kv_full", i)] + s(0) + [("wait", "v_full", i), ("wait", "do_full", g), dp(0)]
            for j in range(n):
                mma += [("wait", "p_full", g + j), ("async", [("do_empty", g + j)])]
                if j + 1 < n:
                    mma += s(j + 1) + [("wait", "do_full", g + j + 1), ("wait", "dp_read", g + j), dp(j + 1)]
                mma += [("wait", "ds_full", g + j), ("async", [("ds_empty", g + j), ("qdo_empty", g + j)] + last(j, "acc_full"))]
                warp += [("arrive", "join", len(warp)), ("wait", "join", len(warp)), ("wait", "st_full", g + j),
                         ("arrive", "p_full", g + j), ("wait", "dp_full", g + j), ("arrive", "dp_read", g + j)]
                warp += [("wait", "ds_empty", g + j - 1)] if g + j else []
                warp.append(("arrive", "ds_full", g + j))
        warp.append(("wait", "acc_full", i))
        g += n
    item(len(sizes))           # there is none any more
    if kernel == "CtlDkv":
        tma.append(("wait", "k_free", len(sizes) - 1))
    return [tma, mma] + [warp] * WARPS


def _explore(kernel, bars, progs):
    """None, or what goes wrong in some interleaving."""
    count = {op[1]: WARPS for op in progs[-1] if op[0] == "arrive"}
    count["item_empty"] = WARPS + 1
    issued = [[sum(op[0] == "async" for op in p[:i]) for i in range(len(p) + 1)] for p in progs]

    def prefix(lists):                     # arrivals per barrier after the first i of them
        out = [{}]
        for arrivals in lists:
            cur = dict(out[-1])
            for kind, j in arrivals:
                cur[kind, j % bars[kind]] = cur.get((kind, j % bars[kind]), 0) + 1
            out.append(cur)
        return out

    done_arr = [prefix([op[1] for op in p if op[0] == "async"]) for p in progs]
    warp_arr = [prefix([[op[1:]] if op[0] == "arrive" else [] for op in p]) for p in progs]
    start = ((0,) * len(progs), (0,) * len(progs))
    seen, todo = {start}, [start]
    while todo:
        done, pcs = todo.pop()

        def phases(kind, j):
            key = (kind, j % bars[kind])
            return sum(done_arr[a][done[a]].get(key, 0) + warp_arr[a][pcs[a]].get(key, 0)
                       for a in range(len(progs))) // count.get(kind, 1)

        nxt = []
        for a, prog in enumerate(progs):
            if done[a] < issued[a][pcs[a]]:
                nxt.append((done[:a] + (done[a] + 1,) + done[a + 1:], pcs))
            if pcs[a] == len(prog):
                continue
            op = prog[pcs[a]]
            if op[0] == "wait":
                phase, over = op[2] // bars[op[1]], phases(*op[1:])
                if over % 2 == phase % 2:  # the barrier is in a phase of the awaited parity: not over yet
                    continue
                if over <= phase:
                    return f"{kernel}: the wait for {op[1]} of tile {op[2]} ends early"
            nxt.append((done, pcs[:a] + (pcs[a] + 1,) + pcs[a + 1:]))
        if not nxt and any(pc < len(p) for pc, p in zip(pcs, progs)):
            return f"{kernel}: stuck at " + ", ".join(str(p[pc]) for pc, p in zip(pcs, progs) if pc < len(p))
        for s in nxt:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


@pytest.mark.parametrize("kernel,sizes", [("CtlDq", (1,)), ("CtlDq", (4,)), ("CtlDq", (2, 1, 2)), ("CtlDq", (1, 1, 1, 1)),
                                          ("CtlDkv", (1,)), ("CtlDkv", (3,)), ("CtlDkv", (2, 1, 1)), ("CtlDkv", (1, 1, 1, 1))])
def test_every_interleaving_comes_to_its_end(kernel, sizes):
    bars = _bars(kernel)
    assert _explore(kernel, bars, _programs(kernel, sizes, bars)) is None


def test_the_model_sees_a_phase_that_is_overtaken_and_a_tile_that_nobody_frees():
    bars = _bars("CtlDq")
    one = dict(bars, ds_full=1)
    assert "stuck" in _explore("CtlDq", one, _programs("CtlDq", (4,), one))
    progs = _programs("CtlDq", (2, 2), bars)
    progs[1] = [(op, [e for e in ev if e[0] != "q_free"]) if op == "async" else (op, ev, *j) for op, ev, *j in progs[1]]
    assert "stuck" in _explore("CtlDq", bars, progs)
