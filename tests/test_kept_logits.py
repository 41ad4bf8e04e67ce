"""The allowance for logits that calls with gradients keep (host side; the kernels are in test_gpu_logp.py)."""
import subprocess
import sys
import textwrap

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
