"""GPU: double joins on a device with little memory left.

The exact form's request buffer (64 requests of 16 bytes per window) shrinks to
what fits, the cells past its end going to the FP64 kernel, and where one of its
other buffers does not fit the join runs without it.  Each join runs in a process
of its own that holds the device's memory but for a stated rest: enough for the
FP64 kernels' buffers, too little for the exact form's.  The results are those of
the same join with the memory free.
"""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = """
import sys
sys.path.insert(0, sys.argv[1])
import numpy as np, torch, scamp_gb300
kind, n, m, k, mib = sys.argv[2], *map(int, sys.argv[3:])
rng = np.random.default_rng(n)
x = np.cumsum(rng.standard_normal(n))

def join(y):
    if kind == "1nn":
        r = scamp_gb300.join(y, None, m, precision="double")["profile_a"]
    else:
        r = scamp_gb300.join(y, None, m, "ALL_NEIGHBORS", "double", threshold=0.5,
                             max_matches=k)["knn_a"]
    return scamp_gb300.unpack_profile(r)

join(x[:4000])                            # the kernels are loaded
torch.zeros(1, device="cuda")
free = torch.cuda.mem_get_info()[0]
held = torch.empty(free - (mib << 20), dtype=torch.uint8, device="cuda")
got = join(x)
del held
torch.cuda.empty_cache()
want = join(x)
assert np.max(np.abs(got[0].astype(np.float64) - want[0])) <= 2e-7  # float32 of the same r
assert np.mean(got[1] != want[1]) <= 1e-4                           # equal r aside
print("same")
"""


@pytest.mark.parametrize("kind,n,m,k,mib", [
    ("1nn", 1 << 19, 128, 0, 256),   # 512 MiB of requests
    ("knn", 1 << 16, 128, 64, 96)])  # three lists of 32 MiB and requests
def test_little_memory(gpu_engine, kind, n, m, k, mib):
    pytest.importorskip("torch")
    r = subprocess.run([sys.executable, "-c", CHILD, os.path.join(ROOT, "gpu-scrimp-large_gb300"),
                        kind, str(n), str(m), str(k), str(mib)],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stdout + r.stderr


def test_requests_do_not_depend_on_earlier_joins(gpu_engine):
    """A join verifies what is worth it at its size, whatever buffer an earlier
    join has left: a square wave (no bound separates its cells) asks for all it
    may."""
    a = (np.arange(60000) // 25 % 2).astype(float)

    def verified():
        return gpu_engine.join(a, None, 256, precision="double")["counters"]["verifications"]

    before = verified()
    gpu_engine.join(np.cumsum(np.random.default_rng(1).standard_normal(1 << 18)), None, 64,
                    precision="double")
    assert 0 < before and verified() <= 1.2 * before
