"""Launches whose static and dynamic shared memory exceed the default 48 KB
together but not each alone, each in a process of its own (an earlier launch
with more would leave the kernel's limit raised); and launches of one kernel
with different amounts from several host threads."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

COUNTS = """
import sys
import numpy as np
from oracle import oracle as O
from trajsimimeasures_b200 import datagen as D, engine
m, n, longest = sys.argv[1], int(sys.argv[2]), int(sys.argv[3])
rng = np.random.Generator(np.random.PCG64(9))
pts, off, lens = D._walks(rng, np.r_[rng.integers(1, 7, n - 1), longest], 2e-4)
s = engine.TrajSet.from_packed(pts, off, lens)
_, cnt = engine.matrix(m, s, s, eps=3e-2)
ia = np.r_[rng.integers(0, n, 4000), np.full(n, n - 1), np.arange(n)]
ib = np.r_[rng.integers(0, n, 4000), np.arange(n), np.full(n, n - 1)]
want = O.pairs_idx(O.pairs_f32, {"edr": 1, "lcss": 2}[m], pts, off, lens, ia, ib, eps=3e-2)[1]
assert np.array_equal(cnt.cpu().numpy()[ia, ib], want)
print("EQUAL")
"""


@pytest.mark.parametrize("measure", ["edr", "lcss"])
@pytest.mark.parametrize("n,longest", [(9, 1100), (1000, 500), (2000, 280)])
def test_counts_between_the_two_limits(measure, n, longest):
    r = subprocess.run([sys.executable, "-c", COUNTS, measure, str(n), str(longest)], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "EQUAL" in r.stdout, r.stderr


@pytest.mark.parametrize("measure", ["dtw", "hausdorff"])
def test_host_threads_do_not_lower_each_others_limit(measure):
    import threading

    import numpy as np
    import torch
    from trajsimimeasures_b200 import datagen as D, engine
    rng = np.random.Generator(np.random.PCG64(10))
    sets = [engine.TrajSet.from_packed(*D._walks(rng, np.r_[2, 3, longest], 2e-4)) for longest in (700, 1400, 1000, 900)]
    outs = [torch.empty((3, 3), dtype=torch.float32, device="cuda") for _ in sets]
    failed = []

    def work(s, out, stream):
        try:
            for _ in range(3000):
                engine.matrix_raw(measure, s, s, out=out, stream=stream)
            stream.synchronize()
        except Exception as e:  # noqa: BLE001 (reported by the test)
            failed.append(str(e))
    for s in sets:
        s.order_by_length()
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(s, o, torch.cuda.Stream())) for s, o in zip(sets, outs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed
