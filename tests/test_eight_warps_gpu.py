"""The kNN screen with eight epilogue warps (B2K_TC_EW=8, read once a process):
answers agree with the oracle, and whatever pass seeds a row's lists publishes a
threshold that cuts them."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = r"""
import os
import sys
import numpy as np
import oracle
from mlxlearn_b200.index import build_index

k = int(sys.argv[1])
rng = np.random.default_rng(k)
X = rng.standard_normal((17_000, 24)).astype(np.float32)
index = build_index(X)
for m in (200, 2_100):  # queries as they come, and grouped
    Q = rng.standard_normal((m, 24)).astype(np.float32)
    ed, ei = oracle.knn(X, Q, k)
    entries = {}
    for seed in "01":
        os.environ["B2K_SEED"] = seed
        dist, idx = index.query(Q, k, mode="bf16", stats=True)
        assert np.array_equal(idx, ei) and np.array_equal(dist, ed), (m, seed)
        entries[seed] = index.last_stats["list_entries"]
        assert (index.last_stats["seed_ms"] > 0) == (seed == "1" and k > 16)
    if k > 16:
        assert entries["1"] < 0.8 * entries["0"], (m, entries)
"""


@pytest.mark.parametrize("k", [16, 17, 32, 33, 50, 64])
def test_eight_epilogue_warps(k):
    env = dict(os.environ, B2K_TC_EW="8")
    r = subprocess.run([sys.executable, "-c", SCRIPT, str(k)], env=env, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
