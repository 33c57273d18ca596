"""Batches whose screen lists pass their memory budget, or find no memory, are
answered block by block with the same results."""
import os
import subprocess
import sys

import numpy as np
import pytest

import oracle
from mlxlearn_b200.index import build_index

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d,k,mode", [(9000, 24, 20, "bf16"), (9000, 5, 3, "auto"),
                                        (3000, 40, 64, "tf32"), (9000, 24, 20, "fp32"),
                                        (9000, 24, 10, "bf16")])
def test_blocks_agree(monkeypatch, n, d, k, mode):
    rng = np.random.default_rng(n + d)
    X = rng.standard_normal((n, d)).astype(np.float32)
    index = build_index(X)
    whole = index.query(X, k, exclude_self=True, mode=mode, stats=True)
    stats = index.last_stats
    monkeypatch.setenv("B2K_KNN_LIST_MB", "16")
    part = index.query(X, k, exclude_self=True, mode=mode, stats=True)
    for a, b in zip(whole, part):
        assert np.array_equal(a, b)
    assert index.last_stats["mode_used"] == stats["mode_used"]
    ed, ei = oracle.knn(X, X, k, exclude_self=True)
    assert np.array_equal(part[1], ei) and np.array_equal(part[0], ed)


def test_no_memory_for_a_block(monkeypatch):
    """Each allocation of a call fails once: the call answers in smaller blocks."""
    rng = np.random.default_rng(5)
    X = rng.standard_normal((9000, 6)).astype(np.float32)
    Q = rng.standard_normal((20_000, 6)).astype(np.float32)
    index = build_index(X)
    dist, idx = index.query(Q, 20)
    ed, ei = oracle.knn(X, Q, 20)
    assert np.array_equal(idx, ei) and np.array_equal(dist, ed)
    for nth in (4, 5):  # after the three arrays of the host call
        monkeypatch.setenv("B2K_FAULT", f"alloc:{nth}")
        d2, i2 = index.query(Q, 20)
        monkeypatch.delenv("B2K_FAULT")
        index.query(Q[:5], 3)  # restarts the count
        assert np.array_equal(i2, ei) and np.array_equal(d2, ed)
    monkeypatch.setenv("B2K_FAULT", "alloc")
    with pytest.raises(MemoryError):
        index.query(Q, 20)


SCRATCH = r"""
import sys
import torch
from mlxlearn_b200.index import NeighborIndex

d, k, m = map(int, sys.argv[1:])
X = torch.randn(4_000, d, device="cuda")
Q = torch.randn(m, d, device="cuda")
index = NeighborIndex.from_device(X)
index.query_device(Q[:1000], k)
before = torch.cuda.mem_get_info()[0]
index.query_device(Q, k)
torch.cuda.synchronize()
print((before - torch.cuda.mem_get_info()[0]) >> 20)
"""


# (a million queries at one split: 16 GB of lists in one block)
@pytest.mark.parametrize("d,k", [(16, 17), (8, 5)])
def test_scratch_of_a_large_batch_is_bounded(d, k):
    r = subprocess.run([sys.executable, "-c", SCRATCH, str(d), str(k), "1000000"], timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout) < 11_000
