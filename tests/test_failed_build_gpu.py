"""An index whose first query runs out of device memory at any of its
allocations answers the next query correctly: nothing half built is kept."""
import numpy as np
import pytest

import oracle
from mlxlearn_b200.index import build_index

pytestmark = pytest.mark.gpu


# 9,000 rows: grouped rows (pivots, the row sort) and grouped queries
@pytest.mark.parametrize("d,mode,k", [(24, "bf16", 5), (6, "bf16", 20), (24, "tf32", 5)])
def test_query_after_a_failed_first_query(monkeypatch, d, mode, k):
    rng = np.random.default_rng(d)
    X = rng.standard_normal((9000, d)).astype(np.float32)
    Q = rng.standard_normal((2100, d)).astype(np.float32)
    ed, ei = oracle.knn(X, Q, k)
    for nth in range(1, 100):
        index = build_index(X)
        index._ensure_device()
        monkeypatch.setenv("B2K_FAULT", f"alloc:{nth}")
        try:
            index.query(Q, k, mode=mode)
        except MemoryError:
            failed = True
        else:
            failed = False
        monkeypatch.delenv("B2K_FAULT")
        dist, idx = index.query(Q, k, mode=mode)
        assert np.array_equal(idx, ei), nth
        assert np.array_equal(dist, ed), nth
        index.close()
        if not failed:
            break
    assert 8 <= nth < 99  # every allocation of the call has failed once
