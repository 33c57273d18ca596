"""Radius rows left unsorted (class counts) hold the sorted rows' entries; every
other nonzero sort flag sorts by distance."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,d", [(1500, 20), (9000, 24), (9000, 5)])
def test_any_order(n, d):
    from mlxlearn_b200 import _lib
    from mlxlearn_b200.index import build_index
    from mlxlearn_b200.radius_result import RadiusCSR

    rng = np.random.default_rng(n + d)
    X, Q = (rng.standard_normal((r, d)).astype(np.float32) for r in (n, 300))
    index = build_index(X)
    handle = index._ensure_device()
    radius = float(np.median(index.query(Q, 20)[0][:, -1]))

    def fetch(flag):
        res = ctypes.c_void_p()
        _lib.check(_lib.load().b2k_radius(handle, Q.ctypes.data, len(Q), radius, 0, 0, 1, flag,
                                          ctypes.byref(res)), "b2k_radius")
        part = RadiusCSR.from_device(res, len(Q), device=0, distances=True)
        return part.indptr, part.indices, part.distances

    ip, ix, dd = fetch(0)
    up, ux, ud = fetch(_lib.RADIUS_ANY_ORDER)
    assert np.array_equal(ip, up)
    for a, b in zip(ip[:-1], ip[1:]):
        order = np.argsort(ux[a:b])
        assert np.array_equal(ux[a:b][order], ix[a:b])
        assert np.array_equal(ud[a:b][order], dd[a:b])
    want = fetch(1)
    for flag in (2, 7, -1):
        assert all(np.array_equal(p, q) for p, q in zip(fetch(flag), want))
    assert any(np.any(np.diff(want[1][a:b]) < 0) for a, b in zip(ip[:-1], ip[1:]))
