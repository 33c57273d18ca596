"""Reference-row gradients of rows picked by very many queries: the sum runs in
ascending pick order and is the same on every run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _fma32(c, e, acc):
    # one rounding of c * e + acc: the product of two fp32 is exact in float64,
    # and the float64 sum is off by at most 2^-53 relative before the rounding
    return (c.astype(np.float64) * e.astype(np.float64) + acc.astype(np.float64)).astype(np.float32)


# bucket sizes around the warp's steps, the warp / block edge (128), the block's
# threads (256) and its stage (2048)
@pytest.mark.parametrize("sizes", [(0, 1, 3, 4, 31, 32, 33, 127, 128, 129), (255, 256, 257, 1000),
                                   (2047, 2048, 2049, 2304, 5000)])
@pytest.mark.parametrize("d", [9, 32, 64, 100, 300])
@pytest.mark.parametrize("squared", [True, False])
def test_big_buckets(sizes, d, squared):
    import torch

    from mlxlearn_b200 import _lib

    rng = np.random.default_rng(len(sizes) + d)
    n, k = len(sizes), 4
    picks = np.repeat(np.arange(n), sizes)
    picks = np.concatenate([picks, np.zeros(-len(picks) % k, np.int64)])
    idx = rng.permutation(picks).reshape(-1, k)
    m = len(idx)
    Q, X = (rng.standard_normal((r, d)).astype(np.float32) for r in (m, n))
    G = rng.standard_normal((m, k)).astype(np.float32)
    E = rng.uniform(0.5, 2.0, (m, k)).astype(np.float32)
    t = {name: torch.from_numpy(a).cuda() for name, a in
         (("Q", Q), ("X", X), ("G", G), ("E", E), ("idx", idx))}
    dX = torch.empty_like(t["X"])
    _lib.check(_lib.load().b2k_knn_backward(
        t["Q"].data_ptr(), m, t["X"].data_ptr(), n, d, k, t["idx"].data_ptr(), t["G"].data_ptr(),
        t["E"].data_ptr(), int(squared), None, dX.data_ptr(),
        torch.cuda.current_stream().cuda_stream), "b2k_knn_backward")
    c = (np.float32(2) * G if squared else G / E).reshape(-1)
    want = np.zeros((n, d), np.float32)
    for pos, row in enumerate(idx.reshape(-1)):
        want[row] = _fma32(c[pos], X[row] - Q[pos // k], want[row])
    got = dX.cpu().numpy()
    # the float64 stand-in for the FMA may double-round: allow one unit in the
    # last place per addition of a bucket, 2^-24 of the magnitudes summed
    size = np.bincount(idx.reshape(-1), minlength=n)[:, None]
    scale = np.abs(c).max() * 12.0
    assert np.all(np.abs(got - want) <= 2.0 ** -24 * scale * np.maximum(size, 1))
    again = torch.empty_like(dX)
    _lib.check(_lib.load().b2k_knn_backward(
        t["Q"].data_ptr(), m, t["X"].data_ptr(), n, d, k, t["idx"].data_ptr(), t["G"].data_ptr(),
        t["E"].data_ptr(), int(squared), None, again.data_ptr(),
        torch.cuda.current_stream().cuda_stream), "b2k_knn_backward")
    assert torch.equal(dX, again)
