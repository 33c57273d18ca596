"""Segment lists of unequal length: reference segments may be left over, query
segments may not."""
import numpy as np
import pytest
import torch


def test_query_segment_without_reference_segment():
    from mlxlearn_b200.autograd import _segments_forward

    with pytest.raises(ValueError, match="reference segment"):
        _segments_forward(torch.zeros(5, 3), torch.zeros(4, 3), (2, 3), (4,), 1, False)


@pytest.mark.gpu
@pytest.mark.parametrize("x_sizes", [(40, 30, 1, 7), (40, 38)])
def test_left_over_reference_segments(x_sizes):
    import oracle
    from mlxlearn_b200.autograd import knn_segments

    rng = np.random.default_rng(0)
    X = rng.standard_normal((sum(x_sizes), 3)).astype(np.float32)
    Q = rng.standard_normal((25, 3)).astype(np.float32)
    Qt = torch.from_numpy(Q).cuda().requires_grad_()
    Xt = torch.from_numpy(X).cuda().requires_grad_()
    dist, idx = knn_segments(Qt, Xt, (20, 5), x_sizes, 2)
    dist.sum().backward()
    for q, x in ((slice(0, 20), slice(0, 40)), (slice(20, 25), slice(40, 40 + x_sizes[1]))):
        assert np.array_equal(idx[q].cpu().numpy(), oracle.knn(X[x], Q[q], 2)[1])
    assert not Xt.grad[40 + x_sizes[1]:].any()


@pytest.mark.gpu
def test_no_segments():
    from mlxlearn_b200.autograd import knn_segments

    dist, idx = knn_segments(torch.zeros(0, 3, device="cuda"), torch.zeros(0, 3, device="cuda"),
                             (), (), 1)
    assert dist.shape == idx.shape == (0, 1)
