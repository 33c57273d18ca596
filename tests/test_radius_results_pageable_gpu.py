"""What the radius estimators return is ordinary host memory: an array that a
program keeps pins nothing."""
import numpy as np
import pytest

from mlxlearn_b200.neighbors import RadiusNeighborsClassifier, RadiusNeighborsRegressor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weights", ["uniform", "distance"])
def test_probabilities_and_means_are_not_page_locked(weights):
    import torch

    rng = np.random.default_rng(3)
    X = rng.standard_normal((3000, 8)).astype(np.float32)
    y = rng.integers(0, 4, 3000)
    Q = rng.standard_normal((500, 8)).astype(np.float32)
    kind = dict(radius=2.5, weights=weights)
    model = RadiusNeighborsClassifier(outlier_label="most_frequent", **kind).fit(X, y)
    proba = model.predict_proba(Q)
    means = RadiusNeighborsRegressor(**kind).fit(X, X[:, 0]).predict(Q)
    for a in (proba, means):
        while a.base is not None and isinstance(a.base, np.ndarray):
            a = a.base
        assert not torch.from_numpy(a).is_pinned()
    assert np.allclose(proba.sum(1), 1.0)
