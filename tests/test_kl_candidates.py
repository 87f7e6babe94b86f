"""Which eigenvalue products a K-term expansion looks at: with every axis's
eigenvalues not increasing, the K largest products in the reference's order
(repeated first-maximum search: by value, equal ones by linear index) are among
those with (m + 1)(n + 1)(k + 1) <= K."""
import numpy as np
import pytest


def _largest(prod, K):
    return np.argsort(-prod, kind="stable")[:K]


@pytest.mark.parametrize("ndim", (2, 3))
@pytest.mark.parametrize("K", (1, 2, 3, 7, 16, 40))
@pytest.mark.parametrize("kind", ("smooth", "steps", "equal axes", "rounding ties"))
def test_pruned_candidates_give_the_same_terms(ndim, K, kind):
    rng = np.random.default_rng(K)
    w = np.cumsum(rng.random((K, 3)) + 0.1, axis=0)
    lam = 4.0 * 0.7 / (4.0 + w * w * 0.49)
    if kind == "steps":                       # runs of equal eigenvalues
        lam = np.ceil(lam * 4.0) / 4.0
    elif kind == "equal axes":
        lam[:, 1] = lam[:, 2] = lam[:, 0]
    elif kind == "rounding ties":             # neighbours an ulp apart: products round together
        lam = 1.0 - np.arange(K)[:, None] * np.finfo(float).eps / 2 * np.ones(3)
    shape = (K,) * ndim
    idx = np.indices(shape).reshape(ndim, -1)
    prod = lam[idx[0], 0] * lam[idx[1], 1]
    if ndim == 3:
        prod = prod * lam[idx[2], 2]
    linear = np.arange(prod.size)
    keep = np.prod(idx + 1, axis=0) <= K
    all_terms = _largest(prod, K)
    pruned = linear[keep][_largest(prod[keep], K)]
    assert np.array_equal(all_terms, pruned)
