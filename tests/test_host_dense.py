"""The host's dense Rayleigh-Ritz (vectorised over contiguous elements) at sizes around its blocks of 8 rows."""
import numpy as np
import pytest


@pytest.mark.parametrize("scale", [1.0, 1e-141])
@pytest.mark.parametrize("m", [1, 2, 3, 7, 8, 9, 16, 17, 24, 63])
def test_rayleigh_ritz_sizes(ks, m, scale):
    """Every pair of a well-conditioned pencil against scipy, also with A so small that the squares of its rotations
    come near underflow. Bounds: the decomposition is backward stable, so the Ritz values are off by at most a small multiple of
    m eps |A| cond(B); cond(B) <= 3 here, and 50 m eps leaves room for the two reductions and the QL sweeps."""
    from scipy.linalg import eigh
    rng = np.random.default_rng(m)
    x = rng.standard_normal((m, m))
    a = (x + x.T) * scale
    q, _ = np.linalg.qr(rng.standard_normal((m, m)))
    b = q @ np.diag(np.linspace(1.0, 3.0, m)) @ q.T
    b = (b + b.T) / 2
    theta, c, _ = ks.rayleigh_ritz(a, b, m)
    tol = 50 * m * np.finfo(float).eps * 3
    norm = np.abs(np.linalg.eigvalsh(a / scale)).max()
    assert np.abs(theta / scale - eigh(a / scale, b, eigvals_only=True)).max() < tol * norm
    assert np.abs(c.T @ b @ c - np.eye(m)).max() < tol
    r = (a / scale) @ c - b @ c * (theta / scale)
    assert np.abs(r).max() < 3 * tol * norm
