"""The hot kernels at the sizes where their tiling can go wrong (edges of tiles and pieces, remainders, the smallest
and largest of a range), against f64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U = 2.0 ** -24  # f32 rounding unit


def f32(a):
    return np.asarray(a, dtype=np.float32).astype(np.float64)


@pytest.mark.parametrize("n,k", [(5, 1), (13, 3), (13, 8), (13, 9), (13, 21), (33, 4), (33, 21)])
def test_block_update_over_solves(ks, oracle, n, k):
    """out_j = sum_i C_ij S_i through whole LOBPCG solves: q = 2k outputs below, at and above the groups of 8 (2 .. 42),
    m up to 63 inputs, fields of one partial slice (n = 5), of fewer slices than SMs (13) and of more (33). The block must
    stay orthonormal, and the updated H X consistent with X (the residual recomputed in f64 from X alone).
    Bounds: a combination of m <= 63 fields is one f32 fmaf chain, off by at most m U per unit vector; H amplifies the
    rounding of X by its norm, at most 3 * 205/72 * 16/9 / (2 h^2) * 2 + max V."""
    h = 0.4 if n > 5 else 0.8
    x, y, z = oracle.grid_points(n, h)
    v = f32(0.5 * (x * x + 1.1 * y * y + 1.3 * z * z))
    rng = np.random.default_rng(n + k)
    guess = rng.uniform(-0.5, 0.5, (k, n ** 3)) * np.exp(-(x * x + y * y + z * z) / 8.0)
    tol = 1e-3
    ev, xs, it, mr = ks.lobpcg(n, h, v, guess, tol=tol, max_iter=400)
    assert mr <= tol, (it, mr)
    gm = xs @ xs.T * h ** 3
    d = 1.0 / np.sqrt(gm.diagonal())
    assert np.abs(gm * np.outer(d, d) - np.eye(k)).max() < 8 * 63 * U
    hnorm = 3 * 205 / 72 * 16 / 9 / h ** 2 + v.max()
    for i in range(k):
        r = oracle.hamiltonian(n, h, xs[i], v) - ev[i] * xs[i]
        assert np.sqrt((r * r).sum() / (xs[i] * xs[i]).sum()) < tol * max(1.0, abs(ev[i])) + 63 * U * hnorm, (i, it)
