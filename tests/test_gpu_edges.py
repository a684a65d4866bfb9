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


@pytest.mark.parametrize("n,m,mt", [(5, 1, 1), (9, 8, 8), (17, 9, 7), (29, 24, 24), (25, 17, 32), (33, 32, 32), (13, 33, 1), (13, 8, 33), (9, 5, 64), (13, 7, 65), (29, 8, 120),
                                    (25, 12, 40), (25, 20, 60), (17, 40, 8), (21, 60, 60), (33, 33, 33)])
@pytest.mark.parametrize("gram_mode", [0, 1])
def test_gram_pieces_match_f64(ks, n, m, mt, gram_mode):
    """S^T [S | T] with one piece and with several (more than 32 rows or columns), every count of row and column groups of
    8, in both forms. Products of one warp's points are summed in f32, two chains of 16 and then one over its slabs (3 at
    most here), the rest in f64: |error| <= (16 + 1 + 3) U |s| |t| by Cauchy-Schwarz; the tensor cores' 3xTF32 form
    (blocks beyond one piece) keeps 2e-6."""
    if gram_mode == 1 and ((m + 7) // 8 * 8 + mt > 128 or m > 64):
        pytest.skip("beyond the tensor-core form's block")
    rng = np.random.default_rng(m + mt)
    s, t = f32(rng.standard_normal((m, n ** 3))), f32(rng.standard_normal((mt, n ** 3)))
    g = ks.gram(n, s, t, gram_mode=gram_mode)
    st = np.concatenate([s, t])
    scale = np.sqrt(np.outer((s * s).sum(1), (st * st).sum(1)))
    err = (np.abs(g - s @ st.T) / scale).max()
    assert err < (2e-6 if gram_mode == 1 and (m > 32 or mt > 32) else 20 * U), err
    if gram_mode == 0:
        assert np.array_equal(g[:, :m], g[:, :m].T)


@pytest.mark.parametrize("n", [31, 47, 49, 63, 64, 65, 95, 97])
def test_stencil_tile_widths(ks, oracle, n):
    """H psi, the Laplacian and the sweeps just below, at and above the tile widths 32, 48 and 64 and their multiples, for
    one vector and for five, and with every z-chunking (down to one plane per chunk) the same bits. Bounds as the
    kernels' other tests: each output is 24 products of neighbouring differences, 1e-6 of the largest term in f32."""
    h, lam = 0.27, -0.4
    x, y, z = oracle.grid_points(n, h)
    rng = np.random.default_rng(n)
    v = f32(-2 * np.exp(-(x * x + y * y + z * z)))
    psi = f32(np.stack([np.exp(-((x - c) ** 2 + y * y + z * z) / 3) + 1e-3 * rng.uniform(-1, 1, n ** 3) for c in (0.0, 0.4, -0.3, 0.7, 0.2)]))
    try:
        ks.clear_stencil_tuning()
        gpu = ks.apply_hamiltonian(n, h, psi, v)
        for i in (0, 4):
            want = oracle.hamiltonian(n, h, psi[i], v)
            assert np.abs(gpu[i] - want).max() < 1e-6 * (np.abs(want).max() + np.abs(v * psi[i]).max())
        one = ks.apply_hamiltonian(n, h, psi[:1], v)
        assert np.array_equal(one[0], gpu[0])
        for chunks in (1, 2, 7, n // 4, n):
            ks.set_stencil_tuning([(n, 1, 1, chunks)])
            assert np.array_equal(ks.apply_hamiltonian(n, h, psi[:1], v), one), chunks
    finally:
        ks.clear_stencil_tuning()
    lap = oracle.laplacian(n, h, psi[1])
    assert np.abs(ks.apply_laplacian(n, h, psi[1]) - lap).max() < 1e-6 * np.abs(lap).max()
    want = oracle.jacobi_precond(n, h, v, lam, psi[2])
    assert np.abs(ks.apply_precond(n, h, v, lam, psi[2]) - want).max() < 2e-6 * np.abs(want).max()


@pytest.mark.parametrize("n", [5, 11, 12, 13, 24, 25, 26, 33, 52])
def test_poisson_level_edges(ks, oracle, n):
    """The Hartree solve where its multigrid levels change: the whole cycle in one CTA (n <= 12), one level above it (13,
    24, 25), two (26, 33, 52), even and odd sizes. Against the f64 solve, with the f32 floor of the single-grid test
    (2e-5 for a potential of order 1), and in no more iterations than a working V-cycle takes (unpreconditioned
    CG on 26^3 takes above 60)."""
    h = 12.0 / n
    x, y, z = oracle.grid_points(n, h)
    s = max(0.8, h)
    rho = (2 * np.pi * s * s) ** -1.5 * np.exp(-((x - 0.5) ** 2 + (y + 0.3) ** 2 + z * z) / (2 * s * s))
    v, it, res = ks.poisson_solve(n, h, rho, tol=1e-7)
    vo, _, _ = oracle.poisson_solve(n, h, f32(rho), tol=1e-11)
    assert it <= 40, it
    assert np.abs(v - vo).max() < 2e-5 * max(1.0, np.abs(vo).max()), (it, res)


@pytest.mark.parametrize("n,m,mt", [(9, 1, 33), (13, 8, 40), (13, 9, 112), (13, 17, 64), (13, 24, 33), (21, 33, 33), (21, 40, 40), (21, 41, 41),
                                    (21, 48, 48), (13, 49, 1), (13, 49, 72), (21, 56, 56), (21, 57, 57), (13, 64, 64)])
def test_tensor_core_gram_shapes(ks, n, m, mt):
    """Every class of N = round16(m) of the tensor-core form against round8(m), with T blocks up to the largest, one stage
    per CTA and several. Bound: hi holds 11 bits, so the dropped lo lo term is below 2^-20 |s| |t|, over uniform mantissas
    a sixth of that in the mean; the two rounded lo operands add 2^-22 each, the truncating sums of a stage's 12 products at
    most 12 times 2^-24: 1.4e-6 together, under the 2e-6 of the other tests."""
    rng = np.random.default_rng(100 * m + mt)
    s, t = f32(rng.standard_normal((m, n ** 3))), f32(rng.standard_normal((mt, n ** 3)))
    g = ks.gram(n, s, t, gram_mode=1)
    st = np.concatenate([s, t])
    scale = np.sqrt(np.outer((s * s).sum(1), (st * st).sum(1)))
    err = (np.abs(g - s @ st.T) / scale).max()
    assert err < 2e-6, err


@pytest.mark.parametrize("m,mt", [(8, 8), (10, 15), (24, 24), (32, 32)])
def test_mixed_form_of_small_blocks_is_the_plain_form(ks, m, mt):
    """Up to 32 columns the mixed form takes the CUDA cores: the same bits as the plain form."""
    rng = np.random.default_rng(m)
    s, t = rng.standard_normal((m, 13 ** 3)), rng.standard_normal((mt, 13 ** 3))
    assert np.array_equal(ks.gram(13, s, t, gram_mode=1), ks.gram(13, s, t, gram_mode=0))


def gaussian_hartree(ks, n):
    """The Hartree potential of an off-centre Gaussian on a 12 Bohr box: (largest error against erf, iterations)."""
    from scipy.special import erf
    h, s = 12.0 / n, 0.8
    ax = (np.arange(n) - (n - 1) / 2) * h
    r = np.sqrt(((ax - 0.5) ** 2)[None, None, :] + ((ax + 0.3) ** 2)[None, :, None] + (ax ** 2)[:, None, None]).ravel()
    v, it, _ = ks.poisson_solve(n, h, (2 * np.pi * s * s) ** -1.5 * np.exp(-r * r / (2 * s * s)), tol=1e-5)
    return np.abs(v - erf(r / (s * np.sqrt(2))) / r).max(), it


@pytest.mark.parametrize("n", [129, 161])
def test_poisson_partials_beyond_one_sum(ks, n):
    """The Hartree solve on both sides of 2048 CTAs of its last sweep: up to there (128^3 has exactly 2048) the direction
    kernel sums their partial pairs itself, beyond a launch of its own does. Bound of the reference's own check: 1e-4. A
    wrong r.z would cost the conjugacy, so the iterations stay what 128^3 takes, within the two that another set of
    coarse grids may add."""
    err, it = gaussian_hartree(ks, n)
    err128, it128 = gaussian_hartree(ks, 128)
    assert err < 1e-4 and err128 < 1e-4, (err, err128)
    assert abs(it - it128) <= 2, (it, it128)
