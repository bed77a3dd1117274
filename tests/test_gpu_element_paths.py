"""The element kernels that condense through the Schur complement, several cells per warp, against the pivoted
elimination of the whole local system (HDG_ELEMENT_FULL_LU), on the same cells.

Both are held to 1e-12 of the largest entry of a cell's block against the exact blocks elsewhere, so here they may
differ by 2e-12 of it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOUND = 2e-12


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    g.build()
    return g.import_package()


def blocks(H, mesh, p, qd, f, tau=1.3, he_tau=False, **kappa):
    fe = H.GenericFiniteElement(H.Dubiner(2, H.RefTetrahedron, p))
    Wh, Vh = H.ScalarFunctionSpace(mesh, fe, quad_degree=qd), H.VectorFunctionSpace(mesh, fe, quad_degree=qd)
    Mh = H.ScalarTraceFunctionSpace(Wh, H.GenericFiniteElement(H.Legendre(1, H.RefTetrahedron, p)))
    K, _, _, _ = H.doassemble(Vh, Wh, Mh, tau, f, he_tau=he_tau, **kappa)
    return K.element_blocks()


def source(H, kind, rng):
    if kind == "sinsin":
        return H.Field.sinsin(2.0, 1.7, 0.6)
    if kind == "bumps":
        k = int(rng.integers(1, 10))  # fewer and more terms than lanes share a point
        return H.Field.bumps(rng.random((k, 2)), 0.05 + 0.2 * rng.random(k), rng.standard_normal(k))
    k = int(rng.integers(1, 40))
    return H.Field.fourier(0.3, rng.uniform(-2, 2, (k, 4)), exponential=kind == "exp_fourier")


def check(a, b):
    for x, y in zip(a, b):
        axes = tuple(range(1, y.ndim))
        scale = np.abs(y).max(axis=axes, keepdims=True)
        assert np.isfinite(x).all()
        assert (np.abs(x - y) <= BOUND * np.maximum(scale, 1e-300)).all()


# 2 cells (less than one warp takes), 8, 18 and 50 (remainders of the cells per warp), 578
@pytest.mark.parametrize("n", [1, 2, 3, 5, 17])
@pytest.mark.parametrize("p,qd", [(1, 2), (2, 3), (2, 4), (3, 6), (4, 9)])
@pytest.mark.parametrize("kind", ["sinsin", "bumps", "fourier", "exp_fourier"])
def test_schur_blocks_match_full_elimination(H, monkeypatch, n, p, qd, kind):
    rng = np.random.default_rng(100 * n + 10 * p + qd)
    mesh = H.rectangle_mesh(H.TriangleCell, (n, n), (0.0, 0.0), (1.0, 1.0))
    mesh.jitter(0.2, 3)
    f, kappa = source(H, kind, rng), np.exp(rng.uniform(-2.3, 2.3, 2 * n * n))
    kw = dict(kappa_cell=kappa if kind != "sinsin" else None, he_tau=kind == "bumps")
    got = blocks(H, mesh, p, qd, f, **kw)
    monkeypatch.setenv("HDG_ELEMENT_FULL_LU", "1")
    check(got, blocks(H, mesh, p, qd, f, **kw))


# kappa a field: an exponential of modes, one that changes its sign (those cells go to the pivoted kernel), bumps, a
# constant
@pytest.mark.parametrize("n", [1, 3, 5, 17])
@pytest.mark.parametrize("p,qd", [(1, 2), (2, 3), (2, 4), (3, 6)])
@pytest.mark.parametrize("kind", ["exp_fourier", "sign", "bumps", "const"])
def test_field_blocks_match_full_elimination(H, monkeypatch, n, p, qd, kind):
    rng = np.random.default_rng(1000 * n + 10 * p + qd)
    mesh = H.rectangle_mesh(H.TriangleCell, (n, n), (0.0, 0.0), (1.0, 1.0))
    mesh.jitter(0.2, 5)
    modes = np.stack([rng.uniform(-1, 1, 17), rng.uniform(-1, 1, 17), rng.uniform(0, 6, 17), 0.2 * rng.standard_normal(17)], 1)
    kappa = {"exp_fourier": H.Field.fourier(0.1, modes, exponential=True),
             "sign": H.Field.fourier(0.0, [[0.5, 0.0, 0.0, 1.0]]),  # cos(pi x): negative for x > 1/2
             "bumps": H.Field.bumps([[0.4, 0.6], [0.5, 0.5]], [0.3, 3.0], [2.0, 1.0]),
             "const": H.Field.const(0.7)}[kind]
    f = source(H, "fourier", rng)
    got = blocks(H, mesh, p, qd, f, kappa=kappa)
    monkeypatch.setenv("HDG_ELEMENT_FULL_LU", "1")
    want = blocks(H, mesh, p, qd, f, kappa=kappa)
    if kind != "sign":
        check(got, want)
        return
    # a cell whose kappa changes its sign may be close to singular: only the definite ones are held to the bound
    # (x < 0.3: no cell that reaches there touches x = 1/2 from n = 5 on); the others took the same kernel
    xy, cells = H.get_vertices_matrix(mesh), H.getcells_matrix(mesh) - 1
    right = xy[cells][:, :, 0].max(axis=1)
    left = right < 0.45
    check([x[left] for x in got], [x[left] for x in want])
    far = xy[cells][:, :, 0].min(axis=1) > 0.55
    if p != 1:  # one cell per warp there: exactly the cells with a negative value are left to it
        for x, y in zip(got, want):
            assert np.array_equal(x[far], y[far])


# phases that are exact multiples of an eighth, a quarter and a half turn, a phase beyond one turn, a zero amplitude
@pytest.mark.parametrize("n", [2, 4, 10])
@pytest.mark.parametrize("p,qd", [(1, 2), (2, 3), (4, 9)])
@pytest.mark.parametrize("f", ["unit", "quarter", "wrapped", "flat", "far"])
def test_fixed_point_fields_at_special_phases(H, monkeypatch, n, p, qd, f):
    mesh = H.rectangle_mesh(H.TriangleCell, (n, n), (-1.0, -1.0), (1.0, 1.0))
    f = {"unit": H.Field.sinsin(2 * np.pi ** 2, 1.0, 1.0),
         "quarter": H.Field.fourier(0.5, [[1.0, 0.0, np.pi / 2, 1.0], [0.0, 4.0, -np.pi, 2.0], [0.5, 0.5, 0.0, 1.0]]),
         "wrapped": H.Field.fourier(0.0, [[1.0, -2.0, 25.0, 1.0], [3.0, 1.0, -40.0, 0.5]]),
         "flat": H.Field.fourier(1.5, [[0.0, 0.0, 0.3, 0.0]]),
         "far": H.Field.bumps([[0.25, 0.25], [40.0, -3.0]], [0.01, 5.0], [1.0, 1e3])}[f]
    got = blocks(H, mesh, p, qd, f)
    monkeypatch.setenv("HDG_ELEMENT_FULL_LU", "1")
    check(got, blocks(H, mesh, p, qd, f))
