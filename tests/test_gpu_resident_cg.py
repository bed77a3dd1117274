"""The Jacobi CG iteration that keeps its state on the chip (one launch per many iterations) against the one with two
kernels per iteration, on the same systems.

Both stop at a relative residual of tol, so each solution is within cond(K) tol of the system's; the trace systems
here have cond(K) < 1e4 (grids up to 64 x 64, kappa = 1, or 16 x 16 with kappa within a decade), so with tol = 1e-12 the
two differ by less than 2e-8 of the norm, whatever the order of their sums."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOUND = 2e-8


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    g.build()
    return g.import_package()


def system(H, n, p, kappa=None):
    mesh = H.rectangle_mesh(H.TriangleCell, (n, n), (0.0, 0.0), (1.0, 1.0))
    fe = H.GenericFiniteElement(H.Dubiner(2, H.RefTetrahedron, p))
    qd = {1: 2, 2: 3, 3: 6, 4: 9}[p]
    Wh, Vh = H.ScalarFunctionSpace(mesh, fe, quad_degree=qd), H.VectorFunctionSpace(mesh, fe, quad_degree=qd)
    Mh = H.ScalarTraceFunctionSpace(Wh, H.GenericFiniteElement(H.Legendre(1, H.RefTetrahedron, p)))
    K, b, _, _ = H.doassemble(Vh, Wh, Mh, 1.0, H.Field.sinsin(3.0, 1.3, 0.7), kappa_cell=kappa)
    H.apply_(K, b, H.Dirichlet(H.TrialFunction(Mh), mesh, "boundary"))
    return K


# one square (most CTAs own no face), sizes around a multiple of the CTAs, more rows than threads, more than 512
# iterations (several launches)
@pytest.mark.parametrize("kind", ["cluster", "grid"])
@pytest.mark.parametrize("n,p", [(1, 1), (1, 4), (3, 2), (5, 3), (16, 4), (33, 1), (64, 1), (40, 2)])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_resident_iteration_matches_the_launched_one(H, monkeypatch, kind, n, p, prec):
    rng = np.random.default_rng(n * 10 + p)
    K = system(H, n, p, np.exp(rng.uniform(-1.1, 1.1, 2 * n * n)) if n == 16 else None)
    precision = H.PREC_MIXED if prec == "mixed" else H.PREC_FP64
    sol = {}
    for k in ("none", kind, kind):
        monkeypatch.setenv("HDG_CG_RESIDENT", k)
        x = H.solve(K, tol=1e-12, precision=precision)
        assert K.stats.converged
        if k in sol:
            assert np.array_equal(sol[k], x)  # repeated solves are bit-identical
        sol[k] = x
    scale = np.linalg.norm(sol["none"])
    assert np.linalg.norm(sol[kind] - sol["none"]) <= BOUND * scale


@pytest.mark.parametrize("kind", ["cluster", "grid"])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_resident_iteration_stops_at_the_cap(H, monkeypatch, kind, prec):
    K = system(H, 20, 2)
    monkeypatch.setenv("HDG_CG_RESIDENT", kind)
    with pytest.raises(H.HDGError) as e:
        H.solve(K, tol=1e-12, maxit=7, precision=H.PREC_MIXED if prec == "mixed" else H.PREC_FP64)
    assert e.value.code == -5 and K.handle
    x = H.solve(K, tol=1e-12)  # the system stays usable
    assert K.stats.converged and np.isfinite(x).all()
