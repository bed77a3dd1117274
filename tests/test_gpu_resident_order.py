"""The resident CG iterations as a cooperative grid: every CTA forms the same scalars from the others' partials, whatever
the order in which they arrive, so a solve repeated many times gives the same bits after the same iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    g.build()
    return g.import_package()


# few rows to a CTA (the partials arrive close together), and more than one launch of iterations
@pytest.mark.parametrize("n,p,prec", [(8, 1, "fp64"), (8, 1, "mixed"), (70, 1, "fp64"), (60, 2, "mixed")])
def test_repeated_solves_give_the_same_bits(H, monkeypatch, n, p, prec):
    monkeypatch.setenv("HDG_CG_RESIDENT", "grid")
    mesh = H.rectangle_mesh(H.TriangleCell, (n, n), (0.0, 0.0), (1.0, 1.0))
    fe = H.GenericFiniteElement(H.Dubiner(2, H.RefTetrahedron, p))
    Wh, Vh = H.ScalarFunctionSpace(mesh, fe), H.VectorFunctionSpace(mesh, fe)
    Mh = H.ScalarTraceFunctionSpace(Wh, H.GenericFiniteElement(H.Legendre(1, H.RefTetrahedron, p)))
    K, b, _, _ = H.doassemble(Vh, Wh, Mh, 1.0, H.Field.sinsin(3.0, 1.3, 0.7))
    H.apply_(K, b, H.Dirichlet(H.TrialFunction(Mh), mesh, "boundary"))
    precision = H.PREC_MIXED if prec == "mixed" else H.PREC_FP64
    first = H.solve(K, tol=1e-11, precision=precision)
    its = K.stats.iterations
    for _ in range(20):
        assert np.array_equal(first, H.solve(K, tol=1e-11, precision=precision))
        assert K.stats.iterations == its
