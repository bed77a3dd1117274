"""Recovery into the TrialFunctions' own arrays: the values of hdg_recover, whatever array the caller put there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    g.build()
    return g.import_package()


@pytest.mark.parametrize("n,p", [(1, 1), (3, 2), (7, 3), (4, 4)])
@pytest.mark.parametrize("form", ["own", "fortran", "float32"])
def test_get_usigma_fills_the_callers_arrays(H, n, p, form):
    mesh = H.rectangle_mesh(H.TriangleCell, (n, n), (0.0, 0.0), (1.0, 1.0))
    fe = H.GenericFiniteElement(H.Dubiner(2, H.RefTetrahedron, p))
    qd = {1: 2, 2: 3, 3: 6, 4: 9}[p]
    Wh, Vh = H.ScalarFunctionSpace(mesh, fe, quad_degree=qd), H.VectorFunctionSpace(mesh, fe, quad_degree=qd)
    Mh = H.ScalarTraceFunctionSpace(Wh, H.GenericFiniteElement(H.Legendre(1, H.RefTetrahedron, p)))
    K, b, K_e, b_e = H.doassemble(Vh, Wh, Mh, 1.0, H.MANUFACTURED_F)
    H.apply_(K, b, H.Dirichlet(H.TrialFunction(Mh), mesh, "boundary"))
    uhat = H.solve(K, b)
    q, u, uc = K.recover()
    fns = [H.TrialFunction(V) for V in (Vh, Wh, Mh)]
    for t in fns:
        if form == "fortran":
            t.m_values = np.asfortranarray(t.m_values)
        elif form == "float32":
            t.m_values = t.m_values.astype(np.float32)
    held = [t.m_values for t in fns]
    H.get_usigma_(*fns, uhat, K_e, b_e, mesh)
    for t, before, want in zip(fns, held, (q, u, np.transpose(uc, (0, 2, 1)))):
        assert t.m_values is before  # filled in place
        assert np.array_equal(t.m_values, want.astype(before.dtype))
    cf = mesh._topology()[2] - 1  # the trace values are the faces' own
    nt = p + 1
    assert np.array_equal(uc, uhat.reshape(-1, nt)[cf])
