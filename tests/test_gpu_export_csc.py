"""The CSC export, column by column on the device and in pieces: against the sum of the element blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    return g.import_package()


# one cell pair, odd and even face counts, and (at 2 million entries to a piece) one piece, several, the last one short
@pytest.mark.parametrize("p,n", [(1, 1), (4, 1), (2, 7), (3, 30), (1, 280), (2, 160), (3, 96), (4, 121)])
@pytest.mark.parametrize("base", [0, 1])
def test_csc_export_is_the_sum_of_the_element_blocks(H, p, n, base):
    import scipy.sparse as sp
    mesh = H.rectangle_mesh(H.TriangleCell, (n, n), (0.0, 0.0), (1.0, 1.0))
    qd = {1: 2, 2: 3, 3: 6, 4: 9}[p]
    fe = H.GenericFiniteElement(H.Dubiner(2, H.RefTetrahedron, p))
    Wh, Vh = H.ScalarFunctionSpace(mesh, fe, quad_degree=qd), H.VectorFunctionSpace(mesh, fe, quad_degree=qd)
    Mh = H.ScalarTraceFunctionSpace(Wh, H.GenericFiniteElement(H.Legendre(1, H.RefTetrahedron, p)))
    S = H.doassemble(Vh, Wh, Mh, 1.0, H.MANUFACTURED_F)[0]
    colptr, rowval, nzval, rhs = S.csc(base)
    assert colptr[0] == base and colptr[-1] == S.nnz + base
    At, bt, _, _ = S.element_blocks()
    cf = mesh._topology()[2]
    cf = cf - cf.min()
    nt, m = p + 1, 3 * (p + 1)
    d = (cf[:, :, None] * nt + np.arange(nt)).reshape(len(cf), m)
    K = sp.coo_matrix((At.ravel(), (np.repeat(d, m, axis=1).ravel(), np.tile(d, (1, m)).ravel())),
                      shape=(S.ndofs, S.ndofs)).tocsc()
    K.sort_indices()
    np.testing.assert_array_equal(colptr - base, K.indptr)
    np.testing.assert_array_equal(rowval - base, K.indices)
    np.testing.assert_allclose(nzval, K.data, rtol=0, atol=4 * 2.0 ** -53 * np.abs(At).max())
    b = np.bincount(d.ravel(), bt.ravel(), S.ndofs)
    np.testing.assert_allclose(rhs, b, rtol=0, atol=4 * 2.0 ** -53 * np.abs(bt).max())
    L = H._lib
    only = np.full(S.nnz, 7.0)  # any array may be left out
    L.check(L.load().hdg_system_get_csc(S._h, base, None, None, L.dptr(only), None), S.ctx)
    np.testing.assert_array_equal(only, nzval)
