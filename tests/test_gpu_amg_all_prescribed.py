"""Multigrid on systems whose trace is prescribed on every face: the hierarchy has no coarse rows, P0' no entries."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    g.build()
    return g.import_package()


def triangle_files(root, cells):
    """The .node, .edge and .ele files of one triangle of the unit square, or of both."""
    nodes = ["0.0 0.0", "1.0 0.0", "0.0 1.0", "1.0 1.0"][:cells + 2]
    tri = ["1 2 3", "2 4 3"][:cells]
    edges = ["1 2 1", "2 3 %d" % (cells == 1), "3 1 1", "2 4 1", "4 3 1"][:3 if cells == 1 else 5]
    for ext, lines in (("node", nodes), ("ele", tri), ("edge", edges)):
        text = "".join("%d %s\n" % (k + 1, ln) for k, ln in enumerate(lines))
        root.with_suffix("." + ext).write_text("%d 0 0\n" % len(lines) + text)
    return str(root)


# one triangle (all its faces are on the boundary); a square whose diagonal is prescribed too
@pytest.mark.parametrize("cells", [1, 2])
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_the_solution_is_the_prescribed_trace(H, tmp_path, cells, p, prec):
    mesh = H.parse_mesh_triangle(triangle_files(tmp_path / "m", cells))
    fe = H.GenericFiniteElement(H.Dubiner(2, H.RefTetrahedron, p))
    qd = {1: 2, 2: 3, 3: 6, 4: 9}[p]
    Wh, Vh = H.ScalarFunctionSpace(mesh, fe, quad_degree=qd), H.VectorFunctionSpace(mesh, fe, quad_degree=qd)
    Mh = H.ScalarTraceFunctionSpace(Wh, H.GenericFiniteElement(H.Legendre(1, H.RefTetrahedron, p)))
    K, _, _, _ = H.doassemble(Vh, Wh, Mh, 1.0, H.Field.const(1.0))
    want = np.random.default_rng(p).uniform(-1, 1, K.ndofs)
    for again in range(2):  # the second solve keeps the hierarchy
        if again:
            K.reassemble(1.0, H.Field.const(2.0))
        K.apply_dirichlet(np.arange(1, K.ndofs + 1), want)
        got = H.solve(K, tol=1e-12, preconditioner=H.PRECOND_AMG,
                      precision=H.PREC_MIXED if prec == "mixed" else H.PREC_FP64)
        # the matrix is a multiple of the identity: the solver's tolerance and a rounding of the product
        assert np.linalg.norm(got - want) <= 1e-11 * np.linalg.norm(want)
