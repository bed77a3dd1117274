"""The rows of the condensed blocks: a constant trace is the trace of a constant u without a flux, so a row's entries for
the constants of the three faces add up to (tau' - 1) |e_f| int mu_i, tau' = tau, or to 0 where He carries tau."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    g.build()
    return g.import_package()


# (kappa a field at p = 4 takes the pivoted kernel, whose entries are not tied to each other)
@pytest.mark.parametrize("n", [1, 3, 17])
@pytest.mark.parametrize("p,qd,kappa", [(p, qd, k) for p, qd in ((1, 2), (2, 3), (2, 4), (3, 6), (4, 9))
                                        for k in ("one", "cell", "field") if not (p == 4 and k == "field")])
@pytest.mark.parametrize("tau,he_tau", [(1.0, False), (3.0, True), (3.0, False)])
def test_constants_add_up(H, n, p, qd, kappa, tau, he_tau):
    rng = np.random.default_rng(n + p)
    mesh = H.rectangle_mesh(H.TriangleCell, (n, n), (0.0, 0.0), (1.0, 1.0))
    mesh.jitter(0.2, 3)
    kw = {"one": {}, "cell": dict(kappa_cell=np.exp(rng.uniform(-9, 9, 2 * n * n))),
          "field": dict(kappa=H.Field.fourier(0.1, rng.uniform(-1, 1, (5, 4)), exponential=True))}[kappa]
    fe = H.GenericFiniteElement(H.Dubiner(2, H.RefTetrahedron, p))
    Wh, Vh = H.ScalarFunctionSpace(mesh, fe, quad_degree=qd), H.VectorFunctionSpace(mesh, fe, quad_degree=qd)
    Mh = H.ScalarTraceFunctionSpace(Wh, H.GenericFiniteElement(H.Legendre(1, H.RefTetrahedron, p)))
    Ate = H.doassemble(Vh, Wh, Mh, tau, H.Field.const(1.0), he_tau=he_tau, **kw)[0].element_blocks()[0]
    nt = p + 1
    const = Ate.reshape(-1, 3, nt, 3, nt)[..., 0]  # [cell][f][i][g]
    for f in range(3):
        others = const[:, f, :, (f + 1) % 3] + const[:, f, :, (f + 2) % 3]
        own = const[:, f, :, f]
        assert np.array_equal(Ate, Ate.transpose(0, 2, 1))
        if tau == 1.0 or he_tau:
            assert np.array_equal(own, -others)
            continue
        xy, cells = H.get_vertices_matrix(mesh), H.getcells_matrix(mesh) - 1
        a, b = [(1, 2), (2, 0), (0, 1)][f]
        length = np.linalg.norm(xy[cells[:, a]] - xy[cells[:, b]], axis=1)
        want = np.zeros_like(own)
        want[:, 0] = (tau - 1.0) * length
        # the sum of the others, the length, the product and the integral of mu_i are each to a few roundings
        assert (np.abs(own + others - want) <= 8 * 2.0 ** -52 * (np.abs(others) + want[:, :1])).all()
