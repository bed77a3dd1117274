"""The continuous-Galerkin CG with its vectors resident on the chip against the one with two kernels per iteration.

Both stop at a relative residual of 1e-12; the stiffness matrices here have cond(K) < 1e4 after Jacobi's scaling (grids up
to 40 x 40, kappa within a decade), so the solutions differ by less than 2e-8 of the norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOUND = 2e-8


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    g.build()
    return g.import_package()


def system(H, n, order, f, kappa=None):
    mesh = H.rectangle_mesh(H.TriangleCell, (n, n), (0.0, 0.0), (1.0, 1.0))
    mesh.jitter(0.2, 9)
    Wh = H.ScalarFunctionSpace(mesh, H.ContinuousLagrange(2, H.RefTetrahedron, order), update_face_data=False)
    u_h = H.TrialFunction(Wh)
    dh = H.DofHandler([u_h], mesh)
    K, b = H.doassemble_cg(Wh, H.create_sparsity_pattern(dh), dh, f, kappa_cell=kappa)
    H.apply_(K, b, H.Dirichlet(u_h, dh, "boundary", lambda x: x[0]))
    return K


# 4 dofs (CTAs without a row), rows around a multiple of the CTAs and of a slice, more rows than threads in a CTA
@pytest.mark.parametrize("kind", ["cluster", "grid"])
@pytest.mark.parametrize("n,order", [(1, 1), (1, 2), (3, 1), (6, 2), (21, 1), (40, 2)])
def test_resident_iteration_matches_the_launched_one(H, monkeypatch, kind, n, order):
    rng = np.random.default_rng(n)
    kappa = np.exp(rng.uniform(-1.1, 1.1, 2 * n * n))
    f = H.Field.bumps(rng.random((3, 2)), 0.2, [1.0, -2.0, 0.5])
    sol = {}
    for k in ("none", kind):
        monkeypatch.setenv("HDG_CG_RESIDENT", k)  # taken when the system is created
        K = system(H, n, order, f, kappa)
        sol[k] = H.solve(K, tol=1e-12)
        assert K.stats.converged
        assert np.array_equal(sol[k], H.solve(K, tol=1e-12))  # bit-identical when repeated
    assert np.linalg.norm(sol[kind] - sol["none"]) <= BOUND * np.linalg.norm(sol["none"])


@pytest.mark.parametrize("kind", ["none", "cluster", "grid"])
def test_cap_and_zero_right_hand_side(H, monkeypatch, kind):
    monkeypatch.setenv("HDG_CG_RESIDENT", kind)
    K = system(H, 12, 2, H.Field.const(1.0))
    with pytest.raises(H.HDGError) as e:
        H.solve(K, tol=1e-12, maxit=5)
    assert e.value.code == -5 and K.handle if hasattr(K, "handle") else e.value.code == -5
    assert np.isfinite(H.solve(K, tol=1e-12)).all() and K.stats.converged
    mesh = K.mesh
    Wh = H.ScalarFunctionSpace(mesh, H.ContinuousLagrange(2, H.RefTetrahedron, 1), update_face_data=False)
    u_h = H.TrialFunction(Wh)
    dh = H.DofHandler([u_h], mesh)
    Z, b = H.doassemble_cg(Wh, H.create_sparsity_pattern(dh), dh, H.Field.const(0.0))
    H.apply_(Z, b, H.Dirichlet(u_h, dh, "boundary", lambda x: 0.0))
    assert not H.solve(Z).any() and Z.stats.iterations == 0 and Z.stats.converged
