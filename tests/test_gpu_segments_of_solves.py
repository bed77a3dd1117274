"""The cut of the rows into segments, per solve: beyond a wave of blocks a cut for the FP64 iteration and one for the FP32
one, and a new cut of the rows that are left once problems have finished.  A solution's true residual, from the exported
matrix, is the solver's own criterion."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    g.build()
    return g.import_package()


def matrix(H, pr):
    """The trace matrix and right-hand side of one problem alone, after apply!."""
    mesh = H.rectangle_mesh(H.TriangleCell, (pr.n, pr.n), (0.0, 0.0), (1.0, 1.0))
    if pr.jitter:
        mesh.jitter(pr.jitter, pr.seed)
    fe = H.GenericFiniteElement(H.Dubiner(2, H.RefTetrahedron, pr.p))
    Wh, Vh = H.ScalarFunctionSpace(mesh, fe, quad_degree=pr.qd()), H.VectorFunctionSpace(mesh, fe, quad_degree=pr.qd())
    Mh = H.ScalarTraceFunctionSpace(Wh, H.GenericFiniteElement(H.Legendre(1, H.RefTetrahedron, pr.p)))
    K, b, _, _ = H.doassemble(Vh, Wh, Mh, 1.0, pr.f)
    H.apply_(K, b, H.Dirichlet(H.TrialFunction(Mh), mesh, "boundary"))
    return K.to_scipy()


# rows beyond 1216 segments of 1024 in two problems or more (one alone with Jacobi may take the resident iteration): a large
# one beside a small one, which finishes early; several of one size and small ones; a total just above the limit
@pytest.mark.parametrize("shapes", [[(400, 2), (5, 2)], [(300, 1), (300, 1), (300, 1), (300, 1), (20, 1), (7, 1)],
                                    [(330, 2), (130, 2), (16, 2)]])
@pytest.mark.parametrize("pc,prec", [("jacobi", "fp64"), ("jacobi", "mixed"), ("amg", "fp64"), ("amg", "mixed")])
def test_true_residuals(H, shapes, pc, prec):
    tol = 1e-4 if pc == "jacobi" else 1e-9
    probs = [H.Problem(n=n, p=p, f=H.MANUFACTURED_F, jitter=0.2, seed=k) for k, (n, p) in enumerate(shapes)]
    B = H.Batch(H.default_context(), probs, precision=H.PREC_MIXED if prec == "mixed" else H.PREC_FP64)
    for again in range(2):  # the second solve starts from the restored table
        st = B.solve(tol=tol, preconditioner=H.PRECOND_AMG if pc == "amg" else H.PRECOND_JACOBI)
        assert all(s.converged for s in st)
        its = [s.iterations for s in st]
        if again:
            assert its == first
        first = its
    for pr, sol in zip(probs, B.solutions()):
        K, b = matrix(H, pr)
        # FP64 stops on the recursive residual, which is the true one to rounding (well below tol here)
        assert np.linalg.norm(b - K @ sol[0]) <= 1.01 * tol * np.linalg.norm(b)


def test_the_precision_of_a_solve_picks_the_cut(H):
    """One system solved in turn by iterations with different cuts: each solve repeats to the bit."""
    probs = [H.Problem(n=400, p=2, f=H.MANUFACTURED_F, jitter=0.2, seed=1), H.Problem(n=9, p=2, f=H.MANUFACTURED_F)]
    B = H.Batch(H.default_context(), probs, precision=H.PREC_MIXED)
    seen = {}
    for pc in ("jacobi", "amg", "jacobi", "amg"):
        B.solve(tol=1e-4, preconditioner=H.PRECOND_AMG if pc == "amg" else H.PRECOND_JACOBI)
        x = np.concatenate([s[0] for s in B.solutions()])
        if pc in seen:
            assert np.array_equal(seen[pc], x)
        seen[pc] = x
