"""Trace systems whose rows are cut into one wave of long segments: FP64 and mixed ones, alone and as an uneven batch."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    return g.import_package()


# rows beyond 1216 segments of 1024: one problem; a large one beside small ones
@pytest.mark.parametrize("shapes", [[(400, 2)], [(400, 2), (5, 2), (33, 2), (60, 2)], [(330, 4), (3, 4)]])
def test_precisions_and_single_solves_agree(H, shapes):
    probs = [H.Problem(n=n, p=p, f=H.MANUFACTURED_F, jitter=0.2, seed=k) for k, (n, p) in enumerate(shapes)]
    sols = []
    for prec in (H.PREC_FP64, H.PREC_MIXED):
        B = H.Batch(H.default_context(), probs, precision=prec)
        assert all(s.converged for s in B.solve(tol=1e-11, preconditioner=H.PRECOND_AMG))
        sols.append([np.concatenate([np.ravel(a) for a in sol]) for sol in B.solutions()])
    for pr, a, b in zip(probs, *sols):
        assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(a)
        alone = H.Batch(H.default_context(), [pr])
        assert alone.solve(tol=1e-11, preconditioner=H.PRECOND_AMG)[0].converged
        c = np.concatenate([np.ravel(x) for x in alone.solutions()[0]])
        assert np.linalg.norm(a - c) <= 1e-8 * np.linalg.norm(a)
