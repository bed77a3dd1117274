"""Recovery of systems whose outputs are staged in several pieces of 32 MB: every cell's values, whichever arrays are
asked for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    g.build()
    return g.import_package()


# 480 bytes a cell at p = 4: a piece is 69905 cells; 72200 and 142578 cells are two and three pieces, 2 x 187^2 is within one
@pytest.mark.parametrize("n,p", [(187, 4), (190, 4), (267, 4), (300, 1)])
def test_every_piece(H, n, p):
    L = H._lib
    B = H.Batch(H.default_context(), [H.Problem(n=n, p=p, f=H.MANUFACTURED_F, jitter=0.2, seed=2)])
    assert B.solve(tol=1e-3, preconditioner=H.PRECOND_AMG)[0].converged
    b = B.bins[0]
    uhat, q, u = b.solution()[0]  # from [q; u] as the device holds it
    nc, nw, nt = b.mesh.ncells, b.nw, b.nt
    trace = uhat.reshape(-1, nt)[b.mesh._topology()[2] - 1]  # cells x 3 x nt
    for ask in ((1, 1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1), (0, 1, 1)):
        for by_function in (0, 1):
            got = [np.full(s, np.nan) for s in ((nc, 2 * nw), (nc, nw), (nc, nt, 3) if by_function else (nc, 3, nt))]
            L.check(L.load().hdg_recover_into(b.h, *[L.dptr(a) if on else None for a, on in zip(got, ask)], by_function),
                    H.default_context().handle)
            for a, want, on in zip(got, (q, u, trace.transpose(0, 2, 1) if by_function else trace), ask):
                assert np.array_equal(a, want) if on else np.isnan(a).all()
