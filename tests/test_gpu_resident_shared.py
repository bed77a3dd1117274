"""The resident CG iteration as a grid over the whole chip is for a solve that is alone: solves that share the chip overlap
as launched iterations, which is faster for them all."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    g.build()
    return g.import_package()


def problem(H, n, p, seed):
    rng = np.random.default_rng(seed)
    f = H.Field.bumps(rng.random((4, 2)), 0.05 + 0.1 * rng.random(4), rng.standard_normal(4))
    return H.Problem(n=n, p=p, f=f, jitter=0.2, seed=seed)


def solve(H, probs, prec, tol=1e-8):
    """Solutions, iterations, kernel launches of a batch's second step."""
    B = H.Batch(H.default_context(), probs, precision=prec)
    B.solve(tol=tol)
    before = H.default_context().launches()
    st = B.solve(tol=tol)
    n = H.default_context().launches() - before
    assert all(s.converged for s in st)
    return [np.concatenate([np.ravel(a) for a in s]) for s in B.solutions()], [s.iterations for s in st], n


# a launched iteration is two launches, a resident one 1/512
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_which_batches_take_the_grid(H, prec):
    precision = H.PREC_MIXED if prec == "mixed" else H.PREC_FP64
    four = [problem(H, 64, p, p) for p in (1, 2, 3, 4)]  # each beyond a cluster's rows
    sol, its, n = solve(H, four, precision)
    assert n > 2 * max(its)
    for pr, x, k in zip(four, sol, its):  # alone: the grid
        one, own, m = solve(H, [pr], precision)
        assert m < own[0]
        # both stop at 1e-8; cond(K) is below 1e5 (64 x 64 squares, kappa = 1)
        assert np.linalg.norm(one[0] - x) <= 2e-3 * np.linalg.norm(x)
    # one beside a cluster: the grid
    _, its, n = solve(H, [problem(H, 96, 4, 1), problem(H, 24, 2, 2)], precision)
    assert n < min(its)


def test_solves_from_several_threads(H):
    results, errors = {}, []

    def work(k):
        try:
            ctx = H.Context(0)
            B = H.Batch(ctx, [problem(H, 64, 2, 7)], precision=H.PREC_FP64)
            for _ in range(3):
                assert B.solve(tol=1e-8)[0].converged
            results[k] = np.concatenate([np.ravel(a) for a in B.solutions()[0]])
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors and len(results) == 6
    for x in results.values():
        assert np.linalg.norm(x - results[0]) <= 2e-3 * np.linalg.norm(results[0])


def test_requests_one_at_a_time_and_together(H):
    probs = [problem(H, 64, 2, k) for k in range(6)]
    want = [solve(H, [pr], H.PREC_FP64)[0][0] for pr in probs]
    for max_batch in (1, 32):
        eng = H.Engine(H.default_context(), tol=1e-8, precision=H.PREC_FP64, max_batch=max_batch)
        for together in (False, True):
            ids = []
            for pr in probs:
                ids.append(eng.submit(pr.p, pr.f, mesh=H.batch.host_mesh(pr), quad_degree=pr.qd()))
                if not together:
                    eng.run_until_idle()
            eng.run_until_idle()
            for i, x in zip(ids, want):
                got = np.concatenate([np.ravel(v) for v in eng.result(i)])
                assert np.linalg.norm(got - x) <= 2e-3 * np.linalg.norm(x)
