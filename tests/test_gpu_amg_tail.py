"""The coarse levels of the V-cycle in one cluster per problem: the bits of one launch per phase."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

_SCRIPT = r"""
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import __graft_entry__ as g
H = g.import_package()
out = {}
# one problem (clusters of 16), a few and many (smaller clusters), with one-level and unequal hierarchies among them
for name, shapes in (("one", [(96, 1)]), ("two", [(3, 4), (60, 3)]), ("nine", [(8 + 9 * k, 1 + k % 2) for k in range(9)]),
                     ("sixteen", [(10 + 5 * k, 1 + k % 2) for k in range(16)]), ("thirty", [(9 + 2 * k, 1) for k in range(30)]),
                     ("forty", [(4 + k, 2) for k in range(40)]), ("many", [(6 + k % 23, 1) for k in range(170)])):
    rng = np.random.default_rng(5)
    probs = [H.Problem(n=n, p=p, f=H.MANUFACTURED_F, jitter=0.2, seed=k,
                       kappa_cell=np.exp(rng.uniform(np.log(1e-2), np.log(1e2), 2 * n * n)) if name != "one" else None)
             for k, (n, p) in enumerate(shapes)]
    B = H.Batch(H.default_context(), probs)
    for again in range(2):  # a second assembly makes the image again
        st = B.solve(tol=1e-9, preconditioner=H.PRECOND_AMG)
    assert all(s.converged for s in st)
    out[name + "_its"] = np.array([s.iterations for s in st])
    for k, sol in enumerate(B.solutions()):
        out[f"{name}_{k}"] = np.concatenate([np.ravel(a) for a in sol])
np.savez(sys.argv[2], **out)
"""


def test_cluster_tail_gives_the_bits_of_the_launches(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    (tmp_path / "s.py").write_text(_SCRIPT)
    got = {}
    for rows in ("0", "65536", "300"):
        env = dict(os.environ, HDG_AMG_TAIL_ROWS=rows, HDG_AMG_SWEEP="face")
        r = subprocess.run([sys.executable, str(tmp_path / "s.py"), root, str(tmp_path / f"{rows}.npz")], env=env,
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        got[rows] = np.load(tmp_path / f"{rows}.npz")
    for rows in ("65536", "300"):
        for k in got["0"].files:
            assert got["0"][k].tobytes() == got[rows][k].tobytes(), (rows, k)


_STREAM = r"""
import sys
import numpy as np
sys.path.insert(0, sys.argv[1])
import __graft_entry__ as g
H = g.import_package()
out = {}
for n, p in ((700, 1), (512, 2), (400, 3), (330, 4)):  # level-0 values of 70 to 85 MB
    B = H.Batch(H.default_context(), [H.Problem(n=n, p=p, f=H.MANUFACTURED_F, jitter=0.2, seed=3)])
    st = B.solve(tol=1e-9, preconditioner=H.PRECOND_AMG)
    assert st[0].converged
    out[f"its{p}"] = np.array([st[0].iterations])
    out[f"u{p}"] = np.concatenate([np.ravel(a) for a in B.solutions()[0]])
np.savez(sys.argv[2], **out)
"""


def test_streamed_level0_gives_the_bits_of_the_rows(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    (tmp_path / "s.py").write_text(_STREAM)
    got = {}
    for sweep in ("face", "row"):
        env = dict(os.environ, HDG_AMG_TAIL_ROWS="0", HDG_AMG_SWEEP=sweep)
        r = subprocess.run([sys.executable, str(tmp_path / "s.py"), root, str(tmp_path / f"{sweep}.npz")], env=env,
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        got[sweep] = np.load(tmp_path / f"{sweep}.npz")
    for k in got["row"].files:
        assert got["row"][k].tobytes() == got["face"][k].tobytes(), k
