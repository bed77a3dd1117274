"""What a user of this framework has it do, as cases that can be timed and checked.

Five kinds of work, each through the public entry points:

  poisson   one HDG Poisson problem, new coefficients on a mesh that the program keeps: reassemble, apply_, solve,
            recovery, the squared error against a model solution where the reference's script forms it
  script    the whole flow of the reference's script in one call, system and all (solve_poisson)
  matrix    the first half of that flow: the trace matrix and right-hand side after apply!, as the CSC arrays that a
            program hands to a solver of its own
  batch     independent problems of uneven size and degree as one step (Batch.solve), solutions in host memory
  serve     a burst of requests through the serving engine, a part of them on resident meshes
  lagrange  the continuous-Galerkin script (nodal elements of order 1 and 2)

exact() is the same mathematics in plain torch and numpy, in 64 bits."""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# the quadrature degree of each polynomial degree in the batching and precision workloads (the default p + 1 leaves
# the local systems singular from p = 3 on)
QUAD = {1: 2, 2: 3, 3: 6, 4: 9}


def _package():
    """The package under its importable name (its folder's name has a dot)."""
    if "hdg_gb300" not in sys.modules:
        where = os.path.join(ROOT, "hdiscontinuousgalerkin.jl_gb300")
        spec = importlib.util.spec_from_file_location("hdg_gb300", os.path.join(where, "__init__.py"),
                                                      submodule_search_locations=[where])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["hdg_gb300"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["hdg_gb300"]


def listed():
    return [
        # the reference's HDG script as shipped: 10 x 10 squares, degree 1, direct from mesh to (u, q)
        dict(name="script_10_p1", kind="script", n=10, p=1, kappa="one", jitter=0.0, pc="jacobi", prec="fp64", tol=1e-12),
        # the reference's example size of the repository's own configurations (2048 triangles), a new source each time
        dict(name="poisson_32_p1", kind="poisson", n=32, p=1, kappa="one", jitter=0.0, pc="jacobi", prec="fp64",
             tol=1e-12),
        # an ordinary distorted mesh of odd size, a coefficient per cell, the mixed-precision iteration
        dict(name="poisson_97_p4_mixed", kind="poisson", n=97, p=4, kappa="cell", jitter=0.2, pc="jacobi", prec="mixed",
             tol=1e-10),
        # degree 4 with the multigrid preconditioner and Gaussian bumps as the source
        dict(name="poisson_181_p4_amg", kind="poisson", n=181, p=4, kappa="cell", jitter=0.2, pc="amg", prec="mixed",
             tol=1e-10),
        # the plain method scaled up (131072 triangles, FP64): Jacobi, and multigrid
        dict(name="poisson_256_p2", kind="poisson", n=256, p=2, kappa="one", jitter=0.0, pc="jacobi", prec="fp64",
             tol=1e-12),
        dict(name="poisson_256_p2_amg", kind="poisson", n=256, p=2, kappa="one", jitter=0.0, pc="amg", prec="fp64",
             tol=1e-12),
        # the largest single problem of the configurations: 524288 distorted triangles, degree 3, the coefficient and
        # the source as sums of 64 random Fourier modes
        dict(name="poisson_512_p3_field", kind="poisson", n=512, p=3, kappa="field", jitter=0.2, pc="amg", prec="mixed",
             tol=1e-10),
        # the assembled system for a solver of the user's own
        dict(name="matrix_96_p3", kind="matrix", n=96, p=3, kappa="cell", jitter=0.2),
        # the uneven batch: n log-uniform in [8, 128], degrees 1 to 4, a coefficient per cell over four decades
        dict(name="batch_64_amg", kind="batch", count=64, nmax=128, pc="amg", tol=1e-10),
        # a burst of requests as the serving engine meets them
        dict(name="serve_20", kind="serve", count=20, nmax=64, pc="amg", tol=1e-10),
        # the reference's continuous-Galerkin script as shipped, and scaled up
        dict(name="lagrange_10_p1", kind="lagrange", n=10, p=1, kappa="one", jitter=0.0, tol=1e-12),
        dict(name="lagrange_256_p2", kind="lagrange", n=256, p=2, kappa="one", jitter=0.0, tol=1e-12),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["poisson"] * 6 + ["script", "matrix", "batch", "serve", "lagrange", "lagrange"])
    if kind in ("batch", "serve"):
        count = size(4, 64) if kind == "batch" else rng.randint(3, 20)
        return dict(kind=kind, count=count, nmax=rng.randint(24, 128 if kind == "batch" else 64), pc="amg", tol=1e-10)
    if kind == "lagrange":
        return dict(kind=kind, n=size(6, 256), p=rng.randint(1, 2), kappa=rng.choice(["one", "cell"]),
                    jitter=rng.choice([0.0, 0.2]), tol=1e-12)
    p = rng.randint(1, 4)
    if kind == "matrix":
        return dict(kind=kind, n=size(8, 110), p=p, kappa=rng.choice(["one", "cell"]), jitter=0.2)
    if kind == "script":
        return dict(kind=kind, n=size(6, 64), p=p, kappa=rng.choice(["one", "cell"]), jitter=0.2, pc="jacobi",
                    prec="fp64", tol=1e-12 if p < 3 else 1e-11)
    pc = rng.choice(["jacobi", "amg"])
    prec = rng.choice(["fp64", "mixed"])
    # the degree-4 rule has negative weights, under which a strongly varying field can leave a coarse cell indefinite
    kappa = rng.choice(["one", "cell", "field"] if p < 4 else ["one", "cell"])
    # the conjugate gradients' work grows like n^3 with Jacobi and n^2 with multigrid
    n = size(8, 128 if pc == "jacobi" else 320)
    return dict(kind=kind, n=n, p=p, kappa=kappa, jitter=rng.choice([0.0, 0.2]), pc=pc, prec=prec, tol=1e-10)


# ---- inputs, from the case and the seed alone (plain numbers, shared with exact()) ------------------------------
def _rng(seed):
    return np.random.default_rng([20240611, int(seed) & 0xFFFFFFFF])


def _grid(n):
    """Nodes (x fastest) and triangles of the n x n unit square with right diagonals, 0-based."""
    t = np.arange(n + 1) / n
    xy = np.stack([np.tile(t, n + 1), np.repeat(t, n + 1)], axis=1)
    j, i = np.divmod(np.arange(n * n), n)
    a = j * (n + 1) + i
    b, c, d = a + 1, a + n + 1, a + n + 2
    cells = np.stack([np.stack([a, b, c], 1), np.stack([b, d, c], 1)], axis=1).reshape(-1, 3)
    return xy, cells


def _coordinates(case, rng):
    """Interior nodes moved by up to jitter * h."""
    n = case["n"]
    xy, _ = _grid(n)
    inner = np.all((xy > 1e-9) & (xy < 1 - 1e-9), axis=1)
    xy[inner] += case["jitter"] / n * rng.uniform(-1.0, 1.0, (int(inner.sum()), 2))
    return xy


def _fourier(rng, scale, modes=64):
    """Random modes (kx, ky, phase, amplitude) of wavelength >= 0.1."""
    ang, rad = rng.uniform(0, 2 * math.pi, modes), 10.0 * np.sqrt(rng.uniform(0, 1, modes))
    return np.stack([rad * np.cos(ang), rad * np.sin(ang), rng.uniform(0, 2 * math.pi, modes),
                     scale * rng.standard_normal(modes) / math.sqrt(32.0)], axis=1)


def _inputs(case, seed):
    """Coordinates, source, coefficient: dict(xy, f, kappa) with f and kappa as (kind, parameters) or an array."""
    rng = _rng(seed)
    xy = _coordinates(case, rng)
    if case["kappa"] == "one":  # the manufactured source 2 pi^2 sin(pi x) sin(pi y), scaled and with other wave numbers
        kx, ky = rng.uniform(0.8, 2.5, 2)
        return dict(xy=xy, f=("sinsin", (math.pi ** 2 * (kx * kx + ky * ky) * rng.uniform(0.5, 2.0), kx, ky)), kappa=None)
    if case["kappa"] == "field":
        return dict(xy=xy, f=("fourier", _fourier(rng, 10.0)), kappa=("exp_fourier", _fourier(rng, 1.0)))
    centres, widths = rng.random((8, 2)), 0.03 + 0.12 * rng.random(8)
    f = ("bumps", (centres, widths, 10.0 * rng.standard_normal(8)))
    return dict(xy=xy, f=f, kappa=np.exp(rng.uniform(math.log(1e-1), math.log(1e1), 2 * case["n"] ** 2)))


def _field(H, spec):
    kind, prm = spec
    if kind == "sinsin":
        return H.Field.sinsin(*prm)
    if kind == "bumps":
        return H.Field.bumps(*prm)
    return H.Field.fourier(0.0, prm, exponential=kind == "exp_fourier")


def _draw_problem(rng, nmax):
    """One problem of the batching workload: size, degree, bumps, coefficient per cell over four decades."""
    n = int(round(math.exp(rng.uniform(math.log(8), math.log(nmax)))))
    p = int(rng.integers(1, 5))
    bumps = (rng.random((8, 2)), 0.03 + 0.12 * rng.random(8), 10.0 * rng.standard_normal(8))
    return n, p, bumps, np.exp(rng.uniform(math.log(1e-2), math.log(1e2), 2 * n * n)), int(rng.integers(1 << 30))


# ---- the passes ---------------------------------------------------------------------------------------------------
def _options(H, case):
    return dict(tol=case["tol"], preconditioner=H.PRECOND_AMG if case["pc"] == "amg" else H.PRECOND_JACOBI)


def _precision(H, case):
    return H.PREC_MIXED if case.get("prec") == "mixed" else H.PREC_FP64


def prepare(case, seed):
    H = _package()
    st = dict(H=H, kind=case["kind"], case=case)
    if case["kind"] in ("batch", "serve"):
        # the sizes and degrees belong to the case, the meshes and coefficients to the seed
        shape, rng = np.random.default_rng([7, case["count"], case["nmax"]]), _rng(seed)
        problems = []
        for _ in range(case["count"]):
            n, p, _, _, _ = _draw_problem(shape, case["nmax"])
            _, _, bumps, _, mesh_seed = _draw_problem(rng, 8)
            kappa = np.exp(rng.uniform(math.log(1e-2), math.log(1e2), 2 * n * n))
            problems.append(H.Problem(n=n, p=p, f=H.Field.bumps(*bumps), kappa_cell=kappa, jitter=0.2, seed=mesh_seed))
        ctx = H.default_context()
        if case["kind"] == "batch":
            st["batch"] = H.Batch(ctx, problems)
            return st
        st["engine"] = H.Engine(ctx, tol=case["tol"], preconditioner=H.PRECOND_AMG)
        st["problems"] = problems
        meshes = [H.batch.host_mesh(pr) for pr in problems]
        # seven of ten requests are on meshes that the engine holds
        st["on"] = [dict(mesh_id=st["engine"].add_resident(m, pr.p)) if k % 10 < 7 else dict(mesh=m)
                    for k, (m, pr) in enumerate(zip(meshes, problems))]
        return st
    new = _inputs(case, seed)
    mesh = H.rectangle_mesh(H.TriangleCell, (case["n"], case["n"]), (0.0, 0.0), (1.0, 1.0))
    mesh.set_coordinates(new["xy"])
    st["mesh"], st["f"] = mesh, _field(H, new["f"])
    st["kappa"] = {}
    if isinstance(new["kappa"], np.ndarray):
        st["kappa"] = dict(kappa_cell=new["kappa"])
    elif new["kappa"] is not None:
        st["kappa"] = dict(kappa=_field(H, new["kappa"]))
    if case["kind"] == "lagrange":
        Wh = H.ScalarFunctionSpace(mesh, H.ContinuousLagrange(2, H.RefTetrahedron, case["p"]), update_face_data=False)
        u_h = H.TrialFunction(Wh)
        dh = H.DofHandler([u_h], mesh)
        st["dbc"] = H.Dirichlet(u_h, dh, "boundary", lambda x: 0.0)
        st["K"], _ = H.doassemble_cg(Wh, H.create_sparsity_pattern(dh), dh, st["f"], **st["kappa"])
        return st
    if case["kind"] == "script":
        return st
    fe = H.GenericFiniteElement(H.Dubiner(2, H.RefTetrahedron, case["p"]))
    qd = QUAD[case["p"]]
    Wh, Vh = H.ScalarFunctionSpace(mesh, fe, quad_degree=qd), H.VectorFunctionSpace(mesh, fe, quad_degree=qd)
    Mh = H.ScalarTraceFunctionSpace(Wh, H.GenericFiniteElement(H.Legendre(1, H.RefTetrahedron, case["p"])))
    st["h"] = [H.TrialFunction(V) for V in (Vh, Wh, Mh)]
    st["dbc"] = H.Dirichlet(st["h"][2], mesh, "boundary")
    st["K"], st["b"], st["Ke"], st["be"] = H.doassemble(Vh, Wh, Mh, 1.0, st["f"], precision=_precision(H, case),
                                                        **st["kappa"])
    return st


class _Held(np.ndarray):
    """A view of the page-locked memory of a batch, which it keeps alive (the memory goes with the batch)."""
    owner = None


def _held(array, owner):
    v = array.view(_Held)
    v.owner = owner
    return v


def run(st):
    H, case = st["H"], st["case"]
    kind = st["kind"]
    if kind == "script":
        uhat, q, u, _ = H.solve_poisson(st["mesh"], case["p"], st["f"], quad_degree=QUAD[case["p"]],
                                        precision=_precision(H, case), **st["kappa"], **_options(H, case))
        return dict(uhat=uhat, q=q, u=u)
    if kind == "poisson":
        K = st["K"]
        K.reassemble(1.0, st["f"], **st["kappa"])
        H.apply_(K, st["b"], st["dbc"])
        uhat = H.solve(K, st["b"], precision=_precision(H, case), **_options(H, case))
        sigma_h, u_h, uhat_h = st["h"]
        H.get_usigma_(sigma_h, u_h, uhat_h, uhat, st["Ke"], st["be"], st["mesh"])
        out = dict(uhat=uhat, q=sigma_h.m_values, u=u_h.m_values)
        if case["kappa"] == "one":
            out["error"] = H.errornorm(u_h, H.MANUFACTURED_U)
        return out
    if kind == "matrix":
        K = st["K"]
        K.reassemble(1.0, st["f"], **st["kappa"])
        H.apply_(K, st["b"], st["dbc"])
        colptr, rowval, nzval, rhs = K.csc()
        return dict(colptr=colptr, rowval=rowval, nzval=nzval, rhs=rhs)
    if kind == "lagrange":
        K = st["K"]
        K.assemble(st["f"], **st["kappa"])
        H.apply_(K, None, st["dbc"])
        return dict(u=H.solve(K, tol=case["tol"]))
    if kind == "batch":
        B = st["batch"]
        B.solve(download=True, **_options(H, case))
        # the page-locked arrays that the step filled, whole, per degree
        out = {}
        for b in B.bins:
            out["uhat%d" % b.p], out["qu%d" % b.p] = (_held(a, B) for a in b.enable_download())
        return out
    eng = st["engine"]
    ids = [eng.submit(pr.p, pr.f, pr.kappa_cell, **on) for pr, on in zip(st["problems"], st["on"])]
    eng.run_until_idle()
    return [eng.result(i) for i in ids]


# ---- the work that no implementation is without -------------------------------------------------------------------
def _one(n, p, cells_only=False):
    nc, nf = 2 * n * n, 3 * n * n + 2 * n
    nw, nt = (p + 1) * (p + 2) // 2, p + 1
    # nodes, connectivity, coefficient in; u_hat, q, u out
    by = 16 * (n + 1) ** 2 + 24 * nc + 8 * nc + 8 * (nf * nt + 3 * nw * nc)
    # per cell: factorise an nw x nw symmetric system, solve for 3 nt + 1 columns, form the condensed block
    m = 3 * nt
    fl = nc * (nw ** 3 / 3 + 2 * nw * nw * (m + 1) + nw * m * (m + 1)) + nc * 2 * 3 * nw * (m + 1)
    # and at least one product with the trace matrix per grid line that information has to cross
    fl += 0 if cells_only else 2 * 5 * nf * nt * nt
    return by, fl


def work(case):
    if case["kind"] in ("batch", "serve"):
        shape = np.random.default_rng([7, case["count"], case["nmax"]])
        both = [_one(*_draw_problem(shape, case["nmax"])[:2]) for _ in range(case["count"])]
        return {"bytes": sum(b for b, _ in both), "flops": sum(f for _, f in both)}
    n, p = case["n"], case["p"]
    if case["kind"] == "lagrange":
        nd, nl, nc = (p * n + 1) ** 2, (p + 1) * (p + 2) // 2, 2 * n * n
        return {"bytes": 16 * (n + 1) ** 2 + 24 * nc + 8 * nd, "flops": nc * (6 * nl * nl * 3 + 2 * nl * nl)}
    by, fl = _one(n, p, cells_only=case["kind"] == "matrix")
    if case["kind"] == "matrix":
        nnz = (15 * n * n + 2 * n) * (p + 1) ** 2
        by += 16 * nnz
    return {"bytes": by, "flops": fl}


# ---- the same in plain torch and numpy ------------------------------------------------------------------------------
def _strang(order):
    if order == 2:
        return np.array([[1 / 6, 1 / 6], [1 / 6, 2 / 3], [2 / 3, 1 / 6]]), np.full(3, 1 / 6)
    if order == 3:
        a, b, c = 0.659027622374092, 0.231933368553031, 0.109039009072877
        return np.array([[a, b], [a, c], [b, a], [b, c], [c, a], [c, b]]), np.full(6, 1 / 12)
    a, b, c, d = 0.873821971016996, 0.063089014491502, 0.501426509658179, 0.249286745170910
    e, f, g = 0.636502499121399, 0.310352451033785, 0.053145049844816
    pts = [[a, b], [b, a], [b, b], [c, d], [d, c], [d, d], [e, f], [e, g], [f, e], [f, g], [g, e], [g, f]]
    return np.array(pts), 0.5 * np.repeat([0.050844906370207, 0.116786275726379, 0.082851075618374], [3, 3, 6])


def _volume_rule(order):
    """Strang's rules up to order 6, Grundmann and Moeller's above."""
    if order <= 6:
        return _strang(order)
    s = (order - 1) // 2
    d, pts, w = 2 * s + 1, [], []
    for i in range(s + 1):
        wi = (-1.0) ** i * 2.0 ** (-2 * s) * float(d + 2 - 2 * i) ** d / (math.factorial(i) * math.factorial(d + 2 - i))
        for p2 in range(s - i + 1):
            for p1 in range(s - i - p2 + 1):
                pts.append([(2 * p1 + 1) / (d + 2 - 2 * i), (2 * p2 + 1) / (d + 2 - 2 * i)])
                w.append(wi)
    return np.array(pts), 0.5 * np.array(w) / sum(w)


def _jacobi(x, n, al, be):
    a, b = np.ones_like(x), ((2 + al + be) * x + (al - be)) / 2
    if n == 0:
        return a
    for k in range(2, n + 1):
        a1 = 2 * k * (k + al + be) * (2 * k - 2 + al + be)
        a2 = (2 * k - 1 + al + be) * (al + be) * (al - be)
        a3 = (2 * k - 2 + al + be) * (2 * k - 1 + al + be) * (2 * k + al + be)
        a4 = 2 * (k - 1 + al) * (k - 1 + be) * (2 * k + al + be)
        a, b = b, ((a2 + a3 * x) * b - a4 * a) / a1
    return b


def _dubiner(p, x, y):
    """[nw][points], orthonormal on the reference triangle, degree by degree."""
    out = []
    for c in range(p + 1):
        for n in range(c, -1, -1):
            m = c - n
            xi, eta = 2 * x / (1 - y) - 1, 2 * y - 1
            v = _jacobi(xi, n, 0, 0) * _jacobi(eta, m, 2 * n + 1, 0) * ((1 - eta) / 2) ** n
            out.append(2 * v / math.sqrt(2 / ((2 * n + 1) * (m + n + 1))))
    return np.array(out)


def _gradient(fun, x, y):
    """By the complex step, which takes no difference."""
    h = 1e-40
    return np.imag(fun(x + 1j * h, y + 0j)) / h, np.imag(fun(x + 0j, y + 1j * h)) / h


EDGE_ENDS = (((1.0, 0.0), (0.0, 1.0)), ((0.0, 1.0), (0.0, 0.0)), ((0.0, 0.0), (1.0, 0.0)))


def _first_seen(keys):
    """Numbers 0, 1, ... in the order in which the keys first come."""
    _, first, inv = np.unique(keys, return_index=True, return_inverse=True)
    rank = np.empty(len(first), np.int64)
    rank[np.argsort(first)] = np.arange(len(first))
    return rank[inv]


def _faces(cells, nn):
    """Faces of each cell (local edges 2-3, 3-1, 1-2) numbered at first visit, their orientation, the boundary ones."""
    v = np.stack([cells[:, [1, 2]], cells[:, [2, 0]], cells[:, [0, 1]]], axis=1)
    faces = _first_seen((v.min(2).astype(np.int64) * nn + v.max(2)).ravel()).reshape(-1, 3)
    return faces, v[:, :, 1] > v[:, :, 0], np.nonzero(np.bincount(faces.ravel()) == 1)[0]


def _evaluate(spec, x, y):
    """A field at torch points."""
    kind, prm = spec
    if kind == "sinsin":
        return prm[0] * torch.sin(prm[1] * math.pi * x) * torch.sin(prm[2] * math.pi * y)
    if kind == "bumps":
        return sum(float(a) * torch.exp(-((x - float(c[0])) ** 2 + (y - float(c[1])) ** 2) / (2 * float(s) ** 2))
                   for c, s, a in zip(*prm))
    g = sum(float(a) * torch.cos(2 * math.pi * (float(kx) * x + float(ky) * y) + float(ph)) for kx, ky, ph, a in prm)
    return torch.exp(g) if kind == "exp_fourier" else g


def _cg(rows, cols, vals, b, n):
    """Jacobi-preconditioned conjugate gradients to the last digits, then once more on the remaining residual."""
    A = torch.sparse_coo_tensor(torch.stack([rows, cols]), vals, (n, n)).coalesce()
    i = A.indices()
    dinv = torch.zeros(n, dtype=b.dtype, device=b.device)
    on = i[0] == i[1]
    dinv[i[0][on]] = 1 / A.values()[on]
    A = A.to_sparse_csr()
    x = torch.zeros_like(b)
    for goal in (1e-14, 1e-4):
        r = b - A @ x
        stop = (goal * r.norm()) ** 2
        y, z = torch.zeros_like(b), dinv * r
        p, rz = z.clone(), r @ z
        for k in range(60000):
            q = A @ p
            alpha = rz / (p @ q)
            y += alpha * p
            r -= alpha * q
            z = dinv * r
            rz, old = r @ z, rz
            p = z + (rz / old) * p
            if k % 32 == 31 and not bool(r @ r > stop):
                break
        x = x + y
    return x


def _exact_hdg(case, seed, device):
    new, p = _inputs(case, seed), case["p"]
    xy, (_, cells) = new["xy"], _grid(case["n"])
    nc, nw, nt = len(cells), (p + 1) * (p + 2) // 2, p + 1
    m, n, qd = 3 * nt, 3 * nw, QUAD[p]
    faces, orient, boundary = _faces(cells, len(xy))
    nf = int(faces.max()) + 1
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=device)  # noqa: E731
    pts, w = _volume_rule(qd)
    N = _dubiner(p, pts[:, 0], pts[:, 1])
    dN = _gradient(lambda x, y: _dubiner(p, x, y), pts[:, 0], pts[:, 1])
    s, fw = np.polynomial.legendre.leggauss(qd)
    s, fw = (s + 1) / 2, fw / 2
    mu = np.array([math.sqrt(2 * k + 1) * _jacobi(2 * s - 1, k, 0, 0) for k in range(nt)])
    on_edge = [_dubiner(p, (1 - s) * a[0] + s * b[0], (1 - s) * a[1] + s * b[1]) for a, b in EDGE_ENDS]
    D = T(np.stack([(g * w) @ N.T for g in dN]))                      # int d_l phi_i phi_j
    C = T(np.stack([(e * fw) @ e.T for e in on_edge]))
    F = T(np.stack([[(e[:, ::-1] * fw) @ mu.T, (e * fw) @ mu.T] for e in on_edge]))  # [face][orientation]
    Hm = T((mu * fw) @ mu.T)
    tN, tw, tp = T(N), T(w), T(pts)
    outs = []
    for lo in range(0, nc, 65536):
        c = slice(lo, min(nc, lo + 65536))
        X = T(xy[cells[c]])
        k = len(X)
        J = torch.stack([X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]], dim=2)
        det = J[:, 0, 0] * J[:, 1, 1] - J[:, 0, 1] * J[:, 1, 0]
        adj = torch.stack([torch.stack([J[:, 1, 1], -J[:, 0, 1]], 1), torch.stack([-J[:, 1, 0], J[:, 0, 0]], 1)], 1)
        wn = torch.stack([torch.stack([J[:, 1, 1] - J[:, 1, 0], J[:, 0, 0] - J[:, 0, 1]], 1),
                          torch.stack([-J[:, 1, 1], J[:, 0, 1]], 1), torch.stack([J[:, 1, 0], -J[:, 0, 0]], 1)], 1)
        le = wn.norm(dim=2)
        Q = X[:, :1] + torch.einsum("cab,qb->cqa", J, tp)
        ki = torch.ones(k, len(w), dtype=torch.float64, device=device)
        if isinstance(new["kappa"], np.ndarray):
            ki = ki / T(new["kappa"][c])[:, None]
        elif new["kappa"] is not None:
            ki = 1 / _evaluate(new["kappa"], Q[:, :, 0], Q[:, :, 1])
        be = torch.einsum("cq,q,iq,c->ci", _evaluate(new["f"], Q[:, :, 0], Q[:, :, 1]), tw, tN, det)
        A = torch.einsum("cq,q,iq,jq,c->cij", ki, tw, tN, tN, det)
        B = torch.einsum("clx,lij->cxij", adj, D)
        Fo = torch.stack([F[f][T(orient[c][:, f].astype(np.int64))] for f in range(3)], dim=2)  # [cell][nw][face][nt]
        E = torch.einsum("cfx,cifj->cxifj", wn, Fo).reshape(k, 2 * nw, m)
        Fe = (le[:, None, :, None] * Fo).reshape(k, nw, m)
        Me = torch.zeros(k, n, n, dtype=torch.float64, device=device)
        Me[:, :nw, :nw] = A
        Me[:, nw:2 * nw, nw:2 * nw] = A
        Me[:, :2 * nw, 2 * nw:] = -B.reshape(k, 2 * nw, nw)
        Me[:, 2 * nw:, :2 * nw] = B.reshape(k, 2 * nw, nw).transpose(1, 2)
        Me[:, 2 * nw:, 2 * nw:] = torch.einsum("cf,fij->cij", le, C)
        right = torch.zeros(k, n, m + 1, dtype=torch.float64, device=device)
        right[:, :2 * nw, :m], right[:, 2 * nw:, :m], right[:, 2 * nw:, m] = -E, Fe, be
        X = torch.linalg.solve(Me, right)
        AB = torch.cat([E, Fe], dim=1).transpose(1, 2) @ X
        for f in range(3):
            AB[:, f * nt:(f + 1) * nt, f * nt:(f + 1) * nt] -= le[:, f, None, None] * Hm
        AB[:, :, m] *= -1
        outs.append((X, AB))
    X, AB = (torch.cat([o[i] for o in outs]) for i in (0, 1))
    gd = (T(faces)[:, :, None] * nt + torch.arange(nt, device=device)).reshape(nc, m)
    nd = nf * nt
    fixed = torch.zeros(nd, dtype=torch.bool, device=device)
    fixed[(T(boundary)[:, None] * nt + torch.arange(nt, device=device)).ravel()] = True
    rows, cols = gd[:, :, None].expand(nc, m, m).reshape(-1), gd[:, None, :].expand(nc, m, m).reshape(-1)
    vals = AB[:, :, :m].reshape(-1)
    b = torch.zeros(nd, dtype=torch.float64, device=device).index_add_(0, gd.reshape(-1), AB[:, :, m].reshape(-1))
    if case["kind"] == "matrix":
        K = torch.sparse_coo_tensor(torch.stack([cols, rows]), vals, (nd, nd)).coalesce()  # column by column
        (cols, rows), vals = K.indices(), K.values().clone()
        diag = (vals[rows == cols].abs().sum() / nd)
        vals[fixed[rows] | fixed[cols]] = 0
        vals[(rows == cols) & fixed[rows]] = diag
        b[fixed] = 0
        return dict(colptr=None, rowval=None, nzval=vals.cpu(), rhs=b.cpu())
    free = ~(fixed[rows] | fixed[cols])
    one = torch.nonzero(fixed).ravel()
    b[fixed] = 0
    uhat = _cg(torch.cat([rows[free], one]), torch.cat([cols[free], one]),
               torch.cat([-vals[free], torch.ones(len(one), dtype=torch.float64, device=device)]), -b, nd)
    qu = (X[:, :, :m] @ uhat[gd][:, :, None])[:, :, 0] + X[:, :, m]
    out = dict(uhat=uhat.cpu(), q=qu[:, :2 * nw].cpu(), u=qu[:, 2 * nw:].cpu())
    if case["kind"] == "poisson" and case["kappa"] == "one":
        Xc = T(xy[cells])
        J = torch.stack([Xc[:, 1] - Xc[:, 0], Xc[:, 2] - Xc[:, 0]], dim=2)
        Q = Xc[:, :1] + torch.einsum("cab,qb->cqa", J, tp)
        d = qu[:, 2 * nw:] @ tN - _evaluate(("sinsin", (1.0, 1.0, 1.0)), Q[:, :, 0], Q[:, :, 1])
        det = J[:, 0, 0] * J[:, 1, 1] - J[:, 0, 1] * J[:, 1, 0]
        out["error"] = float((d * d * tw * det[:, None]).sum())
    return out


def _nodal(k, x, y):
    """Nodal basis of order 1 or 2 on the reference triangle: vertices, then the midpoints of the local edges."""
    a = np.array([1 - x - y, x, y])
    if k == 1:
        return a
    return np.concatenate([a * (2 * a - 1), 4 * np.array([a[1] * a[2], a[2] * a[0], a[0] * a[1]])])


def _exact_lagrange(case, seed, device):
    new, k = _inputs(case, seed), case["p"]
    xy, (_, cells) = new["xy"], _grid(case["n"])
    faces, _, boundary = _faces(cells, len(xy))
    entities = cells if k == 1 else np.concatenate([cells, len(xy) + faces], axis=1)
    dofs = _first_seen(entities.ravel()).reshape(entities.shape)
    outer = np.isin(faces, boundary)
    fixed = [dofs[:, [1, 2]][outer[:, 0]], dofs[:, [2, 0]][outer[:, 1]], dofs[:, [0, 1]][outer[:, 2]]]
    if k == 2:
        fixed.append(dofs[:, 3:][outer])
    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=device)  # noqa: E731
    fixed = T(np.unique(np.concatenate([f.ravel() for f in fixed])))
    pts, w = _volume_rule(k + 1)
    N = T(_nodal(k, pts[:, 0], pts[:, 1]))
    G = T(np.stack(_gradient(lambda x, y: _nodal(k, x, y), pts[:, 0], pts[:, 1])))
    X, tw = T(xy[cells]), T(w)
    J = torch.stack([X[:, 1] - X[:, 0], X[:, 2] - X[:, 0]], dim=2)
    det = J[:, 0, 0] * J[:, 1, 1] - J[:, 0, 1] * J[:, 1, 0]
    g = torch.einsum("clx,liq->cxiq", torch.linalg.inv(J), G)
    kap = T(new["kappa"]) if new["kappa"] is not None else torch.ones_like(det)
    Ke = torch.einsum("cxiq,cxjq,q,c->cij", g, g, tw, det * kap)
    Q = X[:, :1] + torch.einsum("cab,qb->cqa", J, T(pts))
    fe = torch.einsum("cq,iq,q,c->ci", _evaluate(new["f"], Q[:, :, 0], Q[:, :, 1]), N, tw, det)
    gd, nd, nl = T(dofs), int(dofs.max()) + 1, dofs.shape[1]
    rows, cols = gd[:, :, None].expand(-1, nl, nl).reshape(-1), gd[:, None, :].expand(-1, nl, nl).reshape(-1)
    off = torch.zeros(nd, dtype=torch.bool, device=device)
    off[fixed] = True
    free = ~(off[rows] | off[cols])
    b = torch.zeros(nd, dtype=torch.float64, device=device).index_add_(0, gd.reshape(-1), fe.reshape(-1))
    b[fixed] = 0
    u = _cg(torch.cat([rows[free], fixed]), torch.cat([cols[free], fixed]),
            torch.cat([Ke.reshape(-1)[free], torch.ones(len(fixed), dtype=torch.float64, device=device)]), b, nd)
    return dict(u=u.cpu())


def exact(case, seed):
    if case["kind"] in ("batch", "serve"):
        return None  # dozens of systems with a contrast of 1e4: minutes with this iteration
    device = "cuda" if torch.cuda.is_available() else "cpu"
    return (_exact_lagrange if case["kind"] == "lagrange" else _exact_hdg)(case, seed, device)
