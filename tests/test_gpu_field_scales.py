"""Fields that are sums, on domains and with bumps of very different size: the element kernels hold them in fixed point
where that costs no digits, and what one problem of a system needs changes nothing in another.

Against the pivoted kernel, which evaluates in FP64, with the bound of the element paths' tests (2e-12 of a cell's block)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
BOUND = 2e-12


@pytest.fixture(scope="module")
def H():
    import __graft_entry__ as g
    g.build()
    return g.import_package()


def square(H, n, size, ctx="default"):
    mesh = H.rectangle_mesh(H.TriangleCell, (n, n), (0.0, 0.0), (size, size), ctx=ctx)
    mesh.jitter(0.2, 3)
    return mesh


def system(H, mesh, p, f, kappa=None, tau=1.0, he_tau=False):
    fe = H.GenericFiniteElement(H.Dubiner(2, H.RefTetrahedron, p))
    qd = {1: 2, 2: 3, 3: 6, 4: 9}[p]
    Wh, Vh = H.ScalarFunctionSpace(mesh, fe, quad_degree=qd), H.VectorFunctionSpace(mesh, fe, quad_degree=qd)
    Mh = H.ScalarTraceFunctionSpace(Wh, H.GenericFiniteElement(H.Legendre(1, H.RefTetrahedron, p)))
    return H.doassemble(Vh, Wh, Mh, tau, f, kappa=kappa, he_tau=he_tau)[0]


def blocks(H, mesh, p, f, kappa=None):
    return system(H, mesh, p, f, kappa).element_blocks()


def check(a, b):
    for x, y in zip(a, b):
        scale = np.abs(y).max(axis=tuple(range(1, y.ndim)), keepdims=True)
        assert np.isfinite(x).all()
        assert (np.abs(x - y) <= BOUND * np.maximum(scale, 1e-300)).all()


NEAR = ([0.5, 0.4], 0.1, 1.0)


def bumps(H, *b):
    return H.Field.bumps([x[0] for x in b], [x[1] for x in b], [x[2] for x in b])


# a bump switched off by its amplitude, or by its distance: the field without it, to the bit
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("far", [1e4, 1e9, 1e12, 1e15, 1e18, 1e300])
@pytest.mark.parametrize("amplitude", [0.0, 3.0])
def test_a_bump_that_is_off_changes_nothing(H, p, far, amplitude):
    mesh = square(H, 5, 1.0)
    with_it = blocks(H, mesh, p, bumps(H, NEAR, ([far, -far], 0.5, amplitude)))
    for x, y in zip(with_it, blocks(H, mesh, p, bumps(H, NEAR))):
        assert np.array_equal(x, y)


# a far bump wide enough to matter beside a near one; a narrow one near the origin of a large domain
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("far", [1e2, 1e4, 1e9, 1e15, 1e19])
@pytest.mark.parametrize("as_kappa", [False, True])
def test_wide_far_bumps(H, monkeypatch, p, far, as_kappa):
    mesh, f = square(H, 5, 1.0), bumps(H, NEAR, ([far, 0.0], 0.8 * far, 2.0))
    args = (mesh, p) + ((H.Field.const(1.0), f) if as_kappa else (f,))
    got = blocks(H, *args)
    monkeypatch.setenv("HDG_ELEMENT_FULL_LU", "1")
    check(got, blocks(H, *args))


# Lengths scaled by a power of two, tau against them: every number of the element kernels is the unit square's times a
# power of two, so the blocks are to the bit
@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("log2", [-60, -40, -7, 9, 40, 70])
@pytest.mark.parametrize("kind", ["bumps", "fourier", "exp_fourier", "narrow"])
def test_domains_of_any_size(H, p, log2, kind):
    def at(size):
        rng = np.random.default_rng(p)
        modes = rng.uniform(-2, 2, (9, 4))
        modes[:, :2] /= size
        f = {"bumps": bumps(H, ([0.5 * size, 0.4 * size], 0.1 * size, 1.0), ([0.1 * size, 0.9 * size], 0.3 * size, -2.0)),
             "narrow": bumps(H, ([2.0 ** -8 * size, 2.0 ** -9 * size], 2.0 ** -7 * size, 1.0)),
             "fourier": H.Field.fourier(0.3, modes),
             "exp_fourier": H.Field.fourier(0.3, modes, exponential=True)}[kind]
        mesh = square(H, 40 if kind == "narrow" else 7, 1.0)
        mesh.set_coordinates(size * H.get_vertices_matrix(mesh))
        return system(H, mesh, p, f, tau=1.0 / size, he_tau=True).element_blocks()

    size, nw = 2.0 ** log2, (p + 1) * (p + 2) // 2
    for x, y, q, u in zip(at(size), at(1.0), (1.0, size ** 2, 1.0 / size, size), (1.0, size ** 2, 1.0, size ** 2)):
        y = y.copy()
        if y.shape[1] == 3 * nw:  # K_e, b_e: the rows of q, then of u
            y[:, :2 * nw] *= q
            y[:, 2 * nw:] *= u
        else:
            y *= u
        # what a bump's tail leaves near the end of the exponent's range: the recovery's products below 2^-1022 go, up to 20
        # of them times 30, and are divided by det J (2^-120 / 1600): 3e-266, where the largest entry is 5e-22 and more
        assert ((x == y) | (np.maximum(np.abs(x), np.abs(y)) <= 1e-244 * np.abs(y).max())).all()


# many turns over the domain
@pytest.mark.parametrize("p", [2, 3])
@pytest.mark.parametrize("turns", [50.0, 1e3, 1e6])
def test_fast_modes(H, monkeypatch, p, turns):
    # a phase of that many turns is known to 2 pi turns 2^-52 in FP64
    mesh, f = square(H, 5, 1.0), H.Field.fourier(0.0, [[turns, 0.3 * turns, 0.2, 1.0], [1.0, 2.0, 0.0, 0.5]])
    got = blocks(H, mesh, p, f)
    monkeypatch.setenv("HDG_ELEMENT_FULL_LU", "1")
    want = blocks(H, mesh, p, f)
    for x, y in zip(got, want):
        assert np.abs(x - y).max() <= max(BOUND, 20 * turns * 2.0 ** -52) * np.abs(y).max()


@pytest.mark.parametrize("p", [1, 2, 3, 4])
@pytest.mark.parametrize("other", [1e-9, 1e3, 1e9])
@pytest.mark.parametrize("as_kappa", [False, True])
def test_problems_of_a_union_do_not_share_a_scale(H, p, other, as_kappa):
    f = bumps(H, NEAR, ([0.2, 0.2], 0.07, -0.5), ([0.6, 0.3], 2.0, 3.0))
    args = (p,) + ((H.Field.const(1.0), f) if as_kappa else (f,))
    parts = [square(H, 6, other, ctx=None), square(H, 5, 1.0, ctx=None)]
    union = blocks(H, H.concat_meshes(H.default_context(), parts), *args)
    alone = blocks(H, square(H, 5, 1.0), *args)
    if as_kappa and p == 1:  # two cells of a tile may leave it together: those to the bound
        check([x[-50:] for x in union], alone)
        return
    for x, y in zip(union, alone):
        assert np.array_equal(x[-50:], y)


@pytest.mark.parametrize("p", [1, 2, 3, 4])
def test_coordinates_set_large_and_then_small(H, p):
    f = bumps(H, NEAR, ([0.2, 0.2], 0.07, -0.5))
    mesh = square(H, 5, 1.0)
    xy = H.get_vertices_matrix(mesh)
    want = blocks(H, mesh, p, f)
    K = system(H, mesh, p, f)
    for size in (1e9, 1.0, 1e-6, 1.0):
        mesh.set_coordinates(size * xy)
        K.reassemble(resident=True)
        if size == 1.0:
            for x, y in zip(K.element_blocks(), want):
                assert np.array_equal(x, y)
