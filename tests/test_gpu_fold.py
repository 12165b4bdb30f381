"""The parity-folded transforms and the increment form of the step against the
general path.  A basis with two modes swapped is the same basis to the scheme
but not in ascending order, so it takes the general path."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def _params(sg, N, nac, nch, etd2=0, dt=0.005, kk=(1.0, 1.0, 1.0)):
    p = sg.default_params()
    p.nx = p.ny = p.nz = N + 4
    p.xmax, p.ymax, p.zmax = 0.5 * N, 0.45 * N, 0.55 * N
    p.nac, p.nch, p.elastic, p.etd2, p.dt = nac, nch, 0, etd2, dt
    p.kkx, p.kky, p.kkz = kk
    return p


def _swapped(n):
    d, v, vi = cases.eigen_variant(n, 3)
    q = np.arange(n)
    q[:2] = 1, 0
    return d[q], np.ascontiguousarray(v[:, q]), np.ascontiguousarray(vi[q])


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# half edges: 4, 5 (odd block), 18 and 19 (one inverse tile and two), 36 and 37
# (one forward tile and two), 66
EDGES = [4, 5, 31, 33, 68, 70, 128]


@pytest.mark.parametrize("N", EDGES)
def test_fp64_folded_products(N, sclet_lib):
    """One folded product each way against the dense sum in numpy: sums of n
    terms in another order, n 2^-53 at most, about sqrt(n) 2^-53 as they fall."""
    sg = sclet_lib
    s = sg.Solver(_params(sg, N, 1, 0), sg.FP64)
    n = s.n
    a = np.random.default_rng(N).standard_normal((n, n, n))
    _, v, vi = cases.eigen_variant(n, 3)
    for inverse, m in ((False, vi), (True, v)):
        got = s.mode_product(a, inverse)
        # the library's own basis is built like the oracle's, sines of arguments up to n pi: 1e-13
        assert _rel(got, np.einsum("pa,cba->pcb", m, a)) <= 1e-12, inverse
    s.close()


@pytest.mark.parametrize("N,nac,nch,etd2", [(4, 1, 0, 0), (5, 2, 1, 1), (31, 4, 1, 0), (33, 3, 0, 1), (68, 1, 1, 0),
                                            (70, 2, 0, 0)])
def test_fp64_steps_match_the_general_path(N, nac, nch, etd2, sclet_lib):
    sg = sclet_lib
    p = _params(sg, N, nac, nch, etd2, kk=(1.0, 0.7, 0.4))
    n = N + 4
    rng = np.random.default_rng(N)
    u0 = rng.uniform(-0.5, 0.5, size=(nac + nch, n, n, n))
    out = []
    for basis in (cases.eigen_variant(n, 3), _swapped(n)):
        s = sg.Solver(p, sg.FP64)
        s.set_eigen(*basis)
        s.set_fields(u0)
        s.step(3)
        out.append(s.get_fields())
        s.close()
    for f in range(nac + nch):
        assert _rel(out[0][f], out[1][f]) <= 1e-12, f


@pytest.mark.parametrize("dt", [0.05, 5.0])
def test_strong_damping_takes_the_full_form(dt, sclet_lib):
    """dt H reaches 1.7 and 170 on the finest modes: below 4 the increment form
    runs, above it the full one; both match the general path."""
    sg = sclet_lib
    p = _params(sg, 20, 2, 0, dt=dt)
    u0 = np.random.default_rng(3).uniform(-0.1, 0.1, size=(2, 24, 24, 24))
    out = []
    for basis in (cases.eigen_variant(24, 3), _swapped(24)):
        s = sg.Solver(p, sg.FP64)
        s.set_eigen(*basis)
        s.set_fields(u0)
        s.step(2)
        out.append(s.get_fields())
        s.close()
    for f in range(2):
        assert _rel(out[0][f], out[1][f]) <= 1e-12, f


# as EDGES, and halves of 64 and 65 (one epilogue column group full, one live
# column more), 128 and 130 (one a'-tile full, a second of two live columns),
# odd blocks, and block edges that are 0, 2 and odd modulo 4
MIXED_EDGES = [4, 5, 6, 31, 68, 75, 124, 126, 252, 253, 256]


@pytest.mark.parametrize("N", MIXED_EDGES)
def test_mixed_folded_products(N, sclet_lib):
    """One folded tensor-core product each way against FP64 sums of the
    FP32-rounded input, at the bound the dense product is held to."""
    sg = sclet_lib
    s = sg.Solver(_params(sg, N, 1, 0), sg.MIXED)
    n = s.n
    a = np.random.default_rng(N).standard_normal((n, n, n)).astype(np.float32).astype(np.float64)
    _, v, vi = cases.eigen_variant(n, 3)
    for inverse, m in ((False, vi), (True, v)):
        want = (a.reshape(-1, n) @ m.T).T.reshape(n, n, n)  # out[a', c, b]
        assert _rel(s.mode_product(a, inverse), want) <= 2e-7, inverse
    s.sync()
    s.close()


@pytest.mark.parametrize("N,nac,nch,etd2,dt", [(5, 2, 1, 1, 0.005), (31, 4, 1, 0, 0.005), (33, 3, 0, 1, 0.02),
                                               (68, 1, 1, 0, 0.005), (126, 1, 0, 0, 0.005), (20, 2, 1, 0, 5.0)])
def test_mixed_steps_are_no_further_from_fp64_than_the_general_path(N, nac, nch, etd2, dt, sclet_lib):
    sg = sclet_lib
    p = _params(sg, N, nac, nch, etd2, dt=dt, kk=(1.0, 0.7, 0.4))
    n = N + 4
    u0 = np.random.default_rng(N).uniform(-0.3, 0.3, size=(nac + nch, n, n, n))
    u0[nac:] = 0.5 + 0.1 * u0[nac:]

    def run(prec, basis):
        s = sg.Solver(p, prec)
        s.set_eigen(*basis)
        s.set_fields(u0)
        s.step(3)
        u = s.get_fields()
        s.sync()
        s.close()
        return u

    exact = run(sg.FP64, cases.eigen_variant(n, 3))
    fold, general = run(sg.MIXED, cases.eigen_variant(n, 3)), run(sg.MIXED, _swapped(n))
    for f in range(nac + nch):
        ef, eg = _rel(fold[f], exact[f]), _rel(general[f], exact[f])
        # the two differ by chance where both are a few roundings of 2^-24
        assert ef <= 1.5 * eg + 3e-8, (f, ef, eg)


def test_basis_can_change_back_and_forth(sclet_lib):
    """set_eigen switches the layout of the slice planes; nothing of one layout
    may be left in the other's zero columns."""
    sg = sclet_lib
    p = _params(sg, 31, 2, 0)
    u0 = np.random.default_rng(1).uniform(-0.3, 0.3, size=(2, 35, 35, 35))
    out = []
    s = sg.Solver(p, sg.MIXED)
    for basis in (cases.eigen_variant(35, 3), _swapped(35), cases.eigen_variant(35, 3), _swapped(35)):
        s.set_eigen(*basis)
        s.set_fields(u0)
        s.step(2)
        out.append(s.get_fields())
    s.sync()
    s.close()
    np.testing.assert_array_equal(out[0], out[2])
    np.testing.assert_array_equal(out[1], out[3])


@pytest.mark.parametrize("precision_name", ["FP64", "MIXED"])
@pytest.mark.parametrize("folded_first", [True, False])
def test_captured_steps_follow_the_basis(folded_first, precision_name, sclet_lib):
    """A step captured for one basis is not replayed for the next: each basis
    launches kernels and matrix layouts of its own.  Bit for bit."""
    sg = sclet_lib
    p = _params(sg, 31, 2, 1)
    u0 = np.random.default_rng(2).uniform(-0.3, 0.3, size=(3, 35, 35, 35))
    bases = [cases.eigen_variant(35, 3), _swapped(35)]
    if not folded_first:
        bases.reverse()
    s = sg.Solver(p, getattr(sg, precision_name))
    for basis in bases + bases[:1]:
        s.set_eigen(*basis)
        s.set_fields(u0)
        s.graph_step(3)
        got = s.get_fields()
        one = sg.Solver(p, getattr(sg, precision_name))
        one.set_eigen(*basis)
        one.set_fields(u0)
        one.step(3)
        np.testing.assert_array_equal(got, one.get_fields())
        one.close()
    s.sync()
    s.close()


def test_ensemble_steps_follow_the_basis(sclet_lib):
    """The same of the graph an ensemble holds over its contexts."""
    sg = sclet_lib
    made = []
    for N in (31, 20):
        p = _params(sg, N, 2, 0)
        u0 = np.random.default_rng(N).uniform(-0.3, 0.3, size=(2, N + 4, N + 4, N + 4))
        made.append((p, u0, sg.Solver(p, sg.MIXED)))
    ens = sg.Ensemble([s for _, _, s in made])
    for basis in (cases.eigen_variant(35, 3), _swapped(35), cases.eigen_variant(35, 3)):
        made[0][2].set_eigen(*basis)
        for _, u0, s in made:
            s.set_fields(u0)
        ens.step(3)
        ens.sync()
        for k, (p, u0, s) in enumerate(made):
            one = sg.Solver(p, sg.MIXED)
            if k == 0:
                one.set_eigen(*basis)
            one.set_fields(u0)
            one.step(3)
            np.testing.assert_array_equal(s.get_fields(), one.get_fields())
            one.close()
    ens.close()
    for _, _, s in made:
        s.close()


@pytest.mark.parametrize("N", [20, 31])
def test_conserved_update_rounds_no_more_than_the_general_path(N, sclet_lib):
    """One update of a conserved field, which is no increment, against the exact
    update of the same state and right-hand side in FP64: with dense sums seven
    roundings of the state's size (three products, the modes' update, three
    products), folded as many at most.  Means over the cells; 3 % for their chance."""
    sg = sclet_lib
    p = _params(sg, N, 0, 1)
    p.ymax = p.zmax = p.xmax
    n = N + 4
    d, v, vi = cases.eigen_variant(n, 3)
    h2 = (p.xmax / N) ** 2
    T = (d[:, None, None] + d[None, :, None] + d[None, None, :]) / h2
    lci, kci, c0 = p.landau[9], p.landau[10], p.landau[5]
    H = lci * (T * T * p.epn2 - kci * T)
    phi = -np.expm1(-p.dt * H) / H

    def transform(m, a):
        return np.einsum("ia,jb,kc,abc->ijk", m, m, m, a, optimize=True)

    err = []
    for basis in ((d, v, vi), _swapped(n)):
        sq = 0.0
        for seed in range(4):
            s = sg.Solver(p, sg.MIXED)
            s.set_eigen(*basis)
            s.set_fields(c0 + 0.05 * np.random.default_rng(seed).uniform(-0.5, 0.5, size=(1, n, n, n)))
            s.transfer()
            s.calc_rhs(1)
            u, rhs = s.get_fields()[0] - c0, s.get_rhs(1)[0]
            assert s.L.sclet_etd_update(s.h) == 0
            got = s.get_fields()[0] - c0
            s.close()
            q = (got - transform(v, np.exp(-p.dt * H) * transform(vi, u) + phi * transform(vi, rhs)))[(slice(2, -2),) * 3]
            sq += np.mean((q - q.mean()) ** 2)  # the mass correction is a uniform shift
        err.append(np.sqrt(sq / 4))
    assert err[0] <= 1.03 * err[1], err


@pytest.mark.parametrize("N", [4, 5, 21])
def test_full_form_runs_side_by_side(N, sclet_lib):
    """Strong damping: order parameters in the full form, their parts unfolded after
    the products, in every run as in a run of its own."""
    sg = sclet_lib
    p = _params(sg, N, 2, 0, dt=5.0)
    u0 = np.random.default_rng(N).uniform(-0.1, 0.1, size=(3 * 2, N + 4, N + 4, N + 4))
    s = sg.Solver(p, sg.MIXED, runs=3)
    s.set_fields(u0)
    s.step(2)
    got = s.get_fields()
    s.close()
    for r in range(3):
        one = sg.Solver(p, sg.MIXED)
        one.set_fields(u0[2 * r:2 * r + 2])
        one.step(2)
        np.testing.assert_array_equal(got[2 * r:2 * r + 2], one.get_fields())
        one.close()
