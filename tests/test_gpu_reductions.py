"""Diagnostics of check_soln_new where the reduction's shapes meet their edges:
owned edges around the 32 x 8 column tile and the eight-plane unit, several
field counts, both energy forms, against numpy, in both precisions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _numpy(p, u, form):
    nac, nch = p.nac, p.nch
    own = u[:, 2:-2, 2:-2, 2:-2]
    h = [p.xmax / own.shape[3], p.ymax / own.shape[2], p.zmax / own.shape[1]]

    def corner(sz, sy, sx):
        t = own
        for ax, s in ((3, sx), (2, sy), (1, sz)):
            n = t.shape[ax]
            t = np.take(t, range(1, n), ax) + s * np.take(t, range(n - 1), ax)
        return t

    av = corner(1, 1, 1) / 8
    g = [corner(1, 1, -1) / (4 * h[0]), corner(1, -1, 1) / (4 * h[1]), corner(-1, 1, 1) / (4 * h[2])]
    kk = [p.kkx, p.kky, p.kkz]
    grad = [0.5 * p.epn2 * sum((kk[a] if f < nac else 1.0) * g[a][f] ** 2 for a in range(3)) for f in range(nac + nch)]
    e2 = av[:nac] ** 2
    s = e2.sum(0)
    a2, a4, a6, gx, th, c0, A = list(p.landau)[:7]
    ch = 0.0
    if form == 1:
        ac = sum(grad) + a2 / 2 * s + a4 / 4 * (e2 ** 2).sum(0) + a6 / 6 * (e2 ** 3).sum(0)
        ac = ac + gx * (s ** 2 - (e2 ** 2).sum(0)) / 2
        if nch:
            d = av[nac] - c0
            ac = ac + A / 2 * d ** 2 - th * d * s
    else:
        ac = sum(grad[:nac]) if nac else 0.0
        if nac:
            s3 = (av[:nac] ** 3).sum(0)
            ac = ac + 1188.0 / 2372 * s - (7128.0 + 12 * 2372) / 2372 / 3 * s3 + (4752.0 + 12 * 2372) / 2372 / 4 * s ** 2
        if nch:
            ch = (grad[nac] + 0.25 * (av[nac] ** 2 - 1) ** 2).sum()
    h3 = h[0] * h[1] * h[2]
    ac = np.sum(ac)
    return np.array([[f.max(), f.min(), (f + 1).sum() * h3, h3 * (ch if form == 0 and i >= nac else ac)]
                     for i, f in enumerate(own)])


@pytest.mark.parametrize("N,nac,nch", [(4, 1, 0), (7, 0, 1), (8, 4, 1), (9, 2, 1), (33, 4, 0), (41, 3, 1), (65, 4, 1)])
@pytest.mark.parametrize("form", [0, 1])
def test_diagnostics_match_numpy(N, nac, nch, form, sclet_lib):
    """FP64 sums of at most 3e5 values, compensated: 1e-13 covers the roundings of
    a cell's forty operations."""
    sg = sclet_lib
    p = sg.default_params()
    n = N + 4
    p.nx = p.ny = p.nz = n
    p.xmax, p.ymax, p.zmax = 0.5 * N, 0.4 * N, 0.6 * N
    p.kkx, p.kky, p.kkz = 1.0, 0.7, 0.4
    p.nac, p.nch, p.elastic = nac, nch, 0
    u = np.random.default_rng(N).uniform(0.2, 0.9, size=(nac + nch, n, n, n)).astype(np.float32).astype(np.float64)
    s = sg.Solver(p, sg.FP64)
    s.set_fields(u)
    got = s.check_soln(form)
    s.close()
    want = _numpy(p, u, form)
    np.testing.assert_array_equal(got[:, :2], want[:, :2])
    np.testing.assert_allclose(got[:, 2:], want[:, 2:], rtol=1e-13)


def _magnitudes(p, u, form):
    """The energies of _numpy with every term taken by its size."""
    q = type(p)()
    for k, _ in p._fields_:
        setattr(q, k, getattr(p, k))
    q.landau[:] = [abs(v) for v in p.landau]
    nac, own = p.nac, u[:, 2:-2, 2:-2, 2:-2]
    if form == 1:
        # the coupling th d s, d = c - c0, is the one term that _numpy subtracts
        e = _numpy(q, u, 1)[:, 3]
        if p.nch:
            h3 = p.xmax * p.ymax * p.zmax / own[0].size
            e = e + 2 * q.landau[4] * h3 * sum((np.abs(own[nac] - q.landau[5]).max() * (f ** 2).sum()) for f in own[:nac])
        return e
    s = (own[:nac] ** 2).sum(0) if nac else 0.0
    h3 = p.xmax * p.ymax * p.zmax / own[0].size
    add = 2 * (7128.0 + 12 * 2372) / 2372 / 3 * (np.abs(own[:nac]) ** 3).sum() if nac else 0.0
    e = _numpy(p, u, 0)[:, 3]
    return np.array([abs(e[f]) + h3 * (add if f < nac else ((own[nac] ** 2 + 1) ** 2).sum()) for f in range(len(own))])


@pytest.mark.parametrize("N,nac,nch", [(4, 1, 0), (7, 0, 1), (8, 4, 1), (9, 2, 1), (33, 4, 0), (41, 3, 1), (65, 4, 1)])
@pytest.mark.parametrize("form", [0, 1])
def test_fp32_diagnostics_match_numpy(N, nac, nch, form, sclet_lib):
    """The FP32 form on the values the state holds: maxima and minima exact, FP64
    sums of the FP32 values, energies to the FP32 roundings of a cell, at most 40
    of 2^-24 of its terms' sizes."""
    sg = sclet_lib
    p = sg.default_params()
    n = N + 4
    p.nx = p.ny = p.nz = n
    p.xmax, p.ymax, p.zmax = 0.5 * N, 0.4 * N, 0.6 * N
    p.kkx, p.kky, p.kkz = 1.0, 0.7, 0.4
    p.nac, p.nch, p.elastic = nac, nch, 0
    u = np.random.default_rng(N).uniform(0.2, 0.9, size=(nac + nch, n, n, n))
    s = sg.Solver(p, sg.MIXED)
    s.set_fields(u)
    u = s.get_fields()
    got = s.check_soln(form)
    s.close()
    want = _numpy(p, u, form)
    np.testing.assert_array_equal(got[:, :2], want[:, :2])
    np.testing.assert_allclose(got[:, 2], want[:, 2], rtol=1e-12)  # pairs of 13 terms: 13^2 2^-49
    assert np.all(np.abs(got[:, 3] - want[:, 3]) <= 40 * 2.0 ** -24 * _magnitudes(p, u, form))


def test_fp32_volume_keeps_more_than_an_fp32_pair(sclet_lib):
    """One cell each of two warps' columns away from -1, the sum 2 + 2^-20 + 2^-43 +
    2^-45: every warp's sum is an exact FP32 pair, theirs together is not."""
    sg = sclet_lib
    p = sg.default_params()
    p.nx = p.ny = p.nz = 12
    p.xmax = p.ymax = p.zmax = 8.0
    p.nac, p.nch, p.elastic = 1, 0, 0
    u = np.full((1, 12, 12, 12), -1.0)
    u[0, 2, 2, 2] = 2.0 ** -20 + 2.0 ** -43
    u[0, 2, 3, 2] = 2.0 ** -45
    s = sg.Solver(p, sg.MIXED)
    s.set_fields(u)
    np.testing.assert_array_equal(s.get_fields(), u)
    assert s.check_soln(1)[0, 2] == 2.0 + 2.0 ** -20 + 2.0 ** -43 + 2.0 ** -45
    s.close()
