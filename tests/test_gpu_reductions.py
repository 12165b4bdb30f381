"""Diagnostics of check_soln_new where the reduction's shapes meet their edges:
owned edges around the 32 x 8 column tile and the eight-plane unit, several
field counts, both energy forms, against numpy.  (The FP32 form of the same walk
is held to the FP64 one by test_gpu_mixed.py's energy curves.)"""
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
