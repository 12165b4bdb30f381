"""Allen-Cahn right-hand side: the kernels without a shared-memory ring (no
gradient tensor, diagonal tensors) against the general one, over block edges
where the faces, the two-cell neighbourhoods and the (x, y) tiles meet."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu


def _rhs(sg, N, nac, nch, precision, lam, kk):
    p = sg.default_params()
    p.nx = p.ny = p.nz = N + 4
    p.xmax = p.ymax = p.zmax = 0.5 * N
    p.nac, p.nch, p.elastic, p.anisotropic = nac, nch, 0, 1
    p.kkx, p.kky, p.kkz = kk
    for m in range(4):
        for k in range(9):
            p.lambda_file[9 * m + k] = float(lam[m][k // 3, k % 3])
    s = sg.Solver(p, precision)
    n = N + 4
    u = np.random.default_rng(N * 10 + nac).uniform(-0.5, 0.5, size=(nac + nch, n, n, n))
    s.set_fields(u)
    s.calc_rhs(1)
    out = s.get_rhs(1)
    s.close()
    return out


@pytest.mark.parametrize("N,nac,nch", [(4, 1, 0), (5, 2, 1), (7, 3, 0), (27, 4, 1), (29, 4, 0), (61, 1, 1)])
@pytest.mark.parametrize("precision_name", ["FP64", "MIXED"])
def test_diagonal_tensors_match_the_general_kernel(N, nac, nch, precision_name, sclet_lib):
    """An off-diagonal entry of 1e-20 sends the run to the general kernel and
    adds less than 1e-18 to any value.  Both sum the same dozen terms of
    magnitude up to 50 into values of about 3 (root mean square), in one order up to the contraction
    of products: a few roundings of 2^-24 (FP32) or 2^-53."""
    sg = sclet_lib
    lam = [np.diag([0.5 + 0.1 * m, 0.2, 0.3 - 0.05 * m]) for m in range(4)]
    off = [a + 1e-20 * (np.ones((3, 3)) - np.eye(3)) for a in lam]
    prec = getattr(sg, precision_name)
    kk = (0.5, 0.6, 0.7)
    got, want = _rhs(sg, N, nac, nch, prec, lam, kk), _rhs(sg, N, nac, nch, prec, off, kk)
    tol = 2e-6 if precision_name == "MIXED" else 4e-15
    for f in range(nac):
        err = np.linalg.norm(got[f] - want[f]) / np.linalg.norm(want[f])
        assert err <= tol, (f, err)
        assert np.max(np.abs(got[f] - want[f])) <= 20 * tol * np.max(np.abs(want[f])), f


@pytest.mark.parametrize("N,nac", [(4, 1), (5, 3), (30, 4)])
@pytest.mark.parametrize("precision_name", ["FP64", "MIXED"])
def test_no_gradient_tensor_is_pointwise_plus_lifting(N, nac, precision_name, sclet_lib):
    """With the Landau plugin and no anisotropic term: LE KE e - LE f'(e) plus
    LE epn2 e(outside) / h^2 per face, against numpy."""
    sg = sclet_lib
    p = sg.default_params()
    n = N + 4
    p.nx = p.ny = p.nz = n
    p.xmax = p.ymax = p.zmax = 0.5 * N
    p.nac, p.elastic = nac, 0
    s = sg.Solver(p, getattr(sg, precision_name))
    u = np.random.default_rng(N).uniform(-0.5, 0.5, size=(nac, n, n, n)).astype(np.float32).astype(np.float64)
    s.set_fields(u)
    s.calc_rhs(1)
    got = s.get_rhs(1)
    s.close()
    a2, a4, a6, g, _, _, _, LE, KE = list(p.landau)[:9]
    i = (np.arange(n) - 2) % N + 2
    lo, hi = (-3) % N + 2, (n - 2) % N + 2
    tol = 1e-6 if precision_name == "MIXED" else 2e-15
    for m in range(nac):
        e = u[m]
        others = sum(u[q] ** 2 for q in range(nac) if q != m)
        want = LE * KE * e - LE * (a2 * e + a4 * e ** 3 + a6 * e ** 5 + 2 * g * e * others)
        w = LE * p.epn2 / 0.25
        for ax in range(3):
            for at, q in ((0, lo), (n - 1, hi)):
                face = np.take(e, q, axis=ax)[np.ix_(i, i)]
                sl = [slice(None)] * 3
                sl[ax] = at
                want[tuple(sl)] += w * face
        assert np.linalg.norm(got[m] - want) <= tol * np.linalg.norm(want), m


@pytest.mark.parametrize("N,nac", [(4, 1), (5, 2), (30, 1)])
def test_variable_mobility_edges(N, nac, tmp_path, sclet_lib, oracle_lib):
    """The variable-mobility kernels' march and face cells where the block's
    edge meets their planes and CTAs, two steps against the oracle: roundings of
    2^-53 in sums of about thirty terms, amplified by h^-4 and the step."""
    from test_gpu_parity import _oracle_vs_gpu
    case = cases.Case(big_n=N, nac=nac, nch=1, elastic=0, steps=2, seed=N, eta_range=(0.0, 0.9), variable_mobility=1,
                      suffix="vme")
    errs, _, _ = _oracle_vs_gpu(tmp_path, sclet_lib, oracle_lib, case, 2)
    assert max(errs) <= 1e-10, errs
