"""The elastic force's fused contraction (z-lines forward, Green tensor, z-lines
backward in one kernel) against the FP64 form's separate passes, and what the
generic passes round."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 8 lines a CTA (32, 64), 16 (192, 256); one grid (1 and 2 fields) and two
@pytest.mark.parametrize("N,nac", [(32, 1), (32, 2), (32, 3), (64, 4), (80, 3), (192, 2), (256, 4)])
def test_fused_contraction(N, nac, sclet_lib):
    """White noise, so every mode pair counts, the planes of 0 and N / 2 too.
    FP32 transforms of N^3 points round by about sqrt(log2 N^3) 2^-24 of the
    force's norm each way, 5e-7 together at 256: 2e-6."""
    sg = sclet_lib
    p = sg.default_params()
    p.nx = p.ny = p.nz = N + 4
    p.xmax = p.ymax = p.zmax = float(N)
    p.nac, p.nch, p.elastic = nac, 1, 1
    rng = np.random.default_rng(N + nac)
    u = rng.standard_normal((nac + 1, N + 4, N + 4, N + 4)) * 0.3
    own = (slice(2, -2),) * 3
    out = {}
    for prec in (sg.FP64, sg.MIXED):
        s = sg.Solver(p, prec)
        s.set_fields(u)
        s.elastic()
        out[prec] = s.get_felas()
        s.close()
    for m in range(nac):
        a, b = out[sg.MIXED][m][own], out[sg.FP64][m][own]
        assert np.linalg.norm(a - b) <= 2e-6 * np.linalg.norm(b), (N, nac, m)


@pytest.mark.parametrize("N", [6, 12, 18, 24])
def test_generic_force_is_scaled_with_one_rounding(N, sclet_lib):
    """A uniform field: every sum of the generic FP32 transforms is exact, so the
    force is the Green tensor's product at k = 0 times 1 / N^3, each rounded once."""
    sg = sclet_lib
    p = sg.default_params()
    p.nx = p.ny = p.nz = N + 4
    p.xmax = p.ymax = p.zmax = float(N)
    p.nac, p.nch, p.elastic = 1, 0, 1

    def force(s, c):
        s.set_fields(np.full((1, N + 4, N + 4, N + 4), c))
        s.elastic()
        f = s.get_felas()[0][2:-2, 2:-2, 2:-2]
        assert np.all(f == f[0, 0, 0])
        return f[0, 0, 0]

    s = sg.Solver(p, sg.FP64)
    b0 = np.float32(force(s, 1.0))
    s.close()
    s = sg.Solver(p, sg.MIXED)
    for m in range(1, 256, 5):
        c = m / 256.0
        x = b0 * np.float32(2.0 * N ** 3 * c)
        assert force(s, c) == np.float32(np.float64(x) * (0.5 / N ** 3)), m
    s.close()


def _force(p, u):
    """Re IFFT(sum_q B_pq FFT(eta_q)) of the owned cells, B evaluated at every wave
    vector of the scheme's convention (0 .. N/2 - 1, then negative)."""
    N, nac = u.shape[-1], len(u)
    C6 = np.array(p.voigt).reshape(6, 6)
    v = np.array([[0, 5, 4], [5, 1, 3], [4, 3, 2]])
    C = C6[v[:, :, None, None], v[None, None]]
    eps = np.array(p.eigenstrain).reshape(4, 3, 3)[:nac]
    sig = np.einsum("ijkl,qkl->qij", C, eps)
    k = np.arange(N)
    k = np.where(k < N // 2, k, k - N).astype(float)
    n = np.stack(np.meshgrid(k, k, k, indexing="ij")[::-1], axis=-1)  # (x, y, z) at [z, y, x]
    r = np.sqrt((n ** 2).sum(-1, keepdims=True))
    r[0, 0, 0] = 1.0
    n /= r
    n[0, 0, 0] = 0.0, 1.0, 0.0
    om = np.linalg.inv(np.einsum("ijkl,...j,...l->...ik", C, n, n))
    w = np.einsum("qij,...j->q...i", sig, n)
    h = np.fft.fftn(u, axes=(1, 2, 3))
    out = []
    for a in range(nac):
        left = np.einsum("...i,...ij->...j", w[a], om)
        out.append(np.fft.ifftn(sum(((sig[a] * eps[q]).sum() - (left * w[q]).sum(-1)) * h[q] for q in range(nac))).real)
    return np.array(out)


# odd edges, whose two middle wave numbers have no mirror of their own, and edges
# whose last tile of lines is partial
@pytest.mark.parametrize("N,nac", [(15, 3), (25, 1), (27, 4), (45, 2), (75, 4), (20, 4), (50, 3), (100, 2)])
@pytest.mark.parametrize("precision_name", ["FP64", "MIXED"])
def test_generic_passes_match_numpy(N, nac, precision_name, sclet_lib):
    """White noise.  Transforms of N^3 points round by about sqrt(log2 N^3) of the
    precision's unit each way: 1e-15 and 5e-7 at 100, with a margin of four
    (FP64: of the direction cosines and their inverse too, 1e-13)."""
    sg = sclet_lib
    p = sg.default_params()
    p.nx = p.ny = p.nz = N + 4
    p.xmax = p.ymax = p.zmax = float(N)
    p.nac, p.nch, p.elastic = nac, 0, 1
    u = (np.random.default_rng(N).standard_normal((nac,) + (N + 4,) * 3) * 0.3).astype(np.float32).astype(np.float64)
    s = sg.Solver(p, getattr(sg, precision_name))
    s.set_fields(u)
    s.elastic()
    got = s.get_felas()[:, 2:-2, 2:-2, 2:-2]
    s.close()
    want = _force(p, u[:, 2:-2, 2:-2, 2:-2])
    tol = 1e-13 if precision_name == "FP64" else 2e-6
    for m in range(nac):
        assert np.linalg.norm(got[m] - want[m]) <= tol * np.linalg.norm(want[m]), m
