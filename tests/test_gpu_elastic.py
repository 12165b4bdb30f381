"""The elastic force's fused contraction (z-lines forward, Green tensor, z-lines
backward in one kernel) against the FP64 form's separate passes."""
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
