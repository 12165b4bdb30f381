"""Ghost cells done in place, tree by tree, against the rule they come from: a
ghost takes the previous value at its image along its first ghost axis (z, y, x)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _exchange(block):
    """The block with its ghosts taken from the block as it was."""
    n = block.shape[0]
    i = np.arange(n)
    ghost = (i < 2) | (i >= n - 2)
    wrap = np.where(i < 2, i + n - 4, np.where(i >= n - 2, i - n + 4, i))
    z, y, x = np.meshgrid(i, i, i, indexing="ij")
    gz, gy = ghost[z], ghost[y]
    return block[np.where(gz, wrap[z], z), np.where(~gz & gy, wrap[y], y), np.where(~gz & ~gy, wrap[x], x)]


def _solver(sg, N, nac, precision, elastic):
    p = sg.default_params()
    p.nx = p.ny = p.nz = N + 4
    p.xmax = p.ymax = p.zmax = float(N)
    p.nac, p.nch, p.elastic = nac, 1, elastic
    s = sg.Solver(p, precision)
    u = np.random.default_rng(N).standard_normal((nac + 1,) + (N + 4,) * 3).astype(np.float32).astype(np.float64)
    s.set_fields(u)
    return s, s.get_fields()


# 4: every owned cell is within two of a face along each axis
@pytest.mark.parametrize("N", [4, 5, 7, 33])
@pytest.mark.parametrize("precision_name", ["FP64", "MIXED"])
def test_field_ghosts(N, precision_name, sclet_lib):
    s, u = _solver(sclet_lib, N, 2, getattr(sclet_lib, precision_name), 0)
    s.transfer()
    got = s.get_fields()
    s.close()
    for f in range(3):
        np.testing.assert_array_equal(got[f], _exchange(u[f]))


@pytest.mark.parametrize("N,nac", [(4, 1), (5, 2), (9, 3), (16, 4)])
@pytest.mark.parametrize("precision_name", ["FP64", "MIXED"])
def test_elastic_ghosts(N, nac, precision_name, sclet_lib):
    """One block exchanged field after field, over two calls."""
    s, _ = _solver(sclet_lib, N, nac, getattr(sclet_lib, precision_name), 1)
    own = (slice(2, -2),) * 3
    block = np.zeros((N + 4,) * 3)
    for call in range(2):
        s.elastic()
        got = s.get_felas()
        for p in range(nac):
            block[own] = got[p][own]
            block = _exchange(block)
            np.testing.assert_array_equal(got[p], block)
    s.close()
