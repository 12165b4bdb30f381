"""The conserved field's mass (k_mass.cu) by its kernels' entry points: target,
sum of the owned cells and shift, where their shapes meet edges, and the
precision their sums are held in.  Inputs are small multiples of powers of two,
so every sum has one exact value."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _entry(sg, name, *args):
    f = getattr(sg.lib(), name)
    f.restype, f.argtypes = ctypes.c_int, args
    return f


PTR = ctypes.c_void_p


def _mass(sg, u, b, bsub, wa, wb):
    """(target, sum before, shifted u): u, b, bsub FP32 blocks, wa, wb FP32 weights
    (their low halves zero); wa None: the owned cells' sum."""
    torch = pytest.importorskip("torch")
    target = _entry(sg, "_ZN5sclet11mass_targetEPKfPKdS1_S1_S3_iPdP11CUstream_st", PTR, PTR, PTR, PTR, PTR,
                    ctypes.c_int, PTR, PTR)
    fix = _entry(sg, "_ZN5sclet8mass_fixEPfiPKdPdS3_P11CUstream_st", PTR, ctypes.c_int, PTR, PTR, PTR, PTR)
    parts = _entry(sg, "_ZN5sclet13mass_partialsEv")()
    dev = lambda a: None if a is None else torch.from_numpy(np.ascontiguousarray(a)).cuda()
    pair = lambda w: None if w is None else np.stack([w, np.zeros_like(w)], axis=-1)
    du, db, ds, dwa, dwb = dev(u), dev(b), dev(bsub), dev(pair(wa)), dev(pair(wb))
    part = torch.full((4 * parts,), float("nan"), dtype=torch.float64, device="cuda")
    res = torch.zeros(4, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    at = lambda t: None if t is None else t.data_ptr()
    n = u.shape[0]
    assert target(at(du), at(dwa), at(db), at(ds), at(dwb), n, part.data_ptr(), None) == 0
    assert fix(at(du), n, part.data_ptr(), part.data_ptr() + 16 * parts, res.data_ptr(), None) == 0
    torch.cuda.synchronize()
    r = res.cpu().numpy()
    return r[0], r[1], du.cpu().numpy()


# a block smaller than a CTA, odd ones, a row of one and of several loads a lane,
# one and several cells a thread
@pytest.mark.parametrize("n", [8, 9, 36, 67, 101, 137])
@pytest.mark.parametrize("corrector", [False, True])
def test_mass_target_and_shift(n, corrector, sclet_lib):
    """Multiples of 2^-10 below 1 (products: of 2^-20): no sum of a block rounds."""
    rng = np.random.default_rng(n)
    draw = lambda: (rng.integers(-1023, 1024, size=(n, n, n)) / 1024.0).astype(np.float32)
    u, b, wb = draw(), draw(), draw()
    bsub, wa = (draw(), None) if corrector else (None, draw())
    own = (slice(2, -2),) * 3
    d = lambda a: a.astype(np.float64)
    T, A, v = _mass(sclet_lib, u, b, bsub, wa, wb)
    want = (d(u)[own].sum() if corrector else (d(wa) * d(u)).sum()) + (d(wb) * (d(b) - (d(bsub) if corrector else 0))).sum()
    assert T == want and A == d(u)[own].sum()
    ref = u.copy()
    ref[own] += np.float32((T - A) / (n - 4.0) ** 3)
    np.testing.assert_array_equal(v, ref)


def test_mass_sums_keep_more_than_an_fp32_pair(sclet_lib):
    """Three cells of one warp whose sum has 51 bits: the pairs of different
    threads are merged in FP64."""
    n = 8
    u = np.zeros((n, n, n), np.float32)
    u[2, 2, 2:5] = 1.0, 2.0 ** -25 + 2.0 ** -48, 2.0 ** -50
    exact = math.fsum(u[2, 2, 2:5].astype(np.float64))
    assert exact == 1.0 + 2.0 ** -25 + 2.0 ** -48 + 2.0 ** -50
    zero = np.zeros_like(u)
    T, A, _ = _mass(sclet_lib, u, zero, zero, None, zero)
    assert T == exact and A == exact
