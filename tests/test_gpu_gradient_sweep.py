"""The alignment gradient of a batch of several wavelengths, on a handle whose
wavelengths have only just been set, with and without a reference calibration.

Reference for IL: every wavelength's frames as a batch of their own on another
handle; with g_l its gradient and S_l = 10^(IL_l / 10) its captured power, the
sweep's S is their sum and its gradient sum(g_l S_l) / S.  The two sides place
the Fourier window alike and round the fields to int16 alike but for the last
bit of a few pixels: 5e-5 of the coefficients, a twentieth of them in the
gradient, so 1e-3 of the gradient's norm in step-normalised coordinates; the IL
within 1e-3 dB.

Reference for MDL, whose weights mix the wavelengths: central differences of
the value, as for a single wavelength: cosine >= 0.99, each component within
5 % of the norm."""
import ctypes as C

import numpy as np
import pytest

from helpers import ref_calibration, set_ref_calibration
from test_gpu_adjoint import KINDS, _case, _get, _grad, _grad_metric, _perturbed, _set, _steps
from digholo_b200 import api

pytestmark = pytest.mark.gpu

LAMBDA = np.array([1564.4e-9, 1565e-9, 1565.9e-9], np.float32)
STEP = np.array([0.1, 0.1, 0.4, 3e-5, 3e-5, 3e-5] * 2)


@pytest.fixture(scope="module")
def lib():
    import digholo_b200
    return digholo_b200.load()


def _open(lib, cfg, frames, calibration=None):
    """A configured handle with its frames set; nothing has run on it."""
    h = lib.digHoloCreate()
    api.configure(lib, h, cfg)
    if calibration is not None:
        set_ref_calibration(lib, h, cfg, "intensity", calibration)
    frames = np.ascontiguousarray(frames)
    assert api.set_batch(lib, h, frames) == 0
    return h, frames


def _wavelengths(lib, h, lams, orders=(0, 0)):
    lams = np.ascontiguousarray(lams, np.float32)
    assert lib.digHoloConfigSetWavelengths(h, lams.ctypes.data_as(C.POINTER(C.c_float)), len(lams)) == 0
    for i, order in enumerate(orders):
        assert lib.digHoloConfigSetWavelengthOrdering(h, i, order) == 0


def _close(a, b):
    a, b = np.ravel(a) * STEP, np.ravel(b) * STEP
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("orders,calibrated,max_mg", [((0, 0), False, 9), ((1, 0), False, 6), ((0, 1), True, 9)])
def test_il_gradient_of_a_sweep(lib, orders, calibrated, max_mg):
    hol = _case(6)
    cfg = _perturbed(hol, 0)
    cfg.max_mg = max_mg
    L, S = len(LAMBDA), 2
    cal = np.repeat(ref_calibration(cfg, "intensity"), L, axis=0) if calibrated else None
    total, want = 0.0, 0.0
    for l, lam in enumerate(LAMBDA):
        one = _perturbed(hol, 0)
        one.max_mg, one.wavelength = max_mg, float(lam)
        h, keep = _open(lib, one, hol.frames[l::L] if orders[0] == 0 else hol.frames[l * S:(l + 1) * S],
                        cal[:1] if calibrated else None)
        g, il = _grad(lib, h)
        lib.digHoloDestroy(h)
        s = 10.0 ** (il / 10.0)
        total, want = total + s, want + s * g
    h, keep = _open(lib, cfg, hol.frames, cal)
    _wavelengths(lib, h, LAMBDA, orders)
    for _ in range(2):   # the array is pending, then in use
        g, il = _grad(lib, h)
        assert abs(il - 10.0 * np.log10(total)) <= 1e-3
        assert _close(g, want / total) <= 1e-3
    # back to one wavelength: again the first evaluation that sees the array
    _wavelengths(lib, h, LAMBDA[1:2])
    got = _grad(lib, h)[0]
    lib.digHoloDestroy(h)
    h, keep = _open(lib, cfg, hol.frames, cal[:1] if calibrated else None)
    assert _close(got, _grad(lib, h)[0]) <= 1e-3
    lib.digHoloDestroy(h)


@pytest.mark.parametrize("orders", [(0, 0), (0, 1)])
def test_mdl_gradient_of_a_sweep(lib, orders):
    hol = _case(33)
    cfg = _perturbed(hol, 0)
    h, keep = _open(lib, cfg, hol.frames)
    _wavelengths(lib, h, LAMBDA, orders)
    assert lib.digHoloB200FreezeWindow(h, 1) == 0
    g = _grad_metric(lib, h, 1)[0]
    steps = _steps(lib, h, cfg)
    entries = [(pol, k) for pol in (0, 1) for k in KINDS[:5]] + [(None, "waist")]
    ga, gf = [], []
    for pol, kind in entries:
        base, d = _get(lib, h, pol or 0, kind), 0.05 * steps[kind]
        vals = []
        for sign in (1, -1):
            _set(lib, h, pol or 0, kind, base + sign * d)
            vals.append(_grad_metric(lib, h, 1)[1])
        _set(lib, h, pol or 0, kind, base)
        gf.append((vals[0] - vals[1]) / (2 * d) * steps[kind])
        ga.append((g[0, 5] + g[1, 5] if pol is None else g[pol, KINDS.index(kind)]) * steps[kind])
    lib.digHoloDestroy(h)
    ga, gf = np.array(ga), np.array(gf)
    norm = np.linalg.norm(gf)
    assert ga @ gf / (np.linalg.norm(ga) * norm) >= 0.99
    assert np.abs(ga - gf).max() <= 0.05 * norm


def test_refused_gradient_leaves_the_whole_batch(lib):
    """A Laguerre-Gaussian output basis is refused after the batch, whose frames of all wavelengths stay."""
    hol = _case(6)
    cfg = _perturbed(hol, 0)
    cfg.max_mg, cfg.basis_type = 4, 1
    h, keep = _open(lib, cfg, hol.frames)
    _wavelengths(lib, h, LAMBDA)
    want = api.run_batch(lib, h, hol.frames)
    g, il = (C.c_float * 12)(), C.c_float()
    assert lib.digHoloB200AutoAlignGradient(h, g, C.byref(il)) == 8
    b, m, p = C.c_int(), C.c_int(), C.c_int()
    cp = lib.digHoloProcessBatch(h, C.byref(b), C.byref(m), C.byref(p))
    lib.digHoloB200AutoAlignGradient(h, g, C.byref(il))
    again = api.read_outputs(lib, h, 6, cp, m.value, p.value, True)
    lib.digHoloDestroy(h)
    assert again["R"].shape == want["R"].shape and np.array_equal(again["R"], want["R"])
    assert np.array_equal(again["coefs"], want["coefs"])
