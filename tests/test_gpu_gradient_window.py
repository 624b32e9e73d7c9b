"""The alignment gradient from the Fourier windows, over window sides, field
sizes, resolutions, polarisations and group counts (odd, even, one; the middle
mode of an odd count meets its own mirror), and the window path against the
pixel path.

Reference: the library's own float fields V and coefficients c, with the
tangents dV of the adjoint formed from the pixels in 64 bits (the beam centre's
through V's own spectrum): grad = 20 / ln 10 Re sum conj(c) dc / sum |c|^2.
Both sides then share the phases of V, on which the small real part of
conj(c) dc depends.  Tolerance, of the gradient's norm in step-normalised
coordinates: FP32 products (1e-7) against a gradient that is 1e-3 of |c| |dc|:
1e-4.  The pixel path rounds the fields to int16 anew (5e-5 of the
coefficients, a twentieth of them in the gradient): 1e-3."""
import ctypes as C
import importlib.util
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

STEP = np.array([0.1, 0.1, 0.4, 3e-5, 3e-5, 3e-5] * 2)   # tilt, defocus, beam centre, waist


@pytest.fixture(scope="module")
def cases():
    path = os.path.join(os.path.dirname(__file__), "..", "perf", "cases.py")
    spec = importlib.util.spec_from_file_location("perf_cases", path)
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


def _case(**over):
    c = dict(name="gradient", frames=8, width=640, height=512, dtype="float32", pols=2, window=128, groups=9, mode=0,
             carrier=0.25, call="gradient", average=1)
    c.update(over)
    return c


def _close(a, b):
    a, b = np.asarray(a, float) * STEP, np.asarray(b, float) * STEP
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("over", [
    dict(groups=1), dict(groups=2), dict(groups=9, frames=1), dict(groups=15, carrier=0.55, frames=301),
    dict(groups=16, carrier=0.55), dict(groups=20, carrier=0.55, dtype="uint16"), dict(groups=5, pols=1),
    dict(groups=6, mode=1), dict(groups=9, mode=1, carrier=0.55), dict(groups=6, window=64, width=320, height=256, pols=1),
    dict(groups=8, window=256, width=1280, height=1024), dict(groups=9, average=2),
    dict(groups=15, window=512, width=2048, height=2048, carrier=0.55, frames=2),   # tables and window beyond shared memory
], ids=lambda o: "-".join("%s%s" % kv for kv in o.items()))
def test_against_fields(cases, over):
    c = _case(**over)
    s = cases.prepare(c, 1)
    assert s.L.digHoloB200SetKeepField32(s.h, 1) == 0
    got = cases.run(s)["gradient"]
    b, p, w, h = C.c_int(), C.c_int(), C.c_int(), C.c_int()
    v = s.L.digHoloB200GetFields32(s.h, C.byref(b), C.byref(p), C.byref(w), C.byref(h))
    shape = (b.value, p.value, h.value, w.value)
    V = np.ctypeslib.as_array(v, shape=(2 * int(np.prod(shape)),)).copy().view(np.complex64).reshape(shape)
    e = cases.Exact(c, 1)
    V = torch.as_tensor(V, device=e.dev).to(torch.complex128)
    assert _close(got, reference(e, c, V, s.device_coefs().to(torch.complex128))) <= 1e-4


def reference(e, c, V, coefs):
    base, out = e.settings(), np.zeros(12)
    k0, u = 2 * np.pi / 1565e-9, np.pi / 180
    x, y = e.t(e.axis(e.nx))[None, :], e.t(e.axis(e.ny))[:, None]
    for p in range(c["pols"]):
        F, (bx, by), (tx, ty) = V[:, p], base["centre"][p], base["tilt"][p]
        # the conjugate of A R, and of A_x R and A_y R: R out, i k in the spectrum, R in
        R = wave(e, p, base)
        spec = torch.fft.fft2(-F.conj() / R)
        kx, ky = (torch.zeros(n, dtype=torch.float64, device=e.dev) for n in (e.nx, e.ny))
        cols = np.arange(e.w) if not e.full else e.cols[p] % e.n
        rows = np.arange(e.h) if not e.full else e.rows[p]
        kx[torch.as_tensor(cols, device=e.dev)] = e.t(e.k[e.cols[p]])
        ky[torch.as_tensor(rows, device=e.dev)] = e.t(e.k[e.rows[p]])
        Fx = -(torch.fft.ifft2(spec * 1j * kx[None, :]) * R).conj()
        Fy = -(torch.fft.ifft2(spec * 1j * ky[:, None]) * R).conj()
        tangents = [F * 1j * k0 * u * (x + bx), F * 1j * k0 * u * (y + by), F * 1j * np.pi / 1565e-9 * (x * x + y * y),
                    Fx + F * 1j * k0 * u * tx, Fy + F * 1j * k0 * u * ty]
        dc = [e.coefs(p, t, base) for t in tangents]
        step = 2e-8
        dc.append((e.coefs(p, F, dict(base, waist=base["waist"] + step)) -
                   e.coefs(p, F, dict(base, waist=base["waist"] - step))) / (2 * step))
        for k, d in enumerate(dc):
            g = float((coefs[:, p].conj() * d).real.sum())
            out[k if k == 5 else 6 * p + k] += 20.0 / np.log(10.0) * g / float((coefs.abs() ** 2).sum())
    return out


def wave(e, p, q):
    """The reference wave: the field of a window that holds one frequency, over that frequency's wave."""
    win = torch.zeros((1, e.h, e.w), dtype=torch.complex128, device=e.dev)
    win[0, 0, 0] = 1.0
    V = e.field(p, win, q)[0]
    col, row = (int(e.cols[p][0]), int(e.rows[p][0])) if e.full else (0, 0)
    ax = torch.arange(e.nx, device=e.dev, dtype=torch.float64)[None, :] * (col / e.nx)
    ay = torch.arange(e.ny, device=e.dev, dtype=torch.float64)[:, None] * (row / e.ny)
    return -V.conj() / torch.exp(2j * np.pi * (ax + ay))


@pytest.mark.parametrize("over", [dict(groups=9), dict(groups=20, carrier=0.55), dict(groups=6, mode=1)],
                         ids=lambda o: "-".join("%s%s" % kv for kv in o.items()))
def test_against_pixels(cases, over):
    """A uniform reference calibration scales every field alike: the same gradient of IL, from the pixels."""
    c = _case(**over)
    s = cases.prepare(c, 2)
    got = cases.run(s)["gradient"].copy()
    cal = np.full((1, c["height"], c["width"]), 20000, dtype=np.uint16)
    assert s.L.digHoloConfigSetRefCalibrationIntensity(s.h, cal.ctypes.data_as(C.POINTER(C.c_ushort)), 1, c["width"], c["height"]) == 0
    assert s.L.digHoloConfigSetRefCalibrationEnabled(s.h, 1) == 0
    assert _close(cases.run(s)["gradient"], got) <= 1e-3
