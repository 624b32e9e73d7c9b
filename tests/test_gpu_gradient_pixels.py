"""The alignment gradient from the pixels, which a reference calibration that
varies over the field asks for, with each of its kernels: four and two columns
a thread (up to 256 rows and 16 groups, 128 rows and 32 groups), one column a
thread (512 rows; 256 rows beyond 16 groups) and the plain one (beyond 32
groups).

Reference: the library's float fields V, calibration planes and coefficients c,
with the tangents dV formed in 64 bits (the beam centre's through the spectrum
of V freed of reference wave and calibration).  Each component 20 / ln 10
Re sum conj(c) dc / sum |c|^2 within the rounding of its FP32 sums, relative to
|c| |dc|: at most 4096 terms in a row, 6e-8 each, growing with the square root
of their number: 4e-6 (the gradient itself is some 1e-3 of it)."""
import ctypes as C

import numpy as np
import pytest
import torch

from helpers import ref_calibration, ref_calibration_planes, set_ref_calibration
from test_gpu_gradient_window import _case, cases, wave   # noqa: F401 (cases: fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,over", [
    ("field", dict(groups=9)), ("intensity", dict(groups=16, carrier=0.55, pols=1)), ("field", dict(groups=6, mode=1)),
    ("field", dict(groups=20, carrier=0.55)), ("field", dict(groups=8, window=256, width=1280, height=1024, frames=3)),
    ("field", dict(groups=20, window=256, width=1280, height=1024, frames=3)),
    ("field", dict(groups=9, window=512, width=2048, height=2048, frames=2)),
    ("intensity", dict(groups=36, carrier=0.55, frames=3)),
], ids=lambda o: o if isinstance(o, str) else "-".join("%s%s" % kv for kv in o.items()))
def test_against_fields(cases, kind, over):   # noqa: F811
    c = _case(**over)
    s = cases.prepare(c, 1)
    cal = ref_calibration(s.cfg, kind)
    set_ref_calibration(s.L, s.h, s.cfg, kind, cal)
    assert s.L.digHoloB200SetKeepField32(s.h, 1) == 0
    got = cases.run(s)["gradient"]
    b, p, w, h = C.c_int(), C.c_int(), C.c_int(), C.c_int()
    v = s.L.digHoloB200GetFields32(s.h, C.byref(b), C.byref(p), C.byref(w), C.byref(h))
    shape = (b.value, p.value, h.value, w.value)
    V = np.ctypeslib.as_array(v, shape=(2 * int(np.prod(shape)),)).copy().view(np.complex64).reshape(shape)
    e = cases.Exact(c, 1)
    V, coefs = (torch.as_tensor(a, device=e.dev).to(torch.complex128) for a in (V, s.device_coefs()))
    planes = torch.as_tensor(ref_calibration_planes(s.L, s.h)[0], device=e.dev).to(torch.complex128)
    assert float(planes.abs().std() / planes.abs().mean()) > 1e-3   # it varies over the pixels, far above the bound
    base, k0, u = e.settings(), 2 * np.pi / 1565e-9, np.pi / 180
    x, y = e.t(e.axis(e.nx))[None, :], e.t(e.axis(e.ny))[:, None]
    unit = 20.0 / np.log(10.0) / float((coefs.abs() ** 2).sum())
    want, bound = np.zeros(12), np.zeros(12)
    for p in range(c["pols"]):
        F, (bx, by), (tx, ty), cp = V[:, p], base["centre"][p], base["tilt"][p], coefs[:, p]
        R = wave(e, p, base) * planes[p]
        spec = torch.fft.fft2(-F.conj() / R)
        k = [torch.zeros(n, dtype=torch.float64, device=e.dev) for n in (e.nx, e.ny)]
        k[0][torch.as_tensor(e.cols[p] % e.n if e.full else np.arange(e.w), device=e.dev)] = e.t(e.k[e.cols[p]])
        k[1][torch.as_tensor(e.rows[p] if e.full else np.arange(e.h), device=e.dev)] = e.t(e.k[e.rows[p]])
        Fx = -(torch.fft.ifft2(spec * 1j * k[0][None, :]) * R).conj()
        Fy = -(torch.fft.ifft2(spec * 1j * k[1][:, None]) * R).conj()
        dc = [e.coefs(p, t, base) for t in (F * 1j * k0 * u * (x + bx), F * 1j * k0 * u * (y + by),
                                            F * 1j * np.pi / 1565e-9 * (x * x + y * y),
                                            Fx + F * 1j * k0 * u * tx, Fy + F * 1j * k0 * u * ty)]
        step = 2e-8
        dc.append((e.coefs(p, F, dict(base, waist=base["waist"] + step)) -
                   e.coefs(p, F, dict(base, waist=base["waist"] - step))) / (2 * step))
        for i, d in enumerate(dc):
            at = i if i == 5 else 6 * p + i   # the waist is one for both polarisations
            want[at] += unit * float((cp.conj() * d).real.sum())
            bound[at] += unit * 4e-6 * float(cp.norm() * d.norm())
    assert (np.abs(np.asarray(got, float) - want) <= bound).all(), (got, want, bound)
