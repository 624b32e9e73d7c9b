"""The alignment gradient beyond 120 mode groups, whose coefficients exceed the
shared memory of the kernel that takes the Fourier windows: from the pixels.

So many modes span the small fields that still fit, the captured power hardly
depends on the alignment, and the gradient is a small remainder of sum conj(c)
dc.  It is compared with the same sum in 64 bits, from the library's float
fields and coefficients, relative to |c| |dc|: FP32 sums of up to 32 pixels x 121
modes (6e-8 each, growing with the square root of their number: 4e-6): 2e-5."""
import ctypes as C

import numpy as np
import pytest
import torch

from test_gpu_gradient_window import _case, cases, wave   # noqa: F401 (cases: fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [dict(mode=1), dict(mode=1, carrier=0.55, pols=1), dict(window=32, width=320, height=256)],
                         ids=["16", "32", "full32"])
@pytest.mark.parametrize("groups", [120, 121])
def test_gradient(cases, groups, over):   # noqa: F811
    c = _case(groups=9, frames=3, **over)
    s = cases.prepare(c, 1)
    assert s.L.digHoloConfigSetBasisGroupCount(s.h, groups) == 0
    assert s.L.digHoloB200SetKeepField32(s.h, 1) == 0
    got = cases.run(s)["gradient"]
    b, p, w, h = C.c_int(), C.c_int(), C.c_int(), C.c_int()
    v = s.L.digHoloB200GetFields32(s.h, C.byref(b), C.byref(p), C.byref(w), C.byref(h))
    shape = (b.value, p.value, h.value, w.value)
    V = np.ctypeslib.as_array(v, shape=(2 * int(np.prod(shape)),)).copy().view(np.complex64).reshape(shape)
    e = cases.Exact(c, 1)
    e.case = dict(c, groups=groups)
    V, coefs = torch.as_tensor(V, device=e.dev).to(torch.complex128), s.device_coefs().to(torch.complex128)
    assert coefs.shape[-1] == groups * (groups + 1) // 2
    base, k0, u = e.settings(), 2 * np.pi / 1565e-9, np.pi / 180
    x, y = e.t(e.axis(e.nx))[None, :], e.t(e.axis(e.ny))[:, None]
    power, waist = float((coefs.abs() ** 2).sum()), 0.0
    for p in range(c["pols"]):
        F, (bx, by), (tx, ty), cp = V[:, p], base["centre"][p], base["tilt"][p], coefs[:, p]
        R = wave(e, p, base)
        spec = torch.fft.fft2(-F.conj() / R)
        k = [torch.zeros(n, dtype=torch.float64, device=e.dev) for n in (e.nx, e.ny)]
        k[0][torch.as_tensor(e.cols[p] % e.n if e.full else np.arange(e.w), device=e.dev)] = e.t(e.k[e.cols[p]])
        k[1][torch.as_tensor(e.rows[p] if e.full else np.arange(e.h), device=e.dev)] = e.t(e.k[e.rows[p]])
        Fx = -(torch.fft.ifft2(spec * 1j * k[0][None, :]) * R).conj()
        Fy = -(torch.fft.ifft2(spec * 1j * k[1][:, None]) * R).conj()
        dc = [e.coefs(p, t, base) for t in (F * 1j * k0 * u * (x + bx), F * 1j * k0 * u * (y + by),
                                            F * 1j * np.pi / 1565e-9 * (x * x + y * y),
                                            Fx + F * 1j * k0 * u * tx, Fy + F * 1j * k0 * u * ty)]
        for i, d in enumerate(dc):
            want = 20.0 / np.log(10.0) * float((cp.conj() * d).real.sum()) / power
            bound = 2e-5 * 20.0 / np.log(10.0) * float(cp.norm() * d.norm()) / power
            assert abs(got[6 * p + i] - want) <= bound, (p, i, got[6 * p + i], want, bound)
        step = 2e-8
        d = (e.coefs(p, F, dict(base, waist=base["waist"] + step)) - e.coefs(p, F, dict(base, waist=base["waist"] - step))) / (2 * step)
        waist += 20.0 / np.log(10.0) * float((cp.conj() * d).real.sum()) / power
        if p == c["pols"] - 1:
            assert abs(got[5] - waist) <= 2e-5 * 20.0 / np.log(10.0) * float(coefs.norm() * d.norm()) * c["pols"] / power
