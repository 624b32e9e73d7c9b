"""The eigen solver at the edges of its shared-memory kernels: one block up to
n = 64, a cluster of eight up to 304 (register tiles change at 128 and 256),
the one-block global-memory kernel beyond.  Against numpy's eigvalsh: the
solver's own stopping interval is 4 eps of the largest eigenvalue and both
reductions are backward stable with a modest multiple of n eps, so 1e-12 of
the largest eigenvalue; eigenvectors by their residual at the same bound.  The
extremes alone, through MDL of a batch's own coefficients: the same bound on
s_min^2 / s_max^2, and the single-precision rounding of the decibels."""
import ctypes as C

import numpy as np
import pytest

from digholo_b200 import api, synth
from helpers import config_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 63, 64, 65, 71, 127, 128, 129, 255, 256, 257, 303, 304, 305])
@pytest.mark.parametrize("kind", ["gram", "diagonal"])
def test_edges(n, kind):
    import digholo_b200
    lib = digholo_b200.load()
    rng = np.random.default_rng(n)
    if kind == "gram":
        b = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        a = b @ b.conj().T
    else:   # repeated and vanishing eigenvalues, no reflector to apply
        a = np.diag(np.arange(n) // 3 % 7).astype(complex)
    g = np.asfortranarray(a)
    w = np.zeros(n)
    v = np.zeros((2, n), complex)
    p = lambda x: x.ctypes.data_as(C.POINTER(C.c_double))
    assert lib.digHoloB200EigenHermitian(n, p(g), p(w), p(v)) == 0
    ref = np.linalg.eigvalsh(a)
    top = max(np.abs(ref).max(), 1e-300)
    assert np.abs(w - ref).max() <= 1e-12 * top
    for e, u in ((w[0], v[0]), (w[-1], v[1])):
        assert abs(np.linalg.norm(u) - 1) <= 1e-12
        assert np.linalg.norm(a @ u - e * u) <= 1e-12 * top * np.sqrt(n)


@pytest.mark.parametrize("groups", [5, 7, 8, 10, 11, 15, 16, 17])
def test_extremes(groups):
    import digholo_b200
    lib = digholo_b200.load()
    kw = dict(synth.WORKLOADS["align_640x512_f32_2pol"])
    kw["frame_count"], kw["max_mg"] = 320, groups
    kw["coefs"] = synth.transfer_coefs(320, 2, groups, 5)
    hol = synth.generate(**kw)
    h = lib.digHoloCreate()
    api.configure(lib, h, config_for(hol, 1))
    c = api.run_batch(lib, h, hol.frames, want_fields=False)["coefs"]
    assert lib.digHoloAutoAlignCalcMetrics(h) == 0
    mdl = float(lib.digHoloAutoAlignGetMetric(h, 1))
    lib.digHoloDestroy(h)
    s2 = np.linalg.svd(c.reshape(320, -1).astype(np.complex128), compute_uv=False) ** 2
    ref = s2[-1] / s2[0]
    assert abs(10 ** (mdl / 10) - ref) <= 1e-12 + 1e-5 * ref, (mdl, 10 * np.log10(ref))
