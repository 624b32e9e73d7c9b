"""The one-launch forward of 128- and 256-pixel-wide FFT windows
(dh_forward_win.cu) at the window heights and kept-column counts it is built
for, both pixel types, an odd number of frames and a batch calibration: its
Fourier windows against the FP64 oracle.  FP32 radix-2 transforms of at most
2^15 points: 15 stages of 2^-24 relative rounding stay below 1e-6."""
import ctypes as C

import numpy as np
import pytest

import digholo_oracle as O
from digholo_b200 import api, synth
from helpers import config_for, rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    import digholo_b200
    return digholo_b200.load()


@pytest.mark.parametrize("window,carrier,wh,dtype,pols", [
    ((128, 64), (0.6, 0.48), (48, 32), "uint16", 2),
    ((128, 128), (0.8, 0.64), (48, 48), "float32", 1),
    ((128, 256), (0.8, 0.64), (48, 96), "uint16", 2),
    ((256, 64), (0.25, 0.2), (32, 16), "float32", 2),
    ((256, 128), (0.02, 0.6), (64, 32), "uint16", 1),     # columns from the DC column on
    ((256, 256), (0.9, 0.1), (80, 80), "float32", 2),     # columns up to the last
    ((256, 256), (0.25, 0.2), (32, 32), "uint16", 2),
    ((256, 256), (0.8, 0.64), (96, 96), "uint16", 1),     # more columns than fit: through the planes
])
@pytest.mark.parametrize("calibrated", [False, True])
def test_windows_vs_oracle(lib, window, carrier, wh, dtype, pols, calibrated):
    hol = synth.generate(frame_count=3, frame_width=640, frame_height=512, pol_count=pols, max_mg=3, waist=300e-6, snr_db=30,
                         window=window, dtype=dtype, seed=21, carrier=carrier)
    cfg = config_for(hol, 1)
    if calibrated:
        rng = np.random.default_rng(4)
        cfg.batch_cal = (rng.uniform(0.5, 1.5, (pols, 3)) * np.exp(1j * rng.uniform(0, 6, (pols, 3)))).astype(np.complex64)
    o = O.process_batch(hol.frames, cfg, quantised=True)
    assert (o["w"], o["h"]) == wh
    h = lib.digHoloCreate()
    api.configure(lib, h, cfg)
    assert lib.digHoloB200SetForwardKernel(h, 5) == 0
    api.run_batch(lib, h, hol.frames, want_fields=False)
    assert lib.digHoloB200GetForwardKernel(h) == 5, lib.digHoloB200GetLastError(h)
    b, p, w, hh = C.c_int(), C.c_int(), C.c_int(), C.c_int()
    wp = lib.digHoloGetFourierPlaneWindow(h, C.byref(b), C.byref(p), C.byref(w), C.byref(hh))
    got = np.ctypeslib.as_array(wp, shape=(2 * o["window"].size,)).copy().view(np.complex64)
    lib.digHoloDestroy(h)
    assert rel_l2(got, o["window"].ravel()) <= 1e-6
