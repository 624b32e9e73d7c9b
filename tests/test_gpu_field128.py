"""The persistent kernel of 128 x 128 full-resolution fields (IFFT windows of
16, 32 and 48 pixels): one unit, more units than multiprocessors, mode-group
counts at the edges of its operand tiles, and fields with no finite scale.

int16 fields: at most 2 LSB from the quantised oracle, at most 1 LSB from the
band kernels (inverse choice 2: another order of the same float sums).
Coefficients: its byte products are exact, so against the int64 overlap of
the same int16 fields only the float sums over the 128 rows remain:
128 x 2^-24 = 7.6e-6 relative at the very worst."""
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


def hologram(carrier, groups, frames, pols, dtype):
    return synth.generate(frame_count=frames, frame_width=640, frame_height=512, pol_count=pols, max_mg=groups, waist=250e-6,
                          snr_db=30, window=(128, 128), carrier=(carrier, 0.8 * carrier), dtype=dtype, seed=77)


def process(lib, cfg, frames, inverse=0):
    h = lib.digHoloCreate()
    api.configure(lib, h, cfg)
    assert lib.digHoloB200SetInverseKernel(h, inverse) == 0
    out = api.run_batch(lib, h, frames)
    out["overlap"] = lib.digHoloB200GetOverlapKernel(h)
    lib.digHoloDestroy(h)
    return out


def integer_overlap(g, cfg, pol):
    """The overlap of the returned int16 fields in 64-bit integers, scaled."""
    x, y = O.ifft_axes(cfg, 128, 128, 16, 16)
    Hx, Hy, sx, sy = O.basis_axes_modes(cfg, pol, x, y)
    fs = 1.0 / g["scale"][pol].astype(np.float64)
    return O.overlap(g["R"][:, pol], g["I"][:, pol], Hx, Hy, sx, sy, fs, cfg.max_mg)


@pytest.mark.parametrize("carrier,groups,frames,pols,dtype", [
    (0.25, 1, 1, 1, "uint16"),       # one unit, one mode
    (0.25, 15, 75, 2, "uint16"),     # 150 units, the widest 16-row operand
    (0.25, 16, 3, 1, "float32"),     # the constant row needs the next operand size
    (0.55, 31, 2, 2, "float32"),
    (0.55, 32, 1, 2, "uint16"),
    (0.55, 4, 149, 1, "uint16"),     # an odd number of units on blocks of one polarisation
    (0.8, 9, 75, 2, "float32"),      # 48-pixel window
    (0.8, 32, 2, 1, "uint16"),
])
def test_fields_and_overlap(lib, carrier, groups, frames, pols, dtype):
    hol = hologram(carrier, groups, frames, pols, dtype)
    cfg = config_for(hol, 0)
    g = process(lib, cfg, hol.frames)
    b = process(lib, cfg, hol.frames, 2)
    # 32 groups with a 32-pixel window exceed shared memory: the FP32 overlap follows
    assert g["overlap"] == (1 if (carrier, groups) == (0.55, 32) else 2)
    for k in ("R", "I"):
        assert np.abs(g[k].astype(int) - b[k]).max() <= 1
    assert np.array_equal(g["summary"][4].view(np.int32)[:, :frames], b["summary"][4].view(np.int32)[:, :frames])
    n = min(frames, 4)
    o = O.process_batch(hol.frames[-n:], cfg, quantised=True)
    for k in ("R", "I"):
        assert np.abs(g[k][-n:].astype(int) - o[k]).max() <= 2
    for p in range(pols):
        assert rel_l2(g["coefs"][:, p], integer_overlap(g, cfg, p)) <= 7.6e-6


@pytest.mark.parametrize("value", [0.0, np.inf, np.nan])
def test_fields_without_a_scale(lib, value):
    """A frame of zeros, or with one infinite or NaN pixel, has no finite
    scale: every pixel that is not a number once scaled is -32768, as the
    reference's conversion gives it; the frames next to it are unharmed."""
    hol = hologram(0.25, 9, 3, 1, "float32")
    cfg = config_for(hol, 0)
    clean = process(lib, cfg, hol.frames)
    frames = hol.frames.copy()
    if value == 0.0:
        frames[1] = 0.0
    else:
        frames[1, 256, 320] = value
    g = process(lib, cfg, frames)
    b = process(lib, cfg, frames, 2)
    for k in ("R", "I"):
        assert (g[k][1] == -32768).all() and (b[k][1] == -32768).all()
        assert np.array_equal(g[k][[0, 2]], clean[k][[0, 2]])
    assert np.array_equal(g["coefs"][[0, 2]], clean["coefs"][[0, 2]])


def test_without_overlap_and_float_fields(lib):
    """No modes (fields only), and the kept float fields beside the int16 ones."""
    hol = hologram(0.55, 6, 3, 2, "uint16")
    cfg = config_for(hol, 0, max_mg=0)
    g = process(lib, cfg, hol.frames)
    h = lib.digHoloCreate()
    api.configure(lib, h, config_for(hol, 0))
    lib.digHoloB200SetKeepField32(h, 1)
    k = api.run_batch(lib, h, hol.frames)
    b, p, w, hh = C.c_int(), C.c_int(), C.c_int(), C.c_int()
    fp = lib.digHoloB200GetFields32(h, C.byref(b), C.byref(p), C.byref(w), C.byref(hh))
    f32 = np.ctypeslib.as_array(fp, shape=(2 * k["R"].size,)).copy().view(np.complex64).reshape(k["R"].shape)
    lib.digHoloDestroy(h)
    assert g["coefs"] is None and np.array_equal(g["R"], k["R"]) and np.array_equal(g["I"], k["I"])
    ex = O.process_batch(hol.frames, config_for(hol, 0), quantised=False)
    assert rel_l2(f32, ex["field_v"]) <= 1e-5
