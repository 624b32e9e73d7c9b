"""The 512-wide full-resolution fields (dh_field512.cu) at its edges: one unit,
fields of 64 rows (one band) and more, mode-group counts at the ends of the
operand tiles, more units than one chunk of the column stage, a frame of
zeros.

int16 fields: at most 1 LSB from the band kernels (the FP32 overlap choice),
another order of the same float sums.  Coefficients against the int64 overlap
of the same int16 fields: exact byte products, so only the float sums over up
to 512 rows remain, 512 x 2^-24 = 3.1e-5 at the very worst; their usual size
is its square root, and 2e-6 is asked for."""
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


def process(lib, cfg, frames, overlap):
    h = lib.digHoloCreate()
    api.configure(lib, h, cfg)
    assert lib.digHoloB200SetOverlapKernel(h, overlap) == 0
    out = api.run_batch(lib, h, frames)
    out["kernel"] = lib.digHoloB200GetInverseKernel(h)
    lib.digHoloDestroy(h)
    return out


@pytest.mark.parametrize("rows,groups,frames,pols,dtype", [
    (64, 1, 1, 1, "uint16"),
    (64, 16, 131, 2, "uint16"),      # 262 units of one band
    (128, 17, 2, 1, "float32"),
    (256, 32, 2, 2, "uint16"),
    (512, 31, 3, 2, "float32"),
    (512, 32, 40, 1, "uint16"),      # several bands per block
])
def test_fields_and_overlap(lib, rows, groups, frames, pols, dtype):
    hol = synth.generate(frame_count=frames, frame_width=512 * pols, frame_height=rows, pol_count=pols, max_mg=groups,
                         waist=300e-6, snr_db=25, window=(512, rows), dtype=dtype, seed=91)
    cfg = config_for(hol, 0)
    frames_in = hol.frames.copy()
    frames_in[-1] = 0
    g = process(lib, cfg, frames_in, 0)
    b = process(lib, cfg, frames_in, 1)
    assert g["kernel"] == 7 and b["kernel"] == 4
    for k in ("R", "I"):
        assert np.abs(g[k].astype(int) - b[k]).max() <= 1
    assert (g["R"][-1] == -32768).all() and (g["I"][-1] == -32768).all()
    n = frames - 1
    if n:
        assert np.array_equal(g["summary"][4].view(np.int32)[:, :n], b["summary"][4].view(np.int32)[:, :n])
        np.testing.assert_allclose(g["summary"][[0, 3, 5]][:, :, :n], b["summary"][[0, 3, 5]][:, :, :n], rtol=1e-5)
    x, y = O.ifft_axes(cfg, 512, rows, 16, 16)
    for p in range(pols):
        Hx, Hy, sx, sy = O.basis_axes_modes(cfg, p, x, y)
        c = O.overlap(g["R"][:n, p], g["I"][:n, p], Hx, Hy, sx, sy, 1.0 / g["scale"][p, :n].astype(np.float64), groups)
        if n:
            assert rel_l2(g["coefs"][:n, p], c) <= 2e-6
