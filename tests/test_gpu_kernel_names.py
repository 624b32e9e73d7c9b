"""Which kernel a batch ran, where one reported number stands for several, and
the band kernels on 48-pixel windows of 128-pixel fields, which the 128 x 128
field kernel takes by itself: asked for by inverse choice 2, with their own
overlaps.

int16 fields within 2 LSB of the quantised oracle, fields relative L2 <= 5e-5,
coefficients <= 1e-4 (split-BF16) or 5e-5 (FP32), as for the other band shapes."""
import ctypes as C

import numpy as np
import pytest
import torch

import digholo_oracle as O
from digholo_b200 import api, synth
from helpers import config_for, rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    import digholo_b200
    return digholo_b200.load()


def _names(lib, h):
    return tuple(lib.digHoloB200GetKernelName(h, stage).decode() for stage in (0, 1))


@pytest.mark.parametrize("window,carrier,mode,dtype,names", [
    (64, 0.25, 0, "float32", ("k_forward_tma", "k_field_full")),
    (128, 0.25, 0, "uint16", ("k_forward_i8", "k_field128")),
    (128, 0.55, 0, "float32", ("k_forward_tma", "k_field128")),
    (128, 0.8, 0, "uint16", ("k_forward_win", "k_field128")),
    (128, 0.8, 1, "uint16", ("k_forward_win", "k_inverse_dft")),
    (128, 0.25, 1, "uint16", ("k_forward_i8", "k_inverse_lo")),
    (256, 0.25, 0, "uint16", ("k_forward_win", "k_field_big")),
    (256, 0.8, 1, "float32", ("planes", "k_inverse_dft")),     # 96 columns: more than k_forward_win holds
])
def test_kernels_of_a_batch(lib, window, carrier, mode, dtype, names):
    hol = synth.generate(frame_count=2, frame_width=640, frame_height=512, pol_count=1, max_mg=3, waist=300e-6, snr_db=30,
                         window=(window, window), dtype=dtype, seed=21, carrier=(carrier, 0.8 * carrier))
    h = lib.digHoloCreate()
    assert _names(lib, h) == ("", "")
    api.configure(lib, h, config_for(hol, mode))
    dev = torch.as_tensor(hol.frames.view(np.int16) if dtype == "uint16" else hol.frames, device="cuda")
    torch.cuda.synchronize()
    for _ in range(4):   # launched, captured, replayed
        p = C.c_void_p(dev.data_ptr())
        if dtype == "uint16":
            assert lib.digHoloSetBatchUint16(h, 2, C.cast(p, C.POINTER(C.c_ushort)), 0) == 0
        else:
            assert lib.digHoloSetBatch(h, 2, C.cast(p, C.POINTER(C.c_float))) == 0
        assert lib.digHoloB200ProcessBatchDevice(h) == 0, lib.digHoloB200GetLastError(h)
        assert _names(lib, h) == names
    lib.digHoloB200Synchronize(h)
    lib.digHoloDestroy(h)


@pytest.mark.parametrize("overlap", [0, 1])
def test_bands_of_48_pixel_windows(lib, overlap):
    hol = synth.generate(frame_count=4, frame_width=640, frame_height=512, pol_count=2, max_mg=9, waist=320e-6, snr_db=30,
                         window=(128, 128), dtype="float32", seed=2999, carrier=(0.6, 0.48))
    cfg = config_for(hol, 0)
    o = O.process_batch(hol.frames, cfg, quantised=True)
    assert (o["w"], o["h"]) == (48, 48)
    h = lib.digHoloCreate()
    api.configure(lib, h, cfg)
    assert lib.digHoloB200SetInverseKernel(h, 2) == 0 and lib.digHoloB200SetOverlapKernel(h, overlap) == 0
    g = api.run_batch(lib, h, hol.frames)
    assert g["coefs"] is not None, lib.digHoloB200GetLastError(h)
    assert _names(lib, h)[1] == "k_field_big" and lib.digHoloB200GetOverlapKernel(h) == (1 if overlap else 2)
    lib.digHoloDestroy(h)
    assert max(np.abs(g["R"].astype(int) - o["R"]).max(), np.abs(g["I"].astype(int) - o["I"]).max()) <= 2
    assert rel_l2(g["field"], o["field"]) <= 5e-5
    assert rel_l2(g["coefs"], o["coefs"]) <= (1e-4 if overlap == 0 else 5e-5)


@pytest.mark.parametrize("inverse", [0, 2])
def test_no_overlap_reported_without_modes(lib, inverse):
    """48-pixel windows without a basis: overlap 0 from the field kernel as from the bands."""
    hol = synth.generate(frame_count=2, frame_width=640, frame_height=512, pol_count=1, max_mg=3, waist=320e-6, snr_db=30,
                         window=(128, 128), dtype="float32", seed=5, carrier=(0.6, 0.48))
    h = lib.digHoloCreate()
    api.configure(lib, h, config_for(hol, 0, max_mg=0))
    assert lib.digHoloB200SetInverseKernel(h, inverse) == 0
    api.run_batch(lib, h, hol.frames)
    assert _names(lib, h)[1] == ("k_field_big" if inverse else "k_field128")
    assert lib.digHoloB200GetInverseKernel(h) == 4 and lib.digHoloB200GetOverlapKernel(h) == 0
    lib.digHoloDestroy(h)
