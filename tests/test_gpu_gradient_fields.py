"""The float fields after an alignment gradient or search, asked for only then:
those of its last batch, exactly as a handle stores them that keeps them from
the start, and not those of an earlier batch."""
import ctypes as C

import numpy as np
import pytest

from digholo_b200 import api
from test_gpu_adjoint import _case, _grad, _handle, _perturbed

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    import digholo_b200
    return digholo_b200.load()


def _fields(lib, h):
    b, p, w, hh = C.c_int(), C.c_int(), C.c_int(), C.c_int()
    f = lib.digHoloB200GetFields32(h, C.byref(b), C.byref(p), C.byref(w), C.byref(hh))
    assert f, "no float fields"
    n = 2 * b.value * p.value * w.value * hh.value
    return np.ctypeslib.as_array(f, shape=(n,)).copy()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("search", [False, True])
def test_fields_asked_for_afterwards(lib, mode, search):
    hol, other = _case(6), _case(6, 78)
    cfg = _perturbed(hol, mode)
    got = []
    for early in (True, False):
        h, keep = _handle(lib, cfg, other.frames)
        if not early:   # an earlier batch's fields are on the handle
            assert lib.digHoloB200SetKeepField32(h, 1) == 0
            api.run_batch(lib, h, other.frames)
            before = _fields(lib, h)
        assert lib.digHoloB200SetKeepField32(h, 1 if early else 0) == 0
        assert api.set_batch(lib, h, hol.frames) == 0
        if search:
            lib.digHoloConfigSetAutoAlignBasisWaist(h, 1 - mode)
            lib.digHoloB200AutoAlignAdjoint(h)
        else:
            _grad(lib, h)
        assert lib.digHoloB200SetKeepField32(h, 1) == 0
        got.append(_fields(lib, h))
        assert np.array_equal(_fields(lib, h), got[-1])
        lib.digHoloDestroy(h)
    assert not np.array_equal(got[1], before)
    assert np.array_equal(got[0], got[1])
