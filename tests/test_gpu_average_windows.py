"""Frame averaging over the window sides where its kernel changes: 1024 values
(two per thread), up to 4096 (eight), beyond (in memory), against the 64-bit
batch path of perf/cases.py.  Tolerance: the batch path's, 5e-5 of the
coefficients' norm (the int16 rounding of the fields)."""
import importlib.util
import os

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cases():
    path = os.path.join(os.path.dirname(__file__), "..", "perf", "cases.py")
    spec = importlib.util.spec_from_file_location("perf_cases", path)
    m = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(m)
    return m


@pytest.mark.parametrize("average", [2, 5])
@pytest.mark.parametrize("window,carrier,side", [(128, 0.25, 16), (256, 0.25, 32), (128, 0.8, 48), (256, 0.55, 64), (256, 0.8, 96)])
def test_sides(cases, window, carrier, side, average):
    c = dict(name="average", frames=5, width=1280, height=1024, dtype="float32", pols=2, window=window, groups=9, mode=0,
             carrier=carrier, call="batch", average=average)
    s = cases.prepare(c, 4)
    got = cases.run(s)
    torch.cuda.synchronize()   # the call only enqueues
    got = got.to(torch.complex128)
    e = cases.Exact(c, 4)
    assert (e.w, e.h) == (side, side)
    ref = e.batch(e.settings())[0]
    assert float((got - ref).norm() / ref.norm()) <= 5e-5
