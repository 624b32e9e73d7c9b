"""Inverse kernels that start under the forward kernel's tail: two batches
alternating on one stream without a wait, through the same window buffer,
give the values of each batch run by itself (exactly: the same kernels)."""
import importlib.util
import os

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("over", [
    dict(mode=1, dtype="uint16"), dict(mode=1, carrier=0.55), dict(mode=1, frames=3), dict(mode=0, dtype="uint16"),
    dict(mode=0, carrier=0.55, pols=1), dict(mode=0, carrier=0.8), dict(mode=1, dtype="uint16", average=4, frames=40),
], ids=lambda o: "-".join("%s%s" % kv for kv in o.items()))
def test_alternating_batches(over):
    path = os.path.join(os.path.dirname(__file__), "..", "perf", "cases.py")
    spec = importlib.util.spec_from_file_location("perf_cases", path)
    cases = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(cases)
    c = dict(name="batch", frames=150, width=640, height=512, dtype="float32", pols=2, window=128, groups=9, mode=0,
             carrier=0.25, call="batch", average=1)
    c.update(over)
    s, other = cases.prepare(c, 1), cases.prepare(c, 2)

    def run(frames):
        s.ptr = frames.ptr
        out = cases.run(s)
        return out

    mine = type("F", (), {"ptr": s.ptr})()
    want = []
    for f in (mine, other):
        out = run(f)
        torch.cuda.synchronize()
        want.append(out.clone())
        torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    for k in range(40):
        last = run(mine if k % 2 == 0 else other)
        if k in (20, 39):
            torch.cuda.synchronize()
            assert torch.equal(last, want[k % 2])
            torch.cuda.synchronize()
