"""Batches on both sides of the lines by which the forward kernel starts the
small blocks of a low-resolution inverse or of the averaging early (room beside
its own blocks, a nearly empty last turn, twelve units per multiprocessor): two
batches alternating on one stream give the values of each by itself, exactly."""
import pytest

from test_gpu_dependent_launch import test_alternating_batches as alternating

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,carrier,frames", [
    ("uint16", 0.25, (98, 147, 150, 1776)), ("uint16", 0.55, (74, 140, 300)), ("float32", 0.25, (147, 295, 300, 400)),
    ("float32", 0.55, (130, 600, 1000)),
], ids=lambda o: str(o).replace(" ", ""))
def test_batches(dtype, carrier, frames):
    for n in frames:
        alternating(dict(mode=1, dtype=dtype, carrier=carrier, pols=1, frames=n))


@pytest.mark.parametrize("dtype,carrier", [("uint16", 0.55), ("float32", 0.25)])
@pytest.mark.parametrize("mode", [0, 1])
def test_averaged(dtype, carrier, mode):
    for n, average in ((2, 8), (50, 2), (150, 4)):
        alternating(dict(mode=mode, dtype=dtype, carrier=carrier, pols=1, frames=n, average=average))
