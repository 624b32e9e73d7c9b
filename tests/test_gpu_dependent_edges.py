"""Batches at the lines below and above which the forward kernel starts the
low-resolution inverse kernel's blocks early (two thirds of the GPU's forward
blocks, twelve units per multiprocessor): two batches alternating on one stream
give the values of each by itself, exactly."""
import pytest
import torch

from test_gpu_dependent_launch import test_alternating_batches as alternating

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,carrier,blocks", [("uint16", 0.25, 1), ("uint16", 0.55, 1), ("float32", 0.25, 2), ("uint16", 0.25, 18)])
@pytest.mark.parametrize("above", [0, 1])
@pytest.mark.parametrize("pols", [1, 2])
def test_at_the_line(dtype, carrier, blocks, above, pols):
    units = 2 * blocks * torch.cuda.get_device_properties(0).multi_processor_count // 3
    alternating(dict(mode=1, dtype=dtype, carrier=carrier, pols=pols, frames=units // pols + above))
