"""Which kernel a decode call launches: one without the split by length wherever the split count is the same for all."""
import pytest
import torch

from tilecadence_b200 import cuda_runtime


@pytest.mark.gpu
@pytest.mark.parametrize("batch,capacity,num_splits,by_length", [
    (1, 8192, 0, False), (1, 32768, 0, False), (4, 4096, 4, False), (2, 1024, 0, False), (4, 4096, 0, True), (16, 2048, 0, True),
    (65, 2048, 0, False)])
def test_even_splits_carry_no_plan(gpu_device, batch, capacity, num_splits, by_length):
    """The instance that plans keeps its share in static shared memory; the other one has none."""
    ops = cuda_runtime.default_ops("decode")
    q = torch.zeros(batch, 1, 32, 128, device=gpu_device, dtype=torch.bfloat16)
    cache = torch.zeros(batch, capacity, 8, 128, device=gpu_device, dtype=torch.bfloat16)
    old = torch.zeros(batch, device=gpu_device, dtype=torch.int32)
    resources = ops.resources(q, cache, old, num_splits, 1, True)
    assert (resources[14] > 0) == by_length


@pytest.mark.gpu
@pytest.mark.parametrize("batch,capacity,one_per_sm", [(1, 8192, False), (4, 4096, False), (10, 2048, True), (17, 2048, True),
                                                       (18, 2048, False), (32, 2048, False)])
def test_the_resources_are_those_of_the_launch(gpu_device, batch, capacity, one_per_sm):
    """Shared memory and CTAs to an SM are reported as a call without promises launches them: 10 to 17 sequences of one
    split each are kept one to an SM."""
    ops = cuda_runtime.default_ops("decode")
    q = torch.zeros(batch, 1, 32, 128, device=gpu_device, dtype=torch.bfloat16)
    cache = torch.zeros(batch, capacity, 8, 128, device=gpu_device, dtype=torch.bfloat16)
    old = torch.zeros(batch, device=gpu_device, dtype=torch.int32)
    resources = ops.resources(q, cache, old, 0, 1, True)
    assert resources[19] == (1 if one_per_sm else 2) and (resources[13] > 114 * 1024) == one_per_sm
