"""The states of newly admitted requests: rows of every size and alignment, more slots than one launch takes, and nothing beside them."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("slots", [[0], [5, 2], list(range(0, 140, 2))])
def test_zero_slots(slots):
    from reinfer_b200 import ops
    shapes = [((3,), torch.int32), ((1,), torch.bfloat16), ((5, 7), torch.bfloat16), ((16, 3, 64), torch.float32), ((33, 1025), torch.float32)]
    tensors = [torch.ones((141,) + s, dtype=d, device=DEV) for s, d in shapes]
    ops.zero_slots(*ops.zero_slots_table(tensors, DEV), slots)
    for t in tensors:
        want = torch.ones_like(t)
        want[slots] = 0
        assert torch.equal(t, want), t.shape
