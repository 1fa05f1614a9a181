"""State slots of new requests: zeros in one launch, nothing else touched."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("shapes,slots", [([(3, 5)], [1]), ([(7, 16), (7, 3, 4)], [0, 6, 3]), ([(70, 33)] * 17, list(range(1, 69))),
                                          ([(2, 40000), (2, 1)], [1]), ([(4, 8)], [2, 2])])
def test_slots_of_every_state(shapes, slots):
    from vllm_oxide_b200 import kernels
    dtypes = (torch.float32, torch.bfloat16, torch.int32)
    states = [torch.full(s, 3, dtype=dtypes[i % 3], device=DEV) for i, s in enumerate(shapes)]
    states.append(torch.full((shapes[0][0] + 1, 9), 3, dtype=torch.bfloat16, device=DEV)[1:])     # not on a 16-byte boundary
    kernels.clear_states(states, slots)
    for t in states:
        want = torch.full_like(t, 3)
        want[slots] = 0
        assert torch.equal(t, want)


@pytest.mark.parametrize("slots", [[-1], [3], [0, 3]])
def test_slots_out_of_range_are_refused(slots):
    from vllm_oxide_b200 import kernels
    t = torch.ones(3, 8, device=DEV)
    with pytest.raises(kernels.KernelError):
        kernels.clear_states([t], slots)
    assert torch.equal(t, torch.ones(3, 8, device=DEV))
