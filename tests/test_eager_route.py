"""Which calls of the linears may go past the dispatcher (ops.runs_eagerly): only those for which it would have done nothing.  On the CPU;
the shape of every answer, or the error, is that of the registered op."""
import pytest
import torch

from torchao_fork_b200 import ops

T = torch.ops.torchao


def _args(bits, device):
    x = torch.empty(3, 64, device=device, dtype=torch.bfloat16)
    if bits == 4:
        return x, torch.empty(8, 1, 32, 4, dtype=torch.int32, device=device), 64, torch.empty(8, 1, 16, 2, dtype=torch.bfloat16, device=device), 100
    return x, torch.empty(8, 1, 1024, dtype=torch.uint8, device=device), torch.empty(100, dtype=torch.bfloat16, device=device)


CALLS = [(4, ops.int4_weight_only_mm, T.b200_int4_weight_only_mm), (8, ops.int8_weight_only_mm, T.b200_int8_weight_only_mm)]


@pytest.mark.parametrize("bits,call,op", CALLS)
def test_other_devices_go_through_the_dispatcher(bits, call, op):
    args = _args(bits, "meta")          # shapes of a model that has no memory yet
    y = call(*args)
    assert y.device.type == "meta" and y.shape == op(*args).shape == (3, 100)
    with pytest.raises(NotImplementedError, match="CPU"):   # (also what a caller may catch: an op that is not there)
        call(*_args(bits, "cpu"))


def test_only_plain_cuda_memory_is_eager():
    with torch.inference_mode():
        inside = torch.ones(2)
    assert tuple(torch._C._dispatch_keys(t).raw_repr() for t in (inside, torch.ones(2))) == ops._plain_keys("CPU")
    for t in (torch.ones(2), torch.ones(2, device="meta"), torch._neg_view(torch.ones(2)), torch._efficientzerotensor(2),
              torch._to_functional_tensor(torch.ones(2))):
        assert not ops.runs_eagerly(t)


@pytest.mark.gpu
def test_plain_cuda_tensors_are_eager_and_wrapped_ones_are_not():
    x = torch.ones(2, device="cuda")
    with torch.inference_mode():
        inside = torch.ones(2, device="cuda")
    assert ops.runs_eagerly(x) and ops.runs_eagerly(x, inside, x.view(2)) and ops.runs_eagerly(inside)
    for t in (torch._neg_view(x), torch._efficientzerotensor(2, device="cuda"), torch._to_functional_tensor(x), x.cpu()):
        assert not ops.runs_eagerly(t) and not ops.runs_eagerly(x, t)
