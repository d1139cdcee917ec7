"""Routers on rows without a number to choose by: the experts that they name exist (the weights of the next kernel are read at them), and
the row's weights are NaN, so that the row's result is too."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from torchao_fork_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("E,top", [(4, 2), (40, 3), (64, 8)])
@pytest.mark.parametrize("value", [float("nan"), float("-inf")])
def test_routers_name_experts_that_exist(E, top, value):
    L, st = _lib.lm(), torch.cuda.current_stream().cuda_stream
    z = torch.randn(9, E, device="cuda")
    z[3] = value
    z[5, 1:] = value          # one number left
    idx, w = torch.full((9, top), -1, dtype=torch.int32, device="cuda"), torch.zeros(9, top, device="cuda")
    for call in (lambda: L.ao_lm_router_topk_logits(z.data_ptr(), 9, E, top, idx.data_ptr(), w.data_ptr(), st),
                 lambda: L.ao_lm_router_topk_renorm_logits(z.data_ptr(), E, None, 9, E, top, -1, idx.data_ptr(), w.data_ptr(), None, st)):
        idx.fill_(-1)
        _lib.lm_check(call(), "router")
        torch.cuda.synchronize()
        assert int(idx.min()) >= 0 and int(idx.max()) < E
        assert w[3].isnan().all()
        ok = torch.ones(9, dtype=torch.bool)
        ok[3] = ok[5] = False
        assert torch.equal(idx[ok].long().cpu(), z[ok].topk(top).indices.cpu()) and not w[ok].isnan().any()
