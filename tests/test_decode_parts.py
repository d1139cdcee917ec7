"""The decode step where only some projections take the fused GEMV (long activations, more than 16 sequences, unquantized lines), against
the same step made of one launch per operation.  Bound: each of the four places per layer that rounds to bf16 in another order (products
summed in another order and rounded) moves the logits by a relative 2^-9 at most; with two layers and independent roundings
sqrt(8) 2^-9 = 0.55 %, doubled for the sums behind the norms: 1.1 % is 39 dB."""
import pytest
import torch

import torchao_fork_b200 as ao
from torchao_fork_b200._models.llama import ModelArgs, Transformer
from torchao_fork_b200._models.llama.decode_engine import DecodeEngine

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)


def _model(quant, inter, batch):
    torch.manual_seed(3)
    cfg = ModelArgs.from_name("tiny-llama3")
    cfg.intermediate_size = inter
    old = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        with torch.device("cuda"):
            m = Transformer(cfg).eval()
    finally:
        torch.set_default_dtype(old)
    config = ao.Int4WeightOnlyConfig(group_size=64) if quant.startswith("int4") else ao.Int8WeightOnlyConfig()
    keep = (lambda mod, name: isinstance(mod, torch.nn.Linear) and not name.endswith("w2")) if quant.endswith("w2 plain") else None
    ao.quantize_(m, config, filter_fn=keep)
    m.setup_caches(batch, 64, device=torch.device("cuda"))
    return m


@pytest.mark.parametrize("quant,inter,batch", [
    ("int8", 5120, 16), ("int4", 5120, 16), ("int8", 10240, 8), ("int4", 1152, 17), ("int8", 1152, 33), ("int4", 1000, 3), ("int4, w2 plain", 1152, 3)])
def test_parts_match_single_launches(quant, inter, batch):
    m = _model(quant, inter, batch)
    if inter == 1000:   # gate and up are not a multiple of 128 rows: two products
        assert m.layers[0].feed_forward.w1.weight.shape[0] == 1000
    torch.manual_seed(4)
    tok = torch.randint(0, m.config.vocab_size, (4, batch), device="cuda")
    out = []
    for fused in (False, True):
        eng = DecodeEngine(m, batch, 0.0, None, fused=fused)
        assert not eng.fused and eng.parts == fused
        eng = eng.capture()
        eng.set_state(tok[0], 0)
        logits = []
        for t in tok:
            eng.tok.copy_(t)
            eng.step()
            logits.append(eng.logits.double())
        out.append(torch.stack(logits))
    ref, got = out
    assert (got - ref).norm().item() < 0.011 * ref.norm().item()
