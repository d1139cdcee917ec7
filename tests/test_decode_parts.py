"""The decode step where only some projections take the fused GEMV (long activations, more than 16 sequences, unquantized lines), against
the same step made of one launch per operation.  Bound: each of the four places per layer that rounds to bf16 in another order (products
summed in another order and rounded) moves the logits by a relative 2^-9 at most; with two layers and independent roundings
sqrt(8) 2^-9 = 0.55 %, doubled for the sums behind the norms: 1.1 % is 39 dB."""
import pytest
import torch

import torchao_fork_b200 as ao
from torchao_fork_b200 import _lib
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


@pytest.mark.parametrize("fused", [False, True])
def test_int8_gemm_and_int4_tickets_keep_apart(fused):
    """int8 layers whose longest product takes the GEMM beside an int4 output projection large enough for the kernel that counts on zeroed
    tickets (3 to 5 sequences): repeated steps give repeated logits, and the tickets are zero after each."""
    torch.manual_seed(5)
    cfg = ModelArgs(block_size=64, vocab_size=49152, n_layer=1, n_head=40, n_local_heads=10, dim=5120, intermediate_size=28672)
    old = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        with torch.device("cuda"):
            m = Transformer(cfg).eval()
    finally:
        torch.set_default_dtype(old)
    ao.quantize_(m, ao.Int4WeightOnlyConfig(group_size=128), filter_fn=lambda mod, name: name == "output")
    ao.quantize_(m, ao.Int8WeightOnlyConfig(), filter_fn=lambda mod, name: isinstance(mod, torch.nn.Linear) and name != "output")
    m.setup_caches(4, 64, device=torch.device("cuda"))
    eng = DecodeEngine(m, 4, 0.0, None, fused=fused)
    # both want the front of a workspace
    assert eng.output.kind == "int4" and eng.layers[0]["w2"].kind == "int8" and eng.layers[0]["w2"].workspace_bytes(4) > 0
    tok, logits = torch.tensor([1, 2, 3, 4], device="cuda"), []
    for _ in range(4):
        eng.set_state(tok, 3)
        eng.step()
        logits.append(eng.logits.clone())
    for other in logits[1:]:
        assert torch.equal(other, logits[0])
    # [partial sums][tickets ..]: the last kilobyte in front of the GEMM's part
    front = int(_lib.lib().ao_b200_int4_mm_workspace_bytes(1, eng.output.np_, eng.output.kp))
    assert not eng.ws[front - (1 << 20) : front].any()


def test_projection_whose_correction_sums_do_not_fit_beside_its_rows():
    """Five rows of 14336 leave room for the sums over groups of 128 but not for those of 64: the step takes that projection's other form."""
    test_parts_match_single_launches("int4", 14336, 5)


@pytest.mark.parametrize("group", [0, 32, 64, 128, 256])
def test_calls_that_fit_are_taken_and_the_others_refused(group):
    L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    seen = set()
    for K in (4096, 8192, 12288, 14336, 20480, 28672, 36864):
        N = 128
        w = torch.randn(N, K, device="cuda").to(torch.bfloat16)
        if group:
            packed, scales = torch.ops.torchao.b200_int4_quantize_pack(w, group, 1e-6, True)
        else:
            q, scales = torch.ops.torchao.b200_int8_quantize(w, 1e-6, True)
            packed = torch.ops.torchao.b200_int8_pack(q)
        for M in (1, 2, 3, 5, 8, 9, 16):
            x, y = torch.randn(M, K, device="cuda").to(torch.bfloat16), torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
            args = (x.data_ptr(), M, K, K, packed.data_ptr(), scales.data_ptr(), N, K)
            tail = (y.data_ptr(), N, N, None, 0.0, None, 0, 0)
            rc = L.ao_b200_int4_gemv_fused(*args, group, *tail, None, 0, st) if group else L.ao_b200_int8_gemv_fused(*args, *tail, st)
            fits = L.ao_b200_gemv_fused_fits(M, K, group)
            seen.add(fits)
            assert rc == (0 if fits else 4), (M, K, group, rc, fits)
    assert seen == {0, 1} and L.ao_b200_gemv_fused_fits(17, 4096, group) == 0
