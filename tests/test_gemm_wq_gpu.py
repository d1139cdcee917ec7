"""The weight-only GEMM (csrc/gemm_wq_tc.cu) where its plan changes: row tiles of 16 to 256 and the steps between them, one CTA or
a pair per tile, one or two issuing warps, odd and short rings, K whose last 128 is half a unit, row blocks without a partner,
tiles shared by many CTAs, whole tiles dealt out.

Bound: weights rounded once to bf16 (int4) and results rounded to bf16 (twice for int8) are relative errors of at most 2^-9 each,
near uniform, so their root mean squares add up to less than 2^-9 sqrt(2 / 3) (1 + small) of the result's; 2^-8 leaves room for
fp32 sums.  Equal calls give equal bits: shares are added in a fixed order."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

import torchao_fork_b200  # noqa: E402,F401

T = torch.ops.torchao


def _check(bits, m, n, k, group):
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    w = torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    if bits == 4:
        packed, sz = T.b200_int4_quantize_pack(w, group, 1e-6, True)
        q = T.b200_int4_unpack(packed)[:n, :k].double().reshape(n, -1, group)
        p = sz.permute(0, 2, 1, 3).reshape(packed.shape[0] * 16, -1, 2)[:n, : k // group].double()
        wd = ((q - 8) * p[..., 0:1] + p[..., 1:2]).reshape(n, k)
        run = lambda: T.b200_int4_weight_only_mm(x, packed, group, sz, n)  # noqa: E731
    else:
        q, scale = T.b200_int8_quantize(w, 1e-6, True)
        packed = T.b200_int8_pack(q)
        wd = q.double() * scale.double()[:, None]
        run = lambda: T.b200_int8_weight_only_mm(x, packed, scale)  # noqa: E731
    y = run()
    ref = x.double() @ wd.t()
    assert y.shape == (m, n)
    assert ((y.double() - ref).norm() / ref.norm()).item() < 2.0 ** -8
    assert (y.double() - ref).abs().max().item() < 0.05 * ref.square().mean().sqrt().item() + 2.0 ** -7 * ref.abs().max().item()
    assert torch.equal(run(), y)


@pytest.mark.parametrize("m", [17, 32, 33, 64, 65, 128, 129, 144, 255, 256, 257, 513])
@pytest.mark.parametrize("bits,n,k,group", [(4, 640, 1088, 64), (4, 384, 512, 256), (8, 640, 1088, 0)])
def test_row_tiles(bits, n, k, group, m):
    _check(bits, m, n, k, group)


@pytest.mark.parametrize("bits,m,n,k,group", [
    (4, 40, 321, 96, 32), (4, 300, 1000, 4096, 32), (4, 1000, 4096, 4096, 128), (8, 1000, 4096, 4096, 0), (8, 300, 2048, 14336, 0),
    (4, 24, 128, 16384, 128), (8, 24, 128, 16384, 0), (4, 5000, 12800, 256, 128), (8, 5000, 12800, 128, 0)])
def test_splits(bits, m, n, k, group):
    _check(bits, m, n, k, group)


@pytest.mark.parametrize("bits", [4, 8])
def test_output_rows_off_16_bytes(bits):
    # N not a multiple of 8: rows of y start at odd places, stored element by element
    _check(bits, 50, 323, 256, 64)
