"""ao_b200_rmsnorm at both sides of the widths where it changes form, with and without a residual, in place, against float64.

Bound: bf16 has 8 significant bits, so a rounding to it is off by 2^-8 of the value at most, just above a power of two; the norm and its product with the
weight are rounded once each: 2^-7, and 2^-20 and less for the row's factor, an fp32 sum of squares.  2^-6.9 holds all of it.  The sum with the residual
is rounded to bf16 first, here as there."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from torchao_fork_b200 import _lib  # noqa: E402


@pytest.mark.parametrize("dim", [8, 288, 4096, 4104, 8192, 8200, 16384, 16392])
@pytest.mark.parametrize("rows", [1, 3, 700])
@pytest.mark.parametrize("residual", [False, True])
def test_rmsnorm(dim, rows, residual):
    gen = torch.Generator(device="cuda").manual_seed(dim + rows)
    make = lambda *s: torch.randn(*s, generator=gen, device="cuda").bfloat16()  # noqa: E731
    x, w, r = make(rows, dim), make(dim), make(rows, dim)
    h = (x.float() + r.float()).bfloat16() if residual else x.clone()
    y, st = torch.empty_like(x), torch.cuda.current_stream().cuda_stream
    p = lambda t: t.data_ptr()  # noqa: E731
    _lib.check(_lib.lib().ao_b200_rmsnorm(p(x), p(r) if residual else None, p(w), p(x) if residual else None, p(y), rows, dim, 1e-5, st), "rmsnorm")
    assert torch.equal(x, h)           # the sum, written in place
    hd = h.double()
    ref = hd * torch.rsqrt(hd.square().mean(-1, keepdim=True) + 1e-5) * w.double()
    assert ((y.double() - ref).abs() <= 2.0 ** -6.9 * ref.abs() + 1e-30).all()
