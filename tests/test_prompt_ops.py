"""The one-launch element-wise steps of the Llama block for prompt rows against the single operations they stand for."""
import pytest
import torch
import torch.nn.functional as F

from torchao_fork_b200._models.llama import model as M

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)


def _rotary(x, f):
    xs, fc = x.float().reshape(*x.shape[:-1], -1, 2), f.view(1, x.shape[1], 1, x.shape[3] // 2, 2)
    return torch.stack([xs[..., 0] * fc[..., 0] - xs[..., 1] * fc[..., 1], xs[..., 1] * fc[..., 0] + xs[..., 0] * fc[..., 1]], -1).flatten(3).type_as(x)


@pytest.mark.parametrize("b,t,h,d,extra", [(1, 1, 1, 8, 0), (2, 37, 5, 64, 64), (1, 700, 32, 128, 2048), (3, 9, 4, 120, 8), (2, 5, 3, 64, 1), (2, 5, 3, 12, 0)])
@torch.no_grad()
def test_rotation_equals_the_single_operations(b, t, h, d, extra):
    # extra: columns beside the heads in a row (1: rows off 16 bytes, d = 12: heads off 16 bytes: the single operations)
    rows = torch.randn(b, t, h * d + extra, device="cuda").to(torch.bfloat16)
    x = rows[..., : h * d].view(b, t, h, d)
    f = torch.randn(t, d // 2, 2, device="cuda").to(torch.bfloat16)
    assert torch.equal(M.apply_rotary_emb(x, f), _rotary(x, f))
    tr = x.transpose(0, 1)
    f2 = torch.randn(b, d // 2, 2, device="cuda").to(torch.bfloat16)
    assert torch.equal(M.apply_rotary_emb(tr, f2), _rotary(tr, f2))


@pytest.mark.parametrize("shape", [(8,), (3, 24), (700, 1, 14336), (5, 7), (0, 8)])
@torch.no_grad()
def test_silu_product_equals_the_single_operations(shape):
    g, u = (torch.randn(shape, device="cuda").to(torch.bfloat16) * 4 for _ in range(2))
    if g.numel() > 8:
        g.view(-1)[:6] = torch.tensor([float("inf"), float("-inf"), float("nan"), -200.0, 3e38, 0.0])
    assert torch.equal(M.silu_mul(g, u).nan_to_num(nan=7.0), (F.silu(g) * u).nan_to_num(nan=7.0))
    assert torch.equal(M.silu_mul(g[..., 1:], u[..., 1:]).nan_to_num(nan=7.0), (F.silu(g) * u)[..., 1:].nan_to_num(nan=7.0))


@pytest.mark.parametrize("rows,dim", [((1,), 8), ((2, 3), 4096), ((1, 700), 5120), ((4,), 12272), ((4,), 12280), ((2,), 100)])
def test_norm_against_float64(rows, dim):
    m = M.RMSNorm(dim, 1e-5).cuda().to(torch.bfloat16)
    x = (torch.randn(*rows, dim, device="cuda") * 3).to(torch.bfloat16)
    with torch.no_grad():
        m.weight.copy_(torch.randn(dim, device="cuda"))
        y = m(x)
    xd = x.double()
    ref = xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-5) * m.weight.double()
    # bf16 has 8 significant bits: rounding moves a value by a relative 2^-8 at most, twice here; one per cent for the fp32 sums
    assert ((y.double() - ref).abs() <= 2.0 ** -7 * 1.01 * ref.abs() + 1e-38).all()
    # with gradients the single operations run, which have the same bound
    z = m(x)
    assert z.requires_grad and ((z.double() - ref).abs() <= 2.0 ** -7 * 1.01 * ref.abs() + 1e-38).all()
