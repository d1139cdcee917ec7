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


@pytest.mark.parametrize("b,t,h,d,s,extra,by_kernel", [(1, 1, 1, 8, 8, 0, True), (2, 37, 3, 64, 40, 64, True), (1, 700, 8, 128, 704, 4096, True),
                                                       (2, 5, 3, 64, 16, 1, False), (1, 6, 2, 12, 8, 0, False)])
@torch.no_grad()
def test_cache_rows_and_shared_heads_equal_the_single_operations(b, t, h, d, s, extra, by_kernel):
    mine, ref = (M.KVCache(b, s, h, d).cuda() for _ in range(2))
    for c in (mine, ref):
        c.k_cache.fill_(3.0), c.v_cache.fill_(5.0)
    rows = torch.randn(b, t, 2 * h * d + extra, device="cuda").to(torch.bfloat16)
    k, v = (rows[..., i * h * d: (i + 1) * h * d].view(b, t, h, d) for i in range(2))
    f = torch.randn(t, d // 2, 2, device="cuda").to(torch.bfloat16)
    pos = torch.randperm(s, device="cuda")[:t]
    pos[0] -= s                                                      # a position from the end
    assert M.kv_rows(mine, pos.int() if h == 3 else pos, k, v, f) == by_kernel   # (both widths of positions)
    ref.update(pos, _rotary(k, f).transpose(1, 2), v.transpose(1, 2))
    if by_kernel:
        assert torch.equal(mine.k_cache, ref.k_cache) and torch.equal(mine.v_cache, ref.v_cache)
    # not for the kernel: other positions, a cache for more sequences, gradients
    assert not M.kv_rows(mine, pos.short(), k, v, f) and not M.kv_rows(M.KVCache(b + 1, s, h, d).cuda(), pos, k, v, f) and not M.kv_rows(None, None, k, v, f)
    with torch.enable_grad():
        assert not M.kv_rows(mine, pos, k.detach().requires_grad_(), v, f)
    for rep in (1, 2, 5):
        ks, vs = M.repeat_heads(ref.k_cache, ref.v_cache, rep)
        assert torch.equal(ks, ref.k_cache.repeat_interleave(rep, dim=1)) and torch.equal(vs, ref.v_cache.repeat_interleave(rep, dim=1))
    kt, vt = ref.k_cache.transpose(1, 2), ref.v_cache.transpose(1, 2)
    assert all(torch.equal(x, y.repeat_interleave(2, dim=1)) for x, y in zip(M.repeat_heads(kt, vt, 2), (kt, vt)))


@pytest.mark.parametrize("where", ["object", "class"])
@torch.no_grad()
def test_a_replaced_update_of_the_cache_is_called(where, monkeypatch):
    """A program that wraps KVCache.update (to record or change what is cached) sees every call, on the object or on the class."""
    att, seen = M.Attention(M.ModelArgs(dim=256, n_head=4, n_local_heads=2)).to("cuda", torch.bfloat16), []
    att.kv_cache = M.KVCache(1, 16, 2, 64).cuda()
    plain = M.KVCache.update

    def update(self, pos, k, v):
        seen.append(pos.numel())
        return plain(self, pos, k, 2 * v)

    x, pos, f = torch.randn(1, 5, 256, device="cuda").to(torch.bfloat16), torch.arange(5, device="cuda"), torch.randn(5, 32, 2, device="cuda").to(torch.bfloat16)
    mask = torch.ones(1, 1, 5, 16, dtype=torch.bool, device="cuda").tril()
    att(x, f, mask, pos)
    v = att.kv_cache.v_cache.clone()
    if where == "object":
        att.kv_cache.update = update.__get__(att.kv_cache)
    else:
        monkeypatch.setattr(M.KVCache, "update", update)
    att(x, f, mask, pos)
    assert seen == [5] and torch.equal(att.kv_cache.v_cache, 2 * v) and v.any()
