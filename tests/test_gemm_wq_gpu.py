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


@pytest.mark.parametrize("m", [2, 3, 8, 9, 12, 16, 17])
@pytest.mark.parametrize("bits,n,k,group", [(4, 16384, 8192, 128), (4, 8192, 16384, 64), (4, 14336, 4096, 32), (8, 16384, 8192, 0), (8, 640, 14336, 0)])
def test_few_rows(bits, n, k, group, m):
    # both sides of the rule that sends calls of up to 16 rows to the GEMM
    _check(bits, m, n, k, group)


@pytest.mark.parametrize("bits,group", [(4, 32), (4, 128), (8, 0)])
@pytest.mark.parametrize("m,n,k", [(1, 128, 64), (8, 640, 1088), (16, 321, 4096), (17, 640, 1088), (40, 1000, 512), (200, 640, 2048)])
def test_residual(bits, group, m, n, k):
    # y = bf16(residual + bf16(x W^T)): the residual's sum of the plain call's result, also in place and with wider rows
    from torchao_fork_b200 import _lib
    k = -(-k // max(group, 1)) * max(group, 1)
    gen = torch.Generator(device="cuda").manual_seed(m + n + k)
    w = torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    if bits == 4:
        packed, scales = T.b200_int4_quantize_pack(w, group, 1e-6, True)
        plain = T.b200_int4_weight_only_mm(x, packed, group, scales, n)
    else:
        q, scales = T.b200_int8_quantize(w, 1e-6, True)
        packed = T.b200_int8_pack(q)
        plain = T.b200_int8_weight_only_mm(x, packed, scales)
    np_, kp = packed.shape[0] * 16, packed.shape[1] * 64
    xp = torch.nn.functional.pad(x, (0, kp - k))
    L = _lib.lib()
    ws = torch.empty(L.ao_b200_mm_residual_workspace_bytes(m, np_, kp, group), dtype=torch.uint8, device="cuda").random_(0, 255)
    h = torch.randn(m, n + 3, generator=gen, device="cuda").to(torch.bfloat16)
    run = lambda res, y: _lib.check(L.ao_b200_mm_residual(  # noqa: E731
        xp.data_ptr(), m, kp, kp, packed.data_ptr(), scales.data_ptr(), np_, kp, group, y.data_ptr(), n, y.stride(0), res.data_ptr(), res.stride(0),
        ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream), "mm_residual")
    y = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    run(h, y)
    inside = h.clone()
    run(inside[:, :n], inside)
    assert torch.equal(inside[:, :n], y) and torch.equal(inside[:, n:], h[:, n:])
    if m > 16:   # the plain call is this GEMM too: the same bits
        assert torch.equal(y, h[:, :n] + plain)
    # below, the plain call may be a kernel that sums in another order: one rounding of the product apart
    assert ((y.double() - h[:, :n].double() - plain.double()).norm() / y.double().norm()).item() < 2.0 ** -7
    assert L.ao_b200_mm_residual(xp.data_ptr(), m, kp, kp, packed.data_ptr(), scales.data_ptr(), np_, kp, group, y.data_ptr(), n, n, h.data_ptr(), n + 3,
                                 ws.data_ptr(), 16, 0) != 0


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("m", [12, 40, 300])
def test_weights_written_by_the_kernel_in_front(bits, m):
    # the weights of a call may be what the launch before it wrote: its result is that of weights long there, time after time
    n, k = 16384, 8192
    x, packed, scales, want = None, [], [], []
    for seed in range(2):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        w = torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16)
        x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16) if x is None else x
        if bits == 4:
            p, sc = T.b200_int4_quantize_pack(w, 128, 1e-6, True)
        else:
            q, sc = T.b200_int8_quantize(w, 1e-6, True)
            p = T.b200_int8_pack(q)
        packed.append(p), scales.append(sc)
        torch.cuda.synchronize()
        want.append(T.b200_int4_weight_only_mm(x, p, 128, sc, n) if bits == 4 else T.b200_int8_weight_only_mm(x, p, sc))
    pw, sw, got = torch.empty_like(packed[0]), torch.empty_like(scales[0]), []
    torch.cuda.synchronize()
    for i in range(24):
        pw.copy_(packed[i % 2])
        sw.copy_(scales[i % 2])
        got.append(T.b200_int4_weight_only_mm(x, pw, 128, sw, n) if bits == 4 else T.b200_int8_weight_only_mm(x, pw, sw))
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % 2]), i


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("m", [1, 2, 3, 8])
@pytest.mark.parametrize("n,k", [(4096, 14336), (8192, 28672), (4096, 8192)])
def test_weights_of_few_rows_written_by_the_kernel_in_front(bits, m, n, k):
    # the same where the call is a GEMV, which starts while the kernel in front of it ends: k of one CTA, and of a cluster's in halves or quarters
    x, packed, scales, want = None, [], [], []
    for seed in range(2):
        gen = torch.Generator(device="cuda").manual_seed(seed)
        w = torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16)
        x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16) if x is None else x
        p, sc = T.b200_int4_quantize_pack(w, 128, 1e-6, True) if bits == 4 else T.b200_int8_quantize(w, 1e-6, True)
        p = p if bits == 4 else T.b200_int8_pack(p)
        packed.append(p), scales.append(sc)
        torch.cuda.synchronize()
        want.append(T.b200_int4_weight_only_mm(x, p, 128, sc, n) if bits == 4 else T.b200_int8_weight_only_mm(x, p, sc))
    pw, sw, got = torch.empty_like(packed[0]), torch.empty_like(scales[0]), []
    torch.cuda.synchronize()
    for i in range(24):
        sw.copy_(scales[i % 2])
        pw.copy_(packed[i % 2])
        got.append(T.b200_int4_weight_only_mm(x, pw, 128, sw, n) if bits == 4 else T.b200_int8_weight_only_mm(x, pw, sw))
    for i, y in enumerate(got):
        assert torch.equal(y, want[i % 2]), i


def test_threads_that_share_a_stream():
    # a call is a staging launch and the GEMM behind it, over one workspace per stream: nobody's launch may come between them
    import threading
    calls, want = [], []
    for i, (bits, m, n, k) in enumerate(((4, 40, 640, 4096), (4, 130, 1024, 2048), (4, 300, 384, 1024), (4, 24, 640, 8192))):
        gen = torch.Generator(device="cuda").manual_seed(i)
        w, x = (torch.randn(r, k, generator=gen, device="cuda").to(torch.bfloat16) for r in (n, m))
        packed, sz = T.b200_int4_quantize_pack(w, 128, 1e-6, True)
        calls.append((x, packed, 128, sz, n))
        want.append(T.b200_int4_weight_only_mm(*calls[-1]))
    bad, start = [], threading.Barrier(len(calls))

    def work(i):
        start.wait()
        for _ in range(100):
            ys = [T.b200_int4_weight_only_mm(*calls[i]) for _ in range(5)]
            if not all(torch.equal(y, want[i]) for y in ys):
                bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("group", [32, 64, 128, 256])
@pytest.mark.parametrize("m", [12, 16])
def test_few_rows_with_infinities_and_huge_values(group, m):
    # sums that overflow with 128 + q in the place of q - 8, and do not with the weights themselves; infinities keep their sign
    n, k = 16384, 8192
    gen = torch.Generator(device="cuda").manual_seed(group + m)
    w = (0.02 * torch.randn(n, k, generator=gen, device="cuda")).to(torch.bfloat16)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    x[0, 77] = torch.inf
    x[1, 4000], x[1, 8191] = -torch.inf, torch.inf
    x[2, 5] = torch.nan
    x[3, ::97] = 3e38
    x[4, 1024:1152] = -2e37
    x[5, 0] = 3.3e38
    x[m - 1, 130], x[m - 1, 131] = torch.inf, torch.inf
    packed, sz = T.b200_int4_quantize_pack(w, group, 1e-6, True)
    q = T.b200_int4_unpack(packed)[:n, :k].double().reshape(n, -1, group)
    p = sz.permute(0, 2, 1, 3).reshape(packed.shape[0] * 16, -1, 2)[:n, : k // group].double()
    wd = ((q - 8) * p[..., 0:1] + p[..., 1:2]).reshape(n, k)
    y = T.b200_int4_weight_only_mm(x, packed, group, sz, n)
    plain = torch.tensor([r for r in range(m) if r not in (0, 1, 2, m - 1)], device="cuda")
    # marked segments meet the weights as they are in bf16, the others unrounded ones.  (Row 4 has equal activations over a whole group: its
    # 16 weight values occur eight times each, so their roundings add up in step, to 8 sqrt(16) / sqrt(128) = 2.8 times what they make of
    # independent terms; against unrounded weights that is 2.8 x 2^-9 sqrt(1 / 3), close to the bound.  So it is not the reference there.)
    ref = torch.where((x[plain].abs() > 2.0 ** 100).any(1, keepdim=True), x[plain].double() @ wd.to(torch.bfloat16).double().t(), x[plain].double() @ wd.t())
    got = y[plain].double()
    assert got.isfinite().all() and (((got - ref).norm(dim=1) / ref.norm(dim=1)) < 2.0 ** -8).all()
    # one infinity: the sign of its weight as it is in bf16 (zero: NaN); two: NaN where the signs differ
    sign = lambda j: wd[:, j].to(torch.bfloat16).sign()  # noqa: E731
    for row, terms in ((0, [(77, 1)]), (1, [(4000, -1), (8191, 1)]), (m - 1, [(130, 1), (131, 1)])):
        s = [sg * sign(j) for j, sg in terms]
        want = torch.where((s[0] != 0) & (s[-1] == s[0]), s[0].float() * torch.inf, torch.full_like(s[0].float(), torch.nan))
        assert torch.equal(y[row].float().isnan(), want.isnan())
        assert torch.equal(y[row].float().nan_to_num(nan=0.0), want.nan_to_num(nan=0.0)), row
    assert y[2].isnan().all()


def test_first_call_of_a_new_thread():
    # a thread without a current context: the tensor maps have to be made all the same (without them the call is a loop of small products)
    import threading
    gen = torch.Generator(device="cuda").manual_seed(3)
    w, x = (torch.randn(r, 512, generator=gen, device="cuda").to(torch.bfloat16) for r in (640, 200))
    packed, sz = T.b200_int4_quantize_pack(w, 128, 1e-6, True)
    want, got = T.b200_int4_weight_only_mm(x, packed, 128, sz, 640), []
    t = threading.Thread(target=lambda: got.append(T.b200_int4_weight_only_mm(x, packed, 128, sz, 640)))
    t.start()
    t.join()
    assert torch.equal(got[0], want)


def test_more_than_four_million_rows():
    m, n, k = (1 << 22) + 300, 128, 64
    gen = torch.Generator(device="cuda").manual_seed(1)
    w = torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16)
    x = torch.randn(m, k, generator=gen, device="cuda", dtype=torch.bfloat16)
    q, scale = T.b200_int8_quantize(w, 1e-6, True)
    packed = T.b200_int8_pack(q)
    y = T.b200_int8_weight_only_mm(x, packed, scale)
    for rows in (slice(0, 700), slice(1 << 21, (1 << 21) + 300), slice(m - 513, m)):
        ref = x[rows].double() @ (q.double() * scale.double()[:, None]).t()
        assert ((y[rows].double() - ref).norm() / ref.norm()).item() < 2.0 ** -8


@pytest.mark.parametrize("bits,group", [(4, 32), (4, 128), (4, 256), (8, 0)])
@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("m,k", [(3, 28672), (8, 28672), (5, 14336), (8, 14336), (8, 8192)])
def test_long_few_rows_with_infinities_huge_and_tiny_values(bits, group, residual, m, k):
    # calls whose k the CTAs of a cluster share: finite results wherever bf16 products with 32-bit sums have them, infinities with the sign of
    # their weight, tiny rows as exact as others
    from torchao_fork_b200 import _lib
    # the sums have to stay below 3.4e38: 296 terms of 0.02 big have a norm of 0.34 big, of up to 127 big 740 big
    n, big = 640, 1e38 if bits == 4 else 1e35
    gen = torch.Generator(device="cuda").manual_seed(m + k + group)
    w = (0.02 * torch.randn(n, k, generator=gen, device="cuda")).to(torch.bfloat16)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    if bits == 4:
        packed, scales = T.b200_int4_quantize_pack(w, group, 1e-6, True)
        p = scales.permute(0, 2, 1, 3).reshape(packed.shape[0] * 16, -1, 2)[:n, : k // group].double()
        wd = ((T.b200_int4_unpack(packed)[:n, :k].double().reshape(n, -1, group) - 8) * p[..., 0:1] + p[..., 1:2]).reshape(n, k)
        wb = wd.to(torch.bfloat16).double()
    else:
        q, scales = T.b200_int8_quantize(w, 1e-6, True)
        packed, wb, wd = T.b200_int8_pack(q), q.double(), q.double() * scales.double()[:, None]
    # the rows, up to eight of them: an infinity, huge values, tiny ones, two infinities, a NaN, a block of huge ones, a single one, an infinity and a huge value
    x[0, 77] = torch.inf
    x[1, ::97] = big
    x[2] = (x[2].float() * 1e-36).to(torch.bfloat16)
    signs = {0: [(77, 1)]}
    if m > 3:
        x[3, k // 2 - 1], x[3, k - 1] = -torch.inf, torch.inf
        x[4, 5] = torch.nan
        signs[3] = [(k // 2 - 1, -1), (k - 1, 1)]
    if m > 5:
        x[5, 1024:1152] = -big / 16
        x[6, k - 8] = big
        x[7, 130], x[7, k - 130] = torch.inf, big
        signs[7] = [(130, 1)]
    if residual:
        res, L = torch.zeros(m, n, dtype=torch.bfloat16, device="cuda"), _lib.lib()
        np_, kp = packed.shape[0] * 16, packed.shape[1] * 64
        ws = torch.empty(L.ao_b200_mm_residual_workspace_bytes(m, np_, kp, group), dtype=torch.uint8, device="cuda")
        y = torch.empty_like(res)
        _lib.check(L.ao_b200_mm_residual(x.data_ptr(), m, k, k, packed.data_ptr(), scales.data_ptr(), np_, kp, group, y.data_ptr(), n, n, res.data_ptr(), n,
                                         ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream), "mm_residual")
    elif bits == 4:
        y = T.b200_int4_weight_only_mm(x, packed, group, scales, n)
    else:
        y = T.b200_int8_weight_only_mm(x, packed, scales)
    for row in range(m):
        got = y[row].double()
        if row in signs:
            s = [sg * wb[:, j].sign() for j, sg in signs[row]]
            want = torch.where((s[0] != 0) & (s[-1] == s[0]), s[0] * torch.inf, torch.full_like(s[0], torch.nan))
            assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(nan=0.0), want.nan_to_num(nan=0.0)), row
        elif row == 4:
            assert got.isnan().all()
        else:
            # the weights of a row of huge values may be met as they are in bf16: 2^-9 sqrt(1 / 3) of each, and the result's rounding(s); equal values
            # over a block add up roundings in step (2.8 times that, against either reference, half of it against their mean)
            xd = x[row].double()
            ref = xd @ wd.t()
            near = min(((got - r).norm() / ref.norm()).item() for r in (ref, xd @ wb.t() if bits == 4 else ref))
            assert got.isfinite().all() and near < 2.0 ** -8, (row, near)


@pytest.mark.parametrize("bits,group", [(4, 32), (4, 128), (8, 0)])
@pytest.mark.parametrize("m", [24, 32, 48, 64, 77, 128, 144, 256, 300])
@pytest.mark.parametrize("residual", [False, True])
def test_last_tile_from_the_accumulators(bits, group, m, residual):
    """28672 x 2048: 16 units a tile and 24 for each CTA or pair of 148 or 74, so every other tile is shared by two with at least eight units behind it, and
    its first owner finishes it from its accumulators if the second one was there before.  By the deal (25 c mod 16) it holds any number of units of it,
    one among them.  Up to 32 rows one CTA, up to 64 two issuing warps, up to 128 two accumulator buffers, from 257 on two row tiles.  Whether that path is taken
    depends on time: equal calls give equal bits all the same.  Bound as above; a wrong tile would show in its 128 columns, so they are looked at by themselves."""
    from torchao_fork_b200 import _lib
    n, k = 28672, 2048
    gen = torch.Generator(device="cuda").manual_seed(m + bits)
    w = torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    if bits == 4:
        packed, scales = T.b200_int4_quantize_pack(w, group, 1e-6, True)
        p = scales.permute(0, 2, 1, 3).reshape(packed.shape[0] * 16, -1, 2)[:n, : k // group].double()
        wd = ((T.b200_int4_unpack(packed)[:n, :k].double().reshape(n, -1, group) - 8) * p[..., 0:1] + p[..., 1:2]).reshape(n, k)
        run = lambda: T.b200_int4_weight_only_mm(x, packed, group, scales, n)  # noqa: E731
    else:
        q, scales = T.b200_int8_quantize(w, 1e-6, True)
        packed, wd = T.b200_int8_pack(q), q.double() * scales.double()[:, None]
        run = lambda: T.b200_int8_weight_only_mm(x, packed, scales)  # noqa: E731
    ref, h = x.double() @ wd.t(), None
    if residual:
        L = _lib.lib()
        h = torch.randn(m, n, generator=gen, device="cuda").to(torch.bfloat16)
        ws = torch.empty(L.ao_b200_mm_residual_workspace_bytes(m, n, k, group), dtype=torch.uint8, device="cuda")

        def run():
            y = torch.empty_like(h)
            _lib.check(L.ao_b200_mm_residual(x.data_ptr(), m, k, k, packed.data_ptr(), scales.data_ptr(), n, k, group, y.data_ptr(), n, n, h.data_ptr(), n,
                                             ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream), "mm_residual")
            return y
        ref = ref + h.double()
    y = run()
    tiles = lambda t: t.reshape(m, n // 128, 128).square().sum((0, 2)).sqrt()  # noqa: E731
    assert (tiles(y.double() - ref) / tiles(ref)).max().item() < 2.0 ** -8
    assert all(torch.equal(run(), y) for _ in range(12))


@pytest.mark.parametrize("m", [511, 512, 513, 640, 769, 1041])
@pytest.mark.parametrize("bits,n,k,group", [(4, 640, 1088, 32), (4, 321, 1088, 64), (4, 8192, 512, 128), (4, 384, 512, 256), (8, 8320, 192, 0), (8, 8192, 64, 0), (8, 640, 1088, 0)])
def test_activations_read_in_place(bits, n, k, group, m):
    # both sides of the line in rows and in outputs; half a unit at the end of k; tiles that end inside and outside of x
    _check(bits, m, n, k, group)


@pytest.mark.parametrize("bits,group", [(4, 64), (8, 0)])
def test_activations_read_in_place_out_of_wider_rows(bits, group):
    # rows further apart than they are long, from an odd multiple of 16 bytes on, with NaN and infinities around them; k shorter than the weights'
    from torchao_fork_b200 import _lib
    gen = torch.Generator(device="cuda").manual_seed(bits)
    n, k, kx, m, ld = 640, 1152, 1096, 700, 1320
    w = torch.randn(n, k, generator=gen, device="cuda").to(torch.bfloat16)
    x = torch.full((m + 2, ld), float("nan"), device="cuda", dtype=torch.bfloat16)
    x[1::2] = float("inf")
    x[1 : m + 1, 24 : 24 + kx] = torch.randn(m, kx, generator=gen, device="cuda").to(torch.bfloat16)
    if bits == 4:
        packed, scales = T.b200_int4_quantize_pack(w, group, 1e-6, True)
        wd = T.b200_int4_dequantize(packed, scales, group).double()[:n]
    else:
        q, scales = T.b200_int8_quantize(w, 1e-6, True)
        packed = T.b200_int8_pack(q)
        wd = q.double() * scales.double()[:, None]
    np_, kp = packed.shape[0] * 16, packed.shape[1] * 64
    L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    y = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    xp = x.data_ptr() + (ld + 24) * 2
    if bits == 4:
        ws = torch.zeros(L.ao_b200_int4_mm_workspace_bytes(m, np_, kp), dtype=torch.uint8, device="cuda")
        _lib.check(L.ao_b200_int4_mm(xp, m, kx, ld, packed.data_ptr(), scales.data_ptr(), np_, kp, group, y.data_ptr(), n, n, ws.data_ptr(), ws.numel(), st), "int4_mm")
    else:
        ws = torch.empty(L.ao_b200_int8_mm_workspace_bytes(m, np_, kp), dtype=torch.uint8, device="cuda").random_(0, 255)
        _lib.check(L.ao_b200_int8_mm(xp, m, kx, ld, packed.data_ptr(), scales.data_ptr(), np_, kp, y.data_ptr(), n, n, ws.data_ptr(), ws.numel(), st), "int8_mm")
    ref = x[1 : m + 1, 24 : 24 + kx].double() @ wd[:, :kx].t()
    assert ((y.double() - ref).norm() / ref.norm()).item() < 2.0 ** -8


@pytest.mark.parametrize("k", [64, 192, 256, 320, 1088, 4160])
@pytest.mark.parametrize("bits,group,m", [(4, 32, 16), (4, 64, 9), (4, 64, 60), (4, 32, 100), (8, 0, 16), (8, 0, 33), (8, 0, 128)])
def test_long_units(bits, group, m, k):
    # units of 256 k whose second half is there, in part or not at all; tiles of one unit and of several, shared and whole
    for n in (128, 640, 16384):
        _check(bits, m, n, k, group)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("m", [3, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(12288, 4096), (12160, 4096), (24576, 4096), (24448, 4096), (8192, 24576), (8064, 24576)])
def test_few_rows_on_both_sides_of_their_lines(bits, m, n, k):
    _check(bits, m, n, k, 128)


@pytest.mark.parametrize("k", [256, 512, 768, 1280, 2048, 2304, 2816, 3328, 4096, 9472, 11008])   # (9472: 37 units, dealt as 39)
@pytest.mark.parametrize("bits,group,m,n", [(4, 128, 17, 1024), (4, 32, 32, 321), (4, 256, 33, 4096), (4, 64, 128, 8192), (8, 0, 17, 1000), (8, 0, 16, 14336), (8, 0, 64, 640)])
def test_small_weights(bits, group, m, n, k):
    # tiles of one owner, of a few, and of as many as they have units (the number: wq_owners)
    _check(bits, m, n, k, group)


@pytest.mark.parametrize("group,m,n,k", [(128, 9, 18432, 4096), (128, 11, 18304, 4096), (64, 9, 24576, 4096), (64, 10, 24448, 4096), (32, 9, 20480, 4096), (32, 10, 20352, 4096),
                                         (256, 12, 14336, 4096), (256, 12, 14464, 4096), (32, 3, 8192, 24576), (64, 8, 8192, 24576), (64, 3, 8192, 24576), (128, 3, 8192, 24576)])
def test_few_rows_by_group_on_both_sides_of_their_lines(group, m, n, k):
    _check(4, m, n, k, group)


@pytest.mark.parametrize("bits,group", [(4, 64), (8, 0)])
@pytest.mark.parametrize("m", [100, 600, 1024])
def test_results_over_the_activations(bits, group, m):
    # y in x's own memory, plain and with the rows themselves as residual: from 512 rows on the GEMM would read them while it writes
    from torchao_fork_b200 import _lib
    n = k = 1024
    gen = torch.Generator(device="cuda").manual_seed(m)
    w = (torch.randn(n, k, generator=gen, device="cuda") / 32).to(torch.bfloat16)
    x = torch.randn(m, k, generator=gen, device="cuda").to(torch.bfloat16)
    L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    if bits == 4:
        packed, scales = T.b200_int4_quantize_pack(w, group, 1e-6, True)
        plain = T.b200_int4_weight_only_mm(x, packed, group, scales, n)
        size, call, rest = L.ao_b200_int4_mm_workspace_bytes, L.ao_b200_int4_mm, (n, k, group)
    else:
        q, scales = T.b200_int8_quantize(w, 1e-6, True)
        packed = T.b200_int8_pack(q)
        plain = T.b200_int8_weight_only_mm(x, packed, scales)
        size, call, rest = L.ao_b200_int8_mm_workspace_bytes, L.ao_b200_int8_mm, (n, k)
    ws = torch.zeros(max(size(m, n, k), L.ao_b200_mm_residual_workspace_bytes(m, n, k, group)), dtype=torch.uint8, device="cuda")
    p = lambda t: t.data_ptr()  # noqa: E731
    for _ in range(5):
        over, both = x.clone(), x.clone()
        _lib.check(call(p(over), m, k, k, p(packed), p(scales), *rest, p(over), n, n, p(ws), ws.numel(), st), "mm")
        _lib.check(L.ao_b200_mm_residual(p(both), m, k, k, p(packed), p(scales), n, k, group, p(both), n, n, p(both), n, p(ws), ws.numel(), st), "mm_residual")
        # (two orders of the same sums, each rounded within 2^-9 of its value: 2^-8 of the whole; a wrong row would be off by its size)
        assert ((over.double() - plain.double()).norm() / plain.double().norm()).item() < 2.0 ** -8
        want = (x.float() + plain.float()).to(torch.bfloat16)
        assert ((both.double() - want.double()).norm() / want.double().norm()).item() < 2.0 ** -7
        assert (over.float() - plain.float()).abs().amax(1).max() < 0.05 * plain.float().abs().max()


@pytest.mark.parametrize("bits,group", [(4, 128), (4, 32), (8, 0)])
@pytest.mark.parametrize("m,n,k", [(17, 28672, 1280), (33, 28672, 768), (64, 28672, 2048), (128, 28672, 1280), (100, 20480, 1536)])
def test_last_tile_from_the_accumulators_of_long_units(bits, group, m, n, k):
    # a few units of 256 k a tile and more tiles than SMs: the neighbour has two units and more to do behind its share of the tile
    _check(bits, m, n, k, group)
