"""Attention of prompt portions (ao_lm_window_attention_prompt) at the sizes of real layers, through the plan's own tiles: many tiles of
keys per tile of rows, windows shorter and longer than the run, earlier positions in the ring, last tiles of every kind, one and two
maps, and a head too large for anything but the plainest tiling.  Against float64.

Bound: queries are rounded to bf16 in front of the product (relative 2^-9 each, near uniform: 2^-9 / sqrt(3) of the scores' norm, which
moves a weight by |s| times that: below 0.4 % at scores of a few units) and the result is rounded once (2^-9 / sqrt(3)): 1 % holds both.
Equal calls give equal bits: nothing is summed in an order that depends on time."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from torchao_fork_b200 import _lib  # noqa: E402

BF16 = 0


def _reference(q, k, v, past, window, keep, lam):
    n, H, maps, d = q.shape
    G = k.shape[1]
    i, j = torch.arange(past, past + n, device="cuda")[:, None], torch.arange(past + n, device="cuda")[None, :]
    hidden = (j > i) | ((i - j >= window) & (j >= keep))
    out = []
    for h in range(H):
        g = h // (H // G)
        parts = [(q[:, h, m].double() @ k[:, g, m].double().t() * d ** -0.5).masked_fill(hidden, -torch.inf).softmax(-1) @ v[:, g].double()
                 for m in range(maps)]
        y = parts[0]
        if maps == 2:
            y = y - lam * parts[1]
            y = y * torch.rsqrt(y.square().mean(-1, keepdim=True) + 1e-6)
        out.append(y)
    return torch.cat(out, 1)


def _run(q, k, v, past, window, keep, lam):
    n, H, maps, d = q.shape
    G, dv = k.shape[1], v.shape[-1]
    L, p = _lib.lm(), lambda t: t.data_ptr()
    tile = ctypes.c_int()
    _lib.lm_check(L.ao_lm_window_attention_prompt_plan(BF16, maps, H, G, d, dv, ctypes.byref(tile)), "plan")
    assert tile.value > 0
    ring = max(window, 1) + 37
    i32 = lambda t: t.to(torch.int32).cuda()  # noqa: E731
    # the positions before the run as the append leaves them: the last `ring` in the ring, the kept ones beside it, rubbish elsewhere
    rk, rv = (torch.full((2, ring, t[0].numel()), 50.0, dtype=torch.bfloat16, device="cuda") for t in (k, v))
    fk, fv = (torch.full((2, keep + 1, t[0].numel()), 50.0, dtype=torch.bfloat16, device="cuda") for t in (k, v))
    old = torch.arange(max(0, past - ring), past, device="cuda")
    kept = torch.arange(min(past, keep + 1), device="cuda")
    for store, first, t in ((rk, fk, k), (rv, fv, v)):
        store[1, old % ring] = t[old].flatten(1)
        first[1, kept] = t[kept].flatten(1)
    kn, vn = k[past:].contiguous(), v[past:].contiguous()
    first = torch.arange(0, n, tile.value)
    back = torch.arange(n)
    slot, pos, bk = i32(back * 0 + 1), i32(back + past), i32(back)
    tf, tc = i32(first), i32((n - first).clamp(max=tile.value))
    out = torch.full((n, H * dv), 9.0, dtype=torch.bfloat16, device="cuda")
    _lib.lm_check(L.ao_lm_window_attention_prompt(
        p(q), p(kn), p(vn), p(rk), p(rv), p(fk), p(fv), ring, keep + 1, BF16, p(slot), p(pos), p(bk), p(tf), p(tc), tf.numel(), maps, H, G, d, dv, window,
        keep, d ** -0.5, lam, int(maps == 2), 1e-6, 1.0, p(out), H * dv, torch.cuda.current_stream().cuda_stream), "prompt")
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("maps,d,dv,H,G", [(1, 128, 128, 4, 2), (2, 64, 128, 2, 2), (2, 64, 128, 4, 1), (1, 256, 128, 2, 1), (2, 48, 96, 2, 1)])
@pytest.mark.parametrize("n,past,window,keep", [
    (520, 0, 4096, 0), (520, 0, 512, 0), (129, 0, 60, 3), (255, 0, 4096, 0), (127, 1, 512, 0), (128, 300, 512, 0), (161, 127, 4096, 5),
    (1, 700, 512, 4), (2, 129, 100, 0), (383, 640, 512, 0), (130, 1000, 512, 2), (640, 63, 129, 1)])
def test_prompt_portions_of_real_sizes(maps, d, dv, H, G, n, past, window, keep):
    gen = torch.Generator(device="cuda").manual_seed(n + past + d)
    q = torch.randn(n, H, maps, d, generator=gen, device="cuda") * 1.5
    k, v = (torch.randn(past + n, G, *w, generator=gen, device="cuda").to(torch.bfloat16) for w in ((maps, d), (dv,)))
    # from one stretch of keys to the next the scores rise, for some rows only: sums that were started have to be rescaled
    k[(past + n) // 2 :, :, :, 0] += 6
    q[::3, :, :, 0] = 12
    ref, got = _reference(q, k, v, past, window, keep, 0.4), _run(q, k, v, past, window, keep, 0.4)
    rows = ((got.double() - ref).square().sum(1) / ref.square().sum(1)).sqrt()
    assert rows.max().item() < 0.02 and ((got.double() - ref).norm() / ref.norm()).item() < 0.01, rows.topk(min(5, n))
    for _ in range(2):
        assert torch.equal(_run(q, k, v, past, window, keep, 0.4), got)


@pytest.mark.parametrize("maps,d,dv", [(1, 128, 128), (2, 64, 128), (1, 16, 80)])
@pytest.mark.parametrize("H,G,n", [(2, 2, 300), (12, 3, 513), (40, 8, 640), (150, 150, 500)])
@pytest.mark.parametrize("scale", [1.0, -1.0, 0.0])
def test_keys_of_a_tile_shared_out_over_one_to_eight_ctas(maps, d, dv, H, G, n, scale):
    """Few tiles to many: eight, four, two shares of a tile's keys and one; some shares hold no key at all.  A negative and a zero factor of the
    scores; result rows of odd length.  Bound as above."""
    gen = torch.Generator(device="cuda").manual_seed(H + n + d)
    q = torch.randn(n, H, maps, d, generator=gen, device="cuda") * 1.5
    k, v = (torch.randn(n, G, *w, generator=gen, device="cuda").to(torch.bfloat16) for w in ((maps, d), (dv,)))
    L, p = _lib.lm(), lambda t: t.data_ptr()
    tile = ctypes.c_int()
    _lib.lm_check(L.ao_lm_window_attention_prompt_plan(BF16, maps, H, G, d, dv, ctypes.byref(tile)), "plan")
    i32 = lambda t: t.to(torch.int32).cuda()  # noqa: E731
    first, back = torch.arange(0, n, tile.value), torch.arange(n)
    slot, pos, tf, tc = i32(back * 0), i32(back), i32(first), i32((n - first).clamp(max=tile.value))
    rk, rv = torch.zeros(1, 4096, G * maps * d, dtype=torch.bfloat16, device="cuda"), torch.zeros(1, 4096, G * dv, dtype=torch.bfloat16, device="cuda")
    for extra in (0, 1):
        out = torch.full((n, H * dv + extra), 9.0, dtype=torch.bfloat16, device="cuda")
        _lib.lm_check(L.ao_lm_window_attention_prompt(
            p(q), p(k), p(v), p(rk), p(rv), None, None, 4096, 0, BF16, p(slot), p(pos), p(pos), p(tf), p(tc), tf.numel(), maps, H, G, d, dv, 4096, 0,
            scale * d ** -0.5, 0.4, int(maps == 2), 1e-6, 1.0, p(out), H * dv + extra, torch.cuda.current_stream().cuda_stream), "prompt")
        torch.cuda.synchronize()
        ref = _reference(q * scale, k, v, 0, 4096, 0, 0.4)
        assert ((out[:, : H * dv].double() - ref).norm() / ref.norm()).item() < 0.01
        assert extra == 0 or bool((out[:, -1] == 9.0).all())


@pytest.mark.parametrize("maps,d,dv,H,G", [(1, 128, 128, 4, 2), (2, 64, 128, 2, 2), (1, 16, 80, 40, 2)])
@pytest.mark.parametrize("n,past,window,keep", [(300, 0, 4096, 0), (520, 40, 100, 3), (700, 0, 512, 0)])
def test_values_that_are_not_finite_reach_only_rows_that_see_them(maps, d, dv, H, G, n, past, window, keep):
    """An infinity or NaN among the values of a key makes the results of the rows that see it, in its column, not finite (with two maps their norm
    spreads it over the row) and no others: a hidden key has no part in a row, whatever the tile that both are in.  Bound as above."""
    gen = torch.Generator(device="cuda").manual_seed(n + d)
    q = torch.randn(n, H, maps, d, generator=gen, device="cuda") * 1.5
    k, v = (torch.randn(past + n, G, *w, generator=gen, device="cuda").to(torch.bfloat16) for w in ((maps, d), (dv,)))
    ref = _reference(q, k, v, past, window, keep, 0.4).view(n, H, dv)
    i, j = torch.arange(past, past + n, device="cuda")[:, None], torch.arange(past + n, device="cuda")[None, :]
    seen = ~((j > i) | ((i - j >= window) & (j >= keep)))
    for at, g, c, value in ((past + n - 1, 0, 3, torch.inf), (past + n - 37, G - 1, dv - 1, torch.nan), (past + 130, 0, 17, -torch.inf), (past + 130, 0, 18, torch.inf),
                            (past + 63, 0, 0, torch.nan), (past + 64, G - 1, 9, -torch.inf), (past + 1, 0, 40, torch.inf), (1, 0, 41, torch.inf)):
        v[at, g, c] = value
    bad = torch.einsum("ij,jgc->igc", seen.double(), (~v.isfinite()).double()) > 0     # [n][G][dv]
    bad = bad.repeat_interleave(H // G, 1)
    if maps == 2:
        bad = bad.any(-1, keepdim=True).expand(n, H, dv)
    assert bad.any() and not bad.all(-1).all()
    got = _run(q, k, v, past, window, keep, 0.4).double().view(n, H, dv)
    spread = got.isfinite() & bad      # (a norm over an infinity makes the row's other columns zero, not NaN)
    assert not spread.any() if maps == 1 else bool((got[spread] == 0).all())
    assert got[~bad].isfinite().all()
    if maps == 1:                      # (a value set to something finite would have been part of the others' norm)
        # columns are independent of one another: those without a bad value are what they were
        err = torch.where(bad, 0.0, got.nan_to_num() - ref)
        assert (err.norm() / ref.norm()).item() < 0.01
    else:
        rows = ~bad.any(-1)
        assert ((got[rows] - ref[rows]).norm() / ref[rows].norm()).item() < 0.01


@pytest.mark.parametrize("maps,d,H,G,n", [(1, 128, 16, 4, 600), (1, 128, 4, 2, 130), (2, 64, 8, 4, 300)])
@pytest.mark.parametrize("captured", [False, True])
def test_inputs_of_the_kernel_in_front_and_calls_behind_each_other(maps, d, H, G, n, captured):
    """The launch may begin while the kernel in front ends.  That kernel writes the queries, keys and values here, and takes its time; calls follow
    one another into buffers that the next copy reads: the same bits as calls with everything at rest between them."""
    dv, L, p = 128, _lib.lm(), lambda t: t.data_ptr()
    gen = torch.Generator(device="cuda").manual_seed(n)
    tile = ctypes.c_int()
    _lib.lm_check(L.ao_lm_window_attention_prompt_plan(BF16, maps, H, G, d, dv, ctypes.byref(tile)), "plan")
    i32 = lambda t: t.to(torch.int32).cuda()  # noqa: E731
    first, back = torch.arange(0, n, tile.value), torch.arange(n)
    slot, pos, tf, tc = i32(back * 0), i32(back), i32(first), i32((n - first).clamp(max=tile.value))
    rk, rv = torch.zeros(1, 1024, G * maps * d, dtype=torch.bfloat16, device="cuda"), torch.zeros(1, 1024, G * dv, dtype=torch.bfloat16, device="cuda")
    sets = [(torch.randn(n, H, maps, d, generator=gen, device="cuda"), *(torch.randn(n, G, *w, generator=gen, device="cuda").to(torch.bfloat16)
                                                                        for w in ((maps, d), (dv,)))) for _ in range(3)]
    q, k, v = (torch.empty_like(t) for t in sets[0])
    out, big = torch.empty(n, H * dv, dtype=torch.bfloat16, device="cuda"), torch.ones(1 << 24, device="cuda")

    def call(one, result):
        q.copy_(one[0]), k.copy_(one[1])
        big.mul_(1.0)
        v.copy_(one[2])
        _lib.lm_check(L.ao_lm_window_attention_prompt(
            p(q), p(k), p(v), p(rk), p(rv), None, None, 1024, 0, BF16, p(slot), p(pos), p(pos), p(tf), p(tc), tf.numel(), maps, H, G, d, dv, 1024, 0,
            d ** -0.5, 0.4, int(maps == 2), 1e-6, 1.0, p(out), H * dv, torch.cuda.current_stream().cuda_stream), "prompt")
        result.copy_(out)

    want = [torch.empty_like(out) for _ in sets]
    for one, result in zip(sets, want):
        call(one, result)
        torch.cuda.synchronize()
    got = [torch.zeros_like(out) for _ in range(6)]
    graph = torch.cuda.CUDAGraph() if captured else None
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=stream) if captured else torch.cuda.stream(stream):
        for i, result in enumerate(got):
            call(sets[i % 3], result)
    with torch.cuda.stream(stream):
        if captured:
            graph.replay()
    stream.synchronize()
    for i, result in enumerate(got):
        assert torch.equal(result, want[i % 3]), i
