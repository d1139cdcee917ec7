"""The row kernels of a prompt (norm, SiLU, rotation, cache rows, repeated heads) may be launched while the kernel in front ends.  That kernel writes
their input here, and what is behind reads their result and writes their input again: the same bits as with everything at rest between the calls."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from torchao_fork_b200._models.llama.model import KVCache, RMSNorm, apply_rotary_emb, kv_rows, repeat_heads, silu_mul  # noqa: E402

BF = dict(dtype=torch.bfloat16, device="cuda")


def _op(name, T, H, d, cache, freqs, norm, pos):
    if name == "norm":
        return lambda x: norm(x.view(T, H * d))
    if name == "silu":
        return lambda x: silu_mul(x, x)
    if name == "rotary":
        return lambda x: apply_rotary_emb(x, freqs)
    if name == "repeat":
        return lambda x: torch.cat([t.flatten() for t in repeat_heads(x.view(1, H, T, d), x.view(1, H, T, d), 2)])

    def rows(x):
        assert kv_rows(cache, pos, x, x, freqs)
        return torch.cat([cache.k_cache.flatten(), cache.v_cache.flatten()])
    return rows


@pytest.mark.parametrize("name", ["norm", "silu", "rotary", "repeat", "rows"])
@pytest.mark.parametrize("T,H,d", [(1, 2, 64), (700, 8, 128)])
@pytest.mark.parametrize("captured", [False, True])
def test_input_of_the_kernel_in_front(name, T, H, d, captured):
    gen = torch.Generator(device="cuda").manual_seed(T)
    sets = [torch.randn(1, T, H, d, generator=gen, device="cuda").to(torch.bfloat16) for _ in range(3)]
    freqs, pos = torch.randn(T, d // 2, 2, generator=gen, device="cuda").to(torch.bfloat16), torch.arange(T, device="cuda")
    cache, norm = KVCache(1, T, H, d, torch.bfloat16).cuda(), RMSNorm(H * d).to(**BF)
    x, big = torch.empty_like(sets[0]), torch.ones(1 << 24, device="cuda")
    op = _op(name, T, H, d, cache, freqs, norm, pos)

    def call(one):
        big.mul_(1.0)
        x.copy_(one)
        return op(x).clone()

    with torch.no_grad():
        want = []
        for one in sets:
            want.append(call(one))
            torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.graph(graph, stream=stream) if captured else torch.cuda.stream(stream):
            got = [call(sets[i % 3]) for i in range(9)]
        with torch.cuda.stream(stream):
            if captured:
                graph.replay()
        stream.synchronize()
    for i, result in enumerate(got):
        assert torch.equal(result, want[i % 3]), i
