"""Which calls of the linears may go past the dispatcher (ops.runs_eagerly): only those for which it would have done nothing.  On the CPU;
the shape of every answer, or the error, is that of the registered op."""
import weakref

import pytest
import torch
from torch.overrides import BaseTorchFunctionMode

from torchao_fork_b200 import ops

T = torch.ops.torchao


def _args(bits, device):
    x = torch.empty(3, 64, device=device, dtype=torch.bfloat16)
    if bits == 4:
        return x, torch.empty(8, 1, 32, 4, dtype=torch.int32, device=device), 64, torch.empty(8, 1, 16, 2, dtype=torch.bfloat16, device=device), 100
    return x, torch.empty(8, 1, 1024, dtype=torch.uint8, device=device), torch.empty(100, dtype=torch.bfloat16, device=device)


CALLS = [(4, ops.int4_weight_only_mm, T.b200_int4_weight_only_mm), (8, ops.int8_weight_only_mm, T.b200_int8_weight_only_mm)]


@pytest.mark.parametrize("bits,call,op", CALLS)
def test_other_devices_go_through_the_dispatcher(bits, call, op):
    args = _args(bits, "meta")          # shapes of a model that has no memory yet
    y = call(*args)
    assert y.device.type == "meta" and y.shape == op(*args).shape == (3, 100)
    with pytest.raises(NotImplementedError, match="CPU"):   # (also what a caller may catch: an op that is not there)
        call(*_args(bits, "cpu"))


def test_only_plain_cuda_memory_is_eager():
    with torch.inference_mode():
        inside = torch.ones(2)
    assert tuple(torch._C._dispatch_keys(t).raw_repr() for t in (inside, torch.ones(2))) == ops._plain_keys("CPU")
    for t in (torch.ones(2), torch.ones(2, device="meta"), torch._neg_view(torch.ones(2)), torch._efficientzerotensor(2),
              torch._to_functional_tensor(torch.ones(2))):
        assert not ops.runs_eagerly(t)


def test_a_tracer_stops_at_the_first_question():
    f = lambda x: x + 1 if ops.runs_eagerly(x) else x * 2  # noqa: E731
    x = torch.randn(3)
    assert torch.equal(torch.compile(f, fullgraph=True, backend="eager")(x), x * 2)


def test_a_function_mode_keeps_its_say(monkeypatch):
    monkeypatch.setattr(ops, "_PLAIN_KEYS", ops._plain_keys("CPU"))
    x = torch.ones(2)
    assert ops.runs_eagerly(x)
    with BaseTorchFunctionMode():
        assert not ops.runs_eagerly(x)


@pytest.mark.gpu
@pytest.mark.parametrize("bits,name", [(4, "torchao::b200_int4_weight_only_mm"), (8, "torchao::b200_int8_weight_only_mm")])
def test_a_profile_names_the_op(bits, name):
    import torchao_fork_b200 as ao
    lin = torch.nn.Linear(128, 128, bias=False, device="cuda", dtype=torch.bfloat16).requires_grad_(False)
    ao.quantize_(lin, ao.Int4WeightOnlyConfig(group_size=64) if bits == 4 else ao.Int8WeightOnlyConfig())
    x = torch.randn(2, 128, device="cuda").bfloat16()
    y = lin(x)
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        assert torch.equal(lin(x), y)
    assert name in {e.name for e in prof.events()}


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 5])
def test_the_blocks_of_the_llama_model_trace_in_one_graph(rows):
    import torchao_fork_b200 as ao
    from torchao_fork_b200._models.llama import ModelArgs
    from torchao_fork_b200._models.llama.model import FeedForward, RMSNorm, apply_rotary_emb
    cfg = ModelArgs.from_name("tiny-llama3")
    torch.manual_seed(0)
    norm, ff = (m.to("cuda", torch.bfloat16).requires_grad_(False) for m in (RMSNorm(cfg.dim), FeedForward(cfg)))
    ao.quantize_(ff, ao.Int4WeightOnlyConfig(group_size=64))
    x = torch.randn(1, rows, cfg.dim, device="cuda").bfloat16()
    q, freqs = torch.randn(1, rows, 4, 128, device="cuda").bfloat16(), torch.randn(rows, 64, 2, device="cuda").bfloat16()
    both = lambda x, q, freqs: (ff(norm(x)), apply_rotary_emb(q, freqs))  # noqa: E731
    torch._dynamo.reset()
    traced, rotated = torch.compile(both, fullgraph=True, backend="aot_eager")(x, q, freqs)
    plain, turned = both(x, q, freqs)
    # the norm adds up in another order: one rounding of its result, 2^-8, and of what follows
    assert torch.equal(rotated, turned) and (traced - plain).float().norm() < 2.0 ** -7 * plain.float().norm()


def test_a_workspace_in_a_graph_is_not_given_back(monkeypatch):
    monkeypatch.setattr(ops, "_WORKSPACES", {})
    monkeypatch.setattr(ops, "_CAPTURED", {})
    cpu, capturing = torch.device("cpu"), [False]
    monkeypatch.setattr(ops, "_capturing", lambda: capturing[0])
    refs = []
    for inside in (False, True):
        capturing[0] = inside
        small = ops._workspace(cpu, 64, "int8", stream=int(inside))
        refs.append(weakref.ref(small))
        capturing[0] = False
        large = ops._workspace(cpu, 128, "int8", stream=int(inside))   # takes the small one's place
        assert large is ops._workspace(cpu, 64, "int8", stream=int(inside)) and large is not small
        del small, large
    assert refs[0]() is None and refs[1]() is not None


@pytest.mark.gpu
def test_a_graph_outlives_the_growth_of_its_workspace():
    # int8, 12 rows by the GEMM, captured on the stream that a larger call uses afterwards
    gen = torch.Generator(device="cuda").manual_seed(0)
    w, x = (torch.randn(r, 8192, generator=gen, device="cuda").bfloat16() for r in (16384, 12))
    q, scale = T.b200_int8_quantize(w, 1e-6, True)
    packed = T.b200_int8_pack(q)
    want, s = T.b200_int8_weight_only_mm(x, packed, scale), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        T.b200_int8_weight_only_mm(x, packed, scale)
        s.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            y = T.b200_int8_weight_only_mm(x, packed, scale)
        T.b200_int8_weight_only_mm(x.repeat(100, 1), packed, scale)
        others = [torch.full((1 << 18,), 3.0, device="cuda") for _ in range(64)]   # what would be allocated in its place
        s.synchronize()
        g.replay()
        s.synchronize()
    assert torch.equal(y, want) and all((t == 3.0).all() for t in others)


@pytest.mark.gpu
def test_plain_cuda_tensors_are_eager_and_wrapped_ones_are_not():
    x = torch.ones(2, device="cuda")
    with torch.inference_mode():
        inside = torch.ones(2, device="cuda")
    assert ops.runs_eagerly(x) and ops.runs_eagerly(x, inside, x.view(2)) and ops.runs_eagerly(inside)
    for t in (torch._neg_view(x), torch._efficientzerotensor(2, device="cuda"), torch._to_functional_tensor(x), x.cpu()):
        assert not ops.runs_eagerly(t) and not ops.runs_eagerly(x, t)


@pytest.mark.gpu
def test_weights_that_are_not_on_the_device_are_refused():
    # the op is registered for CUDA, which the activations alone decide: a host address must not get as far as a launch
    x, packed, group, sz, n = _args(4, "cuda")
    for p, s in ((packed.cpu(), sz), (packed, sz.cpu())):
        with pytest.raises(RuntimeError, match="CUDA"):
            T.b200_int4_weight_only_mm(x, p, group, s, n)
    x, packed, scale = _args(8, "cuda")
    for p, s in ((packed.cpu(), scale), (packed, scale.cpu())):
        with pytest.raises(RuntimeError, match="CUDA"):
            T.b200_int8_weight_only_mm(x, p, s)


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 3, 17, 64])
@pytest.mark.parametrize("bits,call,op", CALLS)
def test_the_native_host_side_gives_what_the_python_one_gives(bits, call, op, rows, monkeypatch):
    host = ops._host()
    assert host is not None, "python -m torchao_fork_b200.build host"
    gen = torch.Generator(device="cuda").manual_seed(rows)
    w = torch.randn(320, 512, generator=gen, device="cuda").bfloat16()
    if bits == 4:
        packed, sz = T.b200_int4_quantize_pack(w, 64, 1e-6, True)
        rest = (packed, 64, sz, 320)
    else:
        q, scale = T.b200_int8_quantize(w, 1e-6, True)
        rest = (T.b200_int8_pack(q), scale)
    native, scratch = (host.int4_mm, ops._int4_scratch) if bits == 4 else (host.int8_mm, ops._int8_scratch)
    big = torch.randn(rows + 1, 1032, generator=gen, device="cuda").bfloat16()
    stream = torch.cuda.Stream()
    for x, taken in ((big[:rows, :512], True), (big[1:, 8:520], True), (big[:rows, :504], True), (big[:rows, 1:513], False), (big[:rows, :511], False),
                     (big[:rows, :1024:2], False), (big[:0, :512], False), (big[:rows, :512].contiguous(), True)):
        y = native(x, *rest, scratch)
        assert (type(y) is torch.Tensor) == taken and (taken or y is None)
        if not taken and x.shape == (1, 512):   # (one row off 16 bytes counts as contiguous and is refused behind Python too)
            continue
        want = op(x, *rest)
        assert torch.equal(call(x, *rest), want) and (not taken or torch.equal(y, want))
        with torch.cuda.stream(stream), torch.inference_mode():
            stream.wait_stream(torch.cuda.default_stream())
            inside = call(x, *rest)
            assert inside.is_inference() and torch.equal(inside, want)
        torch.cuda.default_stream().wait_stream(stream)
    for x in (big[:rows, :512].float(), big[:rows, :512].cpu(), big[0, :512]):
        assert native(x, *rest, scratch) is None
    wrong = big[:rows, :520]
    assert native(wrong, *rest, scratch) is None
    with pytest.raises(RuntimeError):
        call(wrong, *rest)
    monkeypatch.setattr(ops, "_host", lambda: None)
    assert torch.equal(call(big[:rows, :512], *rest), op(big[:rows, :512], *rest))


@pytest.mark.gpu
@pytest.mark.parametrize("recipe", ["int4", "hqq", "int8"])
def test_a_quantized_weight_is_a_parameter_like_any_other(recipe):
    import copy

    import torchao_fork_b200 as ao
    config = ao.Int8WeightOnlyConfig() if recipe == "int8" else ao.Int4WeightOnlyConfig(group_size=64, use_hqq=recipe == "hqq")
    lin = torch.nn.Linear(256, 128, bias=False, device="cuda", dtype=torch.bfloat16)
    x, w = torch.randn(4, 256, device="cuda").bfloat16(), lin.weight.detach().clone()
    ao.quantize_(lin, config)
    p = lin.weight
    assert isinstance(p, torch.nn.Parameter) and not p.requires_grad and p.is_leaf and [n for n, _ in lin.named_parameters()] == ["weight"]
    y = lin(x)
    for other in (copy.deepcopy(lin), torch.nn.Linear(256, 128, bias=False, device="meta", dtype=torch.bfloat16)):
        if other.weight.is_meta:
            other.load_state_dict(lin.state_dict(), assign=True)
        assert isinstance(other.weight, torch.nn.Parameter) and type(other.weight) is type(p) and torch.equal(other(x), y)
    # the dispatcher's way, as under a profile, makes the same
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CPU]) as prof:
        again = torch.nn.Linear(256, 128, bias=False, device="cuda", dtype=torch.bfloat16)
        again.weight = torch.nn.Parameter(w, requires_grad=False)
        ao.quantize_(again, config)
    assert any("b200_int" in e.name for e in prof.events())
    for n in p.tensor_impl.__tensor_flatten__()[0]:
        assert torch.equal(getattr(p.tensor_impl, n), getattr(again.weight.tensor_impl, n))
    # a weight that the config does not fit stays what it was, a parameter of its own
    odd = torch.nn.Linear(250, 128, bias=False, device="cuda", dtype=torch.bfloat16)
    if recipe == "int4":
        ao.quantize_(odd, config)
        assert type(odd.weight) is torch.nn.Parameter


@pytest.mark.parametrize("what", ["missing", "garbage", "of another version", "older than its binding"])
def test_a_host_module_that_does_not_load_counts_as_not_built(what, monkeypatch, tmp_path):
    import os

    from torchao_fork_b200 import _lib, build
    if not os.path.exists(_lib.LIB_PATH) or not os.path.exists(build.host_path()):
        pytest.skip("python -m torchao_fork_b200.build")
    path = tmp_path / "ao_b200_host.so"
    if what == "garbage":
        path.write_bytes(b"\x7fELF" + b"\0" * 200)
    elif what != "missing":
        path = build.host_path()
        monkeypatch.setattr(_lib, "lib", lambda real=_lib.lib(): _Like(real, 4 if what == "of another version" else "older"))
    monkeypatch.setattr(build, "host_path", lambda: str(path))
    with pytest.warns(RuntimeWarning, match="in Python"):
        assert _lib.host() is None


class _Like:
    """The library, but for its version"""
    def __init__(self, real, version):
        self.real, self.ao_b200_abi_version = real, lambda: version

    def __getattr__(self, name):
        return getattr(self.real, name)


def test_the_host_module_of_this_build_is_bound():
    import os

    from torchao_fork_b200 import _lib, build
    if not os.path.exists(_lib.LIB_PATH) or not os.path.exists(build.host_path()):
        pytest.skip("python -m torchao_fork_b200.build")
    assert callable(_lib.host().int4_mm) and callable(_lib.host().int8_mm)


def test_a_build_without_a_cpp_compiler_has_its_libraries(monkeypatch, capsys):
    from torchao_fork_b200 import build
    done = []

    def host(verbose, force):
        done.append("host")
        raise FileNotFoundError("g++")
    monkeypatch.setattr(build, "_build_locked", lambda verbose, force, target: done.append(target) or build.TARGETS[target][1])
    monkeypatch.setattr(build, "_build_host", host)
    assert build.build(target="all") == build.LIB and set(done) == {"lm", "core", "host"}
    assert "not built" in capsys.readouterr().err
    with pytest.raises(FileNotFoundError):     # asked for by name it has to be there
        build.build(target="host")
