"""Int4WeightOnlyConfig(use_hqq=True) on the GPU (csrc/hqq.cu) against the reference's golden
vectors (tests/golden/hqq_*.npz, produced by _choose_qparams_and_quantize_affine_hqq on CPU) and the numpy oracle.
The solver iterates in fp32 with a mean over each group, so agreement is stated as a tolerance: scale bit-exact (no
iteration in it), q identical on >= 99.9 % of the weights and never off by more than one step, zero within a bf16 ulp
(or 1/128 of the scale) on >= 99 % of the groups."""
import glob
import os

import numpy as np
import pytest
import torch

import ao_oracle as o
import torchao_fork_b200 as ao  # noqa: F401
from conftest import GOLDEN
from test_oracle_golden import hqq_agreement
from torchao_fork_b200.quantization import Int4WeightOnlyConfig, quantize_

pytestmark = pytest.mark.gpu
T = torch.ops.torchao
HQQ = sorted(glob.glob(os.path.join(GOLDEN, "hqq_*.npz")))


def bf16_from_bits(b):
    return torch.from_numpy(b.astype(np.int16)).view(torch.bfloat16).cuda()


def f32_of(t):
    return t.float().cpu().numpy()


@pytest.mark.parametrize("path", HQQ, ids=os.path.basename)
def test_hqq_matches_reference_golden(path):
    g = np.load(path)
    q, s, z = T.b200_int4_hqq_quantize(bf16_from_bits(g["w"]), int(g["group_size"]))
    same_q, max_dq, scale_exact, zero_ok = hqq_agreement(q.cpu().numpy().astype(np.uint8), f32_of(s), f32_of(z), g)
    assert scale_exact
    assert same_q >= 0.999 and max_dq <= 1
    assert zero_ok >= 0.99


@pytest.mark.parametrize("shape,gs", [((256, 1024), 128), ((96, 512), 32), ((64, 2048), 256), ((130, 448), 64)])
def test_hqq_matches_oracle_on_seeded_weights(shape, gs):
    torch.manual_seed(shape[0] + gs)
    w = (torch.randn(*shape) * torch.exp(0.5 * torch.randn(*shape))).to(torch.bfloat16)
    q, s, z = T.b200_int4_hqq_quantize(w.cuda(), gs)
    oq, os_, oz = o.hqq_quantize(w.float().numpy(), gs)
    ref = {"q": oq, "scale": o.to_bits(os_), "zero": o.to_bits(oz)}
    same_q, max_dq, scale_exact, zero_ok = hqq_agreement(q.cpu().numpy().astype(np.uint8), f32_of(s), f32_of(z), ref)
    assert scale_exact and same_q >= 0.999 and max_dq <= 1 and zero_ok >= 0.99


def test_quantize_with_use_hqq_runs_the_same_kernels_and_lowers_the_lp_error():
    torch.manual_seed(5)
    lin = torch.nn.Linear(1024, 384, bias=False, dtype=torch.bfloat16, device="cuda")
    with torch.no_grad():
        lin.weight.mul_(torch.exp(torch.randn_like(lin.weight.float())).to(torch.bfloat16))  # heavy tails
    w = lin.weight.detach().clone()
    import copy
    hqq, mm = copy.deepcopy(lin), copy.deepcopy(lin)
    quantize_(hqq, Int4WeightOnlyConfig(group_size=64, use_hqq=True))
    quantize_(mm, Int4WeightOnlyConfig(group_size=64))
    e_hqq = (w.float() - hqq.weight.dequantize().float()).abs().pow(0.7).mean().item()
    e_mm = (w.float() - mm.weight.dequantize().float()).abs().pow(0.7).mean().item()
    assert e_hqq < e_mm
    # the quantized tensor matches the op's plain outputs and goes through the same linear kernels
    q, s, z = T.b200_int4_hqq_quantize(w, 64)
    assert torch.equal(T.b200_int4_unpack(hqq.weight.tensor_impl.packed_weight)[:384, :1024], q)
    x = torch.randn(3, 1024, dtype=torch.bfloat16, device="cuda")
    y = hqq(x)
    ref = x.float() @ hqq.weight.dequantize().float().t()
    assert (10 * torch.log10(ref.pow(2).mean() / (ref - y.float()).pow(2).mean())).item() >= 40.0


def test_hqq_constant_and_zero_groups():
    w = torch.zeros(16, 256, dtype=torch.bfloat16, device="cuda")
    w[1] = 3.0
    w[2, :128] = -1.5
    q, s, z = T.b200_int4_hqq_quantize(w, 128)
    oq, os_, oz = o.hqq_quantize(w.float().cpu().numpy(), 128)
    assert np.array_equal(q.cpu().numpy().astype(np.uint8), oq)
    assert np.array_equal(o.to_bits(f32_of(s)), o.to_bits(os_)) and np.array_equal(o.to_bits(f32_of(z)), o.to_bits(oz))
    deq = (q.float() - 8) * s.float().repeat_interleave(128, 1) + z.float().repeat_interleave(128, 1)
    assert torch.allclose(deq, w.float(), atol=1e-2)


@pytest.mark.parametrize("shape,gs", [((256, 512), 64), ((512, 1024), 128), ((64, 256), 32)])
def test_hqq_device_side_early_stop_equals_the_host_driven_loop(shape, gs):
    """ao_b200_hqq_solve (the early stop of quant_primitives.py:1964-1972 decided by a one-block kernel, no host round
    trip) against the same iterations driven from the host with ao_b200_hqq_step: same number of iterations, bit-identical
    zero."""
    from torchao_fork_b200 import _lib
    from torchao_fork_b200.ops import HQQ_BETA, HQQ_ITERS, HQQ_KAPPA, HQQ_LP_NORM
    torch.manual_seed(3)
    w = (torch.randn(*shape, device="cuda") * torch.rand(shape[0], 1, device="cuda")).to(torch.bfloat16).contiguous()
    w[0, :gs] = 0.25                                   # a constant group
    L = _lib.lib()
    n_groups = shape[0] * shape[1] // gs
    st = torch.cuda.current_stream().cuda_stream
    err = torch.empty(int(L.ao_b200_hqq_blocks(n_groups)), dtype=torch.float32, device="cuda")

    def init():
        scale = torch.empty(n_groups, dtype=torch.float32, device="cuda")
        zero = torch.empty_like(scale)
        _lib.check(L.ao_b200_hqq_init(w.data_ptr(), n_groups, gs, scale.data_ptr(), zero.data_ptr(), st), "init")
        return scale, zero

    scale_h, zero_h = init()
    beta, best, ran = HQQ_BETA, 1e4, 0
    for _ in range(HQQ_ITERS):
        _lib.check(L.ao_b200_hqq_step(w.data_ptr(), n_groups, gs, scale_h.data_ptr(), zero_h.data_ptr(), beta, HQQ_LP_NORM,
                                      err.data_ptr(), st), "step")
        beta *= HQQ_KAPPA
        ran += 1
        current = float(err.sum(dtype=torch.float64)) / w.numel()
        if current < best:
            best = current
        else:
            break
    scale_d, zero_d = init()
    state = torch.empty(2, dtype=torch.float64, device="cuda")
    _lib.check(L.ao_b200_hqq_solve(w.data_ptr(), n_groups, gs, scale_d.data_ptr(), zero_d.data_ptr(), HQQ_BETA, HQQ_KAPPA,
                                   HQQ_LP_NORM, HQQ_ITERS, err.data_ptr(), state.data_ptr(), st), "solve")
    torch.cuda.synchronize()
    flags = state[1:].view(torch.int32).cpu()
    assert int(flags[1]) == ran, (int(flags[1]), ran)
    assert int(flags[0]) == (1 if ran < HQQ_ITERS else int(flags[0]))
    assert torch.equal(zero_d, zero_h) and torch.equal(scale_d, scale_h)
    assert abs(float(state[0]) - best) <= 1e-12 * max(best, 1.0)


@pytest.mark.parametrize("shape,gs", [((4096, 512), 64), ((33, 256), 32), ((130, 448), 64), ((40, 768), 256), ((1, 128), 128)])
@pytest.mark.parametrize("spread", [0.02, 1.0, 30.0])
def test_hqq_search_equals_the_iterations_one_by_one(shape, gs, spread):
    """ao_b200_hqq_search (a group's iterations in registers, the shrinkage evaluated only where it can be positive, Markstein's
    division) against init / solve / finalize, bit for bit: it adds in the same order.  Spreads from where the shrinkage is always
    zero to where it seldom is.  The packed form is the plain one packed, padding zero."""
    from torchao_fork_b200 import _lib
    from torchao_fork_b200 import ops as aops
    torch.manual_seed(7)
    n, k = shape
    w = (spread * torch.randn(*shape, device="cuda") * torch.exp(0.3 * torch.randn(n, 1, device="cuda"))).to(torch.bfloat16)
    w[0, :gs] = 0.25
    L, st, n_groups = _lib.lib(), torch.cuda.current_stream().cuda_stream, n * k // gs
    scale = torch.empty(n_groups, dtype=torch.float32, device="cuda")
    zero, err = torch.empty_like(scale), torch.empty(int(L.ao_b200_hqq_blocks(n_groups)), dtype=torch.float32, device="cuda")
    state = torch.empty(2, dtype=torch.float64, device="cuda")
    q0 = torch.empty(n, k, dtype=torch.int32, device="cuda")
    s0 = torch.empty(n, k // gs, dtype=torch.bfloat16, device="cuda")
    z0 = torch.empty_like(s0)
    _lib.check(L.ao_b200_hqq_init(w.data_ptr(), n_groups, gs, scale.data_ptr(), zero.data_ptr(), st), "init")
    _lib.check(L.ao_b200_hqq_solve(w.data_ptr(), n_groups, gs, scale.data_ptr(), zero.data_ptr(), aops.HQQ_BETA, aops.HQQ_KAPPA, aops.HQQ_LP_NORM,
                                   aops.HQQ_ITERS, err.data_ptr(), state.data_ptr(), st), "solve")
    _lib.check(L.ao_b200_hqq_finalize(w.data_ptr(), n_groups, gs, scale.data_ptr(), zero.data_ptr(), q0.data_ptr(), s0.data_ptr(), z0.data_ptr(), st),
               "finalize")
    q, s, z = T.b200_int4_hqq_quantize(w, gs)
    assert torch.equal(s, s0) and torch.equal(z, z0) and torch.equal(q, q0)
    packed, sz = T.b200_int4_hqq_quantize_pack(w, gs)
    pad = torch.zeros(packed.shape[0] * 16, packed.shape[1] * 64, dtype=torch.int32, device="cuda")
    pad[:n, :k] = q
    assert torch.equal(T.b200_int4_unpack(packed), pad)
    ps, pz = aops.unpack_scales_and_zeros_b200(sz)
    assert torch.equal(ps[:n, : k // gs], s) and torch.equal(pz[:n, : k // gs], z)
    assert not ps[n:].any() and not pz[n:].any() and not ps[:, k // gs :].any()


@pytest.mark.gpu
@pytest.mark.parametrize("gs,seed", [(64, 34), (32, 35), (128, 36), (256, 37)])
def test_packed_words_of_many_weights_equal_the_plain_result(gs, seed):
    """Enough weights that some land within a rounding error of a half: product and sum have to be rounded one after the other in both."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    w = (torch.randn(4096, 4096, device="cuda", generator=g) * 0.05).to(torch.bfloat16)
    packed, _ = T.b200_int4_hqq_quantize_pack(w, gs)
    q, _, _ = T.b200_int4_hqq_quantize(w, gs)
    assert torch.equal(T.b200_int4_unpack(packed)[:4096, :4096], q)


@pytest.mark.gpu
@pytest.mark.parametrize("shape,gs,spread", [((4096, 4096), 64, 0.05), ((1024, 4096), 32, 0.05), ((1024, 4096), 128, 1.0), ((1024, 4096), 256, 0.02),
                                             ((2900, 4096), 32, 30.0), ((2900, 4096), 256, 1.0)])   # (the last two: dealt in pieces, several to a block)
def test_zero_points_of_the_search_equal_those_of_the_steps_in_32_bits(shape, gs, spread):
    """ao_b200_hqq_search against init / solve, the fp32 zero points as they are left in the workspace ([means 64 x 8 bytes][errors 10 x 8 bytes per
    8192 weights][scale][zero points of the last ten iterations]), bit for bit: a product and a sum rounded as one would show in their last bits."""
    from torchao_fork_b200 import _lib
    from torchao_fork_b200 import ops as aops
    g = torch.Generator(device="cuda").manual_seed(gs)
    n, k = shape
    w = (spread * torch.randn(n, k, device="cuda", generator=g)).to(torch.bfloat16)
    L, st, n_groups = _lib.lib(), torch.cuda.current_stream().cuda_stream, n * k // gs
    scale = torch.empty(n_groups, dtype=torch.float32, device="cuda")
    zero, err = torch.empty_like(scale), torch.empty(int(L.ao_b200_hqq_blocks(n_groups)), dtype=torch.float32, device="cuda")
    state = torch.empty(2, dtype=torch.float64, device="cuda")
    args = (aops.HQQ_BETA, aops.HQQ_KAPPA, aops.HQQ_LP_NORM, aops.HQQ_ITERS)
    _lib.check(L.ao_b200_hqq_init(w.data_ptr(), n_groups, gs, scale.data_ptr(), zero.data_ptr(), st), "init")
    _lib.check(L.ao_b200_hqq_solve(w.data_ptr(), n_groups, gs, scale.data_ptr(), zero.data_ptr(), *args, err.data_ptr(), state.data_ptr(), st), "solve")
    ws = torch.empty(int(L.ao_b200_hqq_search_workspace_bytes(n_groups, gs)), dtype=torch.uint8, device="cuda")
    q = torch.empty(n, k, dtype=torch.int32, device="cuda")
    s, z = (torch.empty(n, k // gs, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    _lib.check(L.ao_b200_hqq_search(w.data_ptr(), n, k, gs, *args, ws.data_ptr(), ws.numel(), q.data_ptr(), s.data_ptr(), z.data_ptr(), 0, 0, None, None, st),
               "search")
    ran = int(state[1:].view(torch.int32)[1])
    at = (64 + 10 * (-(-n * k // 8192))) * 8
    own = ws[at : at + 4 * n_groups * 11].view(torch.float32)
    assert torch.equal(own[:n_groups], scale)
    last = (ran - 1) % 10
    assert torch.equal(own[n_groups * (1 + last) : n_groups * (2 + last)].view(torch.int32), zero.view(torch.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("gs", [32, 64, 128, 256])
@pytest.mark.parametrize("shape,iters,kappa", [((3, 512), 1, 1.01), ((37, 768), 9, 1.01), ((601, 2048), 11, 0.97), ((5000, 1024), 33, 1.05)])
def test_groups_at_rest_give_what_their_iterations_would(shape, iters, kappa, gs):
    """Groups that come to rest early, late and never (a spread of row scales from 0.01 to 10, constant groups, a NaN and an infinity), counts of iterations
    around those of a launch, thresholds that fall and that rise: the search's zero points are those of the steps, bit for bit (NaN where those are)."""
    from torchao_fork_b200 import _lib
    from torchao_fork_b200 import ops as aops
    g = torch.Generator(device="cuda").manual_seed(gs + iters)
    n, k = shape
    w = (10 ** (3 * torch.rand(n, 1, device="cuda", generator=g) - 2) * torch.randn(n, k, device="cuda", generator=g)).to(torch.bfloat16)
    w[0, :gs], w[1, :gs] = 0.25, 0.0
    L, st, n_groups = _lib.lib(), torch.cuda.current_stream().cuda_stream, n * k // gs
    args = (aops.HQQ_BETA, kappa, aops.HQQ_LP_NORM, iters)
    for odd in (False, True):
        if odd:
            w[2, 3], w[-1, -1] = float("nan"), float("inf")
        scale = torch.empty(n_groups, dtype=torch.float32, device="cuda")
        zero, err = torch.empty_like(scale), torch.empty(int(L.ao_b200_hqq_blocks(n_groups)), dtype=torch.float32, device="cuda")
        state = torch.empty(2, dtype=torch.float64, device="cuda")
        _lib.check(L.ao_b200_hqq_init(w.data_ptr(), n_groups, gs, scale.data_ptr(), zero.data_ptr(), st), "init")
        _lib.check(L.ao_b200_hqq_solve(w.data_ptr(), n_groups, gs, scale.data_ptr(), zero.data_ptr(), *args, err.data_ptr(), state.data_ptr(), st), "solve")
        ws = torch.empty(int(L.ao_b200_hqq_search_workspace_bytes(n_groups, gs)), dtype=torch.uint8, device="cuda").fill_(0x7F)
        q = torch.empty(n, k, dtype=torch.int32, device="cuda")
        s, z = (torch.empty(n, k // gs, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        _lib.check(L.ao_b200_hqq_search(w.data_ptr(), n, k, gs, *args, ws.data_ptr(), ws.numel(), q.data_ptr(), s.data_ptr(), z.data_ptr(), 0, 0, None, None,
                                        st), "search")
        ran = int(state[1:].view(torch.int32)[1])
        at = (64 + 10 * (-(-n * k // 8192))) * 8
        own = ws[at : at + 4 * n_groups * 11].view(torch.float32)
        last = (ran - 1) % 10
        got = own[n_groups * (1 + last) : n_groups * (2 + last)]
        same = (got.view(torch.int32) == zero.view(torch.int32)) | (got.isnan() & zero.isnan())
        assert bool(same.all()), int((~same).sum())
        assert bool(zero.isnan().any()) == odd


@pytest.mark.gpu
@pytest.mark.parametrize("gs", [32, 64, 128, 256])
@pytest.mark.parametrize("over", [-7, -1, 0, 1, 9])
def test_lists_that_end_inside_a_warp(gs, over):
    """A block's warps race for the last groups of its list, and a warp gets none, some or all of what its lanes could take; whether it fetches at all is one
    answer for all its lanes.  Groups that rest at once beside groups that never do, so that lanes come free one by one; several times over,
    as the race ends otherwise each time, and the numbers must not."""
    n_groups = 8192 // gs * 3 + over   # three blocks' worth, a little less, a little more
    g = torch.Generator(device="cuda").manual_seed(gs + over)
    w = torch.randn(n_groups, gs, device="cuda", generator=g) * (10 ** (3 * torch.rand(n_groups, 1, device="cuda", generator=g) - 2))
    w = w.to(torch.bfloat16)
    from torchao_fork_b200 import _lib
    from torchao_fork_b200 import ops as aops
    L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    scale = torch.empty(n_groups, dtype=torch.float32, device="cuda")
    zero, err = torch.empty_like(scale), torch.empty(int(L.ao_b200_hqq_blocks(n_groups)), dtype=torch.float32, device="cuda")
    state = torch.empty(2, dtype=torch.float64, device="cuda")
    q0 = torch.empty(n_groups, gs, dtype=torch.int32, device="cuda")
    s0, z0 = (torch.empty(n_groups, 1, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    _lib.check(L.ao_b200_hqq_init(w.data_ptr(), n_groups, gs, scale.data_ptr(), zero.data_ptr(), st), "init")
    _lib.check(L.ao_b200_hqq_solve(w.data_ptr(), n_groups, gs, scale.data_ptr(), zero.data_ptr(), aops.HQQ_BETA, aops.HQQ_KAPPA, aops.HQQ_LP_NORM,
                                   aops.HQQ_ITERS, err.data_ptr(), state.data_ptr(), st), "solve")
    _lib.check(L.ao_b200_hqq_finalize(w.data_ptr(), n_groups, gs, scale.data_ptr(), zero.data_ptr(), q0.data_ptr(), s0.data_ptr(), z0.data_ptr(), st),
               "finalize")
    for _ in range(5):
        q, s, z = T.b200_int4_hqq_quantize(w, gs)
        assert torch.equal(s, s0) and torch.equal(z, z0) and torch.equal(q, q0)
