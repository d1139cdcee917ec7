"""Decode GEMVs of 2 .. 16 rows at the lines between their stagings: rows in registers (up to 4, 8 or 16 of up to 512, 1024 or 2048 chunks of eight)
and the loops behind them; short rows, ragged numbers of chunks, a zero row and one of huge values.  Against float64 on the dequantized weight.

Bound: the activations are exact in fp16 but for values 2^-27 below a row's largest, sums are fp32, the normed activation is rounded to bf16 as the
reference rounds it (here too), the result once (int4) or twice (int8): 2^-9 each, 1 % per row holds both with a wide margin."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if not torch.cuda.is_available():
    pytest.skip("needs a CUDA device", allow_module_level=True)

from torchao_fork_b200 import _lib, ops  # noqa: E402

T = torch.ops.torchao


@pytest.mark.parametrize("bits,group", [(8, 0), (4, 32), (4, 64), (4, 128), (4, 256)])
@pytest.mark.parametrize("K", [512, 2048, 4096, 5120, 8192, 14336])
@pytest.mark.parametrize("normed", [False, True])
def test_every_staging(bits, group, K, normed):
    torch.manual_seed(K + bits)
    N, eps = 352, 1e-5
    w = (torch.randn(N, K, device="cuda") * 0.03).to(torch.bfloat16)
    L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    if bits == 4:
        packed, par = T.b200_int4_quantize_pack(w, group, 1e-6, True)
        s, z = (t[:N, : K // group].double().repeat_interleave(group, 1) for t in ops.unpack_scales_and_zeros_b200(par))
        dense = (T.b200_int4_unpack(packed)[:N, :K].double() - 8) * s + z
    else:
        q, par = T.b200_int8_quantize(w, 1e-6, True)
        packed, par, dense = T.b200_int8_pack(q), par.contiguous(), q.double() * par.double().reshape(-1, 1)
    nw = (1 + 0.3 * torch.randn(K, device="cuda")).to(torch.bfloat16)
    ws = torch.zeros(1 << 24, dtype=torch.uint8, device="cuda")
    for M in (2, 4, 5, 8, 9, 16):
        x = (torch.randn(M, K, device="cuda") * torch.exp(torch.randn(M, 1, device="cuda"))).to(torch.bfloat16)
        x[M // 2] = 0
        x[M - 1] *= 1e4
        y = torch.full((M, N), 7.0, dtype=torch.bfloat16, device="cuda")
        common = (x.data_ptr(), M, K, K, packed.data_ptr(), par.data_ptr(), packed.shape[0] * 16, packed.shape[1] * 64)
        tail = (y.data_ptr(), N, N, nw.data_ptr() if normed else None, eps, None, 0, 0)
        if bits == 4:
            rc = L.ao_b200_int4_gemv_fused(*common, group, *tail, ws.data_ptr(), ws.numel(), st)
        else:
            rc = L.ao_b200_int8_gemv_fused(*common, *tail, st)
        if rc == 4 and M * K > 8 * 4096:
            continue                       # activations that fit no staging are refused
        _lib.check(rc, "gemv_fused")
        xd = x.double()
        ref = ((x.float() * nw.float()).to(torch.bfloat16).double() * torch.rsqrt(xd.square().mean(1, keepdim=True) + eps) if normed else xd) @ dense.t()
        err = (y.double() - ref).norm(dim=1) / ref.norm(dim=1).clamp(min=1e-30)
        assert bool((y[M // 2] == 0).all())
        err[M // 2] = 0
        assert err.max().item() < 0.01, (M, err)


@pytest.mark.parametrize("bits,group", [(8, 0), (4, 32), (4, 128), (4, 256)])
@pytest.mark.parametrize("N,K", [(1184, 8192), (2400, 14336), (336, 28672), (4096, 13824), (160, 8448)])
def test_long_activations_shared_out_over_clusters(bits, group, N, K):
    """Products of 2 .. 9 rows whose k the CTAs of a cluster share (halves or quarters), with and without a residual, beside the shapes and row
    counts that are not shared; more and fewer strips than clusters, an out width that ends inside a strip.  Equal calls give equal bits.  Bound as above."""
    if bits == 4 and K % group:
        pytest.skip("group does not divide k")
    torch.manual_seed(N + K)
    n = N - 3                                # the last rows of the last strip are padding
    w = (torch.randn(N, K, device="cuda") * 0.03).to(torch.bfloat16)
    w[n:] = 0
    L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    if bits == 4:
        packed, par = T.b200_int4_quantize_pack(w, group, 1e-6, True)
        s, z = (t[:N, : K // group].double().repeat_interleave(group, 1) for t in ops.unpack_scales_and_zeros_b200(par))
        dense = (T.b200_int4_unpack(packed)[:N, :K].double() - 8) * s + z
    else:
        q, par = T.b200_int8_quantize(w, 1e-6, True)
        packed, par, dense = T.b200_int8_pack(q), par.contiguous(), q.double() * par.double().reshape(-1, 1)
    np_, kp = packed.shape[0] * 16, packed.shape[1] * 64
    for M in (2, 3, 5, 8, 9):
        x = (torch.randn(M, K, device="cuda") * torch.exp(torch.randn(M, 1, device="cuda"))).to(torch.bfloat16)
        ref = x.double() @ dense.t()[:, :n]
        res = torch.randn(M, n + 5, device="cuda").to(torch.bfloat16)
        for residual in (False, True):
            if residual:
                need = int(L.ao_b200_mm_residual_workspace_bytes(M, np_, kp, group))
                if need == 0:
                    continue                 # not a shape of that call
            else:
                need = int((L.ao_b200_int4_mm_workspace_bytes if bits == 4 else L.ao_b200_int8_mm_workspace_bytes)(M, np_, kp))
            ys = []
            for _ in range(2):
                y = torch.full((M, n + 5), 7.0, dtype=torch.bfloat16, device="cuda")
                ws = torch.zeros(max(need, 16), dtype=torch.uint8, device="cuda")
                common = (x.data_ptr(), M, K, K, packed.data_ptr(), par.data_ptr(), np_, kp)
                if residual:
                    rc = L.ao_b200_mm_residual(*common, group, y.data_ptr(), n, n + 5, res.data_ptr(), n + 5, ws.data_ptr(), ws.numel(), st)
                elif bits == 4:
                    rc = L.ao_b200_int4_mm(*common, group, y.data_ptr(), n, n + 5, ws.data_ptr(), ws.numel(), st)
                else:
                    rc = L.ao_b200_int8_mm(*common, y.data_ptr(), n, n + 5, ws.data_ptr(), ws.numel(), st)
                _lib.check(rc, "mm")
                ys.append(y)
            assert torch.equal(ys[0], ys[1]) and bool((y[:, n:] == 7.0).all())
            got = y[:, :n].double() - (res[:, :n].double() if residual else 0)
            err = (got - ref).norm(dim=1) / (ref.norm(dim=1) + (res[:, :n].double().norm(dim=1) if residual else 0))
            assert err.max().item() < 0.01, (M, residual, err)
