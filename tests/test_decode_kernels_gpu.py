"""The kernels of a decode step -- streaming linear layers in FP8 and bf16 -- against float64."""
import pytest
import torch

from gpuk_b200 import cabi
from oracle import fp8_linear_oracle as fo

E4M3 = torch.float8_e4m3fn


def _ptr(t):
    return t.data_ptr()


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _status_ok():
    cabi.check(cabi.lib.gpuk_fp8_linear_status())


@pytest.mark.gpu
@pytest.mark.parametrize("k_split", [0, 1, 3, 8])
@pytest.mark.parametrize("m,n,k", [(1, 128, 8), (16, 256, 64), (17, 128, 72), (32, 384, 1000), (31, 1280, 4096), (9, 16384, 2048)])
def test_bf16_linear(m, n, k, k_split):
    """Tokens on both sides of the 16-column tile, k that ends inside a step (8, 72, 1000), fewer steps than parts, tiles below and above
    the number of SMs.  fp32 sums of exact products, one rounding: one bf16 step."""
    g = torch.Generator().manual_seed(m + n + k)
    x, w = torch.randn(m, k, generator=g).bfloat16(), torch.randn(n, k, generator=g).bfloat16()
    dx, dw = x.cuda(), w.cuda()
    out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    cabi.check(cabi.lib.gpuk_linear_skinny(_ptr(dx), _ptr(dw), _ptr(out), m, n, k, k_split, _stream()))
    _status_ok()
    assert fo.within_one_bf16_step(out.cpu(), x.double() @ w.double().t())


@pytest.mark.gpu
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("m,n,k", [(8, 1536, 8192), (8, 1664, 8192), (9, 128, 64), (16, 256, 192), (17, 256, 4160), (32, 10240, 1024)])
def test_fp8_linear_around_the_dispatch(m, n, k, packed):
    """The weight size and the token count at which the entry point changes kernels, k with an odd number of 64-byte blocks, and an
    output and channel scales that are aligned for single elements only."""
    import gpuk_b200 as gpuk
    g = torch.Generator().manual_seed(m + n + k)
    x, w = (torch.randn(m, k, generator=g) * 100).clamp_(-448, 448).to(E4M3), (torch.randn(n, k, generator=g) * 100).clamp_(-448, 448).to(E4M3)
    xs, ws = torch.rand(m, 1, generator=g) * 0.02 + 1e-3, torch.rand(1, n, generator=g) * 0.02 + 1e-3
    want = fo.fp8_linear_reference(x, xs, w, ws)
    dx, dxs, dw, dws = x.cuda(), xs.cuda(), w.cuda(), ws.cuda()
    if packed:
        dw = gpuk.fp8_pack_weight(dw)
    got = gpuk.fp8_linear(dx, dxs, dw, dws, packed=packed)
    assert fo.within_one_bf16_step(got.cpu(), want)
    out = torch.full((m * n + 1,), float("nan"), dtype=torch.bfloat16, device="cuda")
    shifted = torch.cat([dws.view(-1)[:1], dws.view(-1)])[1:]
    again = gpuk.fp8_linear(dx, dxs, dw, shifted, out[1:].view(m, n), packed=packed)
    _status_ok()
    assert torch.equal(again.view(torch.int16), got.view(torch.int16)) and bool(torch.isnan(out[0]))


def test_refused_shapes():
    f = cabi.lib.gpuk_linear_skinny
    assert f(16, 16, 16, 33, 128, 64, 0, None) == cabi.ERR_UNSUPPORTED and f(16, 16, 16, 8, 100, 64, 0, None) == cabi.ERR_UNSUPPORTED
    assert f(16, 16, 16, 8, 128, 12, 0, None) == cabi.ERR_UNSUPPORTED and f(16, 16, 16, 8, 128, 64, 9, None) == cabi.ERR_INVALID_ARGUMENT
    assert f(16, 8, 16, 8, 128, 64, 0, None) == cabi.ERR_INVALID_ARGUMENT and f(None, 16, 16, 8, 128, 64, 0, None) == cabi.ERR_INVALID_ARGUMENT
    assert f(16, 16, 16, 0, 128, 64, 0, None) == cabi.OK
