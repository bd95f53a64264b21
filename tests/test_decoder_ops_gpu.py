"""The decoder's own kernels between its projections, against the PyTorch operators they replace."""
import pytest
import torch
import torch.nn.functional as F

import gpuk_b200
from gpuk_b200 import _native, cabi

pytestmark = pytest.mark.gpu


def _rope(x, cos, sin):
    x1, x2 = x[..., 0::2], x[..., 1::2]
    cos, sin = cos.unsqueeze(-2), sin.unsqueeze(-2)
    return torch.cat((x1 * cos - x2 * sin, x2 * cos + x1 * sin), dim=-1).type_as(x)


@pytest.mark.parametrize("batch,t,heads,kv,hd,positions", [
    (1, 1, 8, 1, 128, [0]), (5, 1, 16, 4, 128, [39]), (2, 3, 4, 2, 16, [7, 0, 39]), (3, 17, 6, 3, 48, list(range(5, 22))), (1, 2, 2, 1, 64, [-1, -40])])
def test_rope_append_equals_the_operator_chain(batch, t, heads, kv, hd, positions):
    """One thread per 16 elements: one and several parts per head, one head and many, positions at both ends of the cache and
    counted from its end.  The arithmetic is the chain's, rounding for rounding, so the bits are the same."""
    g = torch.Generator(device="cuda").manual_seed(hd * 100 + t)
    max_seq = 40
    qkv = torch.randn(batch * t, (heads + 2 * kv) * hd, generator=g, device="cuda").bfloat16()
    freqs = torch.outer(torch.arange(max_seq * 2).float(), 1.0 / (10000.0 ** (torch.arange(0, hd, 2).float() / hd)))
    cos, sin = freqs.cos().cuda(), freqs.sin().cuda()
    pos = torch.tensor(positions, device="cuda")
    caches = [torch.randn(batch + 1, kv, max_seq, hd, generator=g, device="cuda").bfloat16() for _ in range(2)]
    want_k, want_v = (c.clone() for c in caches)
    q, k, v = qkv.view(batch, t, heads + 2 * kv, hd).split([heads, kv, kv], dim=2)
    want_q = _rope(q, cos[pos], sin[pos])
    want_k[:batch, :, pos] = _rope(k, cos[pos], sin[pos]).transpose(1, 2)
    want_v[:batch, :, pos] = v.transpose(1, 2)
    got = _native.rope_append(qkv, cos, sin, pos, caches[0], caches[1], heads)
    assert torch.equal(got.view(want_q.shape), want_q)
    assert torch.equal(caches[0], want_k) and torch.equal(caches[1], want_v)


def test_rope_append_writes_nothing_outside_the_cache():
    qkv = torch.ones(1, 3 * 16, device="cuda").bfloat16()
    cos = torch.ones(20, 8, device="cuda")
    caches = [torch.zeros(2, 1, 4, 16, device="cuda").bfloat16() for _ in range(2)]
    for at in (4, 19, 20, -5):
        _native.rope_append(qkv, cos, cos, torch.tensor([at], device="cuda"), caches[0], caches[1], 1)
        assert cabi.lib.gpuk_fp8_linear_status() == cabi.ERR_INVALID_ARGUMENT
    assert not caches[0].any() and not caches[1].any()


@pytest.mark.parametrize("rows,f", [(1, 8), (3, 2048), (37, 4104), (2, 28672)])
def test_silu_mul_equals_the_operators(rows, f):
    """Same roundings as silu, then multiply; the exponential may differ in the last fp32 bit, so a value in a thousand may
    round the other way: one bf16 step of the product (2^-7 relative at most)."""
    x = (torch.randn(rows, 2 * f, generator=torch.Generator(device="cuda").manual_seed(f), device="cuda") * 4).bfloat16()
    want = F.silu(x[:, :f]) * x[:, f:]
    got = _native.silu_mul(x)
    assert float((got != want).float().mean()) <= 1e-3
    assert torch.all((got.float() - want.float()).abs() <= want.float().abs() * 2.0 ** -7)


def test_shapes_that_are_not_built_are_refused():
    x = torch.zeros(2, 24, device="cuda").bfloat16()
    with pytest.raises(RuntimeError, match="multiple of 8"):
        _native.silu_mul(x)
    with pytest.raises(RuntimeError, match="contiguous CUDA tensor"):
        _native.silu_mul(x.cpu())
    assert cabi.lib.gpuk_silu_mul(None, None, 0, 8, None) == cabi.OK
    assert gpuk_b200._native is _native


@pytest.mark.parametrize("rows,f", [(1, 8), (3, 2048), (1, 2056), (1200, 4104)])
def test_silu_mul_at_the_ends_of_a_chunk_and_of_the_range(rows, f):
    """One and two vectors a thread, rows that end inside a chunk; infinities, NaN, zeros of both signs, quotients that leave the range."""
    special = torch.tensor([float("inf"), float("-inf"), float("nan"), 0.0, -0.0, -88.5, -89.0, -104.0, 88.0, 3e38, -3e38, 1e-39, -70.0, -1e-31, 2e30, 1.0])
    g = torch.Generator().manual_seed(rows + f)
    x = torch.randn(rows, 2 * f, generator=g) * 3
    x[0, :min(f, 16)] = special[:min(f, 16)]
    x = x.bfloat16().cuda()
    a, b = x.split(f, -1)
    want, got = F.silu(a) * b, _native.silu_mul(x)
    nan = want.isnan()
    assert torch.equal(got.isnan(), nan) and torch.equal(got[~nan].view(torch.int16), want[~nan].view(torch.int16))


def test_silu_of_every_bf16():
    """All 65536 inputs times one: the bits of the operator, NaN where it is."""
    a = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).view(torch.bfloat16).cuda()
    got, want = _native.silu_mul(torch.cat([a, torch.ones_like(a)]).view(1, -1))[0], F.silu(a) * torch.ones_like(a)
    nan = want.isnan()
    assert torch.equal(got.isnan(), nan) and torch.equal(got[~nan].view(torch.int16), want[~nan].view(torch.int16))
