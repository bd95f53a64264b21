"""The kernels of a decode step -- streaming linear layers in FP8 and bf16, attention over the KV cache for one and for many new tokens -- against float64."""
import pytest
import torch

import gpuk_b200 as gpuk
from gpuk_b200 import _native, cabi
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
@pytest.mark.parametrize("m,n,k", [(1, 128, 8), (16, 256, 64), (17, 128, 72), (32, 384, 1000), (31, 1280, 4096), (9, 16384, 2048), (24, 6144, 2048),
                                   (32, 4352, 4096), (4, 19072, 1024), (17, 18944, 1024)])
def test_bf16_linear(m, n, k, k_split):
    """Tokens on both sides of the 16-column tile, k that ends inside a step (8, 72, 1000), fewer steps than parts, tiles below and above
    the number of SMs, and numbers of them that clusters of six or eight would not fit.  fp32 sums of exact products, one rounding: one bf16 step."""
    g = torch.Generator().manual_seed(m + n + k)
    x, w = torch.randn(m, k, generator=g).bfloat16(), torch.randn(n, k, generator=g).bfloat16()
    dx, dw = x.cuda(), w.cuda()
    out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    cabi.check(cabi.lib.gpuk_linear_skinny(_ptr(dx), _ptr(dw), _ptr(out), m, n, k, k_split, _stream()))
    _status_ok()
    assert fo.within_one_bf16_step(out.cpu(), x.double() @ w.double().t())


@pytest.mark.gpu
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("m,k_split", [(32, 8), (16, 8), (32, 3)])
def test_more_clusters_than_tensor_memory_holds(m, k_split, fp8):
    """One step a part, or two: rings so short that shared memory and registers would let more CTAs on an SM than it has columns for."""
    n, k = 128 * 400, 1024 if fp8 else 512
    ops = _fused_operands(m, n, k, fp8, torch.Generator().manual_seed(m))
    x, xs, w, ws = ops
    want = x.double() @ w.double().t() * (xs.double() * ws.double() if fp8 else 1.0)
    for _ in range(3):
        out = torch.full((m, n), float("nan"), dtype=torch.bfloat16, device="cuda")
        if fp8:
            gpuk.fp8_linear(x, xs, w, ws, out, k_split=k_split if k_split != 3 else 4)
        else:
            cabi.check(cabi.lib.gpuk_linear_skinny(_ptr(x), _ptr(w), _ptr(out), m, n, k, k_split, _stream()))
        _status_ok()
        assert fo.within_one_bf16_step(out.cpu(), want.cpu())


@pytest.mark.gpu
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("m,n,k", [(8, 1536, 8192), (8, 1664, 8192), (8, 4096, 8192), (7, 4224, 8192), (9, 128, 64), (16, 256, 192), (17, 256, 4160), (32, 10240, 1024)])
def test_fp8_linear_around_the_dispatch(m, n, k, packed):
    """The weight size and the token count at which the entry point changes kernels, k with an odd number of 64-byte blocks, and an
    output and channel scales that are aligned for single elements only."""
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


def _fused_operands(m, n, k, fp8, g):
    """x, its scales, w, its scales, as the native calls take them."""
    if not fp8:
        return torch.randn(m, k, generator=g).bfloat16().cuda(), None, (torch.randn(n, k, generator=g) / k ** 0.5).bfloat16().cuda(), None
    x, w = (torch.randn(m, k, generator=g) * 100).clamp_(-448, 448).to(E4M3), (torch.randn(n, k, generator=g) * 100).clamp_(-448, 448).to(E4M3)
    return x.cuda(), (torch.rand(m, 1, generator=g) * 0.01 + 1e-3).cuda(), w.cuda(), (torch.rand(1, n, generator=g) * 0.01 + 1e-3).div_(k ** 0.5).cuda()


def _streamed(x, xs, w, ws):
    """The projection alone, by the same kernel: `w` repeated until the entry point leaves the warp-level kernel out."""
    if xs is None:
        return _native.linear(x, w)
    reps = 1 if x.shape[0] > 8 else -(-((32 << 20) + 1) // w.numel())
    return gpuk.fp8_linear(x, xs, w.repeat(reps, 1), ws.repeat(1, reps))[:, :w.shape[0]].contiguous()


@pytest.mark.gpu
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("m,f,k", [(1, 64, 64), (8, 192, 1024), (16, 4096, 2048), (17, 64, 4160), (32, 7168, 1024)])
def test_swiglu(m, f, k, fp8):
    """One tile and many, both column counts: the projection in float64, its two halves rounded, silu rounded, product rounded -- each of the four
    roundings can fall the other way by a step: 2^-7 of the projection's larger half carries through as at most four steps of the result."""
    ops = _fused_operands(m, 2 * f, k, fp8, torch.Generator().manual_seed(m + f))
    got = _native.swiglu(*ops)
    _status_ok()
    y = ops[0].double() @ ops[2].double().t() * (ops[1].double() * ops[3].double() if fp8 else 1.0)
    a, b = y.bfloat16().double().split(f, -1)
    want = (a / (1 + torch.exp(-a))).bfloat16().double() * b
    assert bool(((got.double() - want).abs() <= 4 * 2.0 ** -8 * want.abs() + 1e-5).all())
    same = _native.silu_mul(_streamed(*ops))
    if m > 8 or not fp8:      # the same parts of k
        assert torch.equal(got.view(torch.int16), same.view(torch.int16))
    else:                     # cut elsewhere: a step apart in a few places, no more
        assert float((got.view(torch.int16) == same.view(torch.int16)).float().mean()) > 0.99


@pytest.mark.gpu
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("batch,t,heads,kv,k,positions", [(1, 1, 8, 1, 64, [0]), (32, 1, 16, 4, 2048, [39]), (3, 5, 4, 2, 1024, [7, 0, 39, 38, 12]), (1, 2, 2, 1, 4160, [-1, -40]),
                                                         (2, 2, 2, 1, 1024, [38, 3])])
def test_qkv_rope(batch, t, heads, kv, k, positions, fp8):
    """Against the projection and gpuk_rope_append: both ends of the cache, positions from its end."""
    g = torch.Generator().manual_seed(batch + heads)
    ops = _fused_operands(batch * t, (heads + 2 * kv) * 128, k, fp8, g)
    freqs = torch.outer(torch.arange(80).float(), 1.0 / (10000.0 ** (torch.arange(0, 128, 2).float() / 128)))
    cos, sin, pos = freqs.cos().cuda(), freqs.sin().cuda(), torch.tensor(positions).cuda()
    caches = [torch.randn(batch + 1, kv, 40, 128, generator=g).bfloat16().cuda() for _ in range(2)]
    start, mine = [c.clone() for c in caches], [c.clone() for c in caches]
    q = _native.qkv_rope(*ops, cos, sin, pos, *mine, heads)
    _status_ok()
    want = _native.rope_append(_streamed(*ops), cos, sin, pos, *caches, heads)
    written = pos % 40
    for c, s in zip(mine, start):      # nothing but the sequences' own positions
        left = c.clone()
        left[:batch, :, written] = s[:batch, :, written]
        assert torch.equal(left, s)
    for a, b in zip((q, *(c[:batch, :, written] for c in mine)), (want, *(c[:batch, :, written] for c in caches))):
        if batch * t > 8 or not fp8:      # the same parts of k
            assert torch.equal(a, b)
        else:      # sums in another order of k: a projection may fall one bf16 step aside, and a rotated pair with it by the larger of the two
            assert float((a.float() - b.float()).abs().max()) <= 2.0 ** -7 * float(b.float().abs().max()) and float((a == b).float().mean()) > 0.99


@pytest.mark.gpu
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("k_split", [1, 2, 8])
@pytest.mark.parametrize("m", [3, 16, 27])
def test_epilogues_round_as_the_separate_calls(m, k_split, fp8):
    """The same parts of k on both sides: the same bits."""
    k, heads, kv = 2048 + 64, 4, 2
    g = torch.Generator().manual_seed(m)
    n = (heads + 2 * kv) * 128
    x, xs, w, ws = _fused_operands(m, n, k, fp8, g)
    scales = (_ptr(xs), _ptr(ws)) if fp8 else (None, None)

    def projection():
        out = torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
        if fp8:      # so many channels that few tokens go to this kernel too
            reps = -(-((32 << 20) + 1) // w.numel()) if m <= 8 else 1
            return gpuk.fp8_linear(x, xs, w.repeat(reps, 1), ws.repeat(1, reps), k_split=k_split)[:, :n].contiguous()
        cabi.check(cabi.lib.gpuk_linear_skinny(_ptr(x), _ptr(w), _ptr(out), m, n, k, k_split, _stream()))
        return out
    y = projection()
    act = torch.empty(m, n // 2, dtype=torch.bfloat16, device="cuda")
    cabi.check(cabi.lib.gpuk_swiglu_skinny(_ptr(x), scales[0], _ptr(w), scales[1], _ptr(act), m, n, k, k_split, _stream()))
    assert torch.equal(act, _native.silu_mul(y))
    cos, sin, pos = torch.randn(80, 64, generator=g).cuda(), torch.randn(80, 64, generator=g).cuda(), torch.tensor([17], device="cuda")
    caches = [torch.zeros(m, kv, 40, 128, dtype=torch.bfloat16, device="cuda") for _ in range(4)]
    q = torch.empty(m, heads * 128, dtype=torch.bfloat16, device="cuda")
    cabi.check(cabi.lib.gpuk_qkv_rope_skinny(_ptr(x), scales[0], _ptr(w), scales[1], _ptr(cos), _ptr(sin), _ptr(pos), _ptr(q), _ptr(caches[0]), _ptr(caches[1]), m, 1, heads, kv, k,
                                             80, 40, k_split, _stream()))
    _status_ok()
    assert torch.equal(q, _native.rope_append(y, cos, sin, pos, caches[2], caches[3], heads))
    assert torch.equal(caches[0], caches[2]) and torch.equal(caches[1], caches[3])


def _position_reported_once():
    status = cabi.lib.gpuk_fp8_linear_status
    assert status() == cabi.ERR_INVALID_ARGUMENT and "position" in cabi.last_error() and status() == cabi.OK


@pytest.mark.gpu
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("table_rows,bad", [(80, 40), (80, 80), (80, -41), (80, -81), (20, 25), (20, -30), (80, 1 << 32), (80, -(1 << 33))])
def test_positions_outside_the_cache_or_the_table(table_rows, bad, fused, fp8):
    """Of such a token nothing goes to the caches, its queries are NaN, written in full, and the status call says so, once.  Tokens beside it are as without it."""
    batch, heads, kv, k = 3, 4, 2, 1024
    g = torch.Generator().manual_seed(5)
    ops = _fused_operands(batch * 3, (heads + 2 * kv) * 128, k, fp8, g)
    x, xs, w, ws = ops
    cos, sin = torch.randn(table_rows, 64, generator=g).cuda(), torch.randn(table_rows, 64, generator=g).cuda()
    start = [torch.randn(batch, kv, 40, 128, generator=g).bfloat16().cuda() for _ in range(2)]

    def call(positions):
        pos, caches = torch.tensor(positions).cuda(), [c.clone() for c in start]
        q = torch.full((batch * 3, heads * 128), 7.0, dtype=torch.bfloat16, device="cuda")
        common = (_ptr(cos), _ptr(sin), _ptr(pos), _ptr(q), *map(_ptr, caches), batch, 3, heads, kv)
        if fused:
            cabi.check(cabi.lib.gpuk_qkv_rope_skinny(_ptr(x), _ptr(xs) if fp8 else None, _ptr(w), _ptr(ws) if fp8 else None, *common, k, table_rows, 40, 0, _stream()))
        else:
            qkv = _streamed(*ops)
            cabi.check(cabi.lib.gpuk_rope_append(_ptr(qkv), *common, 128, table_rows, 40, _stream()))
        return q.view(batch, 3, heads * 128), caches
    q, caches = call([3, bad, 7])
    _position_reported_once()
    assert bool(q[:, 1].isnan().all()) and not bool(q[:, 0::2].isnan().any())
    want_q, want = call([3, 5, 7])
    _status_ok()
    assert torch.equal(q[:, 0::2], want_q[:, 0::2])
    for c, d, s in zip(caches, want, start):
        d[:, :, 5] = s[:, :, 5]
        assert torch.equal(c, d)


@pytest.mark.gpu
@pytest.mark.parametrize("splits", [0, 1, 3, 8])
@pytest.mark.parametrize("batch,heads,kv_heads,length,max_seq", [(1, 8, 2, 1, 1), (3, 16, 1, 17, 32), (2, 4, 4, 64, 64), (4, 16, 4, 129, 256), (5, 8, 1, 1000, 1024),
                                                                (40, 64, 8, 80, 256), (16, 4, 1, 700, 704), (2, 128, 8, 1300, 1300), (9, 64, 8, 1600, 1600)])
def test_decode_attention(batch, heads, kv_heads, length, max_seq, splits):
    """One key, ends inside a block of 16, parts of the cluster without keys, 1 to 16 query heads per kv head, both ring depths.  What lies behind
    the keys is NaN.  Probabilities are rounded to bf16 before the second product (a relative 2^-8 each, half of the last of eight bits) and
    the result once more: 2 * 2^-8 of sum(p |v|)."""
    g = torch.Generator().manual_seed(batch + heads + length)
    q = (torch.randn(batch, heads, 128, generator=g) * 2).bfloat16()
    k, v = (torch.randn(batch + 1, kv_heads, max_seq, 128, generator=g).bfloat16() for _ in range(2))
    k[:, :, length:], v[:, :, length:] = float("nan"), float("nan")
    kk, vv = (t[:batch, :, :length].repeat_interleave(heads // kv_heads, 1).double() for t in (k, v))
    p = torch.softmax(torch.einsum("bhd,bhkd->bhk", q.double(), kk) / 128 ** 0.5, -1)
    want, bound = torch.einsum("bhk,bhkd->bhd", p, vv), torch.einsum("bhk,bhkd->bhd", p, vv.abs()) * 2.0 ** -7 + 1e-6
    dq, dk, dv = q.cuda(), k.cuda(), v.cuda()
    out = torch.full_like(dq, float("nan"))
    cabi.check(cabi.lib.gpuk_decode_attention(_ptr(dq), _ptr(dk), _ptr(dv), _ptr(out), batch, heads, kv_heads, 128, length, max_seq, splits, _stream()))
    _status_ok()
    assert bool(((out.cpu().double() - want).abs() <= bound).all())


@pytest.mark.gpu
@pytest.mark.parametrize("batch,t,heads,kv_heads,past", [(1, 2, 2, 1, 0), (1, 128, 4, 4, 0), (2, 129, 8, 2, 127), (1, 257, 17, 1, 0), (3, 40, 4, 2, 300), (1, 300, 2, 1, 1700)])
@pytest.mark.parametrize("order", ["rising", "mixed", "far"])
def test_prefill_attention(batch, t, heads, kv_heads, past, order):
    """Both tiles of a CTA, ends at, before and behind a tile of queries and a block of keys, a ring that wraps, queries of a next sequence in the tile;
    positions in order, and in any order with one that sees no key and one beyond the cache, just so and far outside.  Bound as for one token."""
    g = torch.Generator().manual_seed(batch + t + heads)
    length, max_seq = past + t, past + t + 5
    q = (torch.randn(batch, t, heads, 128, generator=g) * 2).bfloat16()
    k, v = (torch.randn(batch, kv_heads, max_seq, 128, generator=g).bfloat16() for _ in range(2))
    k[:, :, length:], v[:, :, length:] = float("nan"), float("nan")
    pos = torch.arange(past, length)
    if order != "rising":
        pos = pos[torch.randperm(t, generator=g)]
        pos[0], pos[-1] = (-1, length + 3) if order == "mixed" else (-(1 << 32), 1 << 32)      # far: the low halves are positions of the cache
    kk, vv = (x[:, :, :length].repeat_interleave(heads // kv_heads, 1).double() for x in (k, v))
    s = torch.einsum("bthd,bhkd->bhtk", q.double(), kk) / 128 ** 0.5
    p = torch.softmax(s.masked_fill(torch.arange(length) > pos[:, None], float("-inf")), -1).nan_to_num(0.0)
    want, bound = torch.einsum("bhtk,bhkd->bthd", p, vv), torch.einsum("bhtk,bhkd->bthd", p, vv.abs()) * 2.0 ** -7 + 1e-6
    dq, dk, dv, dp = q.cuda(), k.cuda(), v.cuda(), pos.cuda()
    out = torch.full_like(dq, float("nan"))
    cabi.check(cabi.lib.gpuk_prefill_attention(_ptr(dq), _ptr(dk), _ptr(dv), _ptr(dp), _ptr(out), batch, t, heads, kv_heads, 128, length, max_seq, _stream()))
    _status_ok()
    assert bool(((out.cpu().double() - want).abs() <= bound).all())


@pytest.mark.gpu
@pytest.mark.parametrize("hidden", [1, 40, 200, 290])
@pytest.mark.parametrize("splits", [0, 1, 3])
def test_scores_of_minus_infinity(hidden, splits):
    """The first `hidden` keys score -infinity for some heads: whole blocks, warps and parts of the cluster of them, in front of scores far below zero.  They weigh
    nothing; the others as in float64.  Bound as in test_decode_attention."""
    batch, heads, length = 2, 4, 300
    g = torch.Generator().manual_seed(hidden)
    q, k, v = (torch.randn(batch, n, m, 128, generator=g).bfloat16() for n, m in ((1, heads), (1, length), (1, length)))
    q = q.view(batch, heads, 128)
    q[:, :, 0] = 2.0
    k[:, :, :, 0] = -1000.0                                    # so far below zero that nothing is left of a weight measured from there
    k[:, :, :hidden, 0] = float("-inf")

    def reference(limit):
        s = torch.einsum("bhd,bhkd->bhk", q.double(), k.double().expand(-1, heads, -1, -1)) / 128 ** 0.5
        s = s.masked_fill(torch.arange(length) >= limit, float("-inf"))
        p = torch.softmax(s, -1)
        vv = v.double().expand(-1, heads, -1, -1)
        return torch.einsum("bhk,bhkd->bhd", p, vv), torch.einsum("bhk,bhkd->bhd", p, vv.abs()) * 2.0 ** -7 + 1e-6
    dq, dk, dv = q.cuda(), k.cuda(), v.cuda()
    out = torch.full_like(dq, float("nan"))
    cabi.check(cabi.lib.gpuk_decode_attention(_ptr(dq), _ptr(dk), _ptr(dv), _ptr(out), batch, heads, 1, 128, length, length, splits, _stream()))
    want, bound = reference(length)
    assert bool(((out.cpu().double() - want).abs() <= bound).all())
    pos = torch.tensor([length - 1, 294], device="cuda")
    many = torch.full((batch, 2, heads, 128), float("nan"), dtype=torch.bfloat16, device="cuda")
    dq2 = dq.view(batch, 1, heads, 128).expand(-1, 2, -1, -1).contiguous()
    cabi.check(cabi.lib.gpuk_prefill_attention(_ptr(dq2), _ptr(dk), _ptr(dv), _ptr(pos), _ptr(many), batch, 2, heads, 1, 128, length, length, _stream()))
    _status_ok()
    for i, limit in enumerate((length, 295)):
        want, bound = reference(limit)
        assert bool(((many[:, i].cpu().double() - want).abs() <= bound).all())


def test_refused_shapes():
    f, a = cabi.lib.gpuk_linear_skinny, cabi.lib.gpuk_decode_attention
    assert f(16, 16, 16, 33, 128, 64, 0, None) == cabi.ERR_UNSUPPORTED and f(16, 16, 16, 8, 100, 64, 0, None) == cabi.ERR_UNSUPPORTED
    assert f(16, 16, 16, 8, 128, 12, 0, None) == cabi.ERR_UNSUPPORTED and f(16, 16, 16, 8, 128, 64, 9, None) == cabi.ERR_INVALID_ARGUMENT
    assert f(16, 8, 16, 8, 128, 64, 0, None) == cabi.ERR_INVALID_ARGUMENT and f(None, 16, 16, 8, 128, 64, 0, None) == cabi.ERR_INVALID_ARGUMENT
    assert f(16, 16, 16, 0, 128, 64, 0, None) == cabi.OK
    assert a(16, 16, 16, 16, 1, 34, 2, 128, 4, 8, 0, None) == cabi.ERR_UNSUPPORTED      # 17 query heads per kv head
    assert a(16, 16, 16, 16, 1, 8, 2, 64, 4, 8, 0, None) == cabi.ERR_UNSUPPORTED and a(16, 16, 16, 16, 1, 8, 2, 128, 9, 8, 0, None) == cabi.ERR_INVALID_ARGUMENT
    assert a(16, 16, 16, 16, 0, 8, 2, 128, 4, 8, 0, None) == cabi.OK
    b = cabi.lib.gpuk_prefill_attention
    assert b(16, 16, 16, 16, 16, 1, 4, 8, 2, 64, 4, 8, None) == cabi.ERR_UNSUPPORTED and b(16, 16, 16, 16, 16, 1, 4, 8, 3, 128, 4, 8, None) == cabi.ERR_UNSUPPORTED
    assert b(16, 16, 16, 16, 16, 1, 4, 8, 2, 128, 9, 8, None) == cabi.ERR_INVALID_ARGUMENT and b(16, 16, 8, 16, 16, 1, 4, 8, 2, 128, 4, 8, None) == cabi.ERR_INVALID_ARGUMENT
    assert b(16, 16, 16, 16, 16, 1, 0, 8, 2, 128, 4, 8, None) == cabi.OK
    # sizes whose products leave 32 or 64 bits
    big = (1 << 31) - 1
    assert b(16, 16, 16, 16, 16, big, big, big, 1, 128, 4, 8, None) == cabi.ERR_UNSUPPORTED
    r = cabi.lib.gpuk_rope_append
    assert r(16, 16, 16, 16, 16, 16, 16, 1, 1, 1 << 30, 1 << 30, 128, 80, 40, None) == cabi.ERR_UNSUPPORTED
    assert r(16, 16, 16, 16, 16, 16, 16, big, big, 8, 1, 128, 80, 40, None) == cabi.ERR_UNSUPPORTED
    assert cabi.lib.gpuk_silu_mul(16, 16, 1 << 62, 1 << 30, None) == cabi.ERR_UNSUPPORTED
    c = cabi.lib.gpuk_swiglu_skinny
    assert c(16, 16, 16, None, 16, 8, 128, 64, 0, None) == cabi.ERR_INVALID_ARGUMENT and c(16, None, 16, None, 12, 8, 128, 64, 0, None) == cabi.ERR_INVALID_ARGUMENT
    assert c(16, None, 16, None, 16, 33, 128, 64, 0, None) == cabi.ERR_UNSUPPORTED and c(16, None, 16, None, 16, 8, 64, 64, 0, None) == cabi.ERR_UNSUPPORTED
    d = cabi.lib.gpuk_qkv_rope_skinny
    assert d(16, None, 16, None, 16, 16, 16, 16, 16, 16, 33, 1, 8, 1, 64, 80, 40, 0, None) == cabi.ERR_INVALID_ARGUMENT
    assert d(16, None, 16, None, 16, 16, 16, 16, 16, 16, 17, 2, 8, 1, 64, 80, 40, 0, None) == cabi.ERR_UNSUPPORTED
    assert d(16, None, 16, None, 16, 16, None, 16, 16, 16, 1, 1, 8, 1, 64, 80, 40, 0, None) == cabi.ERR_INVALID_ARGUMENT


@pytest.mark.gpu
def test_decoder_takes_the_cache_lengths_it_took():
    """A length beyond the cache means all of it for one token and is refused for several; so is a position beyond it, and a wrong number of positions."""
    import torch.distributed as dist
    from gpuk_b200.tp_model import DecoderArgs, TPDecoder
    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    env = gpuk.GPUKDistEnv(group=None, device_id=0)
    m = TPDecoder(DecoderArgs(dim=512, n_layers=1, n_heads=4, n_kv_heads=2, ffn_dim=1024, vocab_size=256, max_seq_len=64), env, device="cuda:0", fp8=False, max_batch=2)
    m.fill_kv_cache(64)
    one, pos = torch.zeros(2, 1, dtype=torch.long, device="cuda"), torch.tensor([63], device="cuda")
    assert torch.equal(m.forward(one, pos, cache_len=70), m.forward(one, pos, cache_len=64))
    for tokens, positions, n in ((one, torch.tensor([64], device="cuda"), None), (one.expand(2, 2), torch.tensor([62, 63], device="cuda"), 70),
                                 (one, torch.tensor([62, 63], device="cuda"), 64)):
        with pytest.raises(RuntimeError):
            m.forward(tokens, positions, cache_len=n)


@pytest.fixture
def decoder():
    """Makes a decoder on one GPU."""
    import torch.distributed as dist
    from gpuk_b200.tp_model import DecoderArgs, TPDecoder
    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    env = gpuk.GPUKDistEnv(group=None, device_id=0)

    def make(head_dim=128, fp8=False, batch=2, dim=512, **more):
        args = dict(dim=dim, n_layers=2, n_heads=4, n_kv_heads=2, head_dim=head_dim, ffn_dim=1024, vocab_size=256, max_seq_len=64)
        args.update(more)
        m = TPDecoder(DecoderArgs(**args), env, device="cuda:0", fp8=fp8, max_batch=batch)
        m.fill_kv_cache(64)
        return m
    return make


@pytest.mark.gpu
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("head_dim", [128, 64])
def test_decoder_marks_positions_behind_its_cache(decoder, head_dim, fp8):
    """No device read: NaN logits for the token that has no place, those of the others as without it, and the status.  With one: refused."""
    m = decoder(head_dim, fp8)
    keep = [layer[n].clone() for layer in m.layers for n in ("k_cache", "v_cache")]

    def caches():
        return [layer[n] for layer in m.layers for n in ("k_cache", "v_cache")]

    def restore():
        for c, k in zip(caches(), keep):
            c.copy_(k)
    one, three = torch.zeros(2, 1, dtype=torch.long, device="cuda"), torch.arange(6, device="cuda").view(2, 3)
    for bad in (64, 70, 1000, -65, -1000):      # the next step of a full cache among them
        logits = m.forward(one, torch.tensor([bad], device="cuda"), cache_len=65)
        assert bool(logits.isnan().all())
        _position_reported_once()
        assert all(torch.equal(c, k) for c, k in zip(caches(), keep))
        for places in ([10, bad, 12], [bad, 11, 12]):
            logits = m.forward(three, torch.tensor(places, device="cuda"), cache_len=13)
            _position_reported_once()
            i = places.index(bad)
            others = [j for j in range(3) if j != i]
            restore()
            # the bad token leaves the old key in its place: as if it stood behind what the others see
            want = m.forward(three, torch.tensor([40 if p == bad else p for p in places], device="cuda"), cache_len=41)
            restore()
            assert bool(logits[:, i].isnan().all()) and not bool(logits[:, others].isnan().any())
            assert float((logits[:, others].float() - want[:, others].float()).norm()) <= 0.03 * float(want[:, others].float().norm())
        for positions, length in ((torch.tensor([bad]), 64), (torch.tensor([bad]), None), (torch.tensor([bad], device="cuda"), None)):
            with pytest.raises(RuntimeError, match="beyond the KV cache"):
                m.forward(one, positions, cache_len=length)
        with pytest.raises(RuntimeError, match="beyond the KV cache"):
            m.forward(three, torch.tensor([10, bad, 12], device="cuda"))
    assert not bool(m.forward(one, torch.tensor([63], device="cuda"), cache_len=70).isnan().any())
    _status_ok()


def _strided(t):
    """The same values with another order of the two dimensions in the middle or, of a matrix, as columns of a wider one."""
    if t.dim() == 4:
        return t.transpose(1, 2).contiguous().transpose(1, 2)
    return torch.cat([t, t], 1)[:, :t.shape[1]]


@pytest.mark.gpu
@pytest.mark.parametrize("t", [1, 3])
@pytest.mark.parametrize("what", ["caches", "weights", "tables", "everything"])
def test_decoder_takes_tensors_the_kernels_do_not_read(decoder, what, t):
    """Views in the place of caches and weights, tables in another type: what the operators took, they take.  Same values as without, up to the roundings of
    bf16 between the operators."""
    plain, m = decoder(), decoder()
    tokens, pos = torch.arange(2 * t, device="cuda").view(2, t), torch.arange(20, 20 + t, device="cuda")
    want = plain.forward(tokens, pos, cache_len=20 + t)
    for layer in m.layers:
        if what in ("caches", "everything"):
            layer["k_cache"], layer["v_cache"] = _strided(layer["k_cache"]), _strided(layer["v_cache"])
        if what in ("weights", "everything"):
            for name in ("wqkv", "wo", "w13", "w2"):
                layer[name].weight = _strided(layer[name].weight)
    if what in ("tables", "everything"):
        m.cos, m.sin = m.cos.double(), m.sin.double()
    got = m.forward(tokens, pos, cache_len=20 + t)
    _status_ok()
    assert float((got.float() - want.float()).norm()) <= 0.03 * float(want.float().norm())
    for a, b in zip(m.layers, plain.layers):
        for name in ("k_cache", "v_cache"):
            assert float((a[name].float() - b[name].float()).abs().max()) <= 0.06


@pytest.mark.gpu
def test_native_calls_hand_back_what_the_kernels_do_not_read():
    """Odd addresses and strides: None, before any launch; a cache that the library's attention could not read either is refused."""
    x, w = torch.zeros(2, 256, device="cuda").bfloat16(), torch.zeros(257 * 256, device="cuda").bfloat16()
    odd = w[1:1 + 256 * 256].view(256, 256)
    assert _native.linear(x, odd) is None and _native.swiglu(x, None, odd, None) is None and _native.linear(x, w[:65536].view(256, 256).t()) is None
    assert _native.silu_mul(w[1:513].view(2, 256)) is None
    q, pos = torch.zeros(2, 1, 128, device="cuda").bfloat16(), torch.zeros(1, dtype=torch.long, device="cuda")
    cos, flat = torch.zeros(8, 64, device="cuda"), torch.zeros(2 * 4 * 136 + 1, device="cuda").bfloat16()
    fine = flat[:1024].view(2, 1, 4, 128)
    for bad in (flat[1:1025].view(2, 1, 4, 128), flat[:2 * 4 * 132].view(2, 1, 4, 132)[..., :128]):
        for call in (lambda k, v: _native.decode_attention(q, k, v, 4), lambda k, v: _native.prefill_attention(q.view(1, 2, 1, 128), k, v, pos.expand(2).contiguous(), 4),
                     lambda k, v: _native.rope_append(torch.zeros(2, 384, device="cuda").bfloat16(), cos, cos, pos, k, v, 1)):
            with pytest.raises(RuntimeError, match="aligned"):
                call(bad, fine)
            with pytest.raises(RuntimeError, match="aligned"):
                call(fine, bad)
    wide = flat[:2 * 4 * 136].view(2, 1, 4, 136)[..., :128]
    assert _native.decode_attention(q, wide, wide, 4) is None


@pytest.mark.gpu
@pytest.mark.parametrize("length", [32767, 32768, 32769, 32900])
def test_decoder_on_both_sides_of_the_library_s_attention(decoder, length):
    """Few sequences and long contexts: the same step by the operators, up to the roundings of bf16 between them."""
    m = decoder(max_seq_len=33024)
    m.fill_kv_cache(length)
    one, pos = torch.ones(2, 1, dtype=torch.long, device="cuda"), torch.tensor([length - 1], device="cuda")
    got = m.forward(one, pos, cache_len=length)
    _status_ok()
    m.own_elementwise = False
    want = m.forward(one, pos, cache_len=length)
    assert float((got.float() - want.float()).norm()) <= 0.03 * float(want.float().norm())


@pytest.mark.gpu
def test_decoder_takes_the_positions_it_took(decoder):
    """A list and 32-bit positions; what indexes no tensor is refused."""
    m, one = decoder(), torch.zeros(2, 1, dtype=torch.long, device="cuda")
    want = m.forward(one, torch.tensor([30], device="cuda"), cache_len=31)
    for positions in (torch.tensor([30], device="cuda", dtype=torch.int32), torch.tensor([30]), [30], slice(30, 31)):
        got = m.forward(one, positions, cache_len=31)
        assert float((got.float() - want.float()).norm()) <= 0.03 * float(want.float().norm())
    for positions in (torch.tensor([30.0], device="cuda"), torch.tensor([30], device="cuda", dtype=torch.int16)):
        with pytest.raises((RuntimeError, IndexError)):
            m.forward(one, positions, cache_len=31)


@pytest.mark.gpu
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("t", [1, 20])
def test_modes_see_the_decoder_s_operators(decoder, t, fp8):
    m = decoder(fp8=fp8)
    tokens, pos = torch.arange(2 * t, device="cuda").view(2, t), torch.arange(20, 20 + t, device="cuda")
    want = m.forward(tokens, pos, cache_len=20 + t)
    seen = []

    class Mode(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))
    with Mode():
        got = m.forward(tokens, pos, cache_len=20 + t)
    products = [f for f in seen if "mm" in f or "linear" in f]
    assert len(products) == 4 * 2 + 1 and sum("scaled_dot_product" in f for f in seen) == 2 and sum("silu" in f for f in seen) == 2, seen
    assert float((got.float() - want.float()).norm()) <= (0.08 if fp8 else 0.03) * float(want.float().norm())


@pytest.mark.gpu
def test_native_calls_of_other_streams_and_threads():
    """Each kind of call on a stream of its own behind the kernels that make its inputs, from four threads at once: the bits of a call by itself."""
    import threading

    def work(i, results):
        with torch.cuda.stream(torch.cuda.Stream()):
            g = torch.Generator(device="cuda").manual_seed(i % 2)
            for _ in range(5):
                x = torch.randn(5, 1024, generator=g, device="cuda").bfloat16()
                w13, wq = (torch.randn(n, 1024, generator=g, device="cuda").bfloat16() * 0.03 for n in (1024, 1024))
                caches = [torch.randn(5, 2, 40, 128, generator=g, device="cuda").bfloat16() for _ in range(2)]
                cos, pos = torch.randn(80, 64, generator=g, device="cuda"), torch.tensor([11], device="cuda")
                q = _native.qkv_rope(x, None, wq, None, cos, cos, pos, *caches, 4)
                mine = [_native.silu_mul(_native.linear(x, w13)), _native.swiglu(x, None, w13, None), q, *caches, _native.decode_attention(q.view(5, 4, 128), *caches, 12),
                        _native.rope_append(_native.linear(x, wq), cos, cos, pos, *caches, 4),
                        _native.prefill_attention(q.view(1, 5, 4, 128), *caches, torch.arange(5, 10, device="cuda"), 12)]
            torch.cuda.current_stream().synchronize()
            results[i] = [t.clone() for t in mine]
            torch.cuda.current_stream().synchronize()
    alone, together = {}, {}
    for i in range(2):
        work(i, alone)
    threads = [threading.Thread(target=work, args=(i, together)) for i in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    _status_ok()
    for i in range(4):
        assert all(torch.equal(a, b) for a, b in zip(together[i], alone[i % 2]))
