"""The one-GPU epilogue at the sizes where its entry point changes kernels: a warp per row, a CTA per row, persistent CTAs with either ring."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import epilogue_oracle as eo          # noqa: E402
from tests import util                            # noqa: E402


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("quant", [0, 2, 3, 4])
@pytest.mark.parametrize("tokens,vecs", [(512, 256), (511, 256), (515, 255), (1025, 128), (1100, 121), (2050, 64), (2100, 65), (2049, 64), (16390, 8), (131073, 1)])
def test_a_warp_per_row(tokens, vecs, quant, dtype):
    """2 MiB of input and just less; rows that fill the lanes and rows that do not, for each count of vectors a lane; a last CTA with idle warps."""
    hidden = vecs * (16 // dtype.itemsize)
    parts, res, w = util.random_case(1, tokens, hidden, dtype, seed=tokens + hidden + quant)
    static = 0.05 if quant == 4 else None
    got = util.k1(parts[0].cuda(), res.cuda(), w.cuda(), 1e-6, quant, static)
    util.check_against_oracle(got, eo.add_rms_quant(parts[0], res, w, 1e-6, quant, static), quant, exact_residual=True)


@pytest.mark.parametrize("quant", [0, 3])
@pytest.mark.parametrize("tokens,vecs", [(4736, 640), (4735, 641), (4740, 1024), (7104, 1024), (9472, 257), (9475, 640), (4800, 1025)])
def test_persistent_ctas(tokens, vecs, quant):
    """32, 48 and 64 rows per SM; two stages of 512 threads, four of 256, rings that wrap with a ragged last round."""
    parts, res, w = util.random_case(1, tokens, vecs * 8, torch.bfloat16, seed=tokens + vecs + quant)
    got = util.k1(parts[0].cuda(), res.cuda(), w.cuda(), 1e-6, quant)
    util.check_against_oracle(got, eo.add_rms_quant(parts[0], res, w, 1e-6, quant), quant, exact_residual=True)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("quant", [0, 3])
@pytest.mark.parametrize("tokens,vecs", [(1100, 120), (520, 256), (9475, 300), (4740, 768)])
def test_rows_that_are_not_finite(tokens, vecs, quant, dtype):
    """NaN, infinities, sums of squares that overflow and rows of zeros: a warp per row and persistent CTAs give what a CTA per row gives, and the rows beside them are
    as without."""
    from gpuk_b200 import cabi
    hidden = vecs * (16 // dtype.itemsize)
    parts, res, w = util.random_case(1, tokens, hidden, dtype, seed=tokens + vecs)
    x, big = parts[0], torch.finfo(dtype).max
    x[0], res[0] = 0, 0
    x[1, 3], x[2, 5], x[3, 7], x[tokens - 1, hidden - 1] = float("nan"), float("inf"), float("-inf"), float("nan")
    x[4], res[4] = big, 0
    x[5], res[5] = float("inf"), float("-inf")
    got = util.k1(x.cuda(), res.cuda(), w.cuda(), 1e-6, quant)
    cabi.check(cabi.lib.gpuk_set_tuning(b"k1_staged_min_rows", 1 << 40))
    try:
        want = util.k1(x.cuda(), res.cuda(), w.cuda(), 1e-6, quant)
    finally:
        cabi.check(cabi.lib.gpuk_set_tuning(b"k1_staged_min_rows", -1))
    special = [0, 1, 2, 3, 4, 5, tokens - 1]
    rest = torch.ones(tokens, dtype=torch.bool)
    rest[special] = False
    for name, a, b in zip(("residual", "norm", "scale"), got[:2 if quant == 0 else 3], want):
        a, b = a.float(), b.float()
        assert torch.equal(a[special].isnan(), b[special].isnan()), name
        # the root of a sum in another order: a few units of fp32 in it, and so in what is not rounded further; a step of FP8 (1/8); in 16 bits two roundings, of the normalised
        # value and of its product with the weight, each of which can fall the other way by a step (bf16: 1/128)
        step = 0.0 if name == "residual" else 2.0 ** -20 if name == "scale" or dtype == torch.float32 and quant == 0 else 2.0 ** -3 if quant else 2.0 ** -6
        for rows in (special, rest):
            c, d = a[rows].nan_to_num(7.0), b[rows].nan_to_num(7.0)
            assert bool(((c - d).abs() <= d.abs() * step).all()), name
        assert bool(a[rest].isfinite().all())
