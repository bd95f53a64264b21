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
