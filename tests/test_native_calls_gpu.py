"""The direct calls behind allreduce_add_rms_fused and fp8_linear: the same results as the operator, and the operator where it is wanted."""
import pytest
import torch

import gpuk_b200 as gpuk
from gpuk_b200 import _native


@pytest.fixture
def env():
    import torch.distributed as dist
    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    return gpuk.GPUKDistEnv(group=None, device_id=0)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("quant", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("shape", [(1, 1024), (7, 1032), (2, 3, 2048)])
def test_same_as_the_operator(env, shape, quant, dtype):
    x, r = torch.randn(shape, device="cuda").to(dtype), torch.randn(shape, device="cuda").to(dtype)
    w = torch.randn(shape[-1], device="cuda").to(dtype)
    static = torch.full((1,), 0.05, device="cuda") if quant == 4 else None
    rows = x.numel() // shape[-1]

    def call():
        return env.allreduce_add_rms_fused(x, r, w, 1e-6, quant != 0, static_scale=static, quant_type=quant if quant in (1, 2, 3) else None)
    if len(shape) == 3 and quant in (1, 2, 3):       # one scale a row of the first dimension does not do
        with pytest.raises(RuntimeError, match="scale_out has"):
            call()
        return
    got = call()
    want = (torch.empty_like(r), torch.empty_like(x, dtype=got[1].dtype), static if static is not None else torch.empty(max(rows, 1), 1, device="cuda"))
    gpuk.allreduce_rms(0, x, r, w, *want, 1e-6, quant)
    assert got[0].shape == r.shape and got[1].shape == x.shape
    assert torch.equal(got[0], want[0]) and torch.equal(got[1].view(torch.uint8), want[1].view(torch.uint8))
    if quant in (1, 2, 3):
        assert torch.equal(got[2], want[2])
    if quant == 4:
        assert got[2].data_ptr() == static.data_ptr()


@pytest.mark.gpu
def test_policies_that_do_not_go_together_are_refused(env):
    x, w = torch.randn(4, 1024, device="cuda"), torch.ones(1024, device="cuda")
    for policy in (0, 7, -1):
        with pytest.raises(RuntimeError):
            env.allreduce_add_rms_fused(x, x, w, 1e-6, True, quant_type=policy)
    assert env.allreduce_add_rms_fused(x, x, w, 1e-6, False, quant_type=3)[1].dtype == x.dtype


@pytest.mark.gpu
def test_what_is_not_plain_takes_the_operator(env):
    class Sub(torch.Tensor):
        pass
    x, w = torch.randn(4, 1024, device="cuda"), torch.ones(1024, device="cuda")
    call = lambda a, b=x, c=w, q=0, s=None: _native.add_rms(0, a, b, c, 1e-6, q, s)      # noqa: E731
    assert call(x) is not None
    assert call(x.as_subclass(Sub)) is None and call(x, x.t().contiguous().t()) is None and call(x, x.half()) is None
    assert call(x, x.cpu()) is None and call(x, x, w[:512]) is None and call(x, x, w, 9) is None and call(x, x, w, 4) is None
    assert call(x.double(), x.double(), w.double()) is None and call(x[:0], x[:0]) is None
    assert torch.func.vmap(lambda a: torch.zeros(()) if call(a) is None else torch.ones(()))(torch.stack([x, x])).sum() == 0
    seen = []

    class Mode(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))
    with Mode():
        env.allreduce_add_rms_fused(x, x, w, 1e-6)
    assert any("allreduce_rms" in f for f in seen)


@pytest.mark.gpu
def test_fp8_linear_refuses_before_any_launch():
    e = torch.float8_e4m3fn
    x, w, s, c = (torch.zeros(8, 64, device="cuda").to(e), torch.zeros(128, 64, device="cuda").to(e), torch.ones(8, device="cuda"), torch.ones(128, device="cuda"))
    assert gpuk.fp8_linear(x, s, w, c).shape == (8, 128)
    for args in ((x, s[:7], w, c), (x, s, w, c[:127]), (x, s.double(), w, c), (x, s, w.t(), c), (x, s.cpu(), w, c), (x, s, w.cpu(), c)):
        with pytest.raises(RuntimeError):
            gpuk.fp8_linear(*args)
    for out in (torch.empty(8, 128, device="cuda"), torch.empty(8, 127, device="cuda").bfloat16(), torch.empty(8, 128).bfloat16()):
        with pytest.raises(RuntimeError, match="bf16"):
            gpuk.fp8_linear(x, s, w, c, out)
    with pytest.raises(RuntimeError, match="k_split"):
        gpuk.fp8_linear(x, s, w, c, k_split=3)


@pytest.mark.gpu
@pytest.mark.parametrize("m", [8, 20])
def test_fp8_linear_takes_pinned_host_memory(m):
    """Scales, weights and results that the GPU reaches over the link."""
    g = torch.Generator().manual_seed(m)
    x, w = (torch.randn(m, 256, generator=g) * 50).to(torch.float8_e4m3fn).cuda(), (torch.randn(128, 256, generator=g) * 50).to(torch.float8_e4m3fn)
    s, c = torch.rand(m, generator=g), torch.rand(128, generator=g)
    want = gpuk.fp8_linear(x, s.cuda(), w.cuda(), c.cuda())
    out = torch.zeros(m, 128, dtype=torch.bfloat16).pin_memory()
    assert gpuk.fp8_linear(x, s.pin_memory(), w.pin_memory(), c.pin_memory(), out) is not None
    torch.cuda.synchronize()
    assert torch.equal(out, want.cpu())
