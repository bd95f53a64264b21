"""What a program that uses gpuk_b200 has it do on one GPU, as a list of cases and as ranges to draw more from.

Three kinds of work, each through the entry points that a program calls:

* ``epilogue``  ``GPUKDistEnv.allreduce_add_rms_fused`` (``_host`` for results in host memory) in a group of one: residual add, RMSNorm
  and FP8 quantisation behind a row-parallel projection.
* ``linear``    ``gpuk_b200.fp8_linear``: the projection that consumes the FP8 rows of a decode batch.
* ``decoder``   ``TPDecoder.forward``: a decode step on a filled KV cache, or the prefill of empty ones, down to the logits.

Sizes come from the benchmark's configurations (``gpuk_b200/workloads.py``, ``bench.py``) and from the tests' shape lists.  The exchange between
GPUs is not here: it needs several of them, and its emulation inside one GPU is a test and no work of a user.
"""
import math

import torch
import torch.distributed as dist

import gpuk_b200 as gpuk
from gpuk_b200.tp_model import DecoderArgs, TPDecoder

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}
QUANT_NONE, QUANT_240, QUANT_FNUZ, QUANT_448, QUANT_STATIC = range(5)
EPS = 1e-6
STATIC_SCALE = 0.05
STREAM_RMS = 8.0

# the decoder of the benchmark (64 / 8 heads of 128, four layers) and the small one of the tests
LARGE = {"dim": 8192, "layers": 4, "heads": 64, "kv_heads": 8, "ffn": 28672, "vocab": 32768}
SMALL = {"dim": 2048, "layers": 2, "heads": 16, "kv_heads": 4, "ffn": 4096, "vocab": 1024}


def _epilogue(rows, hidden, dtype="bf16", quant=QUANT_448, outliers=False, host=False):
    return {"kind": "epilogue", "rows": rows, "hidden": hidden, "dtype": dtype, "quant": quant, "outliers": outliers, "host": host}


def _linear(tokens, n, k, packed=True):
    return {"kind": "linear", "tokens": tokens, "n": n, "k": k, "packed": packed}


def _decoder(model, batch, new, past, fp8=True):
    return dict(model, kind="decoder", batch=batch, new=new, past=past, fp8=fp8)


def listed():
    return [
        # eight decode tokens with a calibrated per-tensor scale: the smallest call, launch and host latency
        dict(_epilogue(8, 8192, quant=QUANT_STATIC), name="epilogue decode static"),
        # a ragged fp32 batch with the reference's own saturation value
        dict(_epilogue(129, 1024, dtype="f32", quant=QUANT_240), name="epilogue f32 ragged"),
        # a mixed prefill / decode batch, the benchmark's headline message
        dict(_epilogue(1024, 8192), name="epilogue mid"),
        # an odd number of fp16 rows whose norm stays in fp16 (the consumer is a 16-bit GEMM)
        dict(_epilogue(2501, 7168, dtype="f16", quant=QUANT_NONE), name="epilogue f16 plain"),
        # a long prefill with activation outliers: the largest message
        dict(_epilogue(16384, 7168, outliers=True), name="epilogue prefill"),
        # activations that live in pinned host memory, results wanted there
        dict(_epilogue(1024, 8192, host=True), name="epilogue host buffers"),
        # q|k|v of one of eight ranks, eight sequences
        dict(_linear(8, 1280, 8192), name="linear qkv shard"),
        # vocabulary shard for a ragged batch, weights as they come from a checkpoint (row-major)
        dict(_linear(13, 4096, 8192, packed=False), name="linear vocab row-major"),
        # w1|w3 of one of eight ranks at the full decode batch
        dict(_linear(32, 7168, 8192), name="linear ffn shard"),
        # one token for each of four sequences, small model in bf16: an interactive session
        dict(_decoder(SMALL, batch=4, new=1, past=128, fp8=False), name="decoder step small"),
        # one token for each of 32 sequences at context 2048: a loaded server
        dict(_decoder(LARGE, batch=32, new=1, past=2048), name="decoder step"),
        # a prompt of that length
        dict(_decoder(LARGE, batch=1, new=2048, past=0), name="decoder prefill"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("epilogue", "epilogue", "linear", "decoder"))
    if kind == "epilogue":
        dtype = rng.choice(("bf16", "bf16", "bf16", "f16", "f32"))
        hidden = rng.choice((1024, 2048, 4096, 5120, 7168, 8192, 8 * rng.randint(128, 1024)))
        if rng.random() < 0.15:
            return _epilogue(_log_int(rng, 16, 1024), hidden, host=True)
        # never more bytes than the largest listed message
        most = 16384 * 7168 * 2 // (hidden * (4 if dtype == "f32" else 2))
        return _epilogue(_log_int(rng, 1, min(16384, most)), hidden, dtype, rng.choice((QUANT_448, QUANT_448, QUANT_STATIC, QUANT_240, QUANT_FNUZ, QUANT_NONE)),
                         outliers=rng.random() < 0.3)
    if kind == "linear":
        return _linear(rng.randint(1, 32), 128 * _log_int(rng, 1, 56), 64 * _log_int(rng, 16, 128), packed=rng.random() < 0.7)
    heads = rng.choice((8, 16, 32, 64))
    model = {"dim": 128 * heads, "layers": rng.randint(1, 4), "heads": heads, "kv_heads": heads // rng.choice((4, 8)),
             "ffn": 128 * rng.randint(2 * heads, 3 * heads + heads // 2), "vocab": 128 * rng.randint(8, 256)}
    fp8 = rng.random() < 0.75
    if rng.random() < 0.65:
        return _decoder(model, batch=rng.randint(1, 32), new=1, past=_log_int(rng, 16, 2048), fp8=fp8)
    batch = rng.choice((1, 1, 2, 4))
    return _decoder(model, batch=batch, new=_log_int(rng, 8, 2048 // batch), past=0, fp8=fp8)


# ---------------------------------------------------------------------------------------
def _env():
    """The handle on a group of one that every fused call goes through."""
    if not dist.is_initialized():
        dist.init_process_group("gloo", store=dist.HashStore(), rank=0, world_size=1)
    return gpuk.GPUKDistEnv(group=None, device_id=torch.cuda.current_device())


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)


def _prepare_epilogue(case, seed):
    g, dtype = _generator(seed), DTYPES[case["dtype"]]
    rows, hidden = case["rows"], case["hidden"]
    x = _randn(g, rows, hidden)
    if case["outliers"]:      # one value in a thousand twenty times as large
        mask = torch.rand(rows, hidden, generator=g, device="cuda") < 0.001
        x = torch.where(mask, x * 20.0, x)
    state = {"case": case, "env": _env(), "x": x.to(dtype), "residual": _randn(g, rows, hidden).to(dtype),
             "weight": (1.0 + 0.1 * _randn(g, hidden)).to(dtype),
             "static_scale": torch.full((1,), STATIC_SCALE, device="cuda") if case["quant"] == QUANT_STATIC else None}
    if case["host"]:
        state["x"], state["residual"] = state["x"].cpu().pin_memory(), state["residual"].cpu().pin_memory()
        state["out"] = (torch.empty(rows, hidden, dtype=dtype, pin_memory=True), torch.empty(rows, hidden, dtype=torch.float8_e4m3fn, pin_memory=True),
                        torch.empty(rows, 1, dtype=torch.float32, pin_memory=True))
    return state


def _prepare_linear(case, seed):
    g = _generator(seed)
    tokens, n, k = case["tokens"], case["n"], case["k"]

    def quantised(rows):
        v = _randn(g, rows, k)
        amax = v.abs().amax(dim=1, keepdim=True)
        return (v / amax * 448.0).to(torch.float8_e4m3fn), amax / 448.0
    x, x_scale = quantised(tokens)
    w, w_scale = quantised(n)
    return {"case": case, "x": x, "x_scale": x_scale, "w": gpuk.fp8_pack_weight(w) if case["packed"] else w, "w_scale": w_scale.t().contiguous()}


def _prepare_decoder(case, seed):
    args = DecoderArgs(dim=case["dim"], n_layers=case["layers"], n_heads=case["heads"], n_kv_heads=case["kv_heads"], ffn_dim=case["ffn"],
                       vocab_size=case["vocab"], max_seq_len=(case["past"] + case["new"] + 255) // 256 * 256)
    seed %= 1 << 24
    env = _env()
    model = TPDecoder(args, env, device=torch.device("cuda", torch.cuda.current_device()), fp8=case["fp8"], seed=seed, max_batch=case["batch"])
    # in a trained model the residual stream is many times what one layer adds to it; the random layers here add about a quarter
    model.tok_embeddings.mul_(STREAM_RMS / math.sqrt(2.0 / (case["vocab"] + case["dim"])))
    if case["past"]:
        model.fill_kv_cache(case["past"], seed=seed + 1)
    tokens = torch.randint(0, case["vocab"], (case["batch"], case["new"]), generator=_generator(seed), device="cuda")
    return {"case": case, "model": model, "tokens": tokens, "pos": torch.arange(case["past"], case["past"] + case["new"], device="cuda")}


def prepare(case, seed):
    return {"epilogue": _prepare_epilogue, "linear": _prepare_linear, "decoder": _prepare_decoder}[case["kind"]](case, seed)


def run(state):
    case = state["case"]
    if case["kind"] == "linear":
        return gpuk.fp8_linear(state["x"], state["x_scale"], state["w"], state["w_scale"], packed=case["packed"])
    if case["kind"] == "decoder":
        model = state["model"]
        logits = model.forward(state["tokens"], state["pos"], cache_len=case["past"] + case["new"])
        return {"logits": logits, "k": [layer["k_cache"] for layer in model.layers], "v": [layer["v_cache"] for layer in model.layers]}
    if case["host"]:
        return state["env"].allreduce_add_rms_fused_host(state["x"], state["residual"], state["weight"], EPS, state["out"], quant_type=case["quant"])
    quant = case["quant"]
    residual_out, norm_out, scale = state["env"].allreduce_add_rms_fused(
        state["x"], state["residual"], state["weight"], EPS, quant != QUANT_NONE, static_scale=state["static_scale"],
        quant_type=quant if quant in (QUANT_240, QUANT_FNUZ, QUANT_448) else None)
    # without quantisation there are no scales, and a static one is an input
    return (residual_out, norm_out, scale) if quant in (QUANT_240, QUANT_FNUZ, QUANT_448) else (residual_out, norm_out)


# ---------------------------------------------------------------------------------------
def work(case):
    if case["kind"] == "epilogue":
        rows, hidden = case["rows"], case["hidden"]
        es = 4 if case["dtype"] == "f32" else 2
        out = es if case["quant"] == QUANT_NONE else 1
        scales = 4 * rows if case["quant"] in (QUANT_240, QUANT_FNUZ, QUANT_448) else 0
        # about ten operations an element: add, square and sum, two multiplications, maximum, division
        return {"bytes": rows * hidden * (3 * es + out) + hidden * es + scales, "flops": 10 * rows * hidden}
    if case["kind"] == "linear":
        m, n, k = case["tokens"], case["n"], case["k"]
        return {"bytes": n * k + m * k + 2 * m * n + 4 * (m + n), "flops": 2 * m * n * k}
    rows, total = case["batch"] * case["new"], case["past"] + case["new"]
    dim, hd = case["dim"], case["dim"] // case["heads"]
    kv = case["kv_heads"] * hd
    column = (dim + 2 * kv) * dim + 2 * case["ffn"] * dim            # q|k|v and w1|w3: FP8 weights when the activations are
    row = dim * dim + dim * case["ffn"]                              # wo and w2
    w8 = 1 if case["fp8"] else 2
    cache = 2 * 2 * case["batch"] * kv * (total if case["past"] else 2 * case["new"])      # keys and values: read, and the new ones written
    # a new token attends to what is before it
    scores = case["batch"] * (case["new"] * case["past"] + case["new"] * (case["new"] + 1) // 2)
    return {"bytes": case["layers"] * (column * w8 + 2 * row + cache) + case["vocab"] * dim * w8 + 2 * rows * (dim + case["vocab"]),
            "flops": case["layers"] * (2 * rows * (column + row) + 4 * scores * case["heads"] * hd) + 2 * rows * case["vocab"] * dim}


def tolerance(case):
    """About four times what the path differs from itself by with its sums in another order or in wider types."""
    if case["kind"] == "epilogue":
        if case["quant"] != QUANT_NONE:      # one FP8 step in up to one value in a thousand: 2.4e-3
            return {"rel": 0.01, "max": 0.13}
        # one unit in the last place where the reciprocal root of the sum of squares rounds the other way
        return {"rel": 1e-6, "max": 1e-5} if case["dtype"] == "f32" else {"rel": 1e-4, "max": 0.01}
    if case["kind"] == "linear":             # fp32 sums, rounded once to bf16: 6e-5
        return {"rel": 3e-4, "max": 0.016}
    # bf16 roundings between the operators (3e-3), and FP8 codes that flip with them (up to 1.6e-2 in the logits)
    return {"rel": 0.03, "max": 0.5} if case["fp8"] else {"rel": 0.012, "max": 0.06}
