"""Performance cases of the package: what a program that uses it has it do, at the sizes it meets.

listed() is the fixed set, draw() gives further cases of the same ranges, prepare() makes a case's inputs on the
GPU (or in pinned host memory for the host-buffer entry point), run() is one pass through the public entry points.

A case is one of
  chain         softmax_row(scale * A @ B) on device tensors, through matmul_softmax() ("call") or through a
                PreparedCall that the program keeps ("prepared")
  row_softmax   softmax over the last dimension of a matrix
  row_variance  the row variance, broadcast along the row
  host          the chain on host arrays (matmul_softmax_host)
"""
import math

import torch

import welder_typical_chain_b200 as wtc

_TYPES = {"f16": torch.float16, "f32": torch.float32}
_CODES = {"f16": wtc.F16, "f32": wtc.F32}
_SIZE = {"f16": 2, "f32": 4}


def _chain(name, M, N, K, batch=1, dtype="f16", out="", entry="call", rounded=False, shared_b=False, scale=None):
    c = {"path": "chain", "entry": entry, "batch": batch, "M": M, "N": N, "K": K, "in": dtype, "out": out or dtype,
         "rounded": rounded, "shared_b": shared_b, "scale": 1.0 / math.sqrt(K) if scale is None else scale}
    return dict(c, name=name) if name else c


def _rows(name, path, rows, N, dtype):
    c = {"path": path, "rows": rows, "N": N, "dtype": dtype}
    return dict(c, name=name) if name else c


def _host(name, M, N, K):
    c = {"path": "host", "M": M, "N": N, "K": K, "scale": 1.0 / math.sqrt(K)}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest: the decomposed f32 chain of the shipped 128 x 128 x 128 input, one call at a time
        _chain("f32_128x128x128", 128, 128, 128, dtype="f32", scale=1.0),
        # the shape of the shipped f16-native input (f16 operands, f32 probabilities), in a program's loop
        _chain("f16_8192x128x64_to_f32", 8192, 128, 64, out="f32", entry="prepared"),
        # the benchmark's default workload, in a program's loop
        _chain("f16_4096x1024x1024", 4096, 1024, 1024, entry="prepared"),
        # the same chain in the decomposed f32 form: f32 operands, sums and probabilities
        _chain("f32_4096x1024x1024", 4096, 1024, 1024, dtype="f32"),
        # f32 arguments that the chain truncates to f16 before the contraction
        _chain("f32_rounded_4096x1024x1024", 4096, 1024, 1024, dtype="f32", out="f16", rounded=True),
        # attention scores: 8 batches x 8 heads, sequences of 2048 (prefill)
        _chain("attention_64x2048x2048x128", 2048, 2048, 128, batch=64),
        # attention scores of sequences as they come: a length that is no multiple of anything
        _chain("attention_ragged_24x1021x1021x64", 1021, 1021, 64, batch=24),
        # vocabulary-wide probabilities of a whole prompt: the largest
        _chain("vocab_8192x32000x4096", 8192, 32000, 4096),
        # the same for one decode step of sixteen sequences
        _chain("decode_16x32000x4096", 16, 32000, 4096),
        # row softmax of given logits, rows of no particular length
        _rows("row_softmax_f16_12288x5003", "row_softmax", 12288, 5003, "f16"),
        # row variance of activations
        _rows("row_variance_f32_16384x8192", "row_variance", 16384, 8192, "f32"),
        # host arrays in, host array out: what the runner and a caller without device buffers do
        _host("host_4096x1024x1024", 4096, 1024, 1024),
    ]


def _spread(rng, lo, hi, multiple=1):
    """A size between lo and hi, spread over its logarithm."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return max(multiple, v // multiple * multiple)


def draw(rng):
    while True:
        what = rng.choice(["f16"] * 6 + ["f16_ragged"] * 2 + ["f32"] * 3 + ["rounded"] * 2 + ["skinny"] * 2 + ["rows"] * 4 + ["host"])
        if what == "rows":
            dtype = rng.choice(["f16", "f32"])
            rows, N = _spread(rng, 64, 65536), _spread(rng, 32, 50000)
            if rng.random() < 0.5:
                N = max(32, N // 8 * 8)
            if 1e5 <= rows * N <= 2.7e8:
                return _rows(None, rng.choice(["row_softmax", "row_softmax", "row_variance"]), rows, N, dtype)
            continue
        if what == "host":
            M, N, K = _spread(rng, 128, 8192), _spread(rng, 128, 2048, 8), _spread(rng, 64, 1024, 8)
            return _host(None, M, N, K)
        entry = rng.choice(["call", "prepared"])
        batch = rng.choice([1, 1, 1, _spread(rng, 2, 64)])
        shared = batch > 1 and rng.random() < 0.25
        if what == "skinny":          # few rows against a wide matrix
            M, N, K = _spread(rng, 1, 128), _spread(rng, 4096, 40000, 8), _spread(rng, 512, 8192, 8)
            if N * K <= 1.4e8:
                return _chain(None, M, N, K, entry=entry)
            continue
        if what == "f16_ragged":      # any length of row and any contraction length
            M, N, K = _spread(rng, 64, 8192), _spread(rng, 32, 4096), rng.choice([_spread(rng, 16, 1024), rng.choice([64, 128])])
            if 1e6 <= batch * M * N * K <= 2e9 and batch * M * N <= 6e7:
                return _chain(None, M, N, K, batch=batch, shared_b=shared, entry=entry, out=rng.choice(["f16", "f16", "f32"]))
            continue
        if what == "f32":
            M, N, K = _spread(rng, 64, 8192), _spread(rng, 32, 4096), _spread(rng, 16, 2048)
            if rng.random() < 0.6:
                N, K = max(32, N // 8 * 8), max(16, K // 8 * 8)
            if 1e6 <= batch * M * N * K <= 4.3e9 and batch * M * N <= 6e7:
                return _chain(None, M, N, K, batch=batch, dtype="f32", shared_b=shared, entry=entry)
            continue
        M, N, K = _spread(rng, 64, 16384), _spread(rng, 64, 32768, 8), _spread(rng, 32, 4096, 8)
        if 1e6 <= batch * M * N * K <= (1e12 if what == "f16" else 1e11) and batch * M * N <= 2.7e8 and batch * K * max(M, N) <= 2.7e8:
            if what == "rounded":
                return _chain(None, M, N, K, batch=batch, dtype="f32", rounded=True, shared_b=shared, entry=entry, out=rng.choice(["f16", "f32"]))
            return _chain(None, M, N, K, batch=batch, shared_b=shared, entry=entry, out=rng.choice(["f16", "f16", "f32"]))


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)

    def normal(shape, dtype, sigma=1.0):
        t = torch.randn(shape, device="cuda", dtype=dtype, generator=gen)
        return t.mul_(sigma) if sigma != 1.0 else t

    if case["path"] in ("row_softmax", "row_variance"):
        dtype = _TYPES[case["dtype"]]
        X = normal((case["rows"], case["N"]), dtype, 2.0)
        return {"fn": getattr(wtc, case["path"]), "X": X, "out": torch.empty_like(X)}
    if case["path"] == "host":
        # pinned host memory, as a program that calls again and again keeps it
        def pinned(t):
            return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t).numpy()
        A = pinned(normal((case["M"], case["K"]), torch.float16))
        B = pinned(normal((case["K"], case["N"]), torch.float16))
        out = torch.empty((case["M"], case["N"]), dtype=torch.float16, pin_memory=True).numpy()
        return {"A": A, "B": B, "scale": case["scale"], "host_out": out}
    b, M, N, K = case["batch"], case["M"], case["N"], case["K"]
    dtype = _TYPES[case["in"]]
    A = normal((b, M, K) if b > 1 else (M, K), dtype)
    B = normal((b, K, N) if b > 1 and not case["shared_b"] else (K, N), dtype)
    flags = wtc.FLAG_MATMUL_F16 if case["rounded"] else 0
    if case["entry"] == "prepared":
        out = torch.empty((*A.shape[:-1], N), device="cuda", dtype=_TYPES[case["out"]])
        return {"prepared": wtc.PreparedCall(A, B, out, case["scale"], flags=flags)}
    return {"A": A, "B": B, "scale": case["scale"], "out_dtype": _CODES[case["out"]], "flags": flags}


def run(state):
    if "prepared" in state:
        call = state["prepared"]
        call.launch(wtc.current_stream_ptr())
        return call.out
    if "fn" in state:
        return state["fn"](state["X"], out=state["out"])
    if "host_out" in state:
        return wtc.matmul_softmax_host(state["A"], state["B"], state["scale"], out=state["host_out"])
    return wtc.matmul_softmax(state["A"], state["B"], state["scale"], out_dtype=state["out_dtype"], flags=state["flags"])


def work(case):
    """Each input read once and each output written once; the contraction's multiply-adds."""
    if case["path"] in ("row_softmax", "row_variance"):
        n = case["rows"] * case["N"]
        return {"bytes": 2 * n * _SIZE[case["dtype"]], "flops": 4 * n}
    M, N, K = case["M"], case["N"], case["K"]
    if case["path"] == "host":
        return {"bytes": 2 * (M * K + K * N + M * N), "flops": 2 * M * N * K}
    b = case["batch"]
    nb = 1 if case["shared_b"] else b
    return {"bytes": _SIZE[case["in"]] * (b * M * K + nb * K * N) + _SIZE[case["out"]] * b * M * N, "flops": 2 * b * M * N * K}


def tolerance(case):
    """About four times what the outputs differ by from the same chain in 64 bits: f16 results 2.1e-4 (rounded once) to 4.1e-4
    (tiles stored relative to their own maximum and rescaled, values in the subnormal range), f32 chains up to 3.3e-6 (the sums
    of long contractions), row chains 2.1e-4 in f16 and 7e-8 in f32."""
    if case["path"] == "host" or case["path"] == "chain" and case["out"] == "f16":
        return {"rel": 1.8e-3, "max": 5e-3}
    if case["path"] == "chain":
        return {"rel": 1.2e-5, "max": 5e-5}
    return {"rel": 8e-4, "max": 2e-3} if case["dtype"] == "f16" else {"rel": 3e-7, "max": 3e-6}
