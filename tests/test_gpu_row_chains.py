"""The two chains without a matmul (row softmax of a given matrix; row variance broadcast
along the row), through the C ABI against the CPU checker, and through the backend tools
(welder-compiler -> welder-profiler -> verify.py) on the inputs the package ships."""
import os
import subprocess
import sys

import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "welder_typical_chain_b200")
BK = os.path.join(PKG, "backend", "welder", "compiler", "build")


@pytest.mark.parametrize("shape", [(32, 256), (1, 8), (7, 24), (300, 1000), (64, 1024), (5, 2048), (33, 2056), (3, 32000), (2, 4, 520)])
@pytest.mark.parametrize("dtype", ["f32", "f16"])
def test_row_softmax_matches_the_checker(wtc_lib, cuda_dev, shape, dtype):
    import torch
    w = wtc_lib
    rng = np.random.default_rng(sum(shape))
    X = (rng.standard_normal(shape) * 3).astype(np.float16 if dtype == "f16" else np.float32)
    X.reshape(-1, shape[-1])[0, 0] = 11.0                         # one dominant entry
    out = w.row_softmax(torch.from_numpy(X).to(cuda_dev))
    torch.cuda.synchronize()
    got = out.cpu().numpy().reshape(-1, shape[-1])
    res = oracle.compare(got, oracle.row_softmax(X).reshape(-1, shape[-1]))
    assert res["ok"], res
    if dtype == "f32":
        assert np.abs(got.astype(np.float64) - oracle.row_softmax(X).reshape(-1, shape[-1])).max() < 2e-6


@pytest.mark.parametrize("shape", [(32, 256), (1, 8), (7, 24), (300, 1000), (5, 2048), (33, 2056), (3, 32000)])
def test_row_variance_matches_the_checker(wtc_lib, cuda_dev, shape):
    import torch
    w = wtc_lib
    rng = np.random.default_rng(sum(shape) + 1)
    A = (rng.standard_normal(shape) * 2 + 0.5).astype(np.float32)
    out = w.row_variance(torch.from_numpy(A).to(cuda_dev))
    torch.cuda.synchronize()
    ref = oracle.row_variance(A)
    assert np.abs(out.cpu().numpy().astype(np.float64) - ref).max() <= 1e-4 * np.abs(ref).max()
    # other constants than 1/N, f16 elements
    out = w.row_variance(torch.from_numpy(A).to(cuda_dev), mean_factor=0.5 / shape[-1], var_factor=2.0)
    ref = oracle.row_variance(A, 0.5 / shape[-1], 2.0)
    assert np.abs(out.cpu().numpy().astype(np.float64) - ref).max() <= 1e-4 * np.abs(ref).max()
    A16 = A.astype(np.float16)
    out = w.row_variance(torch.from_numpy(A16).to(cuda_dev))
    torch.cuda.synchronize()
    ref = oracle.row_variance(A16)
    assert np.abs(out.cpu().numpy().astype(np.float64) - ref).max() <= 2e-3 * np.abs(ref).max()


def test_row_chain_descriptor_errors_and_empty(wtc_lib, cuda_dev):
    import ctypes as C
    w = wtc_lib
    L = w.lib()
    d = w.RowChainDesc()
    d.struct_size = C.sizeof(w.RowChainDesc)
    d.kind, d.rows, d.N, d.dtype = 7, 4, 4, w.F32
    one = C.c_void_p(256)
    assert L.wtc_row_chain_launch(C.byref(d), one, one, None) == -1 and b"kind" in L.wtc_last_error()
    d.kind, d.rows = w.ROW_SOFTMAX, 0
    assert L.wtc_row_chain_launch(C.byref(d), None, None, None) == 0        # nothing to do
    d.rows, d.ld_in = 4, 2
    assert L.wtc_row_chain_launch(C.byref(d), one, one, None) == -1 and b"stride" in L.wtc_last_error()


@pytest.mark.parametrize("name", ["softmax_row_chain.mlir", "layernorm_variance_chain.mlir"])
@pytest.mark.parametrize("init", ["linear", "random"])
def test_backend_tools_run_and_verify_the_row_chains(tmp_path, name, init):
    out = tmp_path / "c"
    tiles = ["--force-tile-m", "32", "--force-tile-n", "64", "--force-tile-k", "16", "--thread-tile-m", "2", "--thread-tile-n", "2"]
    r = subprocess.run([os.path.join(BK, "welder-compiler"), os.path.join(PKG, "mlir", name), *tiles, "--emit-all-stages", "--output",
                        str(out / "03.after_postbufferize.mlir")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    plan = str(out / "05.out.nvvm.runnable.mlir")
    dump = str(tmp_path / "out.bin")
    r = subprocess.run([os.path.join(BK, "welder-profiler"), plan, "--warmup", "2", "--iters", "5", f"--init={init}", "--seed", "3", "--dump-last-2d", dump],
                       capture_output=True, text=True)
    assert r.returncode == 0 and "avg_ms=" in r.stdout, r.stderr
    v = subprocess.run([sys.executable, os.path.join(PKG, "bench", "verify.py"), "--out", dump, "--plan", plan, "--pattern", init, "--seed", "3",
                        "--rows", "0,1,2,3,7,15,31", "--rtol", "1e-5", "--atol", "1e-7"], capture_output=True, text=True)
    assert v.returncode == 0 and v.stdout.startswith("PASS"), v.stdout + v.stderr


@pytest.mark.parametrize("dtype", ["f32", "f16"])
@pytest.mark.parametrize("rows,N,ld,lead", [
    (70, 1, 1, 0), (9, 7, 7, 3), (33, 31, 31, 1), (40, 63, 63, 0), (40, 65, 65, 5), (5, 127, 131, 2), (9, 257, 257, 0), (13, 1021, 1021, 7), (3, 2047, 2047, 0),
    (3, 2049, 2049, 1), (7, 5003, 5003, 0), (3, 16383, 16383, 4), (2, 32767, 32767, 0), (3, 32769, 32769, 1), (2, 40000, 40000, 0),
    (2, 65537, 65537, 0), (2, 150001, 150001, 3), (2, 300007, 300007, 0),
])
def test_row_chains_of_any_length_start_and_stride(wtc_lib, cuda_dev, rows, N, ld, lead, dtype):
    """Rows that start anywhere: the element-wise ends, the short-row groups, one CTA, a cluster, and rows longer than a
    cluster holds; input and output equally far from a 16-byte boundary, and not.  Nothing outside the rows is written."""
    import ctypes as C
    import torch
    w = wtc_lib
    rng = np.random.default_rng(rows + N)
    t = torch.float16 if dtype == "f16" else torch.float32
    X = (rng.standard_normal((rows, N)) * 2 + 0.5).astype(np.float16 if dtype == "f16" else np.float32)
    src = torch.full((lead + rows * ld + 32,), 9.0, device=cuda_dev, dtype=t)
    src[lead:lead + rows * ld].view(rows, ld)[:, :N] = torch.from_numpy(X).to(cuda_dev)
    x64 = X.astype(np.float64)
    e = np.exp(x64 - x64.max(axis=1, keepdims=True))
    soft = e / e.sum(axis=1, keepdims=True)
    var = np.repeat(((x64 - x64.mean(axis=1, keepdims=True)) ** 2).mean(axis=1, keepdims=True), N, axis=1)
    for kind, ref in ((w.ROW_SOFTMAX, soft), (w.ROW_VARIANCE, var)):
        for off in (lead, lead + 1):
            out = torch.full((off + rows * ld + 32,), 9.0, device=cuda_dev, dtype=t)
            d = w.RowChainDesc()
            d.struct_size = C.sizeof(w.RowChainDesc)
            d.kind, d.rows, d.N, d.ld_in, d.ld_out, d.dtype = kind, rows, N, ld, ld, w.F16 if dtype == "f16" else w.F32
            d.mean_factor = d.var_factor = 1.0 / N
            es = 2 if dtype == "f16" else 4
            assert w.lib().wtc_row_chain_launch(C.byref(d), src.data_ptr() + lead * es, out.data_ptr() + off * es, w.current_stream_ptr()) == 0
            torch.cuda.synchronize()
            host = out.cpu().numpy().astype(np.float64)
            assert (host[:off] == 9).all() and (host[off + rows * ld:] == 9).all()
            got = host[off:off + rows * ld].reshape(rows, ld)
            assert (got[:, N:] == 9).all()
            # f16: the result's own rounding (2^-11, or half a subnormal step); f32: the exponent's rounding (2^-24 * |x - max| * log2 e
            # < 2^-19.5 for |x - max| < 18) and the sums
            tol = 2.0 ** -10 * np.abs(ref) + 2.0 ** -25 if dtype == "f16" else 4e-6 * np.abs(ref)
            assert (np.abs(got[:, :N] - ref) <= tol).all(), (kind, off)


def test_row_softmax_in_place_and_at_the_limits(wtc_lib, cuda_dev):
    import torch
    w = wtc_lib
    for N in (61, 1021, 5003, 40000, 40001):
        X = torch.randn((9, N), device=cuda_dev)
        X[0] = torch.finfo(torch.float32).min                                   # a row of the type's lowest value: uniform
        X[1, 5] = -float("inf")
        X[2, 3] = float("nan")
        X[3] = torch.finfo(torch.float32).min
        X[3, 1] = 0.0
        ref = torch.softmax(X.double(), dim=-1)
        out = w.row_softmax(X, out=X)
        assert out is X
        for r in (0, 1, 3, 4, 8):
            assert torch.allclose(out[r].double(), ref[r], rtol=4e-6, atol=0), (N, r)
        assert torch.isnan(out[2]).all()


@pytest.mark.gpu
def test_more_short_rows_than_a_cluster_grid_could_hold(wtc_lib, cuda_dev):
    """2^28 and a few rows of eight elements: more than an eighth of the largest grid, and still several rows a warp (a CTA a
    row would take a hundred times as long as the traffic)."""
    import torch
    w = wtc_lib
    rows, N = (1 << 28) + 5, 8
    X = torch.zeros(rows, N, device=cuda_dev, dtype=torch.float16)
    for piece in X.split(1 << 24):
        piece.normal_()
    out = torch.empty_like(X)
    w.row_softmax(X, out=out)
    torch.cuda.synchronize()
    for at in (0, rows // 2, rows - 1000):
        P = X[at:at + 1000].double().softmax(-1)
        assert bool((out[at:at + 1000].double() - P).abs().le(2.0 ** -11 * P + 2.0 ** -24).all())
    start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    start.record()
    w.row_softmax(X, out=out)
    end.record()
    torch.cuda.synchronize()
    assert start.elapsed_time(end) < 10 * 2 * X.numel() * 2 / 6e9       # ten times what 6 TB/s take


@pytest.mark.parametrize("N", [64, 61, 1024, 4096, 5000, 5003, 16384, 32000, 40000])
def test_f32_row_softmax_far_from_zero(wtc_lib, cuda_dev, N):
    """Equal values of any size give equal probabilities, values of 1e9 and more one-hot rows, whatever the alignment."""
    import torch
    w = wtc_lib
    for value in (torch.finfo(torch.float32).min, torch.finfo(torch.float32).max, 3e38, 1e10, -1e10, 1e7):
        out = w.row_softmax(torch.full((5, N), value, device=cuda_dev))
        assert bool((out.double() * N - 1).abs().le(2.0 ** -20).all()), value
    X = torch.randn((9, N), device=cuda_dev) * 3e9          # neighbouring f32 values lie 64 and more apart here
    want = torch.softmax(X.double(), -1)
    assert bool((w.row_softmax(X).double() - want).abs().le(2.0 ** -22).all())
