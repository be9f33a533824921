"""f16 chains whose rows TMA cannot take (strides that are no multiple of 16 bytes): padded operand
copies, tensor-core contraction, output rows written from the staging tiles; against the CPU checker,
and against the SIMT kernel, which stays the path of a call without workspace or 16-byte pointers."""
import ctypes as C

import numpy as np
import pytest

from oracle import oracle


def _operands(batch, M, N, K, shared=False, seed=0):
    A = oracle.normal((batch, M, K) if batch > 1 else (M, K), 100 + seed)
    B = oracle.normal((batch, K, N) if batch > 1 and not shared else (K, N), 200 + seed)
    return A, B


def _ref(A, B, scale):
    if A.ndim == 2:
        return oracle.chain(A, B, scale)
    return np.stack([oracle.chain(A[i], B[i] if B.ndim == 3 else B, scale) for i in range(A.shape[0])])


def test_ragged_plans(wtc_lib):
    """Which copies a shape needs; small shapes and rows the SIMT kernel does not take stay as they were."""
    w = wtc_lib
    for (M, N, K), copies, extra in [((1000, 333, 64), "B", 1), ((1000, 328, 61), "A", 1), ((1000, 333, 61), "AB", 1), ((4000, 2305, 64), "B", 1)]:
        p = w.plan_query(w.make_desc(1, M, N, K))
        tiled = N > 2048
        want = 0
        if "A" in copies:
            want += -(-M * (-(-K // 8) * 8) * 2 // 256) * 256
        if "B" in copies:
            want += -(-K * (-(-N // 64) * 64) * 2 // 256) * 256
        if tiled:
            want += M * -(-N // 256) * 8
        assert p.kernel == (w.KERNEL_TC_TILED if tiled else w.KERNEL_TC_CLUSTER)
        assert p.launches == (2 if tiled else 1) + extra and p.workspace_bytes == want
    # padded strides: nothing to copy
    p = w.plan_query(w.make_desc(1, 1000, 333, 64, ldb=336, ldo=336))
    assert p.kernel == w.KERNEL_TC_CLUSTER and p.launches == 1 and p.workspace_bytes == 0
    assert w.plan_query(w.make_desc(1, 100, 70, 64)).kernel == w.KERNEL_SIMT_FUSED
    assert w.plan_query(w.make_desc(1, 1000, 333, 64, flags=w.FLAG_FORCE_SIMT)).kernel == w.KERNEL_SIMT_FUSED
    assert w.plan_query(w.make_desc(1, 500, 60001, 64)).kernel == w.KERNEL_SIMT_FUSED      # refused at launch, as before


def test_padded_rows_of_a_are_read_in_place(wtc_lib):
    """Any K, with rows of A on 16-byte strides: nothing to copy; f32 operands are rounded into such rows, once."""
    w = wtc_lib
    p = w.plan_query(w.make_desc(1, 1000, 1000, 61, lda=64))
    assert (p.kernel, p.launches, p.workspace_bytes) == (w.KERNEL_TC_CLUSTER, 1, 0)
    p = w.plan_query(w.make_desc(1, 1000, 1000, 61, in_dtype=w.F32, flags=w.FLAG_MATMUL_F16))
    same = w.plan_query(w.make_desc(1, 1000, 1000, 64, in_dtype=w.F32, flags=w.FLAG_MATMUL_F16))
    assert p.kernel == w.KERNEL_TC_CLUSTER and p.launches == same.launches == 2
    assert p.workspace_bytes == 1000 * 64 * 2 + -(-61 * 1000 * 2 // 256) * 256


@pytest.mark.gpu
def test_padded_rows_of_a_hide_what_lies_between_them(wtc_lib, cuda_dev):
    """K = 61 in rows of 64: the three elements behind each row are NaN and no part of the sums."""
    import torch
    w = wtc_lib
    M, N, K = 700, 1000, 61
    A, B = _operands(1, M, N, K)
    tA = torch.full((M, 64), float("nan"), device=cuda_dev, dtype=torch.float16)
    tA[:, :K] = torch.from_numpy(A).to(cuda_dev)
    tB = torch.from_numpy(B).to(cuda_dev)
    out = torch.empty((M, N), device=cuda_dev, dtype=torch.float16)
    d = w.make_desc(1, M, N, K, scale=0.1, lda=64)
    assert w.plan_query(d).launches == 1
    assert w.lib().wtc_matmul_softmax_launch(C.byref(d), tA.data_ptr(), tB.data_ptr(), out.data_ptr(), None, 0, w.current_stream_ptr(), None) == 0
    w.check_device_status()
    r = oracle.compare(out.cpu().numpy(), oracle.chain(A, B, 0.1))
    assert r["ok"], r


@pytest.mark.gpu
@pytest.mark.parametrize("N,K,lda", [(1000, 61, 64), (1001, 61, 72), (3001, 65, 72)])
def test_columns_of_a_wider_matrix_as_a(wtc_lib, cuda_dev, N, K, lda):
    """A from the second column of wider rows on, two bytes behind a boundary: copied where the workspace has the room that
    wtc_matmul_softmax_workspace_bytes asks for, and then the bits are those of the same A on its boundary."""
    import torch
    w = wtc_lib
    M = 700
    A, B = _operands(1, M, N, K)
    wide = torch.full((M, lda), float("nan"), device=cuda_dev, dtype=torch.float16)
    wide[:, 1:1 + K] = torch.from_numpy(A).to(cuda_dev)
    tA = torch.full((M, lda), float("nan"), device=cuda_dev, dtype=torch.float16)
    tA[:, :K] = wide[:, 1:1 + K]
    tB = torch.from_numpy(B).to(cuda_dev)
    d = w.make_desc(1, M, N, K, scale=0.1, lda=lda)
    need, planned = w.workspace_bytes(d), w.plan_query(d).workspace_bytes
    assert need == planned + -(-M * ((K + 7) // 8 * 8) * 2 // 256) * 256
    got = []
    for ptr, size in ((tA.data_ptr(), planned), (wide.data_ptr() + 2, need), (wide.data_ptr() + 2, planned)):
        ws = torch.full((size + 256,), 0x7f, device=cuda_dev, dtype=torch.uint8)
        out = torch.empty((M, N), device=cuda_dev, dtype=torch.float16)
        assert w.lib().wtc_matmul_softmax_launch(C.byref(d), ptr, tB.data_ptr(), out.data_ptr(), ws.data_ptr(), size, w.current_stream_ptr(), None) == 0
        w.check_device_status()
        assert bool((ws[size:] == 0x7f).all())
        got.append(out)
    assert torch.equal(got[0], got[1])
    r = oracle.compare(got[2].cpu().numpy(), oracle.chain(A, B, 0.1))      # (the SIMT kernel)
    assert r["ok"], r


@pytest.mark.gpu
@pytest.mark.parametrize("batch,M,N,K,out,kw", [
    (1, 2000, 129, 64, "f16", {}),          # 128-column tiles, one column in the second
    (1, 4000, 127, 33, "f16", {}),          # narrower than a tile, ragged K
    (1, 8200, 255, 63, "f32", {}),          # f32 probabilities, 256-column tile
    (4, 1021, 1021, 64, "f16", {}),
    (24, 1021, 1021, 64, "f16", {}),        # several tiles per CTA
    (24, 700, 1001, 251, "f16", {}),        # the same, ragged K
    (24, 700, 1001, 251, "f16", {"shared": True}),
    (3, 200, 2047, 72, "f32", {}),          # full cluster of eight
    (1, 257, 2049, 64, "f16", {}),          # tiled: one column in the ninth tile
    (2, 300, 3001, 100, "f16", {}),         # tiled, ragged row rescale across tile borders
    (1, 300, 3001, 100, "f32", {}),
    (1, 700, 520, 61, "f16", {}),           # only A is copied: TMA stores
    (1, 700, 1025, 64, "f16", {"acc_dtype": "F16"}),
])
def test_ragged_matches_the_checker(wtc_lib, cuda_dev, batch, M, N, K, out, kw):
    import torch
    w = wtc_lib
    A, B = _operands(batch, M, N, K, kw.get("shared", False))
    tA, tB = torch.from_numpy(A).to(cuda_dev), torch.from_numpy(B).to(cuda_dev)
    acc = getattr(w, kw.get("acc_dtype", "F32"))
    scale = 0.9 / np.sqrt(K)
    odt = w.F16 if out == "f16" else w.F32
    d = w.make_desc(batch, M, N, K, out_dtype=odt, acc_dtype=acc, shared_b=kw.get("shared", False))
    assert w.plan_query(d).kernel in (w.KERNEL_TC_CLUSTER, w.KERNEL_TC_TILED)
    got = w.matmul_softmax(tA, tB, scale, out_dtype=odt, acc_dtype=acc)
    w.check_device_status()
    got = got.cpu().numpy()
    if acc == w.F32:
        r = oracle.compare(got.reshape(-1, N), _ref(A, B, scale).reshape(-1, N))
        assert r["ok"], r
    simt = w.matmul_softmax(tA, tB, scale, out_dtype=odt, acc_dtype=acc, flags=w.FLAG_FORCE_SIMT).cpu().numpy().astype(np.float64)
    # both round the same f32 sums (differing by their order) to the output type: one ulp of it apart (2^-10 relative; twice that is
    # allowed), and with an f16 matmul result one ulp of a logit (2^-10 relative, |logit| < 8) besides
    tol = (2.0 ** -9 if out == "f16" else 2e-5) + (2.0 ** -7 if acc == w.F16 else 0)
    assert (np.abs(got.astype(np.float64) - simt) <= tol * simt + 2.0 ** -23).all()


@pytest.mark.gpu
@pytest.mark.parametrize("batch,M,N,K,rounded", [(1, 300, 3001, 64, False), (2, 257, 2049, 100, False), (1, 16, 4097, 333, False), (1, 700, 2056, 61, False),
                                                 (1, 150, 20001, 72, False), (1, 300, 3001, 251, True), (1, 130, 2304, 67, True)])
def test_long_ragged_rows_round_a_probability_once(wtc_lib, cuda_dev, batch, M, N, K, rounded):
    """f16 probabilities of rows of more than eight column tiles: within half an f16 step of the value in 64 bits, as from the
    SIMT kernel (an f16 value relative to a tile's maximum on the way would cost another half)."""
    import torch
    w = wtc_lib
    gen = torch.Generator(device=cuda_dev)
    gen.manual_seed(N)
    A = torch.randn((batch, M, K) if batch > 1 else (M, K), device=cuda_dev, generator=gen)
    B = torch.randn((batch, K, N) if batch > 1 else (K, N), device=cuda_dev, generator=gen)
    A16, B16 = A.half(), B.half()
    flags = w.FLAG_MATMUL_F16 if rounded else 0
    assert w.plan_query(w.make_desc(batch, M, N, K, w.F32 if rounded else w.F16, w.F16, flags=flags)).kernel == w.KERNEL_TC_TILED
    for scale in (1.0 / K ** 0.5, -0.3):
        P = ((A16.double() @ B16.double()) * scale).softmax(-1)
        got = w.matmul_softmax(A if rounded else A16, B if rounded else B16, scale, out_dtype=w.F16, flags=flags)
        w.check_device_status()
        # half a step of f16 (2^-11 relative, 2^-25 among the subnormals) and the f32 sums of K products below 30
        assert bool((got.double() - P).abs().le((2.0 ** -11 + 2.0 ** -24 * (30 * K ** 0.5 + 16)) * P + 2.0 ** -25).all())


@pytest.mark.gpu
def test_ragged_strided_output_and_neighbours(wtc_lib, cuda_dev):
    """A padded output: the columns between rows, and what lies before and behind, stay untouched; odd row starts."""
    import torch
    w = wtc_lib
    M, N, K = 300, 1021, 64
    A, B = _operands(1, M, N, K)
    tA, tB = torch.from_numpy(A).to(cuda_dev), torch.from_numpy(B).to(cuda_dev)
    for ldo, lead in [(1021, 1), (1023, 0), (1030, 3), (1024, 8)]:
        d = w.make_desc(1, M, N, K, scale=0.1, ldo=ldo)
        buf = torch.full((lead + M * ldo + 64,), 7.0, device=cuda_dev, dtype=torch.float16)
        ws = torch.empty(max(16, w.workspace_bytes(d)), device=cuda_dev, dtype=torch.uint8)
        rc = w.lib().wtc_matmul_softmax_launch(C.byref(d), tA.data_ptr(), tB.data_ptr(), buf.data_ptr() + 2 * lead, ws.data_ptr(), ws.numel(),
                                               w.current_stream_ptr(), None)
        assert rc == 0
        w.check_device_status()
        host = buf.cpu().numpy()
        assert (host[:lead] == 7).all() and (host[lead + M * ldo:] == 7).all()
        rows = host[lead:lead + M * ldo].reshape(M, ldo)
        assert (rows[:, N:] == 7).all()
        r = oracle.compare(rows[:, :N], oracle.chain(A, B, 0.1))
        assert r["ok"], r


@pytest.mark.gpu
def test_ragged_without_workspace_or_alignment(wtc_lib, cuda_dev):
    """A call that brings no workspace, and one whose operands start off a 16-byte boundary, still run."""
    import torch
    w = wtc_lib
    M, N, K = 300, 1021, 64
    A, B = _operands(1, M, N, K)
    ref = oracle.chain(A, B, 0.1)
    tB = torch.from_numpy(B).to(cuda_dev)
    store = torch.empty(M * K + 8, device=cuda_dev, dtype=torch.float16)
    for lead in (0, 1):
        tA = store[lead:lead + M * K].view(M, K)
        tA.copy_(torch.from_numpy(A).to(cuda_dev))
        d = w.make_desc(1, M, N, K, scale=0.1)
        out = torch.empty((M, N), device=cuda_dev, dtype=torch.float16)
        ws = torch.empty(w.workspace_bytes(d), device=cuda_dev, dtype=torch.uint8)
        for ptr, size in ((None, 0), (ws.data_ptr(), ws.numel())):
            out.zero_()
            rc = w.lib().wtc_matmul_softmax_launch(C.byref(d), tA.data_ptr(), tB.data_ptr(), out.data_ptr(), ptr, size, w.current_stream_ptr(), None)
            assert rc == 0
            w.check_device_status()
            r = oracle.compare(out.cpu().numpy(), ref)
            assert r["ok"], (lead, size, r)


@pytest.mark.gpu
def test_rounded_f32_operands_of_ragged_shape(wtc_lib, cuda_dev):
    """f32 arguments truncated to f16, K and N no multiples of 8: the rounded copies have padded rows.  Same contraction
    as the f16 operands' own ragged path, so the same bits."""
    import torch
    w = wtc_lib
    rng = np.random.default_rng(3)
    for batch, M, N, K in ((1, 700, 1001, 251), (3, 300, 333, 100)):
        A = rng.standard_normal((batch, M, K) if batch > 1 else (M, K)).astype(np.float32)
        B = rng.standard_normal((K, N)).astype(np.float32)
        got = w.matmul_softmax(torch.from_numpy(A).to(cuda_dev), torch.from_numpy(B).to(cuda_dev), 0.1, out_dtype=w.F16, flags=w.FLAG_MATMUL_F16)
        w.check_device_status()
        A16, B16 = A.astype(np.float16), B.astype(np.float16)
        same = w.matmul_softmax(torch.from_numpy(A16).to(cuda_dev), torch.from_numpy(B16).to(cuda_dev), 0.1)
        assert torch.equal(got, same)
        r = oracle.compare(got.cpu().numpy().reshape(-1, N), _ref(A16, B16, 0.1).reshape(-1, N))
        assert r["ok"], r


def test_plans_of_few_rows_against_a_wide_matrix(wtc_lib):
    """128-column tiles up to 64 tiles of 256 columns, 256 beyond; a hint or the forced schedule keeps 256."""
    w = wtc_lib
    assert w.plan_query(w.make_desc(1, 16, 4096, 512)).tile_n == 128 and w.plan_query(w.make_desc(1, 16, 16384, 512)).tile_n == 128
    assert w.plan_query(w.make_desc(1, 16, 16640, 512)).tile_n == 256 and w.plan_query(w.make_desc(1, 256, 8200, 512)).tile_n == 256
    assert w.plan_query(w.make_desc(1, 16, 4096, 512, tile_n=256)).tile_n == 256
    assert w.plan_query(w.make_desc(1, 16, 4096, 512, flags=w.FLAG_FORCE_TILED)).tile_n == 256
    p = w.plan_query(w.make_desc(1, 16, 4104, 512))
    assert p.kernel == w.KERNEL_TC_TILED and p.workspace_bytes == 16 * 33 * 8


def test_small_operands_of_long_k_keep_wide_tiles(wtc_lib):
    """Few rows against a wide matrix: 37 to 54 tiles of 256 columns, K beyond 2048 and A of less than 128 KB."""
    w = wtc_lib
    tile = lambda *shape: w.plan_query(w.make_desc(1, *shape)).tile_n
    assert tile(2, 36 * 256 + 8, 2056) == 256 and tile(2, 54 * 256, 2056) == 256 and tile(15, 10240, 4096) == 256
    assert tile(2, 36 * 256, 2056) == 128 and tile(2, 54 * 256 + 8, 2056) == 128
    assert tile(2, 10240, 2048) == 128 and tile(16, 10240, 4096) == 128
    p = w.plan_query(w.make_desc(1, 2, 10240, 4096))
    assert p.workspace_bytes == w.workspace_bytes(w.make_desc(1, 2, 10240, 4096)) == 2 * 40 * 8


def test_pairs_on_request_keep_their_tiles(wtc_lib):
    """WTC_FLAG_PAIR pairs CTAs whenever there are two row blocks: 256-column tiles, whatever the number of tiles."""
    w = wtc_lib
    p = w.plan_query(w.make_desc(1, 256, 4096, 1024, flags=w.FLAG_PAIR))
    assert (p.tile_n, p.stages) == (256, 6) and p.workspace_bytes == 256 * 16 * 8
    assert w.plan_query(w.make_desc(1, 256, 4096, 1024)).tile_n == 128


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,out", [(1, 4096, 520, "f16"), (16, 16384, 64, "f16"), (128, 4104, 1000, "f32"), (129, 4096, 72, "f16"), (40, 4097, 333, "f16")])
def test_few_rows_against_a_wide_matrix(wtc_lib, cuda_dev, M, N, K, out):
    import torch
    w = wtc_lib
    A, B = _operands(1, M, N, K)
    odt = w.F16 if out == "f16" else w.F32
    assert w.plan_query(w.make_desc(1, M, N, K, out_dtype=odt)).tile_n == 128
    got = w.matmul_softmax(torch.from_numpy(A).to(cuda_dev), torch.from_numpy(B).to(cuda_dev), 1 / np.sqrt(K), out_dtype=odt)
    w.check_device_status()
    r = oracle.compare(got.cpu().numpy(), oracle.chain(A, B, 1 / np.sqrt(K)))
    assert r["ok"], r


@pytest.mark.gpu
def test_workspace_sized_for_wide_tiles_still_serves(wtc_lib, cuda_dev):
    import torch
    w = wtc_lib
    M, N, K = 16, 4104, 512
    A, B = _operands(1, M, N, K)
    tA, tB = torch.from_numpy(A).to(cuda_dev), torch.from_numpy(B).to(cuda_dev)
    d = w.make_desc(1, M, N, K, scale=0.04)
    old = M * -(-N // 256) * 8
    assert old < w.workspace_bytes(d)
    ws = torch.empty(old, device=cuda_dev, dtype=torch.uint8)
    out = torch.empty((M, N), device=cuda_dev, dtype=torch.float16)
    assert w.lib().wtc_matmul_softmax_launch(C.byref(d), tA.data_ptr(), tB.data_ptr(), out.data_ptr(), ws.data_ptr(), old, w.current_stream_ptr(), None) == 0
    w.check_device_status()
    r = oracle.compare(out.cpu().numpy(), oracle.chain(A, B, 0.04))
    assert r["ok"], r
    assert w.lib().wtc_matmul_softmax_launch(C.byref(d), tA.data_ptr(), tB.data_ptr(), out.data_ptr(), ws.data_ptr(), old - 8, w.current_stream_ptr(), None) == -3


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,kw", [
    (1000, 333, 64, {}), (1000, 333, 256, {}), (1000, 333, 257, {}), (1000, 333, 320, {}), (700, 1021, 512, {}), (700, 1021, 1023, {}), (300, 3001, 1000, {}),
    (2000, 129, 777, {}), (8200, 1001, 600, {}), (500, 1000, 1001, {}), (400, 3000, 515, {}), (300, 1021, 4001, {}), (700, 1001, 1001, {"rounded": True}),
])
def test_f32_results_of_ragged_chains_are_no_further_off(wtc_lib, cuda_dev, M, N, K, kw):
    """f16 operands, f32 probabilities: the error against 64 bits is at most the SIMT kernel's (the same call with that kernel
    forced), whatever K; sums of more than 256 products are put together from partial ones."""
    import torch
    w = wtc_lib
    flags = w.FLAG_MATMUL_F16 if kw.get("rounded") else 0
    off = {"tc": 0.0, "simt": 0.0}
    for seed in range(3):
        gen = torch.Generator(device=cuda_dev)
        gen.manual_seed(seed)
        A, B = torch.randn(M, K, device=cuda_dev, generator=gen), torch.randn(K, N, device=cuda_dev, generator=gen)
        a, b = (A, B) if flags else (A.half(), B.half())
        scale = 1.0 / K ** 0.5
        P = ((A.half().double() @ B.half().double()) * scale).softmax(-1)
        assert w.plan_query(w.make_desc(1, M, N, K, w.F32 if flags else w.F16, w.F32, flags=flags)).kernel != w.KERNEL_SIMT_FUSED
        for name, extra in (("tc", 0), ("simt", w.FLAG_FORCE_SIMT)):
            got = w.matmul_softmax(a, b, scale, out_dtype=w.F32, flags=flags | extra)
            w.check_device_status()
            off[name] += float((got.double() - P).norm() / P.norm())
    assert off["tc"] <= off["simt"], off


@pytest.mark.gpu
@pytest.mark.parametrize("batch,M,N,K", [(1, 4000, 1021, 601), (6, 500, 1001, 250), (1, 2500, 3001, 65)])
def test_ragged_calls_on_host_buffers(wtc_lib, cuda_dev, batch, M, N, K):
    """Slabs of a ragged call: rows of A and of the output off their 16-byte boundaries, one workspace for all of them."""
    w = wtc_lib
    A, B = _operands(batch, M, N, K)
    for _ in range(2):
        got = w.matmul_softmax_host(A, B, 0.1)
        r = oracle.compare(got.reshape(-1, N), _ref(A, B, 0.1).reshape(-1, N))
        assert r["ok"], r


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,K,kw", [(2000, 1021, 61, {}), (600, 3001, 64, {}), (2000, 1021, 64, {"ldb": 1024})])
def test_operands_ready_with_ragged_rows(wtc_lib, cuda_dev, M, N, K, kw):
    """The loads wait for the call's own copies (if it makes any), the stores for the call before: different operands through
    one workspace into one output, back to back, leave the last call's result."""
    import torch
    w = wtc_lib
    sets = [_operands(1, M, kw.get("ldb", N), K, seed=i) for i in range(5)]
    dev = [(torch.from_numpy(A).to(cuda_dev), torch.from_numpy(B).to(cuda_dev)) for A, B in sets]
    d = w.make_desc(1, M, N, K, scale=0.1, flags=w.FLAG_OPERANDS_READY, **kw)
    ws = torch.empty(max(16, w.workspace_bytes(d)), device=cuda_dev, dtype=torch.uint8)
    out = torch.empty((M, N), device=cuda_dev, dtype=torch.float16)
    torch.cuda.synchronize()
    for _ in range(10):
        for A, B in dev:
            assert w.lib().wtc_matmul_softmax_launch(C.byref(d), A.data_ptr(), B.data_ptr(), out.data_ptr(), ws.data_ptr(), ws.numel(), w.current_stream_ptr(), None) == 0
    w.check_device_status()
    A, B = sets[-1]
    r = oracle.compare(out.cpu().numpy(), oracle.chain(A, np.ascontiguousarray(B[:, :N]), 0.1))
    assert r["ok"], r
