"""The register-tiled f32 chain: sums in ascending k like the row kernel's, so the logits are the same bits and the
probabilities differ by the order of the row sum alone."""
import numpy as np
import pytest

from oracle import oracle


def test_launch_counts(wtc_lib):
    """Rows of more than eight column tiles take a second launch; small chains keep the row kernel."""
    w = wtc_lib
    assert w.plan_query(w.make_desc(1, 4096, 1024, 1024, w.F32, w.F32)).launches == 1
    assert w.plan_query(w.make_desc(1, 4096, 4096, 256, w.F32, w.F32)).launches == 2
    assert w.plan_query(w.make_desc(1, 128, 128, 128, w.F32, w.F32)).launches == 1


def test_plans_describe_the_tile_kernel(wtc_lib):
    """Tile, threads, stages, shared memory, cluster and launches of the kernel that runs, not of the row kernel."""
    w = wtc_lib

    def fields(*shape, **kw):
        p = w.plan_query(w.make_desc(*shape, w.F32, w.F32, **kw))
        return p.tile_m, p.tile_n, p.tile_k, p.cluster_n, p.threads, p.stages, p.launches

    assert fields(1, 4096, 1024, 1024) == (128, 256, 16, 4, 256, 4, 1)
    p = w.plan_query(w.make_desc(1, 4096, 1024, 1024, w.F32, w.F32))
    assert p.smem_bytes == 4 * (4 * 16 * (132 + 256) + (4 + 16 + 2) * 128)       # four stages of A (padded rows) and B, the row statistics
    assert fields(1, 300, 4096, 1024)[3] == 1 and fields(1, 300, 4096, 1024)[6] == 2
    assert fields(1, 128, 128, 128) == (16, 128, 64, 1, 256, 0, 1)
    # batches whose rows do not follow one another: a row softmax each
    d = w.make_desc(3, 300, 4096, 256, w.F32, w.F32)
    assert w.plan_query(d).launches == 2
    d.o_batch_stride = 301 * 4096
    assert w.plan_query(d).launches == 4
    # so many rows that the last tile's would not fit 32 bits
    assert fields(1, 2 ** 31 - 127, 1, 1)[5] == 0 and fields(1, 2 ** 31 - 129, 1, 1)[5] > 0
    # f16 output: rows of more than eight tiles stay with the row kernel
    assert w.plan_query(w.make_desc(1, 300, 4096, 1024, w.F32, w.F16)).stages == 0


@pytest.mark.gpu
@pytest.mark.parametrize("batch,M,N,K,shared", [
    (1, 4096, 1024, 96, False),      # 128 x 256 tiles, clusters of four
    (1, 129, 257, 1001, False),      # one row and one column past a tile, element-wise copies, ragged K
    (1, 1000, 2048, 17, False),      # a full cluster of eight, a K tail of one
    (1, 300, 2049, 64, False),       # logits in the output, then the row softmax in place
    (1, 64, 4096, 333, False),
    (3, 200, 1030, 50, True),        # 64-row or 128-column tiles, B shared, rows no multiple of 16 bytes
    (5, 333, 333, 333, False),
    (2, 64, 3001, 50, False),
    (64, 70, 40, 100, False),         # narrower than a tile
])
def test_f32_tiles_match_the_checker(wtc_lib, cuda_dev, batch, M, N, K, shared):
    import torch
    w = wtc_lib
    assert batch * M * N * K >= 1 << 23
    rng = np.random.default_rng(M + N + K)
    A = rng.standard_normal((batch, M, K) if batch > 1 else (M, K)).astype(np.float32)
    B = rng.standard_normal((batch, K, N) if batch > 1 and not shared else (K, N)).astype(np.float32)
    scale = 2.0 / np.sqrt(K)
    got = w.matmul_softmax(torch.from_numpy(A).to(cuda_dev), torch.from_numpy(B).to(cuda_dev), scale)
    torch.cuda.synchronize()
    got = got.cpu().numpy().reshape(-1, N).astype(np.float64)
    L = scale * np.matmul(A.astype(np.float64), B.astype(np.float64)).reshape(-1, N)
    E = np.exp(L - L.max(axis=1, keepdims=True))
    P = E / E.sum(axis=1, keepdims=True)
    # a logit's error: K roundings of partial sums of size up to ~|scale| sqrt(K) = 2, random in sign, plus the scale's rounding
    # of a logit below 12; the exponential, sum and division add a few ulps
    tol = 2.0 ** -24 * (4 * 2 * np.sqrt(K) + 12 + 16)
    assert np.abs(got / P - 1).max() <= 2 * tol
    res = oracle.compare(got.astype(np.float32), P)
    assert res["ok"], res


@pytest.mark.gpu
def test_f32_tiles_f16_matmul_result_f16_output_and_specials(wtc_lib, cuda_dev):
    import torch
    w = wtc_lib
    rng = np.random.default_rng(9)
    A = rng.standard_normal((300, 96)).astype(np.float32)
    B = rng.standard_normal((96, 515)).astype(np.float32)
    tA, tB = torch.from_numpy(A).to(cuda_dev), torch.from_numpy(B).to(cuda_dev)
    P = oracle.chain(A, B, 0.1)
    r = oracle.compare(w.matmul_softmax(tA, tB, 0.1, out_dtype=w.F16).cpu().numpy(), P)
    assert r["ok"], r
    got = w.matmul_softmax(tA, tB, 0.1, acc_dtype=w.F16).cpu().numpy()
    L = (A.astype(np.float64) @ B.astype(np.float64)).astype(np.float16).astype(np.float64) * 0.1
    E = np.exp(L - L.max(axis=1, keepdims=True))
    # a sum within its rounding error of a tie may go to the neighbouring f16 value: one f16 ulp of a sum below 64 (2^-5), times
    # the scale, times a probability below 0.1
    assert np.abs(got - E / E.sum(axis=1, keepdims=True)).max() <= 2.0 ** -5 * 0.1 * 0.1
    # a column masked with -inf has probability zero, one NaN spoils its own row only
    M2 = tA.clone(); M2[7, 3] = float("nan")
    B2 = tB.abs(); B2[:, 11] = -float("inf")
    out = w.matmul_softmax(M2.abs(), B2, 0.1).cpu().numpy()
    good = np.arange(300) != 7
    assert (out[good][:, 11] == 0).all() and np.isfinite(out[good]).all() and np.isnan(out[7]).all()
