"""Values that a softmax meets beside ordinary ones, through every form of the tensor-core epilogue and the routes into it:
columns masked with -inf, logits far from zero.  Against the same chain in 64 bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain64(A, B, scale):
    L = (A.double() @ B.double()) * scale
    return (L - L.max(-1, keepdim=True).values).softmax(-1)


def _operands(torch, dev, M, N, K, seed):
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    return torch.randn(M, K, device=dev, generator=gen), torch.randn(K, N, device=dev, generator=gen)


# (M, N, K, output, flags, scale): ragged cluster and tiled, narrow tiles, then the aligned forms (128- and 256-column split,
# single tile, relay, tiled, pairs)
_FORMS = [
    (300, 1021, 65, "f16", "", 0.1), (300, 1021, 65, "f32", "", 0.1), (300, 3001, 65, "f16", "", 0.1), (300, 3001, 65, "f32", "", 0.1),
    (9000, 1021, 65, "f16", "", -0.1), (300, 1016, 65, "f16", "", 0.1),
    (16, 4096, 512, "f16", "", 0.1), (16, 4096, 512, "f32", "", 0.1),
    (300, 1024, 64, "f16", "", 0.1), (300, 1024, 64, "f32", "", 0.1), (4096, 1024, 64, "f16", "", 0.1), (9000, 1024, 64, "f16", "", -0.1),
    (9000, 1016, 64, "f16", "", 0.1), (4096, 1024, 64, "f16", "FLAG_EPILOGUE_SPLIT", 0.1), (4096, 1024, 64, "f32", "", 0.1),
    (4096, 4096, 64, "f16", "", 0.1), (4096, 4096, 64, "f32", "", -0.1), (4096, 4096, 256, "f16", "FLAG_PAIR", 0.1),
]


@pytest.mark.parametrize("M,N,K,out,flag,scale", _FORMS)
def test_masked_columns_are_zeros(wtc_lib, cuda_dev, M, N, K, out, flag, scale):
    """An additive mask as the last K row (a column of ones in A, -inf in B), over runs of 64, 128 and 256 columns: whole
    column groups of the epilogue's threads."""
    import torch
    w = wtc_lib
    fA, fB = _operands(torch, cuda_dev, M, N, K, 1)
    flags = getattr(w, flag) if flag else 0
    odt = w.F16 if out == "f16" else w.F32
    for width in (64, 128, 256):
        A, B = fA.half(), fB.half()
        A[:, -1] = 1
        B[-1] = 0
        B[-1, 256:256 + width] = -np.inf if scale > 0 else np.inf
        P = _chain64(A, B, scale)
        assert w.plan_query(w.make_desc(1, M, N, K, out_dtype=odt, flags=flags)).kernel != w.KERNEL_SIMT_FUSED
        got = w.matmul_softmax(A, B, scale, out_dtype=odt, flags=flags)
        w.check_device_status()
        assert not got[:, 256:256 + width].any()
        # f16: one or two roundings of a probability below one; f32: K roundings of a logit below 10 and the exponential's
        tol = 2.0 ** -10 if out == "f16" else 2.0 ** -24 * (10 * K ** 0.5 + 16)
        assert bool((got.double() - P).abs().le(tol * P + 2.0 ** -23).all())
    # a row that is masked throughout is 0 / 0, and the others are none the worse for it
    A[7, -1] = np.inf
    B[-1] = -np.inf if scale > 0 else np.inf
    B[-1, ::2] = -1 if scale > 0 else 1
    got = w.matmul_softmax(A, B, scale, out_dtype=odt, flags=flags)
    w.check_device_status()
    bad = torch.isnan(got).any(-1)
    assert bool(bad[7]) and int(bad.sum()) == 1


@pytest.mark.parametrize("M,N,K,out,flag,scale", _FORMS)
def test_logits_far_from_zero(wtc_lib, cuda_dev, M, N, K, out, flag, scale):
    """Logits of 1e8 to 1e12: one-hot rows, and equal logits give equal probabilities."""
    import torch
    w = wtc_lib
    flags = getattr(w, flag) if flag else 0
    odt = w.F16 if out == "f16" else w.F32
    sign = 1.0 if scale > 0 else -1.0
    for mag in (3000.0, 20000.0):
        A, B = ((x * mag).clamp(-60000, 60000).half() for x in _operands(torch, cuda_dev, M, N, K, 2))
        L = sign * (A.double() @ B.double())
        top = L.topk(2, -1).values
        clear = top[:, 0] - top[:, 1] > 2.0 ** -16 * top[:, 0]         # rows whose largest logit is no tie within f32 sums
        assert clear.float().mean() > 0.9
        got = w.matmul_softmax(A, B, sign, out_dtype=odt, flags=flags)
        w.check_device_status()
        want = torch.nn.functional.one_hot(L.argmax(-1), N)
        assert bool((got.double() - want)[clear].abs().le(2.0 ** -22).all())
        A, B = torch.full_like(A, mag), torch.full_like(B, mag)
        got = w.matmul_softmax(A, B, sign, out_dtype=odt, flags=flags)
        w.check_device_status()
        assert bool((got.double() * N - 1).abs().le(2.0 ** -10 if out == "f16" else 2.0 ** -20).all())


@pytest.mark.parametrize("out", ["f16", "f32"])
@pytest.mark.parametrize("M,N", [(888, 2304), (889, 2304), (3, 5000), (111, 20000), (112, 20000)])
def test_row_rescale_on_both_sides_of_its_rule(wtc_lib, cuda_dev, M, N, out):
    """One vector a thread beyond 888 CTAs, four up to there; a CTA per row, and several."""
    import torch
    w = wtc_lib
    A, B = (x.half() for x in _operands(torch, cuda_dev, M, N, 64, 3))
    odt = w.F16 if out == "f16" else w.F32
    assert w.plan_query(w.make_desc(1, M, N, 64, out_dtype=odt)).kernel == w.KERNEL_TC_TILED
    got = w.matmul_softmax(A, B, 0.125, out_dtype=odt)
    w.check_device_status()
    P = _chain64(A, B, 0.125)
    # f16: the value relative to its tile's maximum and the rescaled one are both rounded
    tol = 2.0 ** -10 if out == "f16" else 2.0 ** -24 * 100
    assert bool((got.double() - P).abs().le(tol * P + 2.0 ** -23).all())
