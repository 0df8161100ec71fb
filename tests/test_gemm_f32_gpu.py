"""The float32 product on the tensor cores (csrc/gemm_f32_split.cu) against 64 bits and against the CUDA-core kernel it takes
the place of: at edges of its tiles and chunks, with strided rows, activations in its epilogue, and operands that are not finite."""
from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def K():
    import toyinfer_b200.kernels as K
    K.library()
    return K


def cuda_cores(K, monkeypatch, fn):
    from toyinfer_b200.kernels import gemm
    with monkeypatch.context() as m:
        m.setattr(gemm, "f32_on_tensor_cores", False)
        return fn()


def operands(M, N, Kd, positive, pad=0):
    g = torch.Generator(device="cuda").manual_seed(M * 7 + N * 3 + Kd)
    x = torch.randn(M, Kd + pad, generator=g, device="cuda")[:, :Kd]
    w = torch.randn(N, Kd + pad, generator=g, device="cuda")[:, :Kd] * Kd ** -0.5
    return (x.abs(), w.abs()) if positive else (x, w)


# tokens at the edges of tiles of 64, 128 and 256; weight rows and contractions at theirs (256 rows, 32 steps), down to one chunk
@pytest.mark.parametrize("M,N,Kd", [(17, 8, 8), (63, 255, 33), (64, 256, 32), (65, 257, 64), (128, 512, 100), (129, 40, 2560), (256, 300, 31),
                                    (257, 1030, 96), (700, 2600, 1000), (40, 2560, 9728), (9, 4096, 2048), (500, 520, 4)])
@pytest.mark.parametrize("positive", [False, True])
def test_product(K, monkeypatch, M, N, Kd, positive):
    pad = -Kd % 4                          # rows start on 16-byte boundaries whatever the contraction's length
    x, w = operands(M, N, Kd, positive, pad if pad else 4)
    want = x.double() @ w.double().T
    got = K.linear(x, w)
    K.check_status()
    off = lambda y: float((y.double() - want).norm() / want.norm())
    # Mixed signs: no further off than the CUDA-core kernel.  The tensor core truncates, so that a sum of one sign loses up to a
    # step of 2^-23 of a chunk's sum with each of its two large MMAs, half a step on average: 2^-23 altogether, on the old
    # kernel's rounding.  (A contraction of one chunk is that loss and little else, whatever the signs.)
    slack = 2.0 ** -23 if positive else 6e-8 if Kd <= 64 else 0.0
    assert off(got) <= 1.05 * off(cuda_cores(K, monkeypatch, lambda: K.linear(x, w))) + slack
    assert torch.equal(got, K.linear(x, w))


@pytest.mark.parametrize("act,limit", [("silu", 0.0), ("gelu_tanh", 0.0), ("clamped_swish", 2.0)])
@pytest.mark.parametrize("M", [33, 130, 300])
def test_gated_epilogue(K, monkeypatch, M, act, limit):
    x, w = operands(M, 602, 200, False)
    got = K.linear_swiglu(x, w, act, limit)
    want = cuda_cores(K, monkeypatch, lambda: K.linear_swiglu(x, w, act, limit))
    torch.testing.assert_close(got, want, rtol=1e-5, atol=4e-6)      # sums of 200 unit products, each side within 1e-6


@pytest.mark.parametrize("act", ["relu2", "gelu"])
def test_pointwise_epilogue(K, monkeypatch, act):
    x, w = operands(77, 300, 96, False)
    torch.testing.assert_close(K.linear_act(x, w, act), cuda_cores(K, monkeypatch, lambda: K.linear_act(x, w, act)), rtol=1e-5, atol=4e-6)


def test_operands_that_are_not_finite(K, monkeypatch):
    x, w = operands(300, 512, 256, False)
    x[3, 5], x[7, 9], w[30, 7] = float("inf"), float("nan"), -float("inf")
    w[11, 3] = 3.4e38                      # finite, but rounds to an infinite bfloat16
    x[:, 3] = x[:, 3].clamp(-1, 1)
    got, want = K.linear(x, w), cuda_cores(K, monkeypatch, lambda: K.linear(x, w))
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[want.isinf()], want[want.isinf()])
    fine = want.isfinite()
    torch.testing.assert_close(got[fine], want[fine], rtol=1e-5, atol=4e-6)


def test_rows_off_the_boundary_take_the_other_kernel(K):
    x, w = operands(40, 96, 64, False)
    base = torch.zeros(96 * 65 + 1, device="cuda")
    odd = base[1:].view(96, 65)[:, :64]
    odd.copy_(w)
    torch.testing.assert_close(K.linear(x, odd), x @ w.T, rtol=1e-5, atol=4e-6)


def microseconds(fn):
    fn()
    times = []
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(4):
            fn()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b) * 250)
    return min(times)


@pytest.mark.parametrize("spoil", ["all nan", "a row nan", "a weight row nan", "all infinite", "a row's end infinite"])
def test_results_that_are_not_finite_cost_little(K, monkeypatch, spoil):
    """Activations that have become NaN or infinite: the results of the CUDA cores, at some times the product's usual cost."""
    x, w = operands(256, 1024, 1024, False)
    usual = microseconds(lambda: K.linear(x, w))
    if spoil == "all nan":
        x[:] = float("nan")
    elif spoil == "a row nan":
        x[100] = float("nan")
    elif spoil == "a weight row nan":
        w[70] = float("nan")
    elif spoil == "all infinite":
        x[:] = float("inf")
    else:
        x[255, 1023] = float("-inf")
    got, want = K.linear(x, w), cuda_cores(K, monkeypatch, lambda: K.linear(x, w))
    K.check_status()
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got[want.isinf()], want[want.isinf()])
    fine = want.isfinite()
    torch.testing.assert_close(got[fine], want[fine], rtol=1e-5, atol=4e-6)
    assert microseconds(lambda: K.linear(x, w)) < 25 * usual + 100     # (a thread a result: 180 times for NaN throughout)


def test_no_weight_rows(K):
    assert K.linear(torch.ones(40, 64, device="cuda"), torch.ones(0, 64, device="cuda")).shape == (40, 0)
