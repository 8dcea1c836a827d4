"""The skinny GEMM (a handful of activation rows, K split over a cluster) against the fp32 statement."""
import pytest
import torch

from dizo_b200.ops import _lib, gemm

pytestmark = pytest.mark.gpu


def _rand(*shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).bfloat16()


def _close(y, ref, K):
    """fp32 sums of K products in another order (2^-24 sqrt(K) relative, generously x16), then one rounding to bf16: an
    8-bit significand, so at most 2^-8 of every element and of the 2-norm."""
    err = ((y.float() - ref).norm() / ref.norm()).item()
    assert err < (2.0 ** -8 if y.dtype == torch.bfloat16 else 0.0) + 16 * K ** 0.5 * 2.0 ** -24, err


@pytest.mark.parametrize("M", [1, 16, 17, 64, 65, 128, 300])
@pytest.mark.parametrize("N,K", [(8, 8), (128, 64), (200, 72), (2048, 2048), (1032, 8200), (25000, 136)])
@pytest.mark.parametrize("splits", [0, 1, 3, 8])
def test_skinny_gemm(M, N, K, splits):
    x, w, r = _rand(M, K, seed=1), _rand(N, K, seed=2, scale=0.05), _rand(M, N, seed=3)
    b = _rand(N, seed=4)
    for dtype, act in ((torch.bfloat16, "relu"), (torch.float32, None)):
        out = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
        gemm._skinny(x, w, out, b, r, gemm.ACT[act], 0.5, splits=splits)
        _lib.check_device_errors()
        _close(out, gemm.linear_reference(x, w, b, act=act, residual=r, scale=0.5, out_dtype=torch.float32), K)


def test_skinny_gemm_in_place_residual_and_strides():
    M, N, K = 5, 264, 512
    wide = _rand(M, 2 * K, seed=5)
    x, w, h = wide[:, K:], _rand(N, K, seed=6, scale=0.05), _rand(M, N, seed=7)
    ref = gemm.linear_reference(x, w, residual=h, out_dtype=torch.float32)
    gemm.linear(x, w, residual=h, out=h)
    _close(h, ref, K)


@pytest.mark.parametrize("M,F,K", [(1, 8, 64), (3, 176, 64), (64, 200, 136), (16, 11008, 4096)])
def test_skinny_swiglu(M, F, K):
    x, w = _rand(M, K, seed=8), _rand(2 * F, K, seed=9, scale=K ** -0.5)
    y = gemm.linear_swiglu(x, w)
    gu = x.float() @ w.float().t()
    ref = torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]
    # __expf and the fast division are good to a few fp32 ulp: far below the bf16 rounding of the result
    _close(y, ref, K)


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K", [(1, 8), (8, 2048), (201, 2056), (1032, 8200), (2048, 11008), (25001, 136)])
def test_gemv(M, N, K):
    x, w, r, b = _rand(M, K, seed=1), _rand(N, K, seed=2, scale=0.05), _rand(M, N, seed=3), _rand(N, seed=4)
    for dtype, act in ((torch.bfloat16, "relu"), (torch.float32, None)):
        out = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
        gemm._gemv(x, w, out, b, r, gemm.ACT[act], 0.5)
        _close(out, gemm.linear_reference(x, w, b, act=act, residual=r, scale=0.5, out_dtype=torch.float32), K)
    if N % 2 == 0:
        out = torch.empty((M, N // 2), dtype=torch.bfloat16, device="cuda")
        gemm._gemv(x, w, out, None, None, 3, 1.0)
        gu = x.float() @ w.float().t()
        _close(out, torch.nn.functional.silu(gu[:, :N // 2]) * gu[:, N // 2:], K)


def test_gemv_limits():
    x, w = _rand(4, 20480, seed=1), _rand(64, 20480, seed=2)
    with pytest.raises(_lib.KernelError):
        gemm._gemv(x, w, torch.empty((4, 64), dtype=torch.bfloat16, device="cuda"), None, None, 0, 1.0)
