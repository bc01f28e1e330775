"""The kernels around the tensor-core products: the product over the rows of both
operands (MN-major), im2col / col2im by rows, the ReLU gradient with its column
sums."""

import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def bf16(*shape, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(*shape, device="cuda", generator=g).to(torch.bfloat16)


@pytest.mark.parametrize("K,M,N", [(8, 8, 8), (63, 32, 24), (65, 64, 72), (130, 136, 264),
                                   (1000, 256, 2304), (5000, 304, 520), (12801, 32, 288),
                                   (700, 2048, 19200)])
def test_product_over_rows(K, M, N):
    """Tiles, boxes and K remainders of every width (the last takes the 256 x 256
    tiles); long K splits.  FP32 accumulation of exact bf16 products: the error
    stays below 1e-5 of the sum of magnitudes."""
    from dgc_b200 import warmstart

    A, B = bf16(K, M, seed=K), bf16(K, N, seed=N + 1)
    got = warmstart.gemm_tn(A, B)
    want = A.double().t() @ B.double()
    scale = (A.double().abs().t() @ B.double().abs()).clamp_min(1.0)
    assert float(((got.double() - want).abs() / scale).max()) < 1e-5


def test_product_over_rows_fallbacks(monkeypatch):
    from dgc_b200 import warmstart

    A, B = bf16(77, 20), bf16(77, 36, seed=1)  # rows off 16 bytes
    want = A.float().t() @ B.float()
    torch.testing.assert_close(warmstart.gemm_tn(A, B), want, rtol=1e-5, atol=1e-4)
    monkeypatch.setenv("DGC_GEMM", "cpasync")
    A, B = bf16(77, 24), bf16(77, 40, seed=1)
    torch.testing.assert_close(warmstart.gemm_tn(A, B), A.float().t() @ B.float(), rtol=1e-5,
                               atol=1e-4)


@pytest.mark.parametrize("B,H,W,C,k,stride", [(2, 7, 9, 2, 3, 2), (3, 8, 8, 8, 3, 1),
                                              (2, 5, 6, 32, 3, 2), (1, 1, 1, 8, 3, 1),
                                              (2, 6, 5, 3, 5, 1), (1, 33, 17, 12, 3, 2)])
def test_im2col_and_its_adjoint(B, H, W, C, k, stride):
    from dgc_b200 import _native, warmstart

    pad = k // 2
    Kp = (k * k * C + 7) // 8 * 8
    x = bf16(B, H, W, C)
    col, Ho, Wo = warmstart._im2col(x, k, stride, pad, Kp)
    want = F.unfold(x.float().permute(0, 3, 1, 2), k, padding=pad, stride=stride)
    want = want.view(B, C, k * k, Ho * Wo).permute(0, 3, 2, 1).reshape(B * Ho * Wo, k * k * C)
    assert torch.equal(col[:, :k * k * C].float(), want)
    assert not col[:, k * k * C:].any()
    g = torch.randn(B * Ho * Wo, Kp, device="cuda")
    dx = torch.empty(B, H, W, C, device="cuda")
    _native.check(_native.lib().dgc_col2im_nhwc_f32(
        g.data_ptr(), B, H, W, C, k, k, stride, pad, Kp, dx.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    gw = g[:, :k * k * C].double().view(B, Ho * Wo, k * k, C).permute(0, 3, 2, 1)
    ref = F.fold(gw.reshape(B, C * k * k, Ho * Wo), (H, W), k, padding=pad, stride=stride)
    torch.testing.assert_close(dx.double(), ref.permute(0, 2, 3, 1), rtol=1e-5, atol=1e-5)
    assert torch.equal(warmstart._col2im(g, (B, H, W, C), k, stride, pad, Kp),
                       dx.to(torch.bfloat16))


@pytest.mark.parametrize("M,C", [(1, 8), (65, 8), (64, 24), (1000, 32), (333, 256), (70000, 64),
                                 (129, 2048)])
@pytest.mark.parametrize("relu", [True, False])
def test_relu_gradient(M, C, relu):
    """g is torch's bit for bit; the FP32 column sums stay within 1e-6 of the sum of
    magnitudes (sums of up to a few hundred terms a thread, then FP64)."""
    from dgc_b200 import warmstart

    gy, y = bf16(M, C, seed=2), bf16(M, C, seed=3)
    gy[0, 0] = -0.0
    y[0, :4] = 0.0
    g, db = warmstart._relu_grad(gy, y, relu)
    want = gy * (y > 0) if relu else gy
    assert torch.equal(g.view(torch.int16), want.view(torch.int16))
    total = want.double().sum(0)
    scale = want.double().abs().sum(0).clamp_min(1e-3)
    assert float(((db.double() - total).abs() / scale).max()) < 1e-6
