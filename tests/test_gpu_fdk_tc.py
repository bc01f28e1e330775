"""The FDK filter's product on the tensor cores against 64-bit arithmetic.

Tolerances, with S = sum_k |h[|u-k|] w[k]|, the sum of magnitudes at an output, and
e = 2^-24: rounded inputs 4 e S (weight and taps); the leading product, per 32 taps
two matrix instructions that each truncate 17 aligned addends, at most 34 e S; U/32
<= 64 FP32 additions, 64 e S; the other products, 2^-8 of it, in one truncating
accumulator of 5 U/16 <= 640 instructions, 2 * 640 * 2^-8 e S; the products left out,
3 e S.  Together below 128 e S at an output.  For white noise the errors of the terms
are independent and the sums of magnitudes are not reached: relative L2 error 2^-20,
below what the smallest product kept (2^-16 of the leading one) would leave.
"""

import numpy as np
import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

E = 2.0**-24


def scan(A, U, V, seed):
    g = torch.Generator().manual_seed(seed)
    p = torch.randn((A, U, V), generator=g).cuda()
    sid = (1000 + 5 * torch.randn(A, generator=g)).cuda()
    sod = (600 + 5 * torch.randn(A, generator=g)).cuda()
    return p, sid, sod


def toeplitz(U, px, alpha):
    from dgc_b200 import _ops

    h = torch.tensor(np.asarray(_ops.fdk_filter_taps(U, px, alpha)), dtype=torch.float64).cuda()
    i = torch.arange(U, device="cuda")
    return h[(i[:, None] - i[None]).abs()]


def weights(p, px, dist, cu, cv):
    A, U, V = p.shape
    u = (torch.arange(U, device="cuda", dtype=torch.float64)[None] - cu.double()[:, None]) * px
    v = (torch.arange(V, device="cuda", dtype=torch.float64)[None] - cv.double()[:, None]) * px
    d = dist.double()[:, None, None]
    return d / (d * d + u[:, :, None] ** 2 + v[:, None, :] ** 2).sqrt()


def close(got, want, magnitudes):
    assert torch.isfinite(got).all()
    assert float(((got.double() - want).abs() - 128 * E * magnitudes).max()) <= 0
    assert float((got.double() - want).norm() / want.norm()) <= 2.0**-20


# edges: 96 rows is the first size; a row tile (128) and one more or less; a column
# tile (256), two, ragged ones; rows that are not 8-element multiples; 2048 rows the
# last (300 columns: no room to turn the rows), 2049 the FP32 product's
SIZES = [(2, 96, 16), (1, 97, 17), (3, 127, 255), (2, 128, 256), (2, 129, 257), (5, 192, 40),
         (1, 187, 521), (2, 768, 100), (1, 2048, 24), (1, 2048, 300), (1, 2049, 24)]


@pytest.mark.parametrize("A,U,V", SIZES)
def test_filter_and_adjoint_match_64_bits(A, U, V):
    from dgc_b200 import _ops

    px, alpha = 0.9, 0.8
    p, sid, sod = scan(A, U, V, U + V)
    H = toeplitz(U, px, alpha)
    w = weights(p, px, sid, torch.full_like(sid, (U - 1) / 2), torch.full_like(sid, (V - 1) / 2))
    c = px * (sid / sod).double()[:, None, None]
    y = _ops.fdk_filter(p, px, sod, sid, alpha)
    close(y, c * (H @ (w * p.double())), c * (H.abs() @ (w * p.double()).abs()))
    g = torch.randn(p.shape, generator=torch.Generator().manual_seed(1)).cuda()
    gp, gsod, gsid = _ops.fdk_filter_backward(g, p, y, px, sod, sid, alpha)
    z = H @ g.double()
    close(gp, c * w * z, c * w * (H.abs() @ g.double().abs()))
    # y = c H(w P): dy/dsod = -y/sod; dy/dsid = y/sid + c H(P dw/dsid), dw/dsid = w r2/(sid dist^2)
    s, o = sid.double(), sod.double()
    gy = (g.double() * y.double()).flatten(1)
    dw = w * (1 - w * w) / s[:, None, None]
    zp = (c * z * p.double() * dw).flatten(1)
    # magnitudes of the summed terms; each carries the error of its y or z, by the L2 bound
    scale = gy.abs().sum(1) / o
    assert float(((gsod.double() + gy.sum(1) / o).abs() - 2.0**-20 * scale).max()) <= 0
    scale = gy.abs().sum(1) / s + zp.abs().sum(1)
    assert float(((gsid.double() - gy.sum(1) / s - zp.sum(1)).abs() - 2.0**-20 * scale).max()) <= 0


def test_frames():
    from dgc_b200 import _ops

    A, U, V, px, alpha = 3, 160, 130, 1.1, 0.9
    p, sid, sod = scan(A, U, V, 3)
    dist, cu, cv = sid * 0.98, torch.tensor([70.0, 79.5, 90.0]).cuda(), torch.tensor([60.0, 64.5, 71.0]).cuda()
    y = _ops.fdk_filter_framed(p, px, sod, sid, alpha, (dist, cu, cv))
    H = toeplitz(U, px, alpha)
    w = weights(p, px, dist, cu, cv)
    c = px * (sid / sod).double()[:, None, None]
    close(y, c * (H @ (w * p.double())), c * (H.abs() @ (w * p.double()).abs()))


def small_workspace(p, px, sod, sid, alpha):
    """The filter with room for its taps alone: the FP32 product."""
    from dgc_b200 import _native

    lib, (A, U, V) = _native.lib(), p.shape
    out = torch.empty_like(p)
    n = (4 * U + 255) // 256 * 256
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    _native.check(lib.dgc_fdk_filter(p.data_ptr(), A, U, V, px, sod.data_ptr(), sid.data_ptr(), alpha,
                                     out.data_ptr(), ws.data_ptr(), n,
                                     torch.cuda.current_stream().cuda_stream))
    return out


def test_values_outside_the_split_take_the_fp32_product():
    """NaN, infinities, values at either end of FP32's range: view by view as the FP32
    product gives them, the other views untouched."""
    from dgc_b200 import _ops

    A, U, V = 7, 130, 70
    p, sid, sod = scan(A, U, V, 4)
    p[1, 5, 6] = float("nan")
    p[2, 129, 69] = float("inf")
    p[3] *= 1e-30
    p[4, 7, 8] = 3e38
    p[5] = 0
    y = _ops.fdk_filter(p, 1.0, sod, sid, 0.8)
    f = small_workspace(p, 1.0, sod, sid, 0.8)
    for a in (1, 2, 3, 4, 5):
        assert torch.equal(torch.nan_to_num(y[a], 7.0, 8.0, 9.0), torch.nan_to_num(f[a], 7.0, 8.0, 9.0))
    assert not torch.isfinite(y[1]).all() and not torch.isfinite(y[2]).all()
    for a in (0, 6):
        one = _ops.fdk_filter(p[a:a + 1].contiguous(), 1.0, sod[a:a + 1], sid[a:a + 1], 0.8)
        assert torch.equal(y[a], one[0])
        assert float((y[a] - f[a]).norm() / f[a].norm()) <= 2.0**-19  # both sides' bounds


def test_chunks_of_views():
    """More views than the split holds at a time: each as in a call of its own."""
    from dgc_b200 import _ops

    A, U, V = 12, 2048, 2000
    p, sid, sod = scan(A, U, V, 5)
    y = _ops.fdk_filter(p, 1.0, sod, sid, 0.8)
    for a in (0, 5, 6, 11):
        one = _ops.fdk_filter(p[a:a + 1].contiguous(), 1.0, sod[a:a + 1], sid[a:a + 1], 0.8)
        assert torch.equal(y[a], one[0])


def test_without_room_for_the_scratch(monkeypatch):
    """No device memory for the split operands: the FP32 product's values and gradients."""
    from dgc_b200 import _ops

    A, U, V = 3, 200, 150
    p, sid, sod = scan(A, U, V, 6)
    g = torch.randn(p.shape, generator=torch.Generator().manual_seed(2)).cuda()
    want = _ops.fdk_filter(p, 1.0, sod, sid, 0.8)
    grads = _ops.fdk_filter_backward(g, p, want, 1.0, sod, sid, 0.8)
    room = _ops._workspace

    def tight(nbytes, device):
        if nbytes > 2048:
            raise torch.cuda.OutOfMemoryError("no room")
        return room(nbytes, device)

    monkeypatch.setattr(_ops, "_workspace", tight)
    y = _ops.fdk_filter(p, 1.0, sod, sid, 0.8)
    assert torch.equal(y, small_workspace(p, 1.0, sod, sid, 0.8))
    assert not torch.equal(y, want)  # the other route
    for got, ref in zip(_ops.fdk_filter_backward(g, p, y, 1.0, sod, sid, 0.8), grads):
        # both sides within 2^-20 of the magnitudes summed; sums of random signs lose
        # at most the square root of their 30000 terms, 2^8, of that
        assert float((got - ref).abs().max()) <= 2.0**-19 * 2.0**8 * float(ref.abs().max())


@pytest.mark.parametrize("U,px", [(96, 1.0), (128, 1.0), (187, 1.0), (768, 3.0), (200, 0.05)])
def test_columns_of_small_values_keep_their_precision(U, px):
    """Every detector column to its own magnitudes, down to the subnormals, beside one of
    ordinary values.  Below FP32's smallest normal number a rounding is 2^-149 at most
    whatever the value: two for a weighted value, one for each of the U products, two
    for the scale."""
    from dgc_b200 import _ops

    A, V, alpha = 2, 64, 0.8
    p, sid, sod = scan(A, U, V, U)
    scale = torch.tensor([1.0] + [2.0 ** -(72 + j) for j in range(1, V)]).cuda()
    H = toeplitz(U, px, alpha)
    w = weights(p, px, sid, torch.full_like(sid, (U - 1) / 2), torch.full_like(sid, (V - 1) / 2))
    c = px * (sid / sod).double()[:, None, None]
    tiny = c * (2 * float(H.abs().sum(1).max()) + U) * 2.0**-149 + 2.0**-148

    def held(got, want, magnitudes):
        assert float(((got.double() - want).abs() - 128 * E * magnitudes - tiny).max()) <= 0

    x = p * scale
    y = _ops.fdk_filter(x, px, sod, sid, alpha)
    held(y, c * (H @ (w * x.double())), c * (H.abs() @ (w * x.double()).abs()))
    gp, _, _ = _ops.fdk_filter_backward(x, x, y, px, sod, sid, alpha)
    held(gp, c * w * (H @ x.double()), c * w * (H.abs() @ x.double().abs()))


def in_room(p, g, y, sod, sid, dist, views):
    """Filter and adjoint (its distance gradients too) of ``views`` views at a time."""
    from dgc_b200 import _native

    lib, (A, U, V) = _native.lib(), p.shape
    out, gp = torch.empty_like(p), torch.empty_like(p)
    gs = [torch.empty_like(sod) for _ in range(3)]
    s = torch.cuda.current_stream().cuda_stream
    n = lib.dgc_fdk_filter_workspace_bytes_at_a_time(A, U, V, 0, views)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    _native.check(lib.dgc_fdk_filter_ex(
        p.data_ptr(), A, U, V, 1.0, sod.data_ptr(), sid.data_ptr(), dist.data_ptr(), None, None, 0.8,
        out.data_ptr(), ws.data_ptr(), n, s))
    n = lib.dgc_fdk_filter_workspace_bytes_at_a_time(A, U, V, 1, views)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    _native.check(lib.dgc_fdk_filter_backward_ex(
        g.data_ptr(), p.data_ptr(), y.data_ptr(), A, U, V, 1.0, sod.data_ptr(), sid.data_ptr(),
        dist.data_ptr(), None, None, 0.8, gp.data_ptr(), *[t.data_ptr() for t in gs], None, None,
        ws.data_ptr(), n, s))
    return [out, gp, *gs]


@pytest.mark.parametrize("U,V", [(192, 17), (129, 97), (300, 203)])
def test_fewer_views_at_a_time_give_the_same_bits(U, V):
    from dgc_b200 import _native, _ops

    A = 7
    p, sid, sod = scan(A, U, V, 8)
    g = torch.randn(p.shape, generator=torch.Generator().manual_seed(3)).cuda()
    dist = sid * 0.97
    y = _ops.fdk_filter_framed(p, 1.0, sod, sid, 0.8, (dist, None, None))
    most = in_room(p, g, y, sod, sid, dist, A)
    assert torch.equal(most[0], y)
    for views in (1, 3, 6):
        assert all(torch.equal(a, b) for a, b in zip(in_room(p, g, y, sod, sid, dist, views), most)), views
    none = in_room(p, g, y, sod, sid, dist, 0)
    assert not torch.equal(none[0], y)
    lib = _native.lib()
    sizes = [lib.dgc_fdk_filter_workspace_bytes_at_a_time(A, U, V, 0, v) for v in (0, 1, 3, A, A + 1)]
    assert sizes == sorted(sizes) and sizes[-1] == sizes[-2] == lib.dgc_fdk_filter_workspace_bytes(A, U, V)


def test_room_for_one_view(monkeypatch):
    """The device has room for one view's split operands: the same bits."""
    from dgc_b200 import _native, _ops

    A, U, V = 5, 200, 150
    p, sid, sod = scan(A, U, V, 6)
    g = torch.randn(p.shape, generator=torch.Generator().manual_seed(2)).cuda()
    want = _ops.fdk_filter(p, 1.0, sod, sid, 0.8)
    grads = _ops.fdk_filter_backward(g, p, want, 1.0, sod, sid, 0.8)
    lib, room = _native.lib(), _ops._workspace
    limit = [lib.dgc_fdk_filter_workspace_bytes_at_a_time(A, U, V, 0, 1)]

    def tight(nbytes, device):
        if nbytes > limit[0]:
            raise torch.cuda.OutOfMemoryError("no room")
        return room(nbytes, device)

    monkeypatch.setattr(_ops, "_workspace", tight)
    assert torch.equal(_ops.fdk_filter(p, 1.0, sod, sid, 0.8), want)
    limit[0] = lib.dgc_fdk_filter_workspace_bytes_at_a_time(A, U, V, 1, 1)
    for a, b in zip(_ops.fdk_filter_backward(g, p, want, 1.0, sod, sid, 0.8), grads):
        assert torch.equal(a, b)


@pytest.mark.parametrize("U,px", [(96, 1.0), (384, 0.9), (2048, 1.3)])
def test_noalloc_is_the_fp32_product(U, px):
    """An impulse gives the taps, one product each: dgc_fdk_filter_noalloc's are those of the
    FP32 product within a rounding of the FP64 taps to FP32 (2^-23 of a tap; an FP64
    error of the DFT, 2^-50 of the largest)."""
    from dgc_b200 import _native

    lib, A, V = _native.lib(), 1, 16
    p = torch.zeros((A, U, V), device="cuda")
    p[0, U // 3] = 1.0
    sid, sod = torch.full((A,), 1000.0, device="cuda"), torch.full((A,), 600.0, device="cuda")
    got, want = torch.empty_like(p), torch.empty_like(p)
    s = torch.cuda.current_stream().cuda_stream
    _native.check(lib.dgc_fdk_filter_noalloc(p.data_ptr(), A, U, V, px, sod.data_ptr(), sid.data_ptr(),
                                             0.8, got.data_ptr(), s))
    n = lib.dgc_fdk_filter_workspace_bytes_at_a_time(A, U, V, 0, 0)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    _native.check(lib.dgc_fdk_filter(p.data_ptr(), A, U, V, px, sod.data_ptr(), sid.data_ptr(), 0.8,
                                     want.data_ptr(), ws.data_ptr(), n, s))
    a, b = got.double(), want.double()
    assert float(b.abs().max()) > 0
    assert float(((a - b).abs() - 2.0**-22 * b.abs() - 2.0**-49 * b.abs().max()).max()) <= 0


@pytest.mark.parametrize("A,U,V", [(3, 192, 130), (5, 300, 96), (2, 768, 300)])
@pytest.mark.parametrize("polls", [0, 1, 2])
def test_waits_that_run_out(A, U, V, polls):
    """Waits inside the tensor-core kernel given up at once (0), or after a poll or two, of
    which some or none then run out: the views come from the FP32 product, and a view
    whose CTAs all got through from the tensor cores -- one of the two, bit for bit, in
    the filter, the projection gradient and the distance gradients.  The next call is
    as if nothing had happened."""
    from dgc_b200 import _native, _ops

    p, sid, sod = scan(A, U, V, 9)
    g = torch.randn(p.shape, generator=torch.Generator().manual_seed(4)).cuda()
    dist = sid * 0.99
    y = _ops.fdk_filter_framed(p, 1.0, sod, sid, 0.8, (dist, None, None))
    fast = in_room(p, g, y, sod, sid, dist, A)
    slow = in_room(p, g, y, sod, sid, dist, 0)
    lib = _native.lib()
    lib.dgc_fdk_limit_waits(polls)
    try:
        got = in_room(p, g, y, sod, sid, dist, A)
        torch.cuda.synchronize()
    finally:
        lib.dgc_fdk_limit_waits(-1)
    for k, (a, f, s) in enumerate(zip(got, fast, slow)):
        for v in range(A):
            assert torch.equal(a[v], s[v]) or (polls and torch.equal(a[v], f[v])), (k, v)
    assert all(torch.equal(a, b) for a, b in zip(in_room(p, g, y, sod, sid, dist, A), fast))
