"""The branches of the FDK filter on the tensor cores beside its plain call: gradients of a
frame, Parker weights, several chunks of views, views that are left to the FP32
product among views that are not, and the route without scratch.

Tolerances as in test_gpu_fdk_tc.py: an element within 128 * 2^-24 of the magnitudes
summed in it, all of them within 2^-20 in L2; a per-view sum of such elements within
2^-20 of its terms' magnitudes, and rounded once to FP32.
"""

import math

import numpy as np
import pytest
import torch

from conftest import rel_l2
from test_gpu_fdk_tc import E, close, scan, toeplitz
from test_gpu_preweight_frame import _offset_geometry, cuda32

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]

PX, ALPHA = 1.1, 0.85


def framed(A, U, V, seed):
    p, sid, sod = scan(A, U, V, seed)
    gen = torch.Generator().manual_seed(seed + 50)
    dist = sid * 0.97 + torch.randn(A, generator=gen).cuda()
    cu = (U - 1) / 2 + 5 * torch.randn(A, generator=gen).cuda()
    cv = (V - 1) / 2 + 3 * torch.randn(A, generator=gen).cuda()
    g = torch.randn(p.shape, generator=gen).cuda()
    return p, g, sod, sid, (dist, cu, cv)


def gradients(p, g, sod, sid, frame, room=None):
    """dgc_fdk_filter_ex and its backward: [y, dP, dsod, dsid, ddist, du, dv]; ``room``: views
    at a time."""
    from dgc_b200 import _native

    lib, (A, U, V) = _native.lib(), p.shape
    room = A if room is None else room
    s = torch.cuda.current_stream().cuda_stream
    y, dp = torch.full_like(p, math.nan), torch.full_like(p, math.nan)
    sums = [torch.full_like(sod, math.nan) for _ in range(5)]
    ptrs = [t.data_ptr() for t in frame]

    def scratch(adjoint):
        n = lib.dgc_fdk_filter_workspace_bytes_at_a_time(A, U, V, adjoint, room)
        return torch.empty(n, dtype=torch.uint8, device="cuda"), n

    ws, n = scratch(0)
    _native.check(lib.dgc_fdk_filter_ex(p.data_ptr(), A, U, V, PX, sod.data_ptr(), sid.data_ptr(), *ptrs,
                                        ALPHA, y.data_ptr(), ws.data_ptr(), n, s))
    ws, n = scratch(1)
    _native.check(lib.dgc_fdk_filter_backward_ex(
        g.data_ptr(), p.data_ptr(), y.data_ptr(), A, U, V, PX, sod.data_ptr(), sid.data_ptr(), *ptrs,
        ALPHA, dp.data_ptr(), *[t.data_ptr() for t in sums], ws.data_ptr(), n, s))
    return [y, dp, *sums]


@pytest.mark.parametrize("A,U,V", [(4, 192, 45), (3, 193, 130), (3, 300, 77), (2, 187, 97), (3, 140, 257)])
def test_gradients_of_a_frame(A, U, V):
    p, g, sod, sid, frame = framed(A, U, V, U)
    got = gradients(p, g, sod, sid, frame)
    P, G, D, cu, cv, o, s = (t.double() for t in (p, g, *frame, sod, sid))
    D, o, s = D[:, None, None], o[:, None, None], s[:, None, None]
    u = (torch.arange(U, device="cuda")[None, :, None] - cu[:, None, None]) * PX
    v = (torch.arange(V, device="cuda")[None, None] - cv[:, None, None]) * PX
    r = (D * D + u * u + v * v).sqrt()
    w, c = D / r, PX * s / o
    H = toeplitz(U, PX, ALPHA)
    y, z = c * (H @ (w * P)), H @ G
    close(got[0], y, c * (H.abs() @ (w * P).abs()))
    close(got[1], c * w * z, c * w * (H.abs() @ G.abs()))
    zp = c * z * P
    terms = [-G * y / o, G * y / s, zp * (u * u + v * v) / r**3, zp * D * u * PX / r**3,
             zp * D * v * PX / r**3]
    for k, term in enumerate(terms):
        want, scale = term.flatten(1).sum(1), term.abs().flatten(1).sum(1)
        assert float(((got[2 + k].double() - want).abs() - 2.0**-20 * scale - E * want.abs()).max()) <= 0, k


@pytest.mark.parametrize("A,U,V", [(7, 192, 33), (5, 257, 129)])
def test_gradients_of_chunks_of_views(A, U, V):
    """However many views at a time, and each view in a call of its own: the same bits."""
    p, g, sod, sid, frame = framed(A, U, V, 3)
    whole = gradients(p, g, sod, sid, frame)
    assert not torch.equal(whole[1], gradients(p, g, sod, sid, frame, room=0)[1])
    for room in (1, 2, 4):
        assert all(torch.equal(a, b) for a, b in zip(gradients(p, g, sod, sid, frame, room), whole)), room
    for a in range(A):
        own = gradients(*(t[a:a + 1].contiguous() for t in (p, g, sod, sid)),
                        [t[a:a + 1].contiguous() for t in frame])
        assert all(torch.equal(x[0], y[a]) for x, y in zip(own, whole)), a


def test_adjoint_of_views_outside_the_split():
    """NaN, infinities, tiny and huge values and zeros in the upstream gradient of some
    views: these as the FP32 product gives them, the others as in a call of their own."""
    A, U, V = 9, 200, 70
    p, g, sod, sid, frame = framed(A, U, V, 8)
    g[1, 5, 6] = math.nan
    g[2, 199, 69] = math.inf
    g[3] *= 1e-30
    g[4, 7, 8] = 3e38
    g[5] = 0
    g[6, :, 3] *= 1e-34
    fast, slow = gradients(p, g, sod, sid, frame), gradients(p, g, sod, sid, frame, room=0)
    # y comes from the tensor cores in `fast`: the sums of g y are compared from the same y
    for a in (1, 2, 3, 4, 5, 6):
        assert torch.equal(torch.nan_to_num(fast[1][a], 7.0, 8.0, 9.0),
                           torch.nan_to_num(slow[1][a], 7.0, 8.0, 9.0)), a
        for k in (4, 5, 6):  # of H(g) alone
            assert torch.equal(torch.nan_to_num(fast[k][a], 7.0, 8.0, 9.0),
                               torch.nan_to_num(slow[k][a], 7.0, 8.0, 9.0)), (k, a)
    assert not torch.isfinite(fast[1][1]).all() and not torch.isfinite(fast[1][2]).all()
    for a in (0, 7, 8):
        own = gradients(*(t[a:a + 1].contiguous() for t in (p, g, sod, sid)),
                        [t[a:a + 1].contiguous() for t in frame])
        assert all(torch.equal(x[0], y[a]) for x, y in zip(own, fast)), a
        assert not torch.equal(fast[1][a], slow[1][a])


def test_the_route_without_scratch_agrees_element_by_element():
    """Both products within their bounds of the exact one, so within twice those of each
    other: a lost split product (2^-16 of the leading one) would not be."""
    A, U, V = 3, 300, 150
    p, g, sod, sid, frame = framed(A, U, V, 6)
    fast, slow = gradients(p, g, sod, sid, frame), gradients(p, g, sod, sid, frame, room=0)
    H = toeplitz(U, PX, ALPHA).abs()
    c = PX * (sid / sod).double()[:, None, None]
    for k, x in ((0, p), (1, g)):
        a, b = fast[k].double(), slow[k].double()
        assert float(((a - b).abs() - 256 * E * c * (H @ x.double().abs())).max()) <= 0
        assert float((a - b).norm() / b.norm()) <= 2.0**-19


@pytest.mark.parametrize("offset", [False, True])
@pytest.mark.parametrize("U,V", [(128, 40), (203, 61)])
def test_parker_weights(offset, U, V, oracle):
    """A short scan, with and without the offset-aware preweight: the weights enter the
    split operand."""
    from dgc_b200 import reconstruct_fdk

    A, px, shape, off = 60, 0.6, (20, 24, 24), (0.3, -0.2, 0.1)
    probe = _offset_geometry(A, U, V, 8)
    if not offset:
        for k in (5, 6, 7):
            probe[k][:] = 0
    shift = np.abs(probe[5]) + np.abs(probe[6])
    reach = np.maximum(probe[3], U - 1 - probe[3]) * px + shift
    fan = float(np.max(np.arctan(reach / (probe[1] - shift))))
    angles = (0.3 + np.linspace(0.0, math.pi + 2 * fan + 0.02, A)).astype(np.float32)
    geom = [angles, *probe[1:]]
    proj = (np.random.default_rng(9).random((A, U, V)) * 4).astype(np.float32)
    vol = reconstruct_fdk(cuda32(proj), *map(cuda32, geom), px, shape, 1.0, volume_offset=off,
                          short_scan=True, offset_preweight=offset)
    gnp = [x.astype(np.float64) for x in geom]
    step = abs(float(angles[-1]) - float(angles[0])) / (A - 1)
    if offset:
        d64, u64, v64 = oracle.preweight_frame(geom, px)
        w64 = oracle.parker_weights(geom[0], geom[1], U, px, d64, u64)
        filt = oracle.fdk_filter(proj * w64[:, :, None], px, gnp[2], gnp[1], 0.8, frame=(d64, u64, v64))
    else:
        w64 = oracle.parker_weights(geom[0], geom[1], U, px)
        filt = oracle.fdk_filter(proj * w64[:, :, None], px, gnp[2], gnp[1], 0.8)
    truth = np.maximum(oracle.backproject(filt, gnp, px, shape, 1.0, off) * step, 0.0)
    assert rel_l2(vol.cpu(), truth) < 1e-5
