"""The backprojector's z blocks and column patches: every depth of block (32, 64, 96 and
128 slices, one block and several, ragged ends), view counts that leave partial groups
of 2, 4, 8 and 32, views that miss some columns.  A voxel's sum over the views has one
order, so every tile gives the same bits, the one-slice blocks' of test_gpu_backproject.py
(which hold the values) among them.
"""

import math

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


def scan(A, U, V, seed, wide):
    g = torch.Generator().manual_seed(seed)
    p = torch.randn((A, U, V), generator=g).cuda()

    def jitter(x, s):
        return (x + s * torch.randn(A, generator=g)).float().cuda()

    angles = torch.arange(A) * 2 * math.pi / A
    u0 = torch.full((A,), (U - 1) / 2)
    if wide:
        u0 = u0 + torch.where(torch.arange(A) % 3 == 0, 0.7 * U, 0.0)  # most columns missed
    return p, [jitter(angles, 0.01), jitter(200.0, 2.0), jitter(130.0, 1.0), jitter(u0, 1.0),
               jitter((V - 1) / 2, 1.0), jitter(0.0, 0.5), jitter(0.0, 0.5), jitter(0.0, 0.5)]


DEPTHS = [1, 31, 32, 33, 64, 65, 95, 96, 97, 128, 129, 160, 192, 193, 257, 400]


@pytest.mark.parametrize("D", DEPTHS)
@pytest.mark.parametrize("px,wide", [(1.0, False), (0.9, True)])
def test_every_block_gives_the_same_bits(D, px, wide):
    from dgc_b200 import _native, _ops

    H, W, A = 7, 13, 35 + D % 36
    U, V = 61, max(16, int(0.9 * D))
    p, geom = scan(A, U, V, D, wide)
    lib = _native.lib()

    def run():
        return _ops.bp_forward(p, *geom, px, D, H, W, 0.8)

    lib.dgc_bp_clear_tile_rules()
    got = run()
    try:
        for kz, cx, cy in ((1, 4, 2), (2, 16, 1), (4, 1, 1), (8, 4, 1), (2 if D > 32 else 1, 8, 1)):
            lib.dgc_bp_clear_tile_rules()
            _native.check(lib.dgc_bp_add_tile_rule(1 << 20, 1 << 20, kz, 0, cx, cy))
            assert torch.equal(run(), got), (kz, cx, cy)
    finally:
        lib.dgc_bp_clear_tile_rules()


def double_reference(p, geom, px, D, H, W, vs):
    """Voxel-driven FDK backprojection (weight (sod + ds_n)^2 / q^2) in float64."""
    A, U, V = p.shape
    z, y, x = torch.meshgrid(*(((torch.arange(n, dtype=torch.float64) - n * 0.5) * vs).cuda()
                               for n in (D, H, W)), indexing="ij")
    out = torch.zeros((D, H, W), dtype=torch.float64, device="cuda")
    for a in range(A):
        th, sid, sod, u0, v0, sx, sy, sz = (float(t[a].double()) for t in geom)
        c, s = math.cos(th), math.sin(th)
        du, dn, dv = sx * c + sy * s, -sx * s + sy * c, sz
        q = sod + dn - (-x * s + y * c)
        t = (sid + dn) / q
        u = (du + t * (x * c + y * s - du)) / px + u0
        v = (dv + t * (z - dv)) / px + v0
        ok = (q > 1e-6) & (u >= 0) & (u < U - 1) & (v >= 0) & (v < V - 1)
        ui, vi = u.floor().clamp(0, U - 2).long(), v.floor().clamp(0, V - 2).long()
        fu, fv = u - ui, v - vi
        P = p[a].double()
        val = ((1 - fu) * ((1 - fv) * P[ui, vi] + fv * P[ui, vi + 1])
               + fu * ((1 - fv) * P[ui + 1, vi] + fv * P[ui + 1, vi + 1]))
        out += torch.where(ok, ((sod + dn) / q) ** 2 * val, torch.zeros_like(val))
    return out


@pytest.mark.parametrize("U,V", [(3, 34), (4, 33), (5, 3), (6, 66), (32, 65), (33, 31), (34, 5), (67, 130)])
def test_quads_of_ragged_detectors(U, V):
    """Detectors whose rows and columns leave partial blocks, threads and row groups of the
    quads.  The border is zero, so the backprojection is continuous at the detector's
    edge and a coordinate's float32 rounding (some 3e-5 pixel at 130) moves a value by no
    more than that times neighbouring data's difference: relative L2 below 1e-4."""
    from dgc_b200 import _ops

    D, H, W, A = V, 9, max(9, U), 12
    p, geom = scan(A, U, V, U + V, False)
    p[:, [0, -1]] = 0
    p[:, :, [0, -1]] = 0
    got = _ops.bp_forward(p, *geom, 1.0, D, H, W, 0.6)
    want = double_reference(p, geom, 1.0, D, H, W, 0.6)
    assert float((got.double() - want).norm() / want.norm()) < 1e-4
