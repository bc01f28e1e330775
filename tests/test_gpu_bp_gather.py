"""The projection gradient of ``backproject`` as a gather (and as a scatter where
the sizes ask for it), alone and beside the geometry gradients, at the sizes
where its tiles, lists and branches change."""

import math

import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu

# The repository's bar for gradients against the FP64 oracle.
GRAD_RTOL = 1e-4
# Gather and scatter add the same FP32 products (same v_idx, weights and upstream
# values) in another order: a pixel's few hundred terms agree to a few 1e-7.
SAME_RTOL = 5e-6

# (D, H, W), U, V, pixel, voxel, sid, sod, offset
CASES = [
    ((20, 33, 35), 9, 31, 1.0, 1.0, 200.0, 120.0, (0.0, 0.0, 0.0)),
    ((20, 33, 35), 48, 32, 1.0, 1.0, 200.0, 120.0, (0.0, 0.0, 0.0)),
    ((31, 32, 32), 33, 33, 1.3, 1.0, 200.0, 120.0, (1.5, -2.0, 0.7)),
    ((40, 34, 70), 2, 65, 0.7, 0.9, 260.0, 160.0, (0.0, 3.0, 0.0)),
    ((64, 40, 33), 40, 97, 0.9, 1.0, 260.0, 160.0, (0.0, 0.0, 0.0)),
    ((150, 32, 33), 21, 257, 1.0, 0.9, 400.0, 240.0, (0.0, 0.0, 0.0)),
    ((250, 32, 32), 19, 780, 0.5, 0.8, 400.0, 240.0, (0.0, 0.0, 0.0)),
    ((40, 130, 129), 50, 60, 1.1, 1.0, 500.0, 300.0, (0.0, 0.0, 0.0)),  # gather for all nine
    ((40, 33, 35), 48, 40, 1.0, 0.8, 126.0, 120.0, (0.0, 0.0, 0.0)),    # voxels below a pixel
    ((40, 64, 64), 12, 24, 1.0, 1.0, 60.0, 150.0, (0.0, 0.0, 0.0)),     # full lists
    ((30, 40, 40), 30, 40, 1.0, 1.0, 45.0, 24.0, (0.0, 0.0, 0.0)),      # source among the voxels
    ((4, 33, 35), 20, 90, 1.0, 1.0, 200.0, 120.0, (0.0, 0.0, 0.0)),     # a slab: scatter
    ((20, 33, 35), 20, 30, 3.0, 1.0, 200.0, 120.0, (0.0, 0.0, 0.0)),    # coarse pixels: scatter
]


def make(case, A=6, seed=11):
    shape, U, V, px, vs, sid, sod, off = case
    rng = np.random.default_rng(seed)
    angles = np.sort(rng.uniform(0, 2 * math.pi, A))
    angles[:3] = [0.0, math.pi / 2, math.pi]
    geom = [angles, sid + rng.normal(0, 1, A), sod + rng.normal(0, 1, A),
            (U - 1) / 2 + rng.normal(0, 1, A), (V - 1) / 2 + rng.normal(0, 1, A),
            *(rng.normal(0, 0.5, A) for _ in range(3))]
    geom = [np.asarray(g, np.float32) for g in geom]
    proj = rng.normal(size=(A, U, V)).astype(np.float32)
    up = rng.normal(size=shape).astype(np.float32)
    return proj, geom, up


def cuda(x):
    return torch.as_tensor(x).cuda()


def gradients(proj, geom, up, case, geometry):
    from cbct_backprojector import backproject

    shape, U, V, px, vs, sid, sod, off = case
    p = cuda(proj).requires_grad_()
    g = [cuda(x).requires_grad_(geometry) for x in geom]
    vol = backproject(p, *g, px, shape, vs, volume_offset=off)
    return torch.autograd.grad(vol, [p, *g] if geometry else [p], grad_outputs=cuda(up))


@pytest.mark.parametrize("case", CASES, ids=str)
def test_projection_gradient(case, oracle):
    shape, U, V, px, vs, sid, sod, off = case
    proj, geom, up = make(case)
    (alone,) = gradients(proj, geom, up, case, False)
    nine = gradients(proj, geom, up, case, True)[0]
    truth, _ = oracle.backproject_backward(up, proj, geom, px, vs, off)
    assert float(np.abs(truth).sum()) > 0.0
    assert rel_l2(alone.cpu(), truth) < GRAD_RTOL
    assert rel_l2(nine.cpu(), truth) < GRAD_RTOL
    assert rel_l2(alone.cpu(), nine.cpu()) < SAME_RTOL


def test_gather_is_reproducible():
    case = CASES[4]
    proj, geom, up = make(case)
    a = gradients(proj, geom, up, case, False)[0]
    for _ in range(3):
        assert torch.equal(a, gradients(proj, geom, up, case, False)[0])


@pytest.mark.parametrize("value", [math.inf, -math.inf, math.nan])
def test_non_finite_voxel_reaches_its_own_pixels_only(value):
    case = CASES[2]
    proj, geom, up = make(case)
    z, y, x = 17, 15, 12
    one = np.zeros_like(up)
    one[z, y, x] = 1.0
    touched = gradients(proj, geom, one, case, False)[0] != 0
    assert 0 < int(touched.sum()) <= 4 * proj.shape[0]
    bad = up.copy()
    bad[z, y, x] = value
    got = gradients(proj, geom, bad, case, False)[0]
    assert torch.equal(~torch.isfinite(got), touched)
    clean = up.copy()
    clean[z, y, x] = 0.0
    want = gradients(proj, geom, clean, case, False)[0]
    assert rel_l2(got[~touched].cpu(), want[~touched].cpu()) < SAME_RTOL


# Scans that are gathered: the smallest depth and detector, tiles of V with one, two and
# three pixels a thread and their remainders, several tiles, one bin, ragged last
# blocks of bins, offsets.
GATHERED = [
    ((48, 33, 35), 30, 48, 1.0, 1.0, 200.0, 120.0, (0.0, 0.0, 0.0)),
    ((49, 40, 34), 41, 65, 1.0, 1.0, 200.0, 120.0, (1.5, -2.0, 0.7)),
    ((64, 32, 33), 2, 96, 0.9, 1.0, 260.0, 160.0, (0.0, 3.0, 0.0)),
    ((60, 50, 32), 38, 97, 0.8, 1.0, 260.0, 160.0, (0.0, 0.0, 0.0)),
    ((120, 34, 40), 50, 193, 1.0, 1.0, 300.0, 180.0, (0.0, 0.0, -2.0)),
    ((330, 32, 33), 21, 529, 1.0, 1.0, 900.0, 540.0, (0.0, 0.0, 0.0)),
    ((250, 33, 32), 19, 1040, 0.5, 1.0, 800.0, 400.0, (0.0, 0.0, 0.0)),
]


def chosen(proj, geom, up, case):
    """dgc_backproject_adjoint's result and whether the views chose the gather (row 0 of the
    view table, which opens the workspace)."""
    from dgc_b200 import _native

    (D, H, W), U, V, px, vs, sid, sod, off = case
    lib, A = _native.lib(), proj.shape[0]
    n = lib.dgc_backproject_adjoint_workspace_bytes(A, D, H, W)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    out = torch.empty(proj.shape, device="cuda")
    g, u = [cuda(x) for x in geom], cuda(up)
    _native.check(lib.dgc_backproject_adjoint(
        u.data_ptr(), A, U, V, *[x.data_ptr() for x in g], px, D, H, W, vs, *off, out.data_ptr(),
        ws.data_ptr(), n, torch.cuda.current_stream().cuda_stream))
    return out, int(ws[36:40].view(torch.int32)[0])


@pytest.mark.parametrize("A", [6, 11])
@pytest.mark.parametrize("case", GATHERED, ids=str)
def test_gathered_scans(case, A, oracle):
    proj, geom, up = make(case, A=A)
    got, gathered = chosen(proj, geom, up, case)
    assert gathered == 1
    truth, _ = oracle.backproject_backward(up, proj, geom, case[3], case[4], case[7])
    assert rel_l2(got.cpu(), truth) < GRAD_RTOL
    assert torch.equal(got, chosen(proj, geom, up, case)[0])


def test_gathered_beside_the_geometry_gradients(oracle):
    """The projection gradient's values, and the geometry gradients as a call for these
    alone gives them (the same march, reduced in a fixed order): bit for bit."""
    from dgc_b200 import _ops

    case = ((100, 128, 129), 60, 120, 1.0, 1.0, 500.0, 300.0, (0.0, 0.0, 0.0))
    proj, geom, up = make(case, A=98)
    assert 128 * 129 * 98 >= 1600000
    nine = gradients(proj, geom, up, case, True)
    again = gradients(proj, geom, up, case, True)
    assert all(torch.equal(a, b) for a, b in zip(nine, again))
    truth, _ = oracle.backproject_backward(up, proj, geom, 1.0, 1.0, case[7])
    assert rel_l2(nine[0].cpu(), truth) < GRAD_RTOL
    alone = _ops.bp_backward(cuda(up), cuda(proj), *[cuda(g) for g in geom], 1.0, 1.0,
                             compute_grad_proj=False)
    assert all(torch.equal(a, b) for a, b in zip(nine[1:], alone[1:]))


def test_non_finite_voxel_of_a_gathered_scan():
    case = GATHERED[1]
    proj, geom, up = make(case)
    z, y, x = 17, 15, 12
    one = np.zeros_like(up)
    one[z, y, x] = 1.0
    touched = gradients(proj, geom, one, case, False)[0] != 0
    bad = up.copy()
    bad[z, y, x] = math.nan
    assert torch.equal(~torch.isfinite(gradients(proj, geom, bad, case, False)[0]), touched)


def change(geom, index, view, value):
    geom = [g.copy() for g in geom]
    geom[index][view] = value
    return geom


@pytest.mark.parametrize("name,case,A,edit", [
    ("magnification 1.1", ((64, 40, 33), 40, 60, 1.0, 1.0, 176.0, 160.0, (0.0, 0.0, 0.0)), 8, None),
    ("voxels of 6 pixels", ((64, 40, 33), 60, 400, 0.25, 1.0, 240.0, 160.0, (0.0, 0.0, 0.0)), 8, None),
    ("a detector past the shadow", ((64, 40, 33), 40, 150, 1.0, 1.0, 260.0, 160.0, (0.0, 0.0, 0.0)), 8, None),
    ("one view of low magnification", ((64, 40, 33), 40, 97, 0.9, 1.0, 260.0, 160.0, (0.0, 0.0, 0.0)), 8, (2, 5, 275.0)),
    ("one view among the voxels", ((64, 40, 33), 40, 97, 0.9, 1.0, 260.0, 160.0, (0.0, 0.0, 0.0)), 8, (2, 5, 12.0)),
    ("few views", ((64, 40, 33), 40, 97, 0.9, 1.0, 260.0, 160.0, (0.0, 0.0, 0.0)), 5, None),
    ("few columns a bin", ((64, 33, 33), 74, 97, 0.9, 1.0, 260.0, 160.0, (0.0, 0.0, 0.0)), 8, None),
    ("a slab", ((47, 40, 33), 40, 70, 0.9, 1.0, 260.0, 160.0, (0.0, 0.0, 0.0)), 8, None),
], ids=lambda x: x if isinstance(x, str) else "")
def test_scans_that_are_scattered(name, case, A, edit, oracle):
    """Where the gather would be the slower one, by the sizes or by any one view."""
    proj, geom, up = make(case, A=A)
    if edit:
        geom = change(geom, *edit)
    got, gathered = chosen(proj, geom, up, case)
    assert gathered == 0
    truth, _ = oracle.backproject_backward(up, proj, geom, case[3], case[4], case[7])
    assert rel_l2(got.cpu(), truth) < GRAD_RTOL


def test_a_view_without_numbers_contributes_nothing():
    case = ((64, 40, 33), 40, 97, 0.9, 1.0, 260.0, 160.0, (0.0, 0.0, 0.0))
    proj, geom, up = make(case, A=8)
    got, gathered = chosen(proj, change(geom, 0, 3, math.nan), up, case)
    assert gathered == 0 and not got[3].any()
    want, gathered = chosen(proj, geom, up, case)
    assert gathered == 1
    assert rel_l2(got[4:].cpu(), want[4:].cpu()) < SAME_RTOL


@pytest.mark.parametrize("geometry", [False, True])
def test_without_room_for_the_columns(geometry, monkeypatch):
    """No device memory for the gather's copy of the volume: the scatter, in the room
    that the view table (and the quads and sums of the geometry gradients) takes."""
    from dgc_b200 import _native, _ops

    case = ((100, 283, 284), 12, 100, 1.0, 1.0, 900.0, 600.0, (0.0, 0.0, 0.0))
    (D, H, W), U, V = case[:3]
    A = 20
    proj, geom, up = make(case, A=A)
    want = gradients(proj, geom, up, case, geometry)
    lib = _native.lib()
    most, least = ((lib.dgc_backproject_backward_workspace_bytes(A, U, V, D, H, W),
                    lib.dgc_backproject_backward_least_workspace_bytes(A, U, V, D, H, W)) if geometry else
                   (lib.dgc_backproject_adjoint_workspace_bytes(A, D, H, W),
                    lib.dgc_backproject_adjoint_least_workspace_bytes(A)))
    assert most >= 4 * D * H * W > least
    asked, room = [], _ops._workspace

    def tight(nbytes, device):
        if nbytes == most:
            asked.append(nbytes)
            raise torch.cuda.OutOfMemoryError("no room")
        return room(nbytes, device)

    monkeypatch.setattr(_ops, "_workspace", tight)
    got = gradients(proj, geom, up, case, geometry)
    assert asked == [most]
    assert rel_l2(got[0].cpu(), want[0].cpu()) < SAME_RTOL
    assert all(torch.equal(a, b) for a, b in zip(got[1:], want[1:]))


def test_least_workspace():
    """dgc_backproject_adjoint in the least workspace, and refused below it."""
    from dgc_b200 import _native

    case = GATHERED[1]
    (D, H, W), U, V, px, vs, sid, sod, off = case
    proj, geom, up = make(case)
    want, gathered = chosen(proj, geom, up, case)
    assert gathered == 1
    lib, A = _native.lib(), proj.shape[0]
    n = lib.dgc_backproject_adjoint_least_workspace_bytes(A)
    ws = torch.empty(n, dtype=torch.uint8, device="cuda")
    out = torch.empty_like(want)
    g, u = [cuda(x) for x in geom], cuda(up)

    def call(nbytes):
        return lib.dgc_backproject_adjoint(
            u.data_ptr(), A, U, V, *[x.data_ptr() for x in g], px, D, H, W, vs, *off, out.data_ptr(),
            ws.data_ptr(), nbytes, torch.cuda.current_stream().cuda_stream)

    assert call(n) == 0
    assert rel_l2(out.cpu(), want.cpu()) < SAME_RTOL
    assert call(n - 256) == 3
