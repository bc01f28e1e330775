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
