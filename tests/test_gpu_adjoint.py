"""The volume gradient of ``project`` with fixed geometry (the adjoint kernel
without gradient sums) and with all nine gradients: edge records at the sizes
where their layout, tiles and cell moves change."""

import numpy as np
import pytest
import torch

from conftest import rel_l2
from test_gpu_forward import GRAD_RTOL, cuda32, random_case, run_project

pytestmark = pytest.mark.gpu

# The two kernels add the same FP32 samples with their weights rounded
# differently (2^-24 a weight) and in another order: a voxel's sum of up to a
# few hundred positive-and-negative terms agrees to a few 1e-7 of its norm.
SAME_RTOL = 5e-6

CASES = [
    # thin volumes (axes of stride 0), both sides of the column rounding, tile edges
    dict(shape=(1, 1, 1)), dict(shape=(1, 5, 4)), dict(shape=(3, 1, 2)), dict(shape=(2, 3, 1)),
    dict(shape=(40, 1, 1)), dict(shape=(15, 9, 31)), dict(shape=(16, 8, 32)),
    dict(shape=(17, 7, 33)), dict(shape=(33, 20, 5)),
    # power-of-two voxels with and without an offset; the general march
    dict(shape=(20, 28, 24), vs=1.0, off=(0.0, 0.0, 0.0)), dict(shape=(20, 28, 24), vs=0.5),
    dict(shape=(20, 28, 24), vs=0.8, off=(0.0, 0.0, 0.0)),
    # steps longer than a voxel move by more than one cell
    dict(shape=(20, 28, 24), vs=1.0, step=1.0), dict(shape=(20, 28, 24), vs=0.5, step=1.7),
    dict(shape=(20, 28, 24), vs=0.8, step=0.05),
]


@pytest.mark.parametrize("options", CASES, ids=lambda o: "-".join(map(str, o.values())))
def test_volume_gradient_alone(options, oracle):
    options = dict(dict(A=7, U=21, V=35, vs=1.0, step=0.37), **options)
    case = random_case(41, **options)
    case["geom"][0][:4] = [0.0, np.pi / 2, np.pi, 3 * np.pi / 2]  # rays along the axes
    out, vol, geom = run_project(case, requires_grad=True)
    rng = np.random.default_rng(3)
    up = cuda32(rng.normal(size=tuple(out.shape)))
    up[0, :3] = 0.0
    nine = torch.autograd.grad(out, [vol, *geom], grad_outputs=up)[0]
    alone_vol = cuda32(case["vol"]).requires_grad_()
    alone_out, _, _ = run_project(case, vol=alone_vol)
    assert torch.equal(alone_out, out)
    (alone,) = torch.autograd.grad(alone_out, [alone_vol], grad_outputs=up)
    truth, _ = oracle.project_backward(up.cpu().numpy(), case["vol"], case["geom"], case["px"],
                                       case["step"], case["vs"], case["off"], mode=1)
    assert float(np.abs(truth).sum()) > 0.0
    assert rel_l2(alone.cpu(), truth) < GRAD_RTOL
    assert rel_l2(nine.cpu(), truth) < GRAD_RTOL
    assert rel_l2(alone.cpu(), nine.cpu()) < SAME_RTOL


@pytest.mark.parametrize("shape,A,U,V", [
    ((9, 8, 7), 8, 40, 30),      # 13 rays a record: one copy of the records
    ((9, 8, 7), 10, 60, 100),    # two, four, eight, sixteen
    ((9, 8, 7), 20, 60, 100), ((9, 8, 7), 40, 60, 100), ((9, 8, 7), 40, 100, 200),
    ((20, 20, 20), 90, 100, 100),  # as many as 512 KB hold
    ((1, 6, 5), 30, 40, 30), ((5, 1, 6), 30, 40, 30), ((2, 3, 40), 30, 60, 30)])
def test_copies_of_the_records(shape, A, U, V):
    """Small volumes under many rays, whose CTAs add into several copies of the records:
    the volume gradient alone and beside the geometry's, against that in a workspace
    of one copy, which adds the same samples."""
    from dgc_b200 import _native

    case = random_case(17, shape=shape, A=A, U=U, V=V, vs=4.0, step=1.3, off=(0.0, 0.0, 0.0))
    out, vol, geom = run_project(case, requires_grad=True)
    up = cuda32(np.random.default_rng(4).normal(size=tuple(out.shape)))
    nine = torch.autograd.grad(out, [vol, *geom], grad_outputs=up)[0]
    alone_vol = cuda32(case["vol"]).requires_grad_()
    alone_out, _, _ = run_project(case, vol=alone_vol)
    (alone,) = torch.autograd.grad(alone_out, [alone_vol], grad_outputs=up)
    D, H, W = shape
    column = (D + 4) // 4 * 4 if D >= 16 else D + 1
    n = 8 * column * (W + 2 if W > 1 else 1) * (H + 2 if H > 1 else 1)
    n = (n + 255) // 256 * 256
    lib, ws, one = _native.lib(), torch.empty(n, dtype=torch.uint8, device="cuda"), torch.empty_like(alone)
    g = [cuda32(x) for x in case["geom"]]

    def call(nbytes):
        return lib.dgc_project_adjoint(
            up.data_ptr(), D, H, W, *[x.data_ptr() for x in g], A, case["px"], U, V, case["step"],
            case["vs"], 0.0, 0.0, 0.0, one.data_ptr(), ws.data_ptr(), nbytes,
            torch.cuda.current_stream().cuda_stream)

    assert call(n) == 0 and call(n - 256) == 3
    assert float(one.abs().sum()) > 0.0
    assert rel_l2(alone.cpu(), one.cpu()) < SAME_RTOL
    assert rel_l2(nine.cpu(), one.cpu()) < SAME_RTOL
