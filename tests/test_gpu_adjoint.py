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
