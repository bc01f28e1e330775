"""The forward march in groups of samples against the march sample by sample (the arm
whose loop the compiler unrolls): the same samples and sums, so the same bits -- for rays
of no, one, two, three, four and many samples, rays through the volume's padding (clamped
coordinates), voxel sizes that divide exactly and that do not, and an offset volume.
"""

import math

import pytest
import torch

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not torch.cuda.is_available(), reason="needs a GPU")]


@pytest.mark.parametrize("shape", [(1, 1, 1), (3, 2, 4), (9, 11, 10), (40, 33, 37)])
@pytest.mark.parametrize("voxel,step,off", [(1.0, 0.5, (0.0, 0.0, 0.0)), (1.0, 1.9, (0.3, -0.2, 0.1)),
                                            (0.7, 0.2, (0.0, 0.0, 0.0)), (2.0, 7.0, (0.0, 0.0, 0.0)),
                                            (0.9, 3.1, (-0.4, 0.2, 0.6))])
def test_groups_give_the_bits_of_single_samples(shape, voxel, step, off):
    from dgc_b200 import _native, _ops

    g = torch.Generator().manual_seed(sum(shape))
    vol = torch.randn(shape, generator=g).cuda()
    A, U, V = 9, 37, 41

    def jitter(x, s):
        return (x + s * torch.randn(A, generator=g)).float().cuda()

    geom = [jitter(torch.arange(A) * 2 * math.pi / A, 0.05), jitter(200.0, 1.0), jitter(120.0, 1.0),
            jitter((U - 1) / 2, 1.0), jitter((V - 1) / 2, 1.0), jitter(0.0, 0.5), jitter(0.0, 0.5),
            jitter(0.0, 0.5)]
    lib = _native.lib()

    def run():
        return _ops.fp_forward(vol, *geom, 1.0, U, V, step, voxel, *off)

    lib.dgc_fp_clear_arm_rules()
    got = run()
    try:
        _native.check(lib.dgc_fp_add_arm_rule(1 << 40, 0, 4, 2, 0))
        want = run()
    finally:
        lib.dgc_fp_clear_arm_rules()
    assert torch.equal(got, want)
    assert float(want.abs().max()) > 0
