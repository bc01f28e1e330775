"""The one-launch validity check of per-view arrays (dgc_check_values) and the
errors that fdk_filter and reconstruct_fdk raise from it."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 255, 256, 257, 1000])
@pytest.mark.parametrize("bad", [math.nan, math.inf, -math.inf, 0.0, -0.0, -3.0])
def test_faults_of_each_array(count, bad):
    from dgc_b200 import _ops

    for where in (0, count - 1):
        for k in (0, 7, 15):
            arrays = [torch.full((count,), 1.0 + i, device="cuda") for i in range(16)]
            arrays[k][where] = bad
            got = _ops.value_faults(arrays)
            assert got == [((not math.isfinite(bad), bad <= 0) if i == k else (False, False))
                           for i in range(16)]
            # the same answers as the reductions it stands for
            assert got[k] == (not bool(torch.isfinite(arrays[k]).all()),
                              bool((arrays[k] <= 0).any()))


def test_errors_come_in_argument_order():
    from cbct_backprojector import fdk_filter, reconstruct_fdk

    A, U, V = 5, 12, 10
    p = torch.rand(A, U, V, device="cuda")
    good = torch.full((A,), 100.0, device="cuda")
    nan = good.clone()
    nan[3] = math.nan
    for sod, sid, frame, message in [
            (nan, torch.ones(3), None, "sod must contain"), (good, nan, None, "sid must contain"),
            (good, -good, (good, good, nan), "sid must contain"),
            (good, good, (0.0, None, None), "frame dist must contain finite positive"),
            (good, good, (None, -1.0, nan), "frame v must contain finite values"),
            (1e39, good, None, "sod must contain"), (good[:2], nan, None, "sod must be a scalar")]:
        with pytest.raises(ValueError, match=message):
            fdk_filter(p, 1.0, sod, sid, frame=frame)
    with pytest.raises(TypeError, match="frame must be"):
        fdk_filter(p, 1.0, good, good, frame=(1.0, 2.0))
    zero = torch.zeros(A, device="cuda")
    angles = torch.arange(A, device="cuda") * 0.1
    with pytest.raises(ValueError, match="only finite"):
        reconstruct_fdk(p, angles, -good, good, nan, zero, zero, zero, zero, 1.0, (4, 4, 4), 1.0)
    with pytest.raises(ValueError, match="positive distances"):
        reconstruct_fdk(p, angles, good, zero, zero, zero, zero, zero, zero, 1.0, (4, 4, 4), 1.0)
    with pytest.raises(ValueError, match="in front of the detector"):
        reconstruct_fdk(p, angles, good, good, zero, zero, zero, -2 * good, zero, 1.0, (4, 4, 4), 1.0,
                        offset_preweight=True)
    for kw in (dict(), dict(offset_preweight=True)):
        with pytest.raises(ValueError, match="short scan must cover"):
            reconstruct_fdk(p, angles, good, good, zero, zero, zero, zero, zero, 1.0, (4, 4, 4), 1.0,
                            short_scan=True, **kw)
