"""Evaluations where the device has memory for the gridded sums' workspace but then not
for the sweep: they take the pair sweep, which needs far less, as they would have
without a grid."""
import numpy as np
import pytest

import hawkes_b200 as hb
from hawkes_b200 import workloads

pytestmark = pytest.mark.gpu

N = 400000


def _engine(loc, t):
    e = hb.CudaHawkes(2, N, hb.CUDA, 0)
    e.setTimesData(t)
    e.updateLocations(-1, loc)
    e.setParameters(workloads.BASE_PARAMS)
    return e


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


def test_the_pair_sweep_takes_over():
    import torch
    loc, t = workloads.uniform(N, 2)
    # every kernel used below is loaded, and what an evaluation allocates measured
    with hb.CudaHawkes(2, 30000, hb.CUDA | hb.NO_TAIL_TRUNCATION, 0) as w:
        x, s = workloads.uniform(30000, 1)
        w.setTimesData(s)
        w.updateLocations(-1, x)
        w.setParameters(workloads.BASE_PARAMS)
        w.getLogLikelihoodAndGradient()
    torch.zeros(1, device="cuda")
    with _engine(loc, t) as e:
        before = _free()
        want = e.getLogLikelihoodAndGradient()
        assert e.lastLaunchEvals() == 0.0
        needed = before - _free()
    assert needed > 300 << 20  # the workspace and, after it, the partial sums
    with _engine(loc, t) as e:
        # all but `needed` less 16 MiB: the last buffers do not fit
        filler = torch.empty(_free() - needed + (16 << 20), dtype=torch.uint8, device="cuda")
        try:
            got = e.getLogLikelihoodAndGradient()
            assert e.lastLaunchEvals() > 0.0
        finally:
            del filler
            torch.cuda.empty_cache()
        assert abs(got[0] - want[0]) <= 1e-12 * abs(want[0])
        np.testing.assert_allclose(got[1], want[1], rtol=1e-9)
        # and with memory again the grid
        e.setParameters(np.asarray(workloads.BASE_PARAMS) * 1.001)
        e.getLogLikelihoodAndGradient()
        assert e.lastLaunchEvals() == 0.0
