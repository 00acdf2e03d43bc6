"""Bounds of the coordinates taken while they are copied in: an outermost event is found
wherever it stands, so that the grid reaches it."""
import numpy as np
import pytest

import hawkes_b200 as hb
from hawkes_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [1, 2])
@pytest.mark.parametrize("n", [24000, 24003, 24005])
def test_outermost_events_anywhere(D, n):
    # positions in and across the copy's blocks of eight values, and in its remainder.
    # An event outside the grid would be pulled to its edge, 6 tauX scales away:
    # P_i of the event moves by its whole self-excitation, far above 1e-12.
    loc, t = workloads.uniform(n, 61, D=D)
    p = np.asarray(workloads.BASE_PARAMS)
    with hb.CudaHawkes(D, n, hb.CUDA, 0) as e, hb.CudaHawkes(D, n, hb.CUDA, 0) as ref:
        ref.setSweepShape(2, 32)  # the pair sweep
        for x in (e, ref):
            x.setTimesData(t)
        for at in [0, 1, 2, 3, 4, 5, 6, 7, 1001, n - 5, n - 3, n - 2, n - 1]:
            x = loc.copy()
            for k in range(D):
                x[at, k] = loc[:, k].max() + 7.0 + k if at % 2 else loc[:, k].min() - 9.0 - k
            out = []
            for eng in (e, ref):
                eng.updateLocations(-1, x)
                eng.setParameters(p)
                ll, g = eng.getLogLikelihoodAndGradient()
                out.append((ll, np.asarray(g), eng.lastLaunchEvals(), eng.getProbsSelfExcite()))
            (la, ga, ea, pa), (lb, gb, eb, pb) = out
            assert ea == 0.0 and eb > 0.0
            assert abs(la - lb) <= 1e-12 * abs(lb)
            np.testing.assert_allclose(ga, gb, rtol=1e-9)
            np.testing.assert_allclose(pa, pb, rtol=1e-12, atol=1e-300)
