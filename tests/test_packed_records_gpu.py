"""Steps that leave events, tauX and tauT alone sweep the records packed before:
against engines that never did, after every kind of change in between."""
import numpy as np
import pytest

import hawkes_b200 as hb
from hawkes_b200 import workloads

pytestmark = pytest.mark.gpu

FP32C = hb.CUDA | hb.COMPENSATED


@pytest.mark.parametrize("flags", [FP32C, hb.CUDA | hb.FLOAT, FP32C | hb.ORDERED],
                         ids=["fp32c", "float", "ordered"])
@pytest.mark.parametrize("n", [300, 5000])
def test_steps_follow_every_change(flags, n):
    # the same kernels on the same records: the same bits, but for the background
    # sums a step keeps from another sweep shape or a moved event's update (1e-9)
    rng = np.random.default_rng(n)
    loc, t = workloads.uniform(n, 3)
    base = np.asarray(workloads.BASE_PARAMS)
    with hb.CudaHawkes(2, n, flags, 0) as e:
        now = {"loc": loc.copy(), "t": t, "p": base.copy()}

        def evaluate():
            e.setParameters(now["p"])
            got = e.getLogLikelihoodAndGradient()[0]
            with hb.CudaHawkes(2, n, flags, 0) as f:
                f.setTimesData(now["t"])
                f.updateLocations(-1, now["loc"])
                f.setParameters(now["p"])
                want = f.getLogLikelihoodAndGradient()[0]
            tol = 1e-9 if flags != hb.CUDA | hb.FLOAT else 2e-5
            assert abs(got - want) <= tol * abs(want)

        def steps():
            for k in (0, 3, 0, 4, 3):
                now["p"][k] *= 1.0 + 0.05 * rng.random()
                evaluate()

        e.setTimesData(t)
        e.updateLocations(-1, now["loc"])
        evaluate()
        steps()
        now["loc"][n // 2] += 0.7  # one event moves and stays
        e.updateLocations(n // 2, now["loc"][n // 2])
        evaluate()
        steps()
        e.storeState()  # one moves and returns
        kept = now["loc"].copy()
        now["loc"][7] -= 0.9
        e.updateLocations(7, now["loc"][7])
        evaluate()
        steps()
        saved = now["p"].copy()
        e.restoreState()
        now["loc"] = kept
        now["p"] = saved
        steps()
        now["p"][1] *= 1.1  # another scaling, and back
        evaluate()
        steps()
        now["p"][1] /= 1.1
        evaluate()
        steps()
        e.batchLogLikelihoodAndGradient(np.stack([now["p"], now["p"] * 1.1]))  # other records
        steps()
        now["t"] = now["t"] * 0.9  # new events
        e.setTimesData(now["t"])
        steps()
        now["loc"] = now["loc"][::-1].copy()
        e.updateLocations(-1, now["loc"])
        steps()
