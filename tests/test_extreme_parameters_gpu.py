"""Parameters whose squares overflow: terms of zero times infinity are not a number and
do not turn into one, other results are the oracle's."""
import numpy as np
import pytest

import hawkes_b200 as hb
import oracle

pytestmark = pytest.mark.gpu

BASE = np.array([1.0, 0.5, 0.01, 1.0, 0.5, 1.0])


def _events(coincident):
    rng = np.random.default_rng(3)
    t = np.sort(rng.uniform(0.0, 400.0, 300))
    loc = rng.uniform(0.0, 20.0, (300, 1))
    if coincident:
        loc[100] = loc[101]
    return loc, t


@pytest.mark.parametrize("step", [False, True], ids=["sweep", "self-excitation step"])
@pytest.mark.parametrize("coincident", [False, True])
def test_sigma_squared_overflows(coincident, step):
    # infinity times the squared distance: no self-excitation, but for events at one
    # place, whose term is not a number
    loc, t = _events(coincident)
    p = BASE.copy()
    with hb.CudaHawkes(1, len(t), hb.CUDA, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        if step:
            e.setParameters(p)
            e.getLogLikelihoodAndGradient()
        p[0] = 1e160
        e.setParameters(p)
        ll, _ = e.getLogLikelihoodAndGradient()
        assert e.lastEvaluationPath == (hb.PATH_SELF_EXCITATION if step else hb.PATH_SWEEP)
    if coincident:
        assert np.isnan(ll)
    else:
        want = oracle.oracle_eval(loc, t, p)["loglik"]
        assert abs(ll - want) <= 1e-12 * abs(want)


@pytest.mark.parametrize("k", [1, 2], ids=["tauX", "tauT"])
def test_background_precision_squared_overflows(k):
    # an event's own background term is infinity times zero
    loc, t = _events(False)
    p = BASE.copy()
    p[k] = 1e160
    with hb.CudaHawkes(1, len(t), hb.CUDA, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        e.setParameters(p)
        ll, g = e.getLogLikelihoodAndGradient()
    assert np.isnan(ll) and np.all(np.isnan(g))
