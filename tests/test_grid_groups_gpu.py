"""Gridded problems of one call that run in several groups: both spline orders, and more
than the workspace holds at once."""
import numpy as np
import pytest

import hawkes_b200 as hb
from hawkes_b200 import workloads

pytestmark = pytest.mark.gpu

FP64 = hb.CUDA
FP32C = hb.CUDA | hb.COMPENSATED


def _single(loc, t, p, flags):
    with hb.CudaHawkes(2, len(t), flags, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        e.setParameters(p)
        ll, g = e.getLogLikelihoodAndGradient()
        assert e.lastLaunchEvals() == 0.0
        return ll, np.asarray(g)


def test_sets_on_both_sides_of_the_higher_order():
    # FP32-compensated: order 16 from 65,536 events on, order 12 below.  The grids' sums
    # are the single evaluations' own; the self-excitation sums of a mixed call are
    # FP32-compensated for all (2^-24 of an event's sum, either sign), in a single large
    # evaluation FP64: the mode's 1e-8 on the log-likelihood, 6e-8 of a gradient
    # component's scale, which is at most some ten times the component here.
    sizes = [70000, 40000, 65536, 65535]
    sets = [workloads.uniform(n, 40 + k) for k, n in enumerate(sizes)]
    P = np.asarray(workloads.BASE_PARAMS) * np.array([1.0, 0.9, 1.2, 1.0, 1.1, 0.9])
    P = np.stack([P * (1 + 0.01 * k) for k in range(len(sizes))])
    with hb.Multiset(2, sizes, FP32C, 0) as m:
        for s, (loc, t) in enumerate(sets):
            m.setData(s, loc, t)
        ll, g = m.logLikelihoodAndGradient(P)
        ll2, g2 = m.logLikelihoodAndGradient(P)
    assert np.array_equal(ll, ll2) and np.array_equal(g, g2)
    for s, (loc, t) in enumerate(sets):
        want = _single(loc, t, P[s], FP64)
        assert abs(ll[s] - want[0]) <= 1e-8 * abs(want[0])
        np.testing.assert_allclose(g[s], want[1], rtol=6e-7)


def test_more_problems_than_the_workspace_holds():
    # about 120 MB a problem: 1.25 GiB hold ten or eleven of the fourteen
    loc, t = workloads.uniform(100000, 50)
    P = workloads.proposals(14, 51)
    P[:, 1:3] = np.asarray(workloads.BASE_PARAMS)[1:3] * np.linspace(0.9, 1.1, 14)[:, None]
    with hb.CudaHawkes(2, len(t), FP64, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        ll, g = e.batchLogLikelihoodAndGradient(P)
        assert e.lastLaunchEvals() == 0.0
        launches = e.lastLaunchStats()[0]
    assert launches >= 20  # two groups of ten kernels
    for k in (0, 8, 9, 10, 11, 13):
        want = _single(loc, t, P[k], FP64)
        assert abs(ll[k] - want[0]) <= 1e-13 * abs(want[0])
        np.testing.assert_allclose(g[k], want[1], rtol=1e-10)


@pytest.mark.parametrize("n", [65536, 90000])
def test_steps_agree_with_full_evaluations_of_another_precision(n):
    # A large FP32-compensated evaluation has FP64 sums, a step in sigma or omega after it
    # the mode's own: 2e-9 of the log-likelihood and 2e-8 of a gradient component's scale
    # (some ten times the component at most here), the mode's error.
    loc, t = workloads.uniform(n, 70)
    p = np.asarray(workloads.BASE_PARAMS)
    q = p * np.array([1.1, 1, 1, 0.9, 1, 1])
    with hb.CudaHawkes(2, n, FP32C, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        e.setParameters(p)
        e.getLogLikelihoodAndGradient()
        e.setParameters(q)
        step = e.getLogLikelihoodAndGradient()
        assert e.lastEvaluationPath == hb.PATH_SELF_EXCITATION
    full = _single(loc, t, q, FP32C)
    assert abs(step[0] - full[0]) <= 2e-9 * abs(full[0])
    np.testing.assert_allclose(step[1], full[1], rtol=2e-7)
