"""The plan of an evaluation follows from its events, parameters and settings, not from
what the engine evaluated before: the same call gives the same bits."""
import numpy as np
import pytest

import hawkes_b200 as hb
from hawkes_b200 import workloads

pytestmark = pytest.mark.gpu

FP64 = hb.CUDA
FP32C = hb.CUDA | hb.COMPENSATED


def _evaluate(e, p):
    """(log-likelihood, gradient, background terms evaluated as pairs)."""
    e.setParameters(p)
    ll, g = e.getLogLikelihoodAndGradient()
    return ll, np.asarray(g), e.lastLaunchEvals()


def test_grid_choice_after_an_fp64_plan():
    # A large FP32-compensated evaluation sweeps in FP64 beside the grid.  A problem just
    # on the pair sweep's side of the choice is taken the same way after it: the edge is
    # found by bisection in tauX (a finer grid costs more) with pair sweeps in between, and
    # the FP64 cut counts up to 1.23 times the pairs, 1.1 times as large a tauX.
    n = 66000
    loc, t = workloads.uniform(n, 3)
    base = np.asarray(workloads.BASE_PARAMS)
    with hb.CudaHawkes(2, n, FP32C | hb.NO_INCREMENTAL, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)

        def at(scale):
            return base * np.array([1, scale, 1, 1, 1, 1])

        pairs, gridded = at(64.0), at(1.0)
        assert _evaluate(e, gridded)[2] == 0.0
        lo, hi = 1.0, 64.0
        while hi / lo > 1.01:
            mid = np.sqrt(lo * hi)
            assert _evaluate(e, pairs)[2] > 0.0
            if _evaluate(e, at(mid))[2] == 0.0:
                lo = mid
            else:
                hi = mid
        edge = at(hi * 1.02)
        assert _evaluate(e, pairs)[2] > 0.0
        ll, g, evals = _evaluate(e, edge)
        assert evals > 0.0
        assert _evaluate(e, gridded)[2] == 0.0
        again = _evaluate(e, edge)
        assert again[2] == evals
        assert again[0] == ll and np.array_equal(again[1], g)


@pytest.mark.parametrize("flags,R", [(FP64, 1), (FP64, 2), (FP32C, 2), (FP32C, 4)])
def test_fixed_events_per_thread_hold_for_every_plan(flags, R):
    # set alone, with the items per SM left to the engine: full sweeps and
    # self-excitation steps, of a few thousand events too
    loc, t = workloads.uniform(3000, 12)
    p = np.asarray(workloads.BASE_PARAMS)
    with hb.CudaHawkes(2, len(t), flags, 0) as e:
        e.setSweepShape(R, 0)
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        e.setParameters(p)
        e.getLogLikelihoodAndGradient()
        assert e.lastEvaluationPath == hb.PATH_SWEEP and e.sweepShape()[0] == R
        e.setParameters(p * np.array([1.1, 1, 1, 1, 1, 1]))
        e.getLogLikelihoodAndGradient()
        assert e.lastEvaluationPath == hb.PATH_SELF_EXCITATION and e.sweepShape()[0] == R


@pytest.mark.parametrize("flags,n", [(FP64, 30000), (FP32C, 40000)])
def test_plan_after_an_event_has_been_far_away(flags, n):
    # An event moves out of the box and back, or another one on its edge moves in: the
    # grid is laid over the present events, as in an engine that has seen no others.
    loc, t = workloads.uniform(n, 13)
    p = np.asarray(workloads.BASE_PARAMS)
    inward = loc.copy()
    edge = int(np.argmin(loc[:, 0]))
    inward[edge] = loc.mean(0)

    def fresh(x):
        with hb.CudaHawkes(2, n, flags, 0) as f:
            f.setTimesData(t)
            f.updateLocations(-1, x)
            return _evaluate(f, p)

    with hb.CudaHawkes(2, n, flags, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        first = _evaluate(e, p)
        assert first[2] == 0.0  # gridded
        e.updateLocations(5, loc[5] - 37.3)
        _evaluate(e, p * 1.1)
        e.updateLocations(5, loc[5])
        back = _evaluate(e, p)
        assert back[0] == first[0] and np.array_equal(back[1], first[1])
        e.updateLocations(edge, inward[edge])
        _evaluate(e, p * 1.1)
        got, want = _evaluate(e, p), fresh(inward)
        assert got[2] == want[2] == 0.0
        assert got[0] == want[0] and np.array_equal(got[1], want[1])


@pytest.mark.parametrize("n,omega,R", [(40000, 1.0, 1), (40000, 0.001, 2), (20000, 0.001, 1)])
def test_strip_height_of_fp64_self_excitation_sweeps(n, omega, R):
    # two rows a thread where the terms are many (8e8 here), one where the sweep is short
    # (2e8 and less)
    loc, t = workloads.uniform(n, 14)
    p = np.asarray(workloads.BASE_PARAMS) * np.array([1, 1, 1, omega, 1, 1])
    with hb.CudaHawkes(2, n, FP64, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        assert _evaluate(e, p)[2] == 0.0  # gridded: self-excitation only
        e.setParameters(p * np.array([1.1, 1, 1, 1, 1, 1]))
        e.getLogLikelihoodAndGradient()
        assert e.lastEvaluationPath == hb.PATH_SELF_EXCITATION and e.sweepShape()[0] == R


@pytest.mark.parametrize("flags,D,n", [(FP64, 2, 12000), (FP64, 1, 20000), (FP32C, 1, 20000),
                                       (FP32C, 2, 30000), (FP32C, 2, 70000)])
def test_crowded_events_keep_the_pair_sweep(flags, D, n):
    # Kernels ten times as wide put all events into a few bins of the grid, whose CTAs
    # then take them one after the other: up to 2.6 times the pair sweep's time.  The
    # larger of these sets are cheaper on the grid at the usual widths.
    loc, t = workloads.uniform(n, 15, D=D)
    p = np.asarray(workloads.BASE_PARAMS)
    wide = p * np.array([1, 0.05, 0.05, 1, 1, 1])
    with hb.CudaHawkes(D, n, flags, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        assert _evaluate(e, wide)[2] > 0.0
        if n > 20000:
            assert _evaluate(e, p)[2] == 0.0
        assert _evaluate(e, wide * 1.001)[2] > 0.0
