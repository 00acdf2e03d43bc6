"""Events recorded by the day or week: the self-excitation window reaches past the gap
between recorded times, so that evaluations are no slower than without a window (where
the window ends before the gap, the finish completes every sum, up to eight times as
slow)."""
import time

import numpy as np
import pytest

import hawkes_b200 as hb
from hawkes_b200 import workloads

pytestmark = pytest.mark.gpu

FP64 = hb.CUDA
FP32C = hb.CUDA | hb.COMPENSATED


def _times(e, p, k):
    """Seconds of an evaluation that moves parameter k, the least of eight."""
    best = np.inf
    for j in range(8):
        p = p.copy()
        p[k] *= 1.001
        e.setParameters(p)
        t0 = time.perf_counter()
        e.getLogLikelihoodAndGradient()
        best = min(best, time.perf_counter() - t0)
    return best


@pytest.mark.parametrize("flags,n,gap,omega,form", [
    (FP64, 20000, 168.0, 0.3, "sorted"), (FP64, 80000, 24.0, 1.0, "sorted"),
    (FP64, 40000, 168.0, 0.3, "series"), (FP32C, 80000, 168.0, 1.0, "sorted")])
def test_recorded_times_are_not_slower_than_without_a_window(flags, n, gap, omega, form):
    rng = np.random.default_rng(9)
    loc = rng.uniform(0.0, 20.0, (n, 2))
    t = np.floor(rng.uniform(0.0, 8760.0, n) / gap) * gap
    if form == "sorted":
        t = np.sort(t)
    else:  # four series after one another
        t = np.concatenate([np.sort(v) for v in np.split(t, 4)])
    p = np.asarray(workloads.BASE_PARAMS).copy()
    p[3] = omega
    times, values = {}, {}
    for name, extra in (("window", 0), ("full", hb.NO_TAIL_TRUNCATION)):
        with hb.CudaHawkes(2, n, flags | extra, 0) as e:
            e.setTimesData(t)
            e.updateLocations(-1, loc)
            e.setParameters(p)
            ll, _ = e.getLogLikelihoodAndGradient()
            values[name] = ll, e.getProbsSelfExcite()
            times[name] = _times(e, p, 2), _times(e, p, 0)  # all anew, a step
    print("\nus:", {k: [round(v * 1e6) for v in t] for k, t in times.items()})
    for a, b in zip(times["window"], times["full"]):
        assert a < 1.3 * b
    (lw, pw), (lf, pf) = values["window"], values["full"]
    if flags == FP64:
        assert abs(lw - lf) <= 1e-13 * abs(lf)
        np.testing.assert_allclose(pw, pf, rtol=1e-12, atol=1e-300)
    else:
        assert abs(lw - lf) <= 1e-8 * abs(lf)
