"""Self-excitation steps on events that come in bursts, whose strips have bands of very
different widths, against full pair sweeps without a window."""
import numpy as np
import pytest

import hawkes_b200 as hb
import oracle
from hawkes_b200 import workloads

pytestmark = pytest.mark.gpu

FP64 = hb.CUDA
FP32C = hb.CUDA | hb.COMPENSATED


def _events(n, bursts, share, rng):
    """share of the events in bursts of four hours, at the ends too."""
    loc = rng.uniform(0.0, 20.0, (n, 2))
    t = rng.uniform(0.0, 8760.0, n)
    m = int(n * share)
    start = np.linspace(0.0, 8756.0, bursts) if bursts > 1 else np.array([4000.0])
    t[:m] = start[np.arange(m) % bursts] + rng.uniform(0.0, 4.0, m)
    return loc, np.sort(t)


@pytest.mark.parametrize("flags", [FP64, FP32C], ids=["fp64", "fp32c"])
@pytest.mark.parametrize("n,bursts,share", [(3000, 1, 0.1), (4097, 3, 0.9), (12001, 1, 0.5),
                                            (20000, 2, 0.3), (33000, 5, 0.1)])
def test_steps_on_bursts(flags, n, bursts, share):
    # FP64: orders of the sums only, 1e-12 and 1e-11 of a component's scale.  FP32-
    # compensated: the mode's error, 2e-9 and 2e-8.
    rng = np.random.default_rng(n)
    loc, t = _events(n, bursts, share, rng)
    p = np.asarray(workloads.BASE_PARAMS)
    P = p * np.exp(0.2 * rng.standard_normal((5, 6)))
    P[:, 1:3] = p[1:3]
    scale = oracle.oracle_eval(loc, t, p, threads=8)["grad_scale"]
    rl, rg = (1e-12, 1e-11) if flags == FP64 else (2e-9, 2e-8)
    with hb.CudaHawkes(2, n, flags, 0) as e, \
            hb.CudaHawkes(2, n, FP64 | hb.NO_INCREMENTAL | hb.NO_TAIL_TRUNCATION, 0) as ref:
        for x in (e, ref):
            x.setTimesData(t)
            x.updateLocations(-1, loc)
            x.setParameters(p)
            x.getLogLikelihoodAndGradient()

        def check(got, q):
            ref.setParameters(q)
            ll, g = ref.getLogLikelihoodAndGradient()
            assert abs(got[0] - ll) <= rl * abs(ll)
            assert np.all(np.abs(got[1] - g) <= rg * scale)

        for q in P[:3]:  # single steps, then all in one call
            e.setParameters(q)
            got = e.getLogLikelihoodAndGradient()
            assert e.lastEvaluationPath == hb.PATH_SELF_EXCITATION
            check(got, q)
        ll, g = e.batchLogLikelihoodAndGradient(P)
        assert e.lastEvaluationPath == hb.PATH_SELF_EXCITATION
        for k in range(len(P)):
            check((ll[k], g[k]), P[k])
