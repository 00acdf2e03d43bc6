"""Small sweeps take their tiles in halves and quarters: against whole tiles (a
fixed sweep shape) and the oracle, at the edges of tiles and of their parts."""
import numpy as np
import pytest

import hawkes_b200 as hb
import oracle
from hawkes_b200 import workloads

pytestmark = pytest.mark.gpu

FP64 = hb.CUDA
FP32C = hb.CUDA | hb.COMPENSATED


@pytest.mark.parametrize("unsorted", [False, True], ids=["sorted", "unsorted"])
@pytest.mark.parametrize("flags", [FP64, FP32C], ids=["fp64", "fp32c"])
@pytest.mark.parametrize("D", [1, 2, 3])
@pytest.mark.parametrize("n", [2, 33, 65, 127, 129, 161, 257, 500, 2048, 2049, 4097])
def test_parts_of_tiles_match_whole_tiles(n, D, flags, unsorted):
    # FP64: the same terms added in another order, n 2^-53 < 5e-13 of a sum of
    # non-negative terms.  FP32-compensated: far-tail terms, at most 2^-10 of an
    # event's own, are added in plain FP32 up to a tile at a time, 128 roundings of
    # 2^-24 each: 8e-9.
    rng = np.random.default_rng([n, D])
    loc, t = workloads.uniform(n, 0, D=D, rng=rng)
    if unsorted:
        t = np.append(rng.permutation(t[:-1]), t[-1])
    p = np.asarray(workloads.BASE_PARAMS) * np.array([1, 1.1, 0.9, 0.2, 1, 1])
    q = p * np.array([1, 1, 1, 1.3, 0.9, 1])  # a self-excitation step: kept background sums
    tol = 1e-12 if flags == FP64 else 1e-8
    out = {}
    for name, shape in (("parts", (0, 0)), ("whole", (2, 8))):
        with hb.CudaHawkes(D, n, flags, 0) as e:
            e.setSweepShape(*shape)
            e.setTimesData(t)
            e.updateLocations(-1, loc)
            out[name] = []
            for params in (p, q, p):
                e.setParameters(params)
                out[name].append(e.getLogLikelihoodAndGradient())
    for params, (la, ga), (lb, gb) in zip((p, q, p), out["parts"], out["whole"]):
        o = oracle.oracle_eval(loc, t, params, threads=8)
        mass = abs(o["loglik"]) + n
        assert abs(la - lb) <= tol * mass
        assert np.all(np.abs(ga - gb) <= tol * o["grad_scale"])
        assert abs(la - o["loglik"]) <= 1e-8 * mass
