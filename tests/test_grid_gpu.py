"""The gridded background sums and the self-excitation window against the pair
sweep and the oracle, over the forms of events they accept."""
import numpy as np
import pytest

import hawkes_b200 as hb
import oracle
from hawkes_b200 import workloads

pytestmark = pytest.mark.gpu

FP64 = hb.CUDA
FP32C = hb.CUDA | hb.COMPENSATED


def _events(form, n, D, rng):
    loc, t = workloads.uniform(n, 0, D=D, rng=rng)
    if form == "unsorted":
        t = np.append(rng.permutation(t[:-1]), t[-1])
    elif form == "far_from_zero":  # coordinates and times of either sign, large offsets
        loc, t = loc - 4000.0, t - 5000.0
    elif form == "one_cell":  # most events within a fraction of a grid cell
        loc[: n - n // 8] = loc[0] + 1e-3 * rng.standard_normal((n - n // 8, D))
    elif form == "ties":
        t = np.floor(t / 50.0) * 50.0
    elif form == "line":  # no extent in one coordinate
        loc[:, -1] = 3.25
    return loc, t


@pytest.mark.parametrize("form", ["plain", "unsorted", "far_from_zero", "one_cell", "ties", "line"])
@pytest.mark.parametrize("D,n", [(1, 30001), (2, 30011)])
def test_gridded_sums_match_the_pair_sweep(form, D, n):
    # A pair's term is off by at most 2.5e-17 and its weighted terms by 1.2e-15 in
    # units of an event's own term, which is at most the event's sum: with
    # rounding, 1e-14 of the per-event scale of each gradient component (the
    # largest over components of |term| / |sum| is about 8) and 1e-15 on the
    # log-likelihood's per-event terms, whose sum cancels up to 100-fold.
    rng = np.random.default_rng([7, D, len(form)])
    loc, t = _events(form, n, D, rng)
    p = np.asarray(workloads.BASE_PARAMS) * np.array([1.0, 0.9, 1.2, 1.0, 1.1, 0.9])
    p[1] = -p[1] if form == "far_from_zero" else p[1]  # a precision's sign drops out squared
    if p[1] < 0 and D == 1:
        p[1] = -p[1]  # odd powers of tauX enter the rate
    out = {}
    for name, shape in (("grid", (0, 0)), ("pairs", (2, 32))):
        with hb.CudaHawkes(D, n, FP64, 0) as e:
            e.setSweepShape(*shape)
            e.setTimesData(t)
            e.updateLocations(-1, loc)
            e.setParameters(p)
            ll, g = e.getLogLikelihoodAndGradient()
            evals = e.lastLaunchEvals()
            out[name] = ll, g, e.getProbsSelfExcite()
            assert (evals == 0.0) == (name == "grid")
            # repeated evaluations give the same bits (new parameters in between)
            e.setParameters(p * 1.05)
            e.getLogLikelihoodAndGradient()
            e.setParameters(p)
            again = e.getLogLikelihoodAndGradient()
            assert again[0] == ll and np.array_equal(again[1], g)
    scale = oracle.oracle_eval(loc, t, p, threads=16)["grad_scale"]
    (la, ga, pa), (lb, gb, pb) = out["grid"], out["pairs"]
    assert abs(la - lb) <= 1e-13 * abs(lb)
    assert np.all(np.abs(ga - gb) <= 1e-14 * scale)
    np.testing.assert_allclose(pa, pb, rtol=1e-13, atol=0)


def test_gridded_batches_and_sets_match_single_evaluations():
    # several grids per launch, more problems than one launch takes, and sets of
    # sizes on both sides of the choice
    rng = np.random.default_rng(9)
    loc, t = workloads.uniform(30000, 0, rng=rng)
    P = workloads.proposals(19, 4)
    with hb.CudaHawkes(2, len(t), FP64, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        ll, g = e.batchLogLikelihoodAndGradient(P)
        for k in (0, 7, 18):
            e.setParameters(P[k])
            l1, g1 = e.getLogLikelihoodAndGradient()
            assert abs(l1 - ll[k]) <= 1e-14 * abs(l1)
            np.testing.assert_allclose(g1, g[k], rtol=1e-11)
    sizes = [40001, 500, 60000, 2000]
    sets = [workloads.uniform(n, 100 + n) for n in sizes]
    with hb.Multiset(2, sizes, FP64, 0) as m:
        for s, (loc, t) in enumerate(sets):
            m.setData(s, loc, t)
        ll, g = m.logLikelihoodAndGradient(P[:4])
    for s, (loc, t) in enumerate(sets):
        with hb.CudaHawkes(2, sizes[s], FP64, 0) as e:
            e.setTimesData(t)
            e.updateLocations(-1, loc)
            e.setParameters(P[s])
            l1, g1 = e.getLogLikelihoodAndGradient()
        assert abs(l1 - ll[s]) <= 1e-13 * abs(l1)
        np.testing.assert_allclose(g1, g[s], rtol=1e-10)


def test_moved_and_restored_events_with_gridded_sums():
    loc, t = workloads.uniform(30000, 21)
    p = np.asarray(workloads.BASE_PARAMS)
    with hb.CudaHawkes(2, len(t), FP64, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        e.setParameters(p)
        first = e.getLogLikelihoodAndGradient()
        e.storeState()
        moved = loc.copy()
        moved[5] = [31.0, -7.0]  # outside the box of the others
        e.updateLocations(5, moved[5])
        near = e.getLogLikelihoodAndGradient()
        assert e.lastEvaluationPath == hb.PATH_INCREMENTAL
        q = p * np.array([1, 1.1, 1, 1, 1, 1])
        e.setParameters(q)  # a sweep with the wider box
        swept = e.getLogLikelihoodAndGradient()
        with hb.CudaHawkes(2, len(t), FP64, 0) as f:
            f.setTimesData(t)
            f.updateLocations(-1, moved)
            f.setParameters(p)
            want = f.getLogLikelihoodAndGradient()
            f.setParameters(q)
            want2 = f.getLogLikelihoodAndGradient()
        assert abs(near[0] - want[0]) <= 1e-13 * abs(want[0])
        assert abs(swept[0] - want2[0]) <= 1e-13 * abs(want2[0])
        np.testing.assert_allclose(swept[1], want2[1], rtol=1e-10)
        e.restoreState()
        e.setParameters(q)
        e.getLogLikelihoodAndGradient()
        e.setParameters(p)
        back = e.getLogLikelihoodAndGradient()
        assert abs(back[0] - first[0]) <= 1e-14 * abs(first[0])


@pytest.mark.parametrize("flags", [FP64, FP32C], ids=["fp64", "fp32c"])
@pytest.mark.parametrize("form", ["plain", "unsorted", "sharp", "pairs", "ties"])
@pytest.mark.parametrize("D", [1, 2, 3])
def test_self_excitation_window_keeps_every_sum(flags, form, D):
    # Every event's self-excitation sum keeps its terms to 2^-60 (FP64) or 2^-36
    # of itself, so P_i agrees with the full sums relatively, also where the
    # sum is tiny: "sharp" kernels (large sigma) and "pairs" (events far from all
    # but one other) are the ones whose sums the finish completes.
    n = 3001
    rng = np.random.default_rng([3, D, len(form)])
    loc, t = _events("unsorted" if form == "unsorted" else "ties" if form == "ties" else "plain",
                     n, D, rng)
    p = np.asarray(workloads.BASE_PARAMS) * np.array([1, 1, 1, 0.5, 1, 1.0])
    if form == "sharp":
        p[0] = 6.0
    if form == "pairs":
        t = np.sort(np.where(np.arange(n) % 2, t, t * 0.02))
    got = {}
    for name, extra in (("window", 0), ("full", hb.NO_TAIL_TRUNCATION)):
        with hb.CudaHawkes(D, n, flags | extra, 0) as e:
            e.setTimesData(t)
            e.updateLocations(-1, loc)
            e.setParameters(p)
            ll, g = e.getLogLikelihoodAndGradient()
            terms = e.lastLaunchStats()[2]
            got[name] = ll, np.asarray(g), e.getProbsSelfExcite(), terms, e.sweepShape()[0]
    (lw, gw, pw, nw, rw), (lf, gf, pf, nf, rf) = got["window"], got["full"]
    # larger strips evaluate more of the terms that are zero
    assert nw <= nf or rw > rf
    if flags == FP64:
        assert abs(lw - lf) <= 1e-13 * abs(lf)
        big = pf > 1e-290
        np.testing.assert_allclose(pw[big], pf[big], rtol=1e-12)
        np.testing.assert_allclose(gw, gf, rtol=1e-9)
    else:
        assert abs(lw - lf) <= 1e-8 * abs(lf)
        big = pf > 1e-30  # above the FP32 terms' underflow
        np.testing.assert_allclose(pw[big], pf[big], rtol=5e-6)


@pytest.mark.parametrize("form,D,n", [("plain", 1, 40000), ("unsorted", 2, 40000),
                                      ("far_from_zero", 2, 40000), ("one_cell", 2, 40000),
                                      ("line", 2, 40000), ("plain", 2, 65535),
                                      ("plain", 2, 65536)])
def test_gridded_fp32_compensated_sums(form, D, n):
    # Below 65,536 events the grid's weighted sums are within 1.4e-10 of themselves;
    # the self-excitation terms carry FP32 roundings (2^-24 of an event's sum, of
    # either sign).  From there on both are as exact as in the FP64 mode.
    rng = np.random.default_rng([11, D, n])
    loc, t = _events(form, n, D, rng)
    p = np.asarray(workloads.BASE_PARAMS) * np.array([1.0, 0.9, 1.2, 1.0, 1.1, 0.9])
    out = {}
    for flags in (FP64, FP32C):
        with hb.CudaHawkes(D, n, flags, 0) as e:
            e.setTimesData(t)
            e.updateLocations(-1, loc)
            e.setParameters(p)
            out[flags] = *e.getLogLikelihoodAndGradient(), e.lastLaunchEvals()
    (lw, gw, _), (lg, gg, evals) = out[FP64], out[FP32C]
    scale = oracle.oracle_eval(loc, t, p, threads=16)["grad_scale"]
    assert evals == 0.0 or form == "unsorted"
    assert abs(lg - lw) <= 1e-8 * abs(lw)
    assert np.all(np.abs(gg - gw) <= 6e-8 * scale)


def test_large_fp32_compensated_evaluations_follow_the_events():
    # the FP64 records such an evaluation sweeps are those of the present events
    loc, t = workloads.uniform(70000, 5)
    p = np.asarray(workloads.BASE_PARAMS)
    moved = loc.copy()
    moved[123] += 0.4
    want = {}
    for name, x in (("first", loc), ("moved", moved)):
        with hb.CudaHawkes(2, len(t), FP64, 0) as f:
            f.setTimesData(t)
            f.updateLocations(-1, x)
            f.setParameters(p)
            want[name] = f.getLogLikelihoodAndGradient()
    with hb.CudaHawkes(2, len(t), FP32C, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, loc)
        e.setParameters(p * 1.1)
        e.getLogLikelihoodAndGradient()
        e.storeState()
        e.updateLocations(123, moved[123])
        e.setParameters(p)
        got = e.getLogLikelihoodAndGradient()
        assert abs(got[0] - want["moved"][0]) <= 1e-8 * abs(want["moved"][0])
        np.testing.assert_allclose(got[1], want["moved"][1], rtol=1e-6)
        assert abs(want["moved"][0] - want["first"][0]) > 1e-7 * abs(want["first"][0])
        e.restoreState()
        e.setParameters(p * 1.05)
        e.getLogLikelihoodAndGradient()
        e.setParameters(p)
        back = e.getLogLikelihoodAndGradient()
        assert abs(back[0] - want["first"][0]) <= 1e-8 * abs(want["first"][0])


@pytest.mark.parametrize("n", [262143, 262144, 262145, 262273])
def test_ranks_of_tied_times(n):
    # Ranks decide which FP32 terms are causal; the FP64 mode compares times.  On
    # both sides of the size up to which each tile adds up the ones before it.
    rng = np.random.default_rng(n)
    t = np.floor(np.sort(rng.uniform(0.0, 40000.0, n)) / 4.0) * 4.0
    loc = rng.uniform(0.0, 3000.0, (n, 1))
    p = np.asarray(workloads.BASE_PARAMS) * np.array([1, 1, 40, 1, 1, 1])
    out = {}
    for flags in (FP64, FP32C):
        with hb.CudaHawkes(1, n, flags, 0) as e:
            e.setSweepShape(2, 64)  # the pair sweep: FP32 terms whatever their number
            e.setTimesData(t)
            e.updateLocations(-1, loc)
            e.setParameters(p)
            out[flags] = e.getLogLikelihoodAndGradient()[0], e.getProbsSelfExcite()
    # a tie counted as causal, or an event left out, moves its P_i by about its size
    assert abs(out[FP64][0] - out[FP32C][0]) <= 1e-8 * abs(out[FP64][0])
    assert np.abs(out[FP64][1] - out[FP32C][1]).max() <= 1e-4
