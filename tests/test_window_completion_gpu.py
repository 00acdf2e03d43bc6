"""The self-excitation window where it is on, and the sums that the finish completes:
events after a pause hold no term inside the window."""
import numpy as np
import pytest

import hawkes_b200 as hb

pytestmark = pytest.mark.gpu

FP64 = hb.CUDA
FP32C = hb.CUDA | hb.COMPENSATED
PARAMS = np.array([1.0, 0.5, 1.0 / 336.0, 1.0, 0.5, 1.0])  # omega = 1


def _events(pause, blocks):
    """20,480 events, ten a unit of time, with a pause before events 4096 (alone), 8192
    (five of one time), 12288 (40 of one time) and 16384 (300 of one time: more than a
    finish block holds); blocks: in shuffled blocks of 512 events."""
    n = 20480
    rng = np.random.default_rng(6)
    step = rng.exponential(0.1, n)
    for i, count in ((4096, 1), (8192, 5), (12288, 40), (16384, 300)):
        step[i] = pause
        step[i + 1:i + count] = 0.0
    t = np.cumsum(step)
    loc = rng.uniform(0.0, 5.0, (n, 1))
    low = np.concatenate([np.arange(i, i + c) for i, c in
                          ((4096, 1), (8192, 5), (12288, 40), (16384, 300))])
    if blocks:
        order = rng.permutation(n // 512 - 1)  # the last stays: its last event ends the time
        order = np.append(order, n // 512 - 1)
        index = (order[:, None] * 512 + np.arange(512)).ravel()
        where = np.empty(n, dtype=int)
        where[index] = np.arange(n)
        return loc[index], t[index], where[low]
    return loc, t, low


def _exact(loc, t, which):
    sigma, a, b, omega, theta, mu0 = PARAMS
    dt = t[which, None] - t[None, :]
    d2 = (loc[which] - loc[:, 0][None, :]) ** 2
    B = np.exp(-0.5 * a * a * d2 - 0.5 * b * b * dt * dt).sum(1) * mu0 * a * b / (2 * np.pi)
    S = np.where(dt > 0, np.exp(-0.5 * sigma ** 2 * d2 - omega * np.abs(dt)), 0).sum(1)
    S *= theta * omega * sigma / np.sqrt(2 * np.pi)
    return S / (B + S)


@pytest.mark.parametrize("blocks", [False, True], ids=["sorted", "blocks"])
@pytest.mark.parametrize("flags,pause", [(FP64, 100.0), (FP32C, 60.0)], ids=["fp64", "fp32c"])
def test_sums_outside_the_window_are_completed(flags, pause, blocks):
    # The window ends at 40 to 45 (FP32-compensated) or about 60 (FP64) exponents, where
    # terms reach to 88 or 750: between half and a tenth of the terms remain, and whole
    # tiles at the edges, of strips of one height at most 0.75.  The completed sums are FP64 sums of exp(): the
    # exponent's rounding, 100 * 2^-52 = 2e-14, and the sum's; the background sum has the
    # mode's rounding, 2^-24 in the FP32-compensated mode.
    loc, t, low = _events(pause, blocks)
    got = {}
    for name, extra in (("window", 0), ("full", hb.NO_TAIL_TRUNCATION)):
        with hb.CudaHawkes(1, len(t), flags | extra, 0) as e:
            e.setTimesData(t)
            e.updateLocations(-1, loc)
            e.setParameters(PARAMS)
            ll, g = e.getLogLikelihoodAndGradient()
            terms = e.lastLaunchStats()[2], e.sweepShape()[0]
            got[name] = ll, np.asarray(g), e.getProbsSelfExcite(), terms
            if name == "window":  # the step's window is the same
                e.setParameters(PARAMS * np.array([1.01, 1, 1, 1, 1, 1]))
                e.getLogLikelihoodAndGradient()
                e.setParameters(PARAMS)
                e.getLogLikelihoodAndGradient()
                step = e.getProbsSelfExcite()
    (lw, gw, pw, (nw, rw)), (lf, gf, pf, (nf, rf)) = got["window"], got["full"]
    assert nw < (0.75 * nf if rw == rf else nf)
    want = _exact(loc, t, low)
    assert np.all(want < (1e-20 if flags == FP32C else 1e-40))
    rtol = 1e-12 if flags == FP64 else 2.0 ** -23
    np.testing.assert_allclose(pw[low], want, rtol=rtol, atol=0)
    np.testing.assert_allclose(step[low], want, rtol=rtol, atol=0)
    # all other events: 2^-60 or 2^-36 of the sum, and the modes' rounding
    np.testing.assert_allclose(pw, pf, rtol=1e-12 if flags == FP64 else 5e-6, atol=0)
    assert abs(lw - lf) <= (1e-13 if flags == FP64 else 1e-8) * abs(lf)
