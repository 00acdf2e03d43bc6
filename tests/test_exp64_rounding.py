"""The FP64 mode's exponential is as good as a correctly rounded one, so that its sums
are no further from exact ones than with the library's exp(), down to the smallest
numbers."""
import numpy as np
import pytest

from test_exp64 import SRC, _constants
import re


def _full():
    text = open(SRC).read()

    def value(name):
        return float.fromhex(re.search(rf"{name} = ([-0-9a-fxp.+]+)[;,]", text).group(1))

    low = re.search(r"kExpLow\[32\] = \{(.*?)\};", text, re.S).group(1)
    low = [int(v.strip().rstrip("u"), 16) for v in low.split(",") if v.strip()]
    return ([0.5] + [value(f"kG{k}") for k in range(3, 7)], value("kInvStep"), value("kStep"),
            value("kStepLow"), (np.array(low, dtype=np.uint64) << np.uint64(32)).view(np.float64))


def test_a_term_is_within_rounding():
    # The kernel's operations on random exponents: one rounding of the result (0.5
    # units in the last place) and those of the polynomial, which is below 0.011, of
    # at most 3 * 0.011 units: 0.54.  A rounding error spread evenly over half a unit
    # either way has a root mean square of 0.2887 units; 0.295 leaves room for the rest.
    ld = np.longdouble
    c, inv, step, step_low, low = _full()
    _, table = _constants()
    table = np.array(table)
    rng = np.random.default_rng(0)
    x = -rng.uniform(0.0, 44.0, 1000000)

    def fma(a, b, d):
        return (ld(1) * a * b + d).astype(np.float64)

    nd = np.rint((ld(1) * x * inv)).astype(np.float64)
    # 64 bits of mantissa hold the difference of the two exactly (n below 2^11)
    r = fma(-nd, step_low, fma(-nd, step, x))
    k = nd.astype(np.int64)
    q = np.full_like(r, c[-1])
    for v in c[-2::-1]:
        q = fma(q, r, v)
    q = fma(q, r, 1.0)
    got = fma(table[k & 31], fma(q, r, low[k & 31]), table[k & 31])
    exact = np.exp(x.astype(ld)) / np.exp2((k >> 5).astype(ld))
    units = np.abs(got - exact) / np.where(exact < 1, ld(2.0) ** -53, ld(2.0) ** -52)
    assert float(units.max()) <= 0.54
    assert float(np.sqrt((units ** 2).mean())) <= 0.295


@pytest.mark.gpu
def test_probabilities_of_short_exponents():
    # One dimension, equal locations, omega = 1 and exponents below 1: S_i is a sum of
    # exponentials whose exponents are exact (times carry 20 bits), P_i = S_i / (B_i +
    # S_i) with B_i = B_ii alone.  A term is off by 0.54 units in the last place at most,
    # 0.29 in the mean square and independently, the sum, the products of the finish
    # and the quotient by some five roundings of the same size: sqrt(6) * 0.29 = 0.71
    # units of at most 2^-52, 1.6e-16, about a mean that the constants shift by up to
    # three more roundings.
    import hawkes_b200 as hb
    n = 400
    rng = np.random.default_rng(4)
    t = np.sort(rng.choice(2 ** 20, size=n, replace=False)) * 2.0 ** -20
    p = np.array([1.0, 1.0, 1e12, 1.0, 1.0, 1.0])
    with hb.CudaHawkes(1, n, hb.CUDA, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, np.zeros((n, 1)))
        e.setParameters(p)
        got = e.getProbsSelfExcite()
    ld = np.longdouble
    dt = (t[:, None] - t[None, :]).astype(ld)
    S = np.where(dt > 0, np.exp(-np.abs(dt)), 0).sum(1) / np.sqrt(2 * np.arccos(ld(-1)))
    B = ld(1e12) / (2 * np.arccos(ld(-1)))
    want = S / (B + S)
    rel = ((got[1:] - want[1:]) / want[1:]).astype(float)
    assert np.std(rel) <= 1.6e-16
    assert abs(np.mean(rel)) <= 3 * 2.0 ** -53


def _probabilities(t, omega=1.0):
    """P_i of events at one place, and in long double."""
    import hawkes_b200 as hb
    p = np.array([1.0, 1.0, 1.0, omega, 1.0, 1.0])
    with hb.CudaHawkes(1, len(t), hb.CUDA, 0) as e:
        e.setTimesData(t)
        e.updateLocations(-1, np.zeros((len(t), 1)))
        e.setParameters(p)
        got = e.getProbsSelfExcite().astype(np.longdouble)
    ld = np.longdouble
    pi = np.arccos(ld(-1))
    dt = (t[:, None] - t[None, :]).astype(ld)
    S = omega * np.where(dt > 0, np.exp(-omega * np.abs(dt)), 0).sum(1) / np.sqrt(2 * pi)
    B = np.exp(-dt * dt / 2).sum(1) / (2 * pi)
    return got, S / (B + S)


@pytest.mark.gpu
def test_sums_of_subnormal_terms():
    # Gaps of 700 to 743 / omega: every sum is one term, most of them subnormal, P_i =
    # prefS S_i / lambda_i with lambda_i = 1 / (2 pi).  S_i and prefS S_i (prefS = 0.4) are
    # each rounded to a multiple of 2^-1074, S_i after the term's own last place; the
    # division multiplies those 1.1 units by 2 pi and rounds once more: 8 units.  The
    # exponent's rounding is at most 745 * 2^-53 relative.
    t = np.concatenate([[0.0], np.cumsum(np.linspace(700.0, 743.0, 87))])
    got, want = _probabilities(t)
    unit = np.longdouble(2.0) ** -1074
    assert np.all(np.abs(got - want) <= 8 * unit + 1e-12 * want)
    assert np.all(got[want > 8 * unit] > 0)


@pytest.mark.gpu
def test_sums_of_subnormal_terms_that_the_finish_completes():
    # Bursts of 640 events, 720 / omega apart: the first event of each has only terms
    # of the burst before, which lie outside the self-excitation window.  640 terms,
    # each rounded to a multiple of 2^-1074, as is their sum.
    rng = np.random.default_rng(8)
    t = np.concatenate([720.0 * k + np.sort(rng.uniform(0.0, 1.0, 640)) for k in range(5)])
    t[::640] = 720.0 * np.arange(5)
    got, want = _probabilities(t)
    unit = np.longdouble(2.0) ** -1074
    first = slice(640, None, 640)
    assert np.all(want[first] < 1e-307)
    assert np.all(np.abs(got[first] - want[first]) <= 700 * unit + 1e-12 * want[first])
    assert np.all(np.abs(got - want)[want > 1e-300] <= 1e-12 * want[want > 1e-300])
