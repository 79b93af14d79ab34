"""The 64-bit integer arithmetic of the FP64 form (wlc_fixfft.cuh, the
rotations of wlc_solve.cu) at the ends of its numbers."""
import numpy as np
import pytest

import oracle
import wlc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [1, 4])
def test_factor_whose_low_half_has_no_negative(L):
    """In this box sin(beta) of the wavevector (9, 20, 21) is 0x1.ba1d1ee4p-1: as a
    factor of 62 fraction bits its low word is 0x80000000.  All of the input
    lies at that wavevector, and a sine off by 2^-30 shows as 1e-9 of the
    result.  Six line transforms and the solve against the oracle: 45 units of
    2^-52 of the largest output, as for any other input."""
    n, dx = 48, (0.14307796224661354, 0.05957622298448444, 0.10527062227864911)
    k = [2 * np.pi / (n * d) * i for d, i in zip(dx, (9, 20, 21))]
    sin_beta = np.hypot(k[0], k[1]) / np.sqrt(k[0] ** 2 + k[1] ** 2 + k[2] ** 2)
    assert int(sin_beta * 2.0 ** 62) & 0xffffffff == 0x80000000
    g = wlc.Instance(n, L, 10, (4, 2, 4), dx, 1.3, (0.5, 0.6, 0.7), (15.0,) * 3, literals=wlc.WLC_LIT_REAL8)
    o = oracle.Oracle((n, n, n), L, 10, (4, 2, 4), dx, 1.3, (0.5, 0.6, 0.7), (15.0,) * 3, real4=0)
    z, y, x = np.meshgrid(*[np.arange(n)] * 3, indexing="ij")
    wave = np.cos(2 * np.pi / n * ((9 * x + 20 * y + 21 * z) % n)).reshape(-1, 1)
    pr = wave * (1.0 + np.arange(g.M))
    ref = o.one_step(3, 1, 1, np.ascontiguousarray(pr.T)).T
    assert np.abs(g.mde_one_step(4, pr) - ref).max() < 1e-14 * np.abs(ref).max()
    o.close()
    g.close()


def _one_step(n, L, pr_of, lit=wlc.WLC_LIT_REAL4):
    g = wlc.Instance(n, L, 10, (4, 2, 4), 1.2 / n, 1.3, (0.5, 0.6, 0.7), (15.0,) * 3, literals=lit)
    rng = np.random.default_rng(700 + n)
    q = g.mde_one_step(4, pr_of(rng.standard_normal((g.nr, g.M)) + 1.0))
    g.close()
    return q


EDGES = [8, 12, 16, 24, 32, 40, 48, 64, 96]


@pytest.mark.parametrize("n", EDGES)
def test_overflow_of_the_literal_correction_is_not_finite(n):
    """Real-4 literals: the first-order correction (from L = 2 on; the couplings
    of L = 1 need none) runs in single precision.
    Where a wavevector's coefficients leave its range (1e39 a point: beyond
    3.4e38 at every wavevector) its sums are infinities and NaNs, and no
    finite number may come out of the lines that they reach.  Well inside the
    range the result is a number."""
    assert np.isfinite(_one_step(n, 2, lambda pr: pr * 1e28)).all()
    assert not np.isfinite(_one_step(n, 2, lambda pr: pr * 1e39)).any()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("n", EDGES)
def test_non_finite_input_with_the_correction(n, bad):
    def put(pr):
        pr[len(pr) // 2 + 3, 0] = bad
        return pr
    assert np.isnan(_one_step(n, 2, put)[:, 0]).all()


def test_diverged_field_is_reported():
    """Propagators that leave the correction's range end in WLC_E_NONFINITE, not in densities."""
    n = 16
    g = wlc.Instance(n, 2, 10, (4, 2, 4), 1.2 / n, 1.3, (0.5, 0.6, 0.7), (15.0,) * 3)
    g.set_fields(np.random.default_rng(1).normal(-1e6, 1e5, size=(3, g.nr)))
    g.MDE_q()
    g.MDE_qstar()
    assert np.abs(g.get_q(1, 5)).max() > 1e20
    with pytest.raises(wlc.WlcError) as e:
        g.density()
    assert e.value.code == -5
    g.close()


@pytest.mark.parametrize("n", EDGES)
def test_small_numbers_with_the_correction(n):
    """The step is linear: inputs scaled by 2^k give outputs scaled by 2^k.  With
    real-4 literals as long as the correction, a few 2^-24 of the result, stays
    in single precision's range (k = -60: to the rounding of the step, 1e-14);
    below, to the size of the correction that is lost, under 1e-6."""
    q = _one_step(n, 2, lambda pr: pr)
    for k, tol in ((-60, 1e-14), (-110, 1e-6), (-140, 1e-6), (-170, 1e-6), (-300, 1e-6), (-800, 1e-6)):
        s = np.ldexp(_one_step(n, 2, lambda pr: np.ldexp(pr, k)), -k)
        assert np.abs(s - q).max() <= tol * np.abs(q).max()


@pytest.mark.parametrize("n", EDGES)
def test_tiny_numbers(n):
    """Down to where doubles themselves lose bits, scaling the input by 2^k scales
    the output: 2^-930 and 2^-990 times numbers over twelve decades, against
    the unscaled step to its rounding (1e-14 of the largest output; the
    smallest subnormal is 2^-84 of the largest number even at k = -990).
    Tiny next to ordinary coefficients, and an input of zeros."""
    def spread(pr):
        return pr * 10.0 ** np.linspace(-12, 0, pr.shape[1])

    q = _one_step(n, 2, spread, wlc.WLC_LIT_REAL8)
    for k in (-930, -990):
        s = np.ldexp(_one_step(n, 2, lambda pr: np.ldexp(spread(pr), k), wlc.WLC_LIT_REAL8), -k)
        assert np.abs(s - q).max() <= 1e-14 * np.abs(q).max()

    def one_tiny(pr):
        pr[:, 0] = np.ldexp(pr[:, 0], -1000)
        return pr

    # as without it
    a, b = _one_step(n, 2, one_tiny), _one_step(n, 2, lambda pr: pr * (np.arange(pr.shape[1]) > 0))
    assert np.abs(a - b).max() <= 1e-14 * np.abs(b).max()
    for lit in (wlc.WLC_LIT_REAL4, wlc.WLC_LIT_REAL8):
        assert not _one_step(n, 2, lambda pr: pr * 0.0, lit).any()
