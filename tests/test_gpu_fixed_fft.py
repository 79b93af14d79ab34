"""The block-floating-point line FFTs of the FP64 form (wlc_fixfft.cuh), at
every compiled grid edge, through wlc_mde_one_step.

* A right-hand side whose planes span twelve decades, against the oracle.
  Each of the six line transforms and the solve round an element by at most
  a few 2^-53 of its line's largest value, in the oracle as here, so the two
  differ by less than 45 units of 2^-52 of the largest output: 1e-14.
* The step is linear and the shared exponents are powers of two, so scaling
  the input by 2^k scales every bit of the output (real-8 literals: the
  single-precision correction of the other mode has a range of its own).
* A not-a-number input makes its coefficient's output not-a-number.
"""
import numpy as np
import pytest

import oracle
import wlc

pytestmark = pytest.mark.gpu

EDGES = [8, 12, 16, 24, 32, 40, 48, 64, 96]


def _case(n, L, lit):
    g = wlc.Instance(n, L, 10, (4, 2, 4), 1.2 / n, 1.3, (0.5, 0.6, 0.7), (15.0,) * 3, literals=lit)
    rng = np.random.default_rng(900 + n)
    pr = rng.standard_normal((g.nr, g.M)) + 1.0
    pr *= (10.0 ** rng.uniform(-12, 0, size=(n, 1, 1, g.M)) * np.ones((n, n, n, g.M))).reshape(g.nr, g.M)
    return g, pr


@pytest.mark.parametrize("lit", [wlc.WLC_LIT_REAL4, wlc.WLC_LIT_REAL8])
@pytest.mark.parametrize("n", EDGES)
def test_wide_range_against_oracle(n, lit):
    L = 1 if n > 24 else 2
    g, pr = _case(n, L, lit)
    o = oracle.Oracle((n, n, n), L, 10, (4, 2, 4), (1.2 / n,) * 3, 1.3, (0.5, 0.6, 0.7), (15.0,) * 3,
                      real4=int(lit == wlc.WLC_LIT_REAL4))
    for g_index, kind in ((4, (3, 1, 1)), (10, (1, -1, 2))):
        ref = o.one_step(*kind, np.ascontiguousarray(pr.T)).T
        q = g.mde_one_step(g_index, pr)
        assert np.abs(q - ref).max() < 1e-14 * np.abs(ref).max()
    o.close()
    g.close()


@pytest.mark.parametrize("n", EDGES)
def test_powers_of_two_scale_exactly(n):
    g, pr = _case(n, 1, wlc.WLC_LIT_REAL8)
    q = g.mde_one_step(3, pr)
    for k in (-600, -1, 37, 600):
        assert np.array_equal(g.mde_one_step(3, np.ldexp(pr, k)), np.ldexp(q, k))
    assert not g.mde_one_step(3, np.zeros_like(pr)).any()
    g.close()


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("n", EDGES)
def test_non_finite_input_stays_non_finite(n, bad):
    g, pr = _case(n, 1, wlc.WLC_LIT_REAL8)
    pr[g.nr // 2 + 3, 0] = bad
    q = g.mde_one_step(3, pr)
    assert np.isnan(q[:, 0]).all()
    g.close()


def test_rotations_without_room_for_their_table():
    """N = 96, L = 11 with real-8 literals is the one size whose column leaves
    no shared memory for the table of cos, sin(m beta) (the rotations then run
    on doubles): one step against the FP32 form, whose rounding (2^-24 an
    operation, some hundred operations in sequence) bounds the difference."""
    n, L = 96, 11
    rng = np.random.default_rng(5)
    M, nr = (L + 1) ** 2, n ** 3
    pr = rng.standard_normal((nr, 1), dtype=np.float32) * rng.uniform(0.1, 1.0, size=(1, M)).astype(np.float32)
    pr = pr.astype(np.float64)
    q = []
    for precision in (wlc.WLC_FP64, wlc.WLC_FP32):
        g = wlc.Instance(n, L, 10, (4, 2, 4), 1.2 / n, 1.3, (0.5, 0.6, 0.7), (15.0,) * 3, literals=wlc.WLC_LIT_REAL8,
                         precision=precision, store_qstar=0, q_checkpoint=3)
        q.append(g.mde_one_step(7, pr))
        g.close()
    assert np.abs(q[0] - q[1]).max() < 200 * 2.0 ** -24 * np.abs(q[0]).max()
