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
