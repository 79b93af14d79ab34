"""The per-point kernels (Theta term, density integrals) where their work
split or their shortcuts change.

* Theta term around the sparsity threshold: a field with ds w = 1 (powers of
  two, so that 1 - ds w is zero in any order of rounding) cancels the rest of the first-order right-hand side exactly, which leaves
  ds sum_j Theta_ij h_j; with the tensor spread log-uniformly over 1e-12..1e-8
  some components are dropped whole, some kept whole and some entry by entry.
  A row sums at most 25 products, in the oracle as here: 50 * 2^-52 of the
  largest value, 1e-14.
* Density integrals of stored slices (several work splits by grid size)
  against the streamed accumulation (another kernel): both FP64 sums of the
  same products, at most M * 2^-52 = 2e-14 apart for L <= 8, and through the
  normalisation twice that: 1e-13.
"""
import numpy as np
import pytest

import oracle
import wlc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,L", [(8, 1), (8, 6), (12, 12), (16, 3)])
def test_theta_threshold(n, L):
    nmax, ns = 8, (4, 2, 2)
    args = (1.2 / n, 1.1, (0.5, 0.5, 0.5), (15.0,) * 3)
    g = wlc.Instance(n, L, nmax, ns, *args, nmu=4.0)
    o = oracle.Oracle((n, n, n), L, nmax, ns, (args[0],) * 3, *args[1:], nmu=4.0)
    rng = np.random.default_rng(10 * n + L)
    m = np.zeros((3, 3, g.nr))
    for a in range(3):
        for b in range(a + 1):
            m[a, b] = m[b, a] = rng.choice([-1, 1], size=g.nr) * 10.0 ** rng.uniform(-12, -8, size=g.nr)
    m[2, 2] = 0.0  # one component absent everywhere
    w = np.full((3, g.nr), 8.0)
    q = rng.standard_normal((g.nr, g.M))
    g.set_fields(w, m)
    g.set_q(1, 0, q)
    o.set_fields(w, m.reshape(9, -1))
    o.set_q(1, 0, np.ascontiguousarray(q.T))
    pr, ref = g.init_pr(1, 1), o.init_pr(1, 1).T
    assert np.abs(ref).max() > 0
    assert np.abs(pr - ref).max() <= 1e-14 * np.abs(ref).max()
    o.close()
    g.close()


@pytest.mark.parametrize("precision", [wlc.WLC_FP64, wlc.WLC_FP32])
@pytest.mark.parametrize("n,L,ns", [(8, 0, (2, 2, 2)), (12, 3, (4, 0, 2)), (40, 2, (2, 2, 2)), (48, 1, (2, 4, 2)),
                                    (64, 1, (2, 2, 2)), (96, 1, (2, 2, 2))])
def test_stored_against_streamed_density(n, L, ns, precision):
    out = []
    for store in (1, 2):
        g = wlc.Instance(n, L, sum(ns), ns, 1.2 / n, 1.3, (0.5, 0.6, 0.7), (15.0, 12.0, 18.0), precision=precision,
                         store_qstar=store)
        g.set_fields(np.random.default_rng(n).normal(0.0, 0.5, size=(3, n ** 3)))
        g.MDE_q()
        g.MDE_qstar()
        out.append(g.density(want_s=True))
        g.close()
    a, b = out
    for key in ("phi", "junction"):
        assert np.abs(a[key] - b[key]).max() <= 1e-13 * np.abs(b[key]).max()
    # the tensor's forms are summed in the compute type, by the same code
    assert np.abs(a["S"] - b["S"]).max() <= 1e-13 * max(np.abs(b["S"]).max(), 1e-300)
    assert abs(a["lnQ"] - b["lnQ"]) <= 1e-13
