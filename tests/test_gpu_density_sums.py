"""The density's sums over coefficients against sums on the host of the same
slices (FP64 products of the stored numbers, exactly rounded sums)."""
import math

import numpy as np
import pytest

import wlc

pytestmark = pytest.mark.gpu

NMAX, NS = 4, (2, 2, 0)


def _simpson(slices, start, n):
    w = [1.0 if j in (0, n) else 4.0 if j % 2 else 2.0 for j in range(n + 1)]
    return sum(a * slices[start + j] for j, a in enumerate(w)) / (3.0 * NMAX)


def _expected(g, dots):
    """phi of the A and B blocks and the junction densities from sum_i q_i q*_i of every slice."""
    n, dx = g.n[0], g.params.dx[0]
    raw = [_simpson(dots, 0, NS[0]), _simpson(dots, NS[0], NS[1])]
    w1 = np.where(np.arange(n) % 2, 4.0, 2.0) * dx / 3.0
    w3 = (w1[:, None, None] * w1[None, :, None] * w1[None, None, :]).ravel()
    f = g.volume / math.fsum(w3 * (raw[0] + raw[1]))
    return np.array(raw) * f, np.array([dots[NS[0]], dots[NMAX]]) * f


def _host_dots(q, p):
    prod = q * p
    return prod.sum(axis=1) if prod.shape[1] < 3 else np.array([math.fsum(r) for r in prod])


@pytest.mark.parametrize("n", [8, 64, 96])
def test_fp32_products_outside_the_range_of_floats(n):
    """Stored FP32 slices of amplitudes over 24 decades up and down: products of
    two coefficients below the smallest and above the largest float, each
    point with its own.  Two coefficients a point, so that a sum of two exact
    products on the host is rounded once: M * 2^-52, the Simpson sums and the
    normalisation, 1e-14 of the point's value."""
    rng = np.random.default_rng(n)
    g = wlc.Instance(n, 1, NMAX, NS, 1.2 / n, 1.3, (0.5,) * 3, (15.0,) * 3, precision=wlc.WLC_FP32)
    g.set_fields(np.zeros((3, g.nr)))
    g.MDE_q()
    g.MDE_qstar()
    dots = []
    scale = 10.0 ** rng.choice([-26, -24, -18, -12, 0, 12, 18, 24], size=(g.nr, 1))
    for s in range(NMAX + 1):
        q, p = [np.zeros((g.nr, 4)) for _ in range(2)]
        for a in (q, p):
            a[:, :2] = (scale * rng.uniform(0.5, 1.0, size=(g.nr, 2))).astype(np.float32)
        g.set_q(1, s, q)
        g.set_q(-1, s, p)
        dots.append(_host_dots(q[:, :2], p[:, :2]))
    d = g.density()
    phi, junc = _expected(g, dots)
    assert (np.abs(d["phi"][:2] - phi) <= 1e-14 * phi).all()
    assert (np.abs(d["junction"][[0, 2]] - junc) <= 1e-14 * junc).all()
    g.close()


@pytest.mark.parametrize("n,store", [(8, 0), (16, 2), (24, 1)])
def test_fp32_densities_of_small_propagators(n, store):
    """A field level of 85 (the split scheme takes any): every product is about
    e^-85, 2^-123, whose rounding error no float holds.  Streamed and stored
    sums against the host's of the same slices: M + 10 roundings of 2^-52."""
    kw = dict(n=n, lmax=1, nmax=NMAX, ns=NS, dx=1.2 / n, loa=1.3, kappa=(0.5,) * 3, chi=(15.0,) * 3,
              precision=wlc.WLC_FP32, scheme=wlc.WLC_SCHEME_SPLIT)
    w = 85.0 + np.random.default_rng(n).normal(0.0, 0.3, size=(3, n ** 3))
    ref = wlc.Instance(store_qstar=1, **kw)
    ref.set_fields(w)
    ref.MDE_q()
    ref.MDE_qstar()
    phi, junc = _expected(ref, [_host_dots(ref.get_q(1, s), ref.get_q(-1, s)) for s in range(NMAX + 1)])
    g = wlc.Instance(store_qstar=store, **kw)
    g.set_fields(w)
    g.MDE_q()
    g.MDE_qstar()
    d = g.density(want_s=store == 2)
    assert (np.abs(d["phi"][:2] - phi) <= 14 * 2.0 ** -52 * phi).all()
    assert (np.abs(d["junction"][[0, 2]] - junc) <= 14 * 2.0 ** -52 * junc).all()
    g.close()
    ref.close()


def test_fp64_sum_is_no_single_chain():
    """121 coefficients whose products are 1 and then 1.5 * 2^-53 each: added one
    after the other every addition rounds up by half a unit of 2^-53, 60 in
    all.  Sums of every fourth product round at most 31 times, join in 2
    additions, and five slices add up and scale in 9: 42 units.  Relative to
    the points whose products but the first are zero and whose sums are exact."""
    n, L = 64, 10
    g = wlc.Instance(n, L, NMAX, NS, 1.2 / n, 1.3, (0.5,) * 3, (15.0,) * 3)
    g.set_fields(np.zeros((3, g.nr)))
    g.MDE_q()
    g.MDE_qstar()
    q = np.zeros((g.nr, g.M))
    q[:, 0] = 1.0
    p = q.copy()
    q[::2, 1:] = 1.0
    p[::2, 1:] = 1.5 * 2.0 ** -53
    for s in range(NMAX + 1):
        g.set_q(1, s, q)
        g.set_q(-1, s, p)
    phi = g.density(want_junction=False)["phi"][:2]
    g.close()
    exact = 120 * 1.5  # units of 2^-53 above 1
    off = (phi[:, ::2] - phi[:, 1::2]) / phi[:, 1::2] * 2.0 ** 53 - exact
    assert np.abs(off).max() <= 42
