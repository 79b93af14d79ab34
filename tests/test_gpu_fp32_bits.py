"""FP32 results keep their bits.

A change in the order of the additions of an FP32 transform moves every
result by some 2^-24, and the partition function of a long chain by as much
as its accumulated rounding; no bound on a single run tells such a move from
the rounding that was there.  So the results themselves are fixed: digests of
one contour step and of a short forward sweep at every compiled grid edge,
recorded from the kernels of commit df35dd0 (nvcc 13.0).  The inputs are
integers over a power of two, the same on every machine.
"""
import hashlib

import numpy as np
import pytest

import wlc

pytestmark = pytest.mark.gpu

DIGESTS = {
    8: ["6983d1afb2863569", "f17f485fb1aa8a98"],
    12: ["df2537d1c7e6477d", "104fd0d01333e943"],
    16: ["3e197515ce16a1bb", "0b33d9631f6e82f4"],
    24: ["613d23efbc745d52", "8f52e8267afb6fa9"],
    32: ["c9de756a5f9300f1", "1c46d53c925c2d1c"],
    40: ["6376c446077907da", "09bfd041b95864ab"],
    48: ["6a6509227ef3dca1", "8bdec3d27a3153f8"],
    64: ["263bc03848099ed0", "d3542ab0b4c9c1f5"],
    96: ["ca1007466e2903bb", "dd596109fa688c62"],
    128: ["db5f52449dbb8777", "b73fc36975d2bbaa"],
}


def _noise(n, k):
    """n values in [-1, 1), multiples of 2^-12 (a linear congruential sequence, no library generator)."""
    x = np.arange(1, n + 1, dtype=np.uint64) * np.uint64(2654435761) + np.uint64(k * 40503 + 12345)
    x ^= x >> np.uint64(13)
    x = (x * np.uint64(1597334677)) & np.uint64(0xffffffff)
    return ((x >> np.uint64(17)) & np.uint64(8191)).astype(np.float64) / 4096.0 - 1.0


def digests(n):
    """Digests of a third-order step (degree 2) and of a sweep of 8 steps (degree 1)."""
    out = []
    for L, nmax, ns in ((2, 8, (2, 4, 2)), (1, 8, (2, 4, 2))):
        g = wlc.Instance(n, L, nmax, ns, 3.0 / n, 1.0, (0.5, 0.625, 0.75), (15.0,) * 3, precision=wlc.WLC_FP32)
        if L == 2:
            q = g.mde_one_step(4, _noise(g.nr * g.M, n).reshape(g.nr, g.M))
        else:
            g.set_fields(_noise(3 * g.nr, n + 1).reshape(3, g.nr))
            g.MDE_q()
            q = g.get_q(1, nmax)
        out.append(hashlib.sha256(q.astype(np.float32).tobytes()).hexdigest()[:16])
        g.close()
    return out


@pytest.mark.parametrize("n", sorted(DIGESTS))
def test_fp32_results_keep_their_bits(n):
    assert digests(n) == DIGESTS[n]
