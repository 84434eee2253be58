"""The FP64 path's noise (Box-Muller with its own logarithm, sine and cosine
on the integer draws) against the oracle's: beads without any force, one step
from rest, so that a step's displacement is the noise times a constant.  20,000
beads give 80,000 draws over all quadrants and table intervals; a few seeds put
draws next to the ends of the range.

Bar: each normal within 8 * 2^-53 relative to the Box-Muller radius bound
(sqrt(2 * 32 * log 2) < 6.7): three roundings of a result in [-6.7, 6.7] from
each of the logarithm, the square root and the trigonometric factor."""
import numpy as np
import pytest

from xmd_gb300 import Engine, synth

pytestmark = pytest.mark.gpu

MASK = (1 << 64) - 1


def normals(seed, n):
    """The reference's draws (rand_gen.h:22-58), in extended precision."""
    s = seed & MASK
    k = np.zeros((n, 4))
    for i in range(n):
        for q in range(4):
            k[i, q] = ((s * 0xd989bcacc137dcd5) & MASK) >> 32
            s ^= s >> 11
            s ^= (s << 31) & MASK
            s ^= s >> 18
    u = k.astype(np.longdouble) / np.longdouble(4294967296.0)
    two_pi = 2 * np.longdouble("3.14159265358979323846264338327950288")
    r1, r2 = np.sqrt(-2 * np.log(u[:, 0])), np.sqrt(-2 * np.log(u[:, 2]))
    return np.stack([r1 * np.cos(two_pi * u[:, 1]), r1 * np.sin(two_pi * u[:, 1]),
                     r2 * np.cos(two_pi * u[:, 3])], axis=1)


@pytest.mark.parametrize("seed", [12345, 1, 0xffffffffffffffff, 0x8000000000000000])
def test_normals(seed):
    n = 20000 if seed == 12345 else 300
    s = synth.make_system([1] * n, 3, native=False, temperature=0.5, avoid_others=False)
    s.r = np.zeros((n, 3)) + np.arange(n)[:, None] * 40.0
    s.atype = np.zeros(n, dtype=np.uint8)
    with Engine(synth.yaml_for("c4")) as e:
        e.add_system(s, seed=seed)
        e.step(1)
        y, _, _ = e.get_history(0)
    # y5 of a bead at rest after one step: c5 h sd N, h = dt^2 / 2, c5 = 1 / 60
    sd = np.sqrt(2.0 * 0.5) * np.sqrt(2.0)
    got = y[5] / (1.0 / 60.0 * 0.005 ** 2 / 2.0 * sd)
    want = normals(seed, n)
    ok = np.isfinite(want).all(axis=1)
    assert ok.sum() >= n - 1
    # four further roundings of the step itself and of the division here
    assert np.abs(got[ok] - want[ok].astype(np.float64)).max() <= 16 * 2.0 ** -53 * 6.7
