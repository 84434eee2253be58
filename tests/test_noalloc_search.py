"""The allocation-free pair search at the edges of its kernels: bead counts
around a warp, a block and a scan block; open, periodic and mixed boxes, with
one, two and many cells per axis; rows longer than shared memory holds; other
length units; beads many boxes away; an output buffer at an odd 4-byte offset;
a cap inside a row.  The pairs, their order and their count equal a brute-force
search with the same rounding of every operation."""
import ctypes

import numpy as np
import pytest

from tests.test_zz_no_alloc import DeviceBuffers
from tests.util import cudart
from xmd_gb300 import abi

pytestmark = pytest.mark.gpu


def brute(r, chain, seq, cell, cutoff):
    out = []
    inv = np.array([1.0 / c if c else 0.0 for c in cell])
    for i in range(len(r)):
        d = r[i + 1:] - r[i]
        d = d - cell * np.rint(d * inv)
        s = np.sqrt((d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2])
        j = np.arange(i + 1, len(r))
        ok = (s < cutoff) & ~((chain[j] == chain[i]) & (np.abs(seq[j] - seq[i]) < 3))
        out.append(np.stack([np.full(ok.sum(), i), j[ok]], axis=1))
    return np.concatenate(out).astype(np.int32)


def case(n, edge, cell, unit=1.0, shift=0.0, seed=0):
    g = np.random.default_rng([n, seed])
    r = g.uniform(-0.5, 0.5, (n, 3)) * edge * unit
    r[::7] += shift * unit          # some beads in other images
    chain = (np.arange(n) // 11).astype(np.int32)
    seq = (np.arange(n) % 11).astype(np.int32)
    return r, chain, seq, np.array(cell, dtype=np.float64) * unit


CASES = [
    # n, edge, cell, cutoff, unit, shift, cap
    (1, 10, (0, 0, 0), 3.0, 1.0, 0.0, None),
    (2, 2, (0, 0, 0), 3.0, 1.0, 0.0, None),
    (33, 6, (0, 0, 0), 3.0, 1.0, 0.0, None),
    (257, 14, (14, 14, 14), 3.0, 1.0, 0.0, None),
    (1023, 20, (20, 20, 20), 3.1, 1.0, 0.0, None),
    (1025, 20, (20, 0, 20), 3.1, 1.0, 20.0, None),
    (700, 8, (5, 8, 11), 4.9, 1.0, 0.0, None),        # one cell, one cell, two cells
    (700, 12, (7, 12, 0), 3.4, 1.0, -36.0, 5000),     # two, three, open; cap inside the list
    (900, 10, (0, 0, 0), 3.2, 1.0, 0.0, 30003),       # rows around 32 and 64 partners, kept and not; cap inside
    (1500, 6, (0, 0, 0), 20.0, 1.0, 0.0, None),       # every pair: rows beyond shared memory
    (1500, 6, (9, 9, 9), 4.0, 1.0, 0.0, 300001),      # long rows, cap inside one
    (900, 20, (20, 20, 20), 3.1, 1e-3, 0.0, None),
    (900, 20, (0, 20, 0), 3.1, 1e4, 0.0, None),
    (600, 20, (20, 20, 20), 3.1, 1.0, 2.0e8, None),   # 10^7 boxes away
    (2100, 3000, (0, 0, 0), 2.0, 1.0, 0.0, None),     # far more cells than the packed form holds
]


@pytest.mark.parametrize("n,edge,cell,cutoff,unit,shift,cap", CASES)
def test_equals_brute_force(n, edge, cell, cutoff, unit, shift, cap):
    lib, rt = abi.load(), cudart()
    r, chain, seq, box = case(n, edge, cell, unit, shift)
    want = brute(r, chain, seq, box, cutoff * unit)
    bufs = DeviceBuffers(rt)
    try:
        d_r, d_c, d_s = bufs.put(r.reshape(-1)), bufs.put(chain), bufs.put(seq)
        k = len(want) + 8 if cap is None else cap
        d_p, d_n = bufs.empty(8 * k + 4), bufs.empty(4)
        out = ctypes.c_void_p(d_p.value + 4)
        for _ in range(2):
            abi.check(lib.xmd_gpu_verlet_pairs_noalloc(d_r, d_c, d_s, n, abi.dptr(box), cutoff * unit, out, k, d_n,
                                                       None))
        assert rt.cudaDeviceSynchronize() == 0
        assert int(bufs.get(d_n, np.int32, 1)[0]) == len(want)
        m = min(len(want), k)
        got = bufs.get(out, np.int32, 2 * m).reshape(m, 2)
    finally:
        bufs.free()
    assert np.array_equal(got, want[:m])
