"""set_state / get_state over the edges of their blocks (256 beads) and pieces
(16384 beads): positions come back as they went in, velocities as (v dt) / dt
with its three roundings, and bead i's generator stands 4 i draws after the
seed."""
import numpy as np
import pytest

from xmd_gb300 import Engine
from xmd_gb300.synth import System

pytestmark = pytest.mark.gpu

M = (1 << 64) - 1
HEAD = 80 + 4 + 56          # a snapshot's header, row capacity and scalars


def _gen(seed, n):
    s, out = seed & M, np.empty(n, dtype=np.uint64)
    for i in range(n):
        out[i] = s
        for _ in range(4):
            s ^= s >> 11
            s ^= (s << 31) & M
            s ^= s >> 18
    return out


def _system(n, rng):
    e = (np.zeros(0, np.int32),)
    none = np.zeros(0)
    return System(n=n, chain=np.zeros(n, np.int32), seq=np.arange(n, dtype=np.int32), atype=np.zeros(n, np.uint8),
                  cell=np.zeros(3), r=rng.normal(size=(n, 3)) * 100.0, tethers=e * 2 + (none,),
                  angles=e * 3 + (none,), dihedrals=e * 4 + (none,), natives=e * 2 + (none,),
                  seed=int(rng.integers(1, 1 << 62)))


@pytest.mark.parametrize("sizes", [(1, 255, 256, 257), (16383, 16384), (16385, 3), (40000,)])
def test_round_trip(sizes):
    rng = np.random.default_rng(sum(sizes))
    e = Engine("")
    systems = [_system(n, rng) for n in sizes]
    for s in systems:
        e.add_system(s)
    for k in range(2):      # the first placement, then a new state in place
        vs = []
        for rep, s in enumerate(systems):
            s.r = rng.normal(size=(s.n, 3)) * 10.0 ** rng.integers(-3, 4)
            vs.append(rng.normal(size=(s.n, 3)) if k else None)
            e.set_state(rep, s.r, vs[-1])
        for rep, s in enumerate(systems):
            r, v, t = e.get_state(rep)
            assert t == 0.0 and np.array_equal(r, s.r)
            want = np.zeros((s.n, 3)) if vs[rep] is None else vs[rep]
            assert (np.abs(v - want) <= 3 * 2.0**-53 * 1.01 * np.abs(want)).all()
            at = HEAD + 184 * s.n
            got = np.frombuffer(e.snapshot(rep)[at:at + 8 * s.n], dtype=np.uint64)
            assert np.array_equal(got, _gen(s.seed, s.n))
