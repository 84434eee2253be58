"""The step kernel's block: bead counts at the edges of its tile (a block of
32, 64 or 128 slots takes 27, 59 or 123 beads), several replicas sharing a
block, and rows so long that a block's pair entries take several passes.

Bars: FP64 forces and energies within 1e-10 of the CPU restatement (the parity
bar of the other tests); the trajectory the same bits for every launch shape,
in both precisions.  (At these native starts the forces cancel, so the mixed
path's relative bar, which test_gpu_parity.py holds it to, says nothing.)"""
import numpy as np
import pytest

from oracle.pyoracle import Oracle
from tests.util import energy_rel, rel_err
from xmd_gb300 import Engine, abi, synth

pytestmark = pytest.mark.gpu

SHAPES = [(32, 0, 16, 1), (32, 0, 16, 4), (64, 0, 16, 2), (64, 0, 16, 4), (128, 0, 16, 2), (128, 0, 16, 4)]


def systems(kind):
    if kind == "dense":
        # every bead charged, native starts: hundreds of entries per bead row
        s = synth.make_system([230], 5, temperature=0.35, start="native")
        s.atype = np.where(np.arange(s.n) % 2 == 0, synth.CHARGED_POS[0], synth.CHARGED_NEG[0]).astype(np.uint8)
        return [s]
    sizes = {"edges27": [27, 28, 26, 1, 2], "edges59": [59, 60, 58, 3], "edges123": [123, 124, 122, 4],
             "small": [5, 4, 3, 2, 1, 31, 32, 33]}[kind]
    return [synth.make_system([n], 40 + k, temperature=0.3 + 0.02 * k, start="native") for k, n in enumerate(sizes)]


@pytest.mark.parametrize("kind", ["edges27", "edges59", "edges123", "small", "dense"])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_block_edges(kind, prec):
    ss = systems(kind)
    y = synth.yaml_for("c4", prec)
    p = abi.parse_params(y)
    with Engine(y) as e:
        for s in ss:
            e.add_system(s)
        for k, s in enumerate(ss):
            F, V = e.eval_forces(k)
            if prec == "fp64":
                Fo, Vo = Oracle(p, s, "port").eval_forces()
                assert rel_err(F, Fo) <= 1e-10, (k, rel_err(F, Fo))
                assert energy_rel(V, Vo).max() <= 1e-10, (k, energy_rel(V, Vo))
        if kind == "dense":
            assert e.stats()["nl_entries"] > 20 * ss[0].n
    want = None
    for shape in SHAPES:
        with Engine(y) as e:
            for s in ss:
                e.add_system(s)
            e.set_tuning(*shape)
            e.step(24)
            got = [e.get_history(k)[0] for k in range(len(ss))]
        if want is None:
            want = got
        for a, b in zip(got, want):
            assert np.array_equal(a, b), shape


def test_extended_start_mixed_force():
    """Extended starts hold triples straight to ~1e-6 rad, whose dihedral
    forces (1 / sin theta) are the largest of a replica: the mixed bar of
    1e-5 of the largest force holds there for every chain."""
    ss = [synth.make_system([90 + 7 * k], 300 + k, temperature=0.35) for k in range(40)]
    F = {}
    for prec in ("fp64", "mixed"):
        with Engine(synth.yaml_for("c4", prec)) as e:
            for s in ss:
                e.add_system(s)
            F[prec] = [e.eval_forces(k)[0] for k in range(len(ss))]
    for m, f in zip(F["mixed"], F["fp64"]):
        assert np.abs(m - f).max() <= 1e-5 * np.abs(f).max()
