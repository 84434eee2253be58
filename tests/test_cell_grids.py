"""The cell build's two grids against the whole-replica tile build: the same
pairs with the same flags, whatever terms set the near and far radii, and
whatever the box (open, periodic, periodic along some axes, so small that an
axis has one cell, so wide that cell coordinates outgrow their packed form),
with no bead charged and with all of them."""
import numpy as np
import pytest

from tests.test_gpu_parity import verlet_pairs, with_engine_key
from xmd_gb300 import Engine, synth

pytestmark = pytest.mark.gpu

A = synth.ANGSTROM
OFF = {"es": "\nconst ES:\n  enabled: false\n", "pauli": "\nPauli exclusion:\n  enabled: false\n"}
PID = "\npseudo-improper dihedral potential:\n  enabled: true\n"
SHORT = "\nneighbor list:\n  cutoff: 14 A\n  skin: 2 A\n"    # the list radius cuts the electrostatic one
NARROW = "\nneighbor list:\n  cutoff: 3 A\n  skin: 1 A\n"    # and the Pauli one

CASES = {
    "open": ("c4", "", None, 1.0, None),
    "periodic": ("c4", "", 90.0, 1.0, None),
    "two-cells": ("c4", "", 52.0, 1.0, None),
    "one-cell": ("c4", "", 30.0, 1.0, None),
    "slab": ("c4", "", 90.0, 1.0, (1, 0, 1)),
    "wide": ("c4", "", None, 4000.0, None),
    "no-charge": ("c4", "", 90.0, 1.0, "none"),
    "all-charged": ("c4", "", 90.0, 1.0, "all"),
    "no-es": ("c4", OFF["es"], 90.0, 1.0, None),
    "no-pauli": ("c4", OFF["pauli"], 90.0, 1.0, None),
    "neither": ("c4", OFF["es"] + OFF["pauli"], 90.0, 1.0, None),
    "pid": ("c4", PID, None, 1.0, None),
    "qa": ("c3", "", 90.0, 1.0, None),
    "short": ("c4", SHORT, 90.0, 1.0, None),
    "narrow": ("c4", NARROW, None, 1.0, None),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_cell_build_equals_tile_build(name):
    base, extra, box, spread, what = CASES[name]
    s = synth.make_system([70, 33, 101, 5], 17, box=None if box is None else box * A, temperature=0.35)
    if spread != 1.0:
        s.r = s.r.copy()
        s.r[s.chain == 2] += spread
    if what == "none":
        s.atype = np.zeros(s.n, dtype=np.uint8)
    elif what == "all":
        s.atype = np.full(s.n, synth.CHARGED_POS[0], dtype=np.uint8)
    elif what is not None:
        s.cell = s.cell * np.array(what, dtype=float)
    got = {}
    for build in ("cell", "tile"):
        y = with_engine_key(synth.yaml_for(base) + extra, f"nl build: {build}")
        with Engine(y) as e:
            e.add_system(s)
            F, V = e.eval_forces(0)
            e.step(30)           # a rebuild or more from moved positions
            got[build] = (verlet_pairs(e, 0, 64 * s.n), F, e.stats()["go_active"])
    assert got["cell"][0] == got["tile"][0]
    assert got["cell"][2] == got["tile"][2]
    assert np.abs(got["cell"][1] - got["tile"][1]).max() <= 1e-10 * max(1.0, np.abs(got["tile"][1]).max())
    if name not in ("neither", "wide", "narrow"):
        assert len(got["cell"][0]) > 0
