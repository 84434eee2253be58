"""The precision of a context may change between calls: what runs after the change
is the same bits as in a context created with that precision.  Without contacts an
FP64 context holds no split positions until it turns mixed."""
import numpy as np
import pytest

from xmd_gb300 import Engine, synth
from xmd_gb300.abi import PREC_FP64, PREC_MIXED, check

pytestmark = pytest.mark.gpu

CODE = {"fp64": PREC_FP64, "mixed": PREC_MIXED}
SYSTEMS = {"open": synth.make_system([90, 70], 4, temperature=0.45, start="native"),
           "periodic": synth.make_system([60, 40], 3, box=60 * 0.2, types="uniform20", temperature=0.35)}


def run(e):
    F, _ = e.eval_forces(0)
    e.step(40)
    y, t, rng = e.get_history(0)
    return F, y, t, rng


@pytest.mark.parametrize("name", sorted(SYSTEMS))
@pytest.mark.parametrize("first,then", [("fp64", "mixed"), ("mixed", "fp64")])
@pytest.mark.parametrize("build", ["auto", "cell"])
def test_changed_precision(name, first, then, build):
    s = SYSTEMS[name]
    got = []
    for prec in (first, then):
        with Engine(synth.yaml_for("c4", prec) + f"  nl build: {build}\n") as e:
            e.add_system(s)
            e.eval_forces(0)
            if prec != then:
                e.step(24)
                check(e.lib.xmd_gpu_set_precision(e.h, CODE[then]))
            e.set_state(0, s.r, np.zeros_like(s.r))
            got.append(run(e))
    for a, b in zip(*got):
        assert np.array_equal(a, b)
