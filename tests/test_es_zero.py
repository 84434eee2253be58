"""Electrostatic pairs without a force: at an infinite permittivity the factor of
a charged pair is zero, and a run is the same bits as without the term."""
import numpy as np
import pytest

from xmd_gb300 import Engine, synth

pytestmark = pytest.mark.gpu

LISTS = "neighbor list:\n  cutoff: 22 A\n  skin: 2 A\n"


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("term", ["const", "relative"])
@pytest.mark.parametrize("box", [None, 80 * 0.2])
def test_zero_factor(prec, term, box):
    s = synth.make_system([90, 70], 4, box=box, temperature=0.35, start="native")
    on = {"const": "const ES:\n  enabled: true\n  permittivity: 1e400 eps_0\n",
          "relative": "const ES:\n  enabled: false\nrelative ES:\n  enabled: true\n  factor: 1e400 eps_0/A\n"}[term]
    got = []
    for es in (on, "const ES:\n  enabled: false\n"):
        with Engine(synth.yaml_for("c4", prec) + LISTS + es) as e:
            e.add_system(s)
            e.step(8)
            got.append(e.get_history(0)[0])
            if es == on:
                assert e.stats()["nl_entries"] > 0
    assert np.array_equal(*got)
