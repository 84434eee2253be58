"""The launch count of a context: what a rebuild pass launched when it ran."""
import pytest

from xmd_gb300 import Engine, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("build", ["cell", "auto", "tile"])
def test_a_leaving_replica_takes_no_launches_with_it(build):
    with Engine(synth.yaml_for("c4", "mixed") + f"  nl build: {build}\n") as e:
        e.reserve(2000, 4, 16000)
        rep = e.add_system(synth.make_system([120], 6, temperature=0.45))
        e.step(64)
        st = e.stats()
        assert st["rebuilds"] >= 3
        e.remove_replica(rep)
        assert e.stats()["launches"] == st["launches"]


def test_a_contacts_rebuild_launches_three_kernels():
    # the lists of the same system with and without contacts: scan, fill and
    # compaction of the free pairs come on top
    s = synth.make_system([60, 40], 3, box=60 * 0.2, types="uniform20", temperature=0.35)
    got = []
    for on in ("true", "false"):
        y = synth.yaml_for("c3", "mixed") + f"quasi-adiabatic potential:\n  enabled: {on}\n"
        with Engine(y) as e:
            e.add_system(s)
            e.eval_forces(0)
            got.append(e.stats()["launches"])
    assert got[0] - got[1] == 3
