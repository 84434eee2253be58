"""The cell build on replicas far from the origin, where FP32 no longer resolves
a bounding box (the shifts lie off the FP32 grid): the same pairs as at the
origin.  Coordinates are multiples of 2^-14, so the shifts are exact and every
FP64 distance the same."""
import numpy as np
import pytest

from tests.test_gpu_parity import verlet_pairs, with_engine_key
from xmd_gb300 import Engine, synth

pytestmark = pytest.mark.gpu

NO_GO = "\nnative contacts:\n  enabled: false\n"


@pytest.mark.parametrize("shift", [(2.0**36 + 3000.0, 0.0, 0.0), (-(2.0**36) - 2900.0, 2.0**35 + 1000.0, 0.0),
                                   (2.0**31 + 100.0, 2.0**33 + 400.0, -(2.0**36) - 4096.0)])
def test_lists_far_from_the_origin(shift):
    rng = np.random.default_rng(12)
    chains, m = 40, 100
    n = chains * m
    none = np.zeros(0, dtype=np.int32)
    r = np.floor(rng.uniform(-15.0, 15.0, (n, 3)) * 2**14) / 2**14
    s = synth.System(
        n=n, chain=np.repeat(np.arange(chains), m).astype(np.int32), seq=np.tile(np.arange(m), chains).astype(np.int32),
        atype=np.full(n, synth.CHARGED_POS[0], dtype=np.uint8), cell=np.zeros(3), r=r,
        tethers=(none, none, np.zeros(0)), angles=(none, none, none, np.zeros(0)),
        dihedrals=(none, none, none, none, np.zeros(0)), natives=(none, none, np.zeros(0)), temperature=0.35, seed=3)
    y = with_engine_key(synth.yaml_for("c4") + NO_GO, "nl build: cell")
    got = []
    for d in (np.zeros(3), np.array(shift)):
        with Engine(y) as e:
            rep = e.add_system(s)
            e.set_state(rep, r + d)
            assert np.array_equal((r + d) - d, r)
            e.eval_forces(rep)
            got.append(verlet_pairs(e, rep, 400 * n))
    assert len(got[0]) > 20 * n
    assert got[0] == got[1]
