"""Mixed runs give what they gave: forces and states recorded with this engine
(commit 9664731, on a GB300) for systems of the other fixtures, in mixed
precision.

Which FP32 rounding a bonded or pair term takes is part of a mixed run's result:
the dynamics amplifies one rounding to 1e-3 of single beads' velocities within
128 steps, so a term restated to better accuracy moves every trajectory as much
as one restated to worse.

Bars.  Forces: the same FP32 terms, added in any order in float-float (2^-47 of
the running sum per addition, some 100 additions, partial sums up to 1000 times
the largest force): 1e-9 of the largest force.  One FP32 rounding of a bond's
length alone moves its force by 1e-4.  States after the run: orders of FP64
operations differ by 1e-15, and where that turns one FP32 rounding it grows to at
most 1e-3 of one bead: 2e-5 in the norm (the FP32 terms' own 5e-6 against FP64,
fourfold), 8e-4 of the largest of a value and the rms in the worst component."""
import numpy as np
import pytest

from tests.util import GOLDEN, load_golden
from xmd_gb300 import Engine

pytestmark = pytest.mark.gpu

STEPS = {"c1_native100": 128, "c2_periodic480": 64, "c2_sparse240": 128, "c2_relsnd480": 64, "c3_qa600": 128}


def replay(name):
    s, y, _ = load_golden(name)
    with Engine(y + "\nengine:\n  precision: mixed\n") as e:
        e.add_system(s)
        F, _ = e.eval_forces(0)
        e.step(STEPS[name])
        r, v, _ = e.get_state(0)
    return {"F": F, "r": r, "v": v}


@pytest.mark.parametrize("name", sorted(STEPS))
def test_recorded_mixed_run(name):
    z = np.load(GOLDEN / "mixed_runs.npz")
    got = replay(name)
    F = z[f"{name}_F"]
    assert np.abs(got["F"] - F).max() <= 1e-9 * max(np.abs(F).max(), 1.0)
    for k in ("r", "v"):
        x, y = got[k], z[f"{name}_{k}"]
        d, rms = np.abs(x - y), np.sqrt((y * y).mean())
        assert np.linalg.norm(x - y) <= 2e-5 * np.linalg.norm(y), (k, np.linalg.norm(x - y) / np.linalg.norm(y))
        assert (d / np.maximum(rms, np.abs(y))).max() <= 8e-4, (k, (d / np.maximum(rms, np.abs(y))).max())
