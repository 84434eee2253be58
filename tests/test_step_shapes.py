"""Launch shapes of the step kernel at a size where 32-slot blocks keep four
threads per slot (below it they take eight): the same bits as 64-slot blocks, and
as the shapes with one and two threads per slot."""
import numpy as np
import pytest

from xmd_gb300 import Engine, synth

pytestmark = pytest.mark.gpu

SHAPES = [(64, 0, 16, 4), (32, 0, 16, 4), (32, 0, 16, 2), (64, 0, 16, 1)]


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_shapes_of_many_blocks(prec):
    # 18,600 beads: 689 blocks of 27 beads, more than the four per SM (mixed; FP64:
    # one) up to which they take eight threads per slot
    one = synth.make_system([290, 20], 8, temperature=0.4, start="native")
    want = None
    for shape in SHAPES:
        with Engine(synth.yaml_for("c4", prec)) as e:
            for k in range(60):
                e.add_system(one, seed=k + 1)
            e.set_tuning(*shape)
            e.step(12)
            got = [e.get_history(k)[0] for k in (0, 1, 31, 59)]
        want = want or got
        for a, b in zip(got, want):
            assert np.array_equal(a, b), shape
