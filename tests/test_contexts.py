"""Two contexts of one process whose kernels need different amounts of shared
memory: the later, smaller one leaves the earlier one's limit alone (the
same trajectory with and without it)."""
import numpy as np
import pytest

from xmd_gb300 import Engine, synth

pytestmark = pytest.mark.gpu

CASES = {   # yaml and sizes of the two contexts, launch shape
    "tile rows": (("c4", "mixed", [1500, 2000]), ("c4", "mixed", [2100]), (64, 0, 16, 4)),
    "contact terms": (("c3", "fp64", [130, 97]), ("c4", "fp64", [130]), (128, 0, 16, 4)),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_smaller_context_after_a_larger(name):
    big, small, shape = CASES[name]

    def engine(cfg, prec, sizes):
        e = Engine(synth.yaml_for(cfg, prec) + "\n")
        e.add_system(synth.make_system(sizes, 3, temperature=0.35, start="native"))
        e.set_tuning(*shape)
        return e
    got = []
    for other in (False, True):
        with engine(*big) as a:
            a.step(2)
            if other:
                with engine(*small) as b:
                    b.step(2)
                    a.eval_forces(0)
                    a.step(40)
            else:
                a.eval_forces(0)
                a.step(40)
            got.append(a.get_history(0)[0])
    assert np.array_equal(*got)
