"""Contexts with reserved capacity while replicas come and go.  A replica's
trajectory does not depend on what the context held before it: the same bits as
alone in a fresh one."""
import time

import numpy as np
import pytest

from xmd_gb300 import Engine, Server, synth

pytestmark = pytest.mark.gpu


def yaml(prec="fp64", build="auto"):
    return synth.yaml_for("c4", prec) + f"  nl build: {build}\n"


def system(n, seed, start="saw"):
    return synth.make_system([n], seed, temperature=0.45, start=start)


def run_alone(y, s, steps):
    with Engine(y) as e:
        e.reserve(2000, 4, 16000)
        rep = e.add_system(s)
        e.step(steps)
        return e.get_history(rep)[0], e.stats()["rebuilds"]


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("build", ["auto", "cell", "tile"])
@pytest.mark.parametrize("emptied", [False, True])
def test_steps_of_an_empty_context(prec, build, emptied):
    # steps while nothing is placed (before the first replica, or after the last
    # one left), then a run over several list rebuilds with the same graphs
    y, s = yaml(prec, build), system(120, 6)
    want, rebuilds = run_alone(y, s, 96)
    assert rebuilds >= 3
    with Engine(y) as e:
        e.reserve(2000, 4, 16000)
        if emptied:
            k = e.add_system(system(70, 7))
            e.step(2)
            e.remove_replica(k)
        e.step(96)
        rep = e.add_system(s)
        e.step(96)
        assert np.array_equal(e.get_history(rep)[0], want)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_finished_replicas_cost_no_step(prec):
    # once every replica has taken its steps, a step kernel only carries the
    # positions over: 48 chains of 500 beads, where a step's arithmetic is most
    # of its time (well over half in both precisions)
    one = system(500, 8, "native")
    with Engine(yaml(prec)) as e:
        for k in range(48):
            e.add_system(one, seed=k + 1)

        def seconds():
            best = 1e9
            for _ in range(5):
                t0 = time.perf_counter()
                e.step(64)
                best = min(best, time.perf_counter() - t0)
            return best

        e.step(64)
        running = seconds()
        for k in range(48):
            e.set_steps(k, 0)
        before = [e.get_history(k)[0] for k in (0, 47)]
        e.step(64)
        done = seconds()
        for k, y in zip((0, 47), before):
            assert np.array_equal(e.get_history(k)[0], y)
    assert done < 0.7 * running, (done, running)


def test_split_positions_only_where_they_are_read():
    # two float4 per bead and buffer hold the mixed path's split positions (and
    # the contacts' sift's): an FP64 context without contacts has none
    per_bead = {}
    for prec in ("fp64", "mixed"):
        with Server(yaml(prec), hbm_budget=64 << 20, max_beads=4000) as srv:
            per_bead[prec] = srv.stats()["bytes_per_bead"]
    assert per_bead["mixed"] - per_bead["fp64"] == pytest.approx(64.0, abs=0.5)
