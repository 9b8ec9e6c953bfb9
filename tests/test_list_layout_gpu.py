"""The neighbour list and the layout a context says it has agree between calls."""

from __future__ import annotations

import numpy as np
import pytest

from beads_b200 import workloads
from beads_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _lists(eng):
    counts, partners = eng.debug_neighbors()
    return counts, [np.sort(row[:c]) for row, c in zip(partners, counts)]


@pytest.mark.parametrize("hand", ["", "schedule", "staged"])
@pytest.mark.parametrize("iterations", [1, 70])
def test_descent_leaves_a_list_in_the_layout_of_the_context(hand, iterations):
    spec = workloads.fit_mixture(n_replicas=1, n=3000, seed=8)[0]

    def go(prepare):
        with Engine(spec) as eng:
            prepare(eng)
            eng.minimize(iterations, 0.002, 100.0)
            staged = eng.list_staged()
            after_descent = _lists(eng)
            eng.eval()
            return staged, after_descent, _lists(eng), eng.state()

    def by_hand(eng):
        assert eng.list_staged()
        if hand == "schedule":
            eng.set_tuning(2, False, 4, True)
        elif hand == "staged":
            eng.set_list_staged(True)

    a, b = go(by_hand), go(lambda eng: eng.set_list_staged(False))
    assert a[0] is (hand != "") and b[0] is False
    for x, y in ((a[1], b[1]), (a[2], b[2])):
        assert np.array_equal(x[0], y[0])
        assert all(np.array_equal(p, q) for p, q in zip(x[1], y[1]))
    for key in ("positions", "forces", "images"):
        assert np.array_equal(a[3][key], b[3][key]), key


def test_steps_captured_before_the_first_evaluation_are_not_replayed_on_another_layout():
    # more slots than whole steps in one kernel take: steps are captured graphs
    spec = workloads.lj_lattice(n_side=53)

    def go(counts_first):
        with Engine(spec) as eng:
            assert eng.list_staged()
            if counts_first:
                eng.launch_counts()
                assert not eng.list_staged()
            eng.profile("step", 3)
            return eng.state()

    a, b = go(True), go(False)
    for key in ("positions", "velocities", "forces", "images"):
        assert np.array_equal(a[key], b[key]), key


def test_staged_contexts_of_different_stage_sizes_run_side_by_side():
    # ~53 and 27 beads per cell: stages above 48 KB, of two sizes
    specs = [workloads.lj_lattice(n_side=15, cutoff=c, check_every=1) for c in (3.6, 2.5)]

    def forces(staged):
        engines = [Engine(s) for s in specs]
        for eng in engines:
            eng.set_list_staged(staged)
            eng.eval()
        engines[0].run(3)
        out = [eng.state() for eng in engines]
        assert all(eng.list_staged() is staged for eng in engines)
        for eng in engines:
            eng.close()
        return out

    for a, b in zip(forces(True), forces(False)):
        for key in ("positions", "forces"):
            assert np.array_equal(a[key], b[key]), key


@pytest.mark.parametrize("n_side", [15, 16, 30, 40])
def test_lists_of_cells_shared_by_several_warps(n_side):
    # cells of 27 beads, 216 cells of 19, 1,331 cells, 3,375 cells: three, three,
    # two and one warp a cell
    spec = workloads.lj_lattice(n_side=n_side, max_neighbors=128)
    out = []
    for by_hand in (True, False):
        with Engine(spec) as eng:
            if by_hand:  # the list build as a kernel of its own
                eng.set_list_staged(False)
                eng.set_tuning(2, False, 4, True)
            eng.eval()
            out.append(eng.debug_neighbors())
    assert np.array_equal(out[0][0], out[1][0])
    assert np.array_equal(out[0][1], out[1][1])
