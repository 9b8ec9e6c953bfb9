"""Corners of the step kernel against the same work launched kernel by kernel."""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from beads_b200 import workloads
from beads_b200.engine import Engine

pytestmark = pytest.mark.gpu

STATE = ("positions", "velocities", "forces", "images")


def _spec(pos, box, seed=1, **kw):
    n = len(pos)
    fields = dict(
        positions=np.asarray(pos, np.float32), types=np.ones(n, np.int32),
        velocities=np.random.default_rng(seed).standard_normal((n, 3)).astype(np.float32),
        masses=np.ones(n, np.float32), box_bound=np.array([np.zeros(3), np.full(3, box)], np.float32),
        rebuild_check_every=1, sort_every_rebuild=2)
    return dataclasses.replace(workloads.lj_lattice(), **(fields | kw))


def _droplet(side, spacing, box, gas, seed=3, **kw):
    """A dense lattice in one corner of a box that is empty but for a gas:
    few beads per cell on average, many in the cells of the droplet."""
    rng = np.random.default_rng(seed)
    drop = (np.indices((side,) * 3).reshape(3, -1).T + 0.5) * spacing
    g = max(1, int(np.ceil(gas ** (1 / 3))))
    sites = (np.indices((g,) * 3).reshape(3, -1).T + 0.5) * (box / g)
    sites = sites[(sites > side * spacing + 2.0).any(1)][:gas].reshape(-1, 3)
    pos = np.concatenate([drop, sites]) + rng.uniform(-0.03, 0.03, (side ** 3 + len(sites), 3))
    return _spec(pos, box, **kw)


def _compare(specs, calls):
    def go(whole):
        with Engine(specs) as eng:
            if not whole:
                eng.set_list_staged(False)
                eng.set_tuning(2, False, 4, True)
            rows = [eng.run(steps, every) for steps, every in calls]
            return rows, [eng.state(r) for r in range(len(specs))]

    a, b = go(True), go(False)
    assert a[0] == b[0]
    for r in range(len(specs)):
        for key in STATE:
            assert np.array_equal(a[1][r][key], b[1][r][key]), (r, key)


SPARSE = {
    # cells of about 22, of about 40, and of more than 256 beads
    "droplet": lambda: [_droplet(8, 1.0, 48.0, 300)],
    "tight_droplet": lambda: [_droplet(9, 0.82, 48.0, 300, sigma=np.array([[0.8]]))],
    "crowd": lambda: [_droplet(9, 0.4, 60.0, 300, sigma=np.array([[0.38]]), dt=0.001,
                               max_neighbors=1024)],
    "droplet_among_dense": lambda: [_droplet(8, 1.0, 48.0, 300, seed=5)]
    + workloads.replica_batch(2, n_min=300, n_max=900, seed=6),
}


@pytest.mark.parametrize("which", list(SPARSE))
def test_crowded_cells_of_sparse_boxes(which):
    _compare(SPARSE[which](), [(20, 10), (15, 0)])


def test_more_shares_of_cells_than_warps():
    # 4,096 cells, shared by more warps than the launch has: some build several
    _compare([workloads.lj_lattice(n_side=44, check_every=1, max_neighbors=128)],
             [(12, 6), (9, 0)])


def test_sizes_around_the_largest_context_that_steps_in_one_kernel():
    # 102,400 slots: 128 of them or fewer beads below, at and above
    sides, base = (102272, 102400, 102401), workloads.lj_lattice(n_side=47, max_neighbors=128)
    for n in sides:
        spec = dataclasses.replace(
            base, positions=base.positions[:n], types=base.types[:n],
            velocities=base.velocities[:n], masses=base.masses[:n], rebuild_check_every=1)
        _compare([spec], [(8, 4)])


@pytest.mark.parametrize("blocks", [1, 3, 100, 60000])
def test_any_number_of_blocks_takes_the_same_steps(blocks):
    """60,000 blocks are more than a GPU holds at once: the launch is refused
    and made with fewer.  The large system has work for that many."""
    large = blocks > 1000
    specs = ([workloads.lj_lattice(n_side=45, check_every=1, max_neighbors=128)] if large else
             [_droplet(8, 1.0, 48.0, 200), workloads.polymer_melt(n_chains=8, beads=40, seed=4,
                                                                  max_neighbors=96)])

    def go(limit):
        with Engine(specs) as eng:
            if limit:
                eng.debug_step_blocks(limit)
            eng.minimize(3, 0.002, 100.0)
            rows = [eng.eval(), eng.run(12, 6)]
            return rows, [eng.state(r) for r in range(len(specs))]

    a, b = go(blocks), go(0)
    assert a[0] == b[0]
    for x, y in zip(a[1], b[1]):
        for key in STATE:
            assert np.array_equal(x[key], y[key]), key


def test_launch_counts_of_a_context_that_steps_in_one_kernel():
    with Engine(workloads.lj_lattice(n_side=8)) as eng:
        assert eng.launch_counts() == {"per_step": 1, "per_rebuild_chain": 0}
        eng.run(5)
        assert eng.launch_counts() == {"per_step": 1, "per_rebuild_chain": 0}
        eng.set_tuning(2, True, 4, True)  # kernel by kernel
        assert eng.launch_counts()["per_step"] == 4


DESCENTS = {
    "fluid": lambda: [_droplet(9, 1.0, 9.6, 0, sort_every_rebuild=3)],
    "no_skin": lambda: [_droplet(7, 1.0, 7.6, 0, cutoff_buffer=0.0, cutoff=2.4)],
    # exclusions, bonded terms, a thermostat, boxes of several sizes and types
    "batch": lambda: [workloads.polymer_melt(n_chains=8, beads=40, seed=4, max_neighbors=128),
                      _droplet(8, 1.0, 48.0, 150, seed=2)]
    + workloads.fit_mixture(n_replicas=2, n=700, seed=3),
}


@pytest.mark.parametrize("which", list(DESCENTS))
@pytest.mark.parametrize("iterations", [1, 63, 64, 65, 129])
def test_descent_gives_the_bits_of_separate_launches(which, iterations, monkeypatch):
    """BEADS_GRAPHS=0 launches every kernel of an iteration by itself."""
    specs = DESCENTS[which]()

    def go(cuts):
        with Engine(specs) as eng:
            for n in cuts:
                eng.minimize(n, 0.004, 50.0)
            states = [eng.state(r) for r in range(len(specs))]
            eng.eval()
            return states, [eng.state(r)["forces"] for r in range(len(specs))]

    cuts = [[iterations], [40, iterations - 40] if iterations > 40 else [iterations]]
    whole = [go(c) for c in cuts]
    monkeypatch.setenv("BEADS_GRAPHS", "0")
    apart = [go(c) for c in cuts]
    for a, b in zip(whole, apart):
        for r in range(len(specs)):
            for key in ("positions", "images"):
                assert np.array_equal(a[0][r][key], b[0][r][key]), (r, key)
            assert np.array_equal(a[1][r], b[1][r]), r


def test_more_than_two_types_step_in_one_kernel_up_to_131072_slots():
    base = workloads.lj_lattice(n_side=48, max_neighbors=128, check_every=1)
    scale = np.array([1.0, 0.9, 1.1])
    spec = dataclasses.replace(
        base, types=(np.arange(base.n) % 3 + 1).astype(np.int32),
        epsilon=np.sqrt(np.outer(scale, scale)), sigma=np.full((3, 3), 1.0))
    with Engine(spec) as eng:
        assert eng.launch_counts()["per_step"] == 1
    _compare([spec], [(8, 4)])
    with Engine(base) as eng:  # one type, the same size: kernel by kernel
        assert eng.launch_counts()["per_step"] > 1
