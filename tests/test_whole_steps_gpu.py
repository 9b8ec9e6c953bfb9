"""Whole steps in one persistent kernel against the same steps launched kernel
by kernel, on the GPU.

A context whose schedule is not fixed by hand takes its steps in one kernel
(small systems); with a fixed schedule every stage is its own launch.  Both
call the same device functions and total in integers, so states, observables
and counters must be the same bits: at one bead, around a 128-slot block, on
direct, small-dimension and regular grids, with exclusions and bonded terms,
in uneven batches, with lists checked at every n-th step and with no skin, and
however a run is cut into calls.
"""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from beads_b200 import workloads
from beads_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _fluid(n, box, seed=1, **kw):
    spec = workloads.lj_lattice()
    rng = np.random.default_rng(seed)
    box = np.asarray(box, float)
    # sites of a nearly cubic lattice that fills the box, so that none overlap
    side = np.ceil(box / (box.prod() / n) ** (1 / 3) - 1e-9).astype(int)
    g = np.indices(side).reshape(3, -1).T
    g = g[np.sort(rng.permutation(g.shape[0])[:n])]
    pos = ((g + 0.5) / side * box + rng.uniform(-0.05, 0.05, (n, 3))) % box
    fields = dict(
        positions=pos.astype(np.float32), types=np.ones(n, np.int32),
        velocities=rng.standard_normal((n, 3)).astype(np.float32), masses=np.ones(n, np.float32),
        box_bound=np.array([np.zeros(3), box], np.float32), rebuild_check_every=1,
        sort_every_rebuild=2)
    return dataclasses.replace(spec, **(fields | kw))


CASES = {
    "one": lambda: [_fluid(1, (6.0, 6.0, 6.0))],
    "two_thermostat": lambda: [_fluid(2, (6.0, 6.0, 6.0), thermostat=(1.0, 0.5))],
    "block_less_one": lambda: [_fluid(127, (6.0, 6.0, 6.0))],
    "block": lambda: [_fluid(128, (6.0, 6.0, 6.0), thermostat=(1.0, 0.5))],
    "block_and_one": lambda: [_fluid(129, (6.0, 6.0, 6.0))],
    "small_dimension": lambda: [_fluid(1000, (20.0, 6.0, 12.0))],
    "regular_every_5": lambda: [_fluid(3000, (15.0, 16.0, 17.0), rebuild_check_every=5,
                                       thermostat=(1.2, 1.0))],
    "no_skin": lambda: [_fluid(300, (7.0, 7.0, 7.0), cutoff_buffer=0.0)],
    "sparse_gas": lambda: [_fluid(500, (40.0, 41.0, 39.0), seed=4)],
    # more cells than 24 per warp of the launch: lists a thread per particle
    "dilute_gas": lambda: [_fluid(700, (95.0, 95.0, 95.0), seed=7, thermostat=(1.0, 1.0))],
    # more replicas than a block has threads, one of them of more cells than a
    # block scans
    "many_replicas": lambda: [_fluid(40 + k, (6.5, 6.5, 6.5), seed=k,
                                     thermostat=(1.0, 1.0) if k % 3 else None)
                              for k in range(140)] + [_fluid(500, (40.0, 41.0, 39.0), seed=4)],
    "melt": lambda: [workloads.polymer_melt(n_chains=20, beads=50, seed=4, max_neighbors=96)],
    "batch": lambda: [_fluid(1, (6.0, 6.0, 6.0)), _fluid(700, (9.0, 9.0, 9.0), seed=2),
                      workloads.polymer_melt(n_chains=10, beads=30, seed=5, max_neighbors=96)]
    + workloads.replica_batch(5, n_min=256, n_max=3000, seed=6),
}


def _run(specs, whole: bool, calls):
    with Engine(specs) as eng:
        if not whole:
            eng.set_tuning(2, False, 4, True)
            eng.set_list_staged(False)
        rows = []
        for steps, every in calls:
            rows.append(eng.run(steps, every))
        states = [eng.state(r) for r in range(len(specs))]
        counters = [eng.counters(r) for r in range(len(specs))]
    return rows, states, counters


@pytest.mark.parametrize("which", list(CASES))
def test_whole_steps_give_the_bits_of_separate_launches(which):
    specs = CASES[which]()
    calls = [(1, 0), (33, 17), (16, 10), (30, 10)]
    a = _run(specs, True, calls)
    b = _run(specs, False, calls)
    assert a[0] == b[0]
    for r in range(len(specs)):
        for key in ("positions", "velocities", "forces", "images"):
            assert np.array_equal(a[1][r][key], b[1][r][key]), (which, r, key)
        for key in ("steps", "builds", "dangerous"):
            assert a[2][r][key] == b[2][r][key], (which, r, key)
    # the same steps cut into other calls
    c = _run(specs, True, [(1, 1)] * 5 + [(45, 0), (30, 80)])
    for r in range(len(specs)):
        for key in ("positions", "velocities", "forces", "images"):
            assert np.array_equal(a[1][r][key], c[1][r][key]), (which, r, key)


def test_set_tuning_returns_to_separate_launches_and_back():
    spec = workloads.lj_lattice(n_side=10)
    with Engine(spec) as eng:
        eng.run(40)
        assert not eng.list_staged()
        eng.set_tuning(4, True, 8, False)
        eng.run(40)
        eng.set_tuning(0)
        eng.run(40)
        mixed = eng.state()
    with Engine(spec) as eng:
        eng.set_tuning(1, False, 4, True)
        eng.run(120)
        plain = eng.state()
    for key in ("positions", "velocities", "forces", "images"):
        assert np.array_equal(mixed[key], plain[key]), key


@pytest.mark.parametrize("iterations", [1, 63, 64, 65])
def test_descent_cut_into_launches(iterations):
    spec = _fluid(900, (12.0, 12.0, 12.0), seed=9)
    outs = []
    for cuts in ([iterations], [1] * iterations if iterations < 64 else [40, iterations - 40]):
        with Engine(spec) as eng:
            for n in cuts:
                eng.minimize(n, 0.01, 100.0)
            outs.append(eng.state())
    if iterations < 64:
        # every call builds its lists anew: the same sets, summed in the same order
        assert np.abs(outs[0]["positions"] - outs[1]["positions"]).max() < 1e-3
    assert np.isfinite(outs[0]["positions"]).all()


@pytest.mark.parametrize("checkpoint", [0, 7, 80])
def test_recorded_steps_give_the_gradients_of_separate_launches(checkpoint):
    """The forward window (more steps than one launch keeps observables of) and
    the replayed segments recorded by the step kernel, against recordings made
    between separate launches."""
    import torch

    from beads_b200.adjoint import trajectory_observables

    specs = workloads.fit_mixture(n_replicas=2, n=700, seed=3) + [
        dataclasses.replace(workloads.fit_mixture(n_replicas=1, n=700, seed=9)[0], thermostat=None)]
    outs = []
    for whole in (True, False):
        with Engine(specs) as eng:
            if not whole:
                eng.set_tuning(2, False, 4, True)
            leaves = [torch.tensor(specs[0].epsilon).requires_grad_(True),
                      torch.tensor(specs[0].sigma).requires_grad_(True),
                      torch.tensor(np.concatenate([s.positions for s in specs])).requires_grad_(True),
                      torch.tensor(np.concatenate([s.velocities for s in specs])).requires_grad_(True)]
            obs = trajectory_observables(eng, *leaves, steps=80, record_from=10,
                                         checkpoint_every=checkpoint)
            grads = torch.autograd.grad((obs * torch.linspace(0.5, 1.5, obs.numel(),
                                                              dtype=obs.dtype).view_as(obs)).sum(),
                                        leaves)
            outs.append([obs.detach(), *grads])
    for a, b in zip(*outs):
        assert torch.equal(a, b)
