"""A barrier of the step kernel that runs out, on the GPU, without faulting it.

The blocks of the step kernel meet at barriers whose waits are bounded.  The
test makes one barrier miss an arrival (a count that nobody completes) with a
short bound: the kernel leaves, the call raises, launches queued behind it leave
at once, and the context, whose step was left half way, takes no further call
that steps or builds lists.
"""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from beads_b200 import workloads
from beads_b200.engine import Engine

pytestmark = pytest.mark.gpu

LIMIT = 1 << 14
STALLED = "did not meet at a barrier"


def _spec():
    return workloads.fit_mixture(n_replicas=1, n=900, seed=4)[0]


def _takes_no_further_call(eng, obs_shape=None):
    calls = [eng.eval, lambda: eng.run(1), lambda: eng.minimize(5, 0.01, 100.0),
             lambda: eng.set_list_staged(True), eng.debug_neighbors, eng.launch_counts,
             lambda: eng.profile("rebuild", 1), lambda: eng.adjoint_forward(4, 1, 2)]
    if obs_shape is not None:
        calls.append(lambda: eng.adjoint_backward(np.ones(obs_shape)))
    for call in calls:
        with pytest.raises(RuntimeError, match=STALLED):
            call()


@pytest.mark.parametrize("how", ["run", "eval", "minimize", "replay"])
def test_a_barrier_that_runs_out_ends_the_context_with_an_error(how):
    with Engine(_spec()) as eng:
        obs = eng.adjoint_forward(12, 5, 4)  # three segments
        before = eng.state()
        eng.debug_stall(LIMIT)
        with pytest.raises(RuntimeError, match=STALLED):
            if how == "run":
                eng.run(64)
            elif how == "eval":
                eng.eval()
            elif how == "minimize":
                eng.minimize(200, 0.01, 100.0)
            else:
                eng.adjoint_backward(np.ones(obs.shape))
        _takes_no_further_call(eng, obs.shape)
        after = eng.state()  # reading the state stays possible
        assert after["positions"].shape == before["positions"].shape
    with Engine(_spec()) as eng:  # other contexts are not affected
        assert np.isfinite(eng.run(20, 20)[0]["pe"])


def test_the_stall_is_reported_where_a_list_has_overflowed_too():
    spec = dataclasses.replace(_spec(), max_neighbors=8)
    with Engine(spec) as eng:
        with pytest.raises(RuntimeError, match="NeighborList overflow"):
            eng.eval()
        eng.debug_stall(LIMIT)
        with pytest.raises(RuntimeError, match=STALLED):
            eng.eval()
        _takes_no_further_call(eng)
