"""Parameter gradients of losses whose gradient on the observables is tiny.

Every particle adds its parameter adjoints to the totals in fixed point (units
of 2^-32, rounded towards minus infinity), so contributions far below one unit
of either sign must leave a total within one unit per contribution of the true
value.
"""

from __future__ import annotations

import dataclasses

import numpy as np
import pytest

from beads_b200 import workloads
from beads_b200.engine import Engine

pytestmark = pytest.mark.gpu

STEPS, RECORD = 12, 5


def _specs(n_types):
    specs = workloads.fit_mixture(n_replicas=2, n=600, seed=17)
    if n_types == 2:
        return specs
    out = []
    for s in specs:
        if n_types == 1:
            types, eps, sig = np.ones(s.n, np.int32), np.array([[1.0]]), np.array([[1.0]])
        else:
            types = (np.arange(s.n) % n_types + 1).astype(np.int32)
            e, g = np.linspace(0.8, 1.1, n_types), np.linspace(0.92, 1.0, n_types)
            eps, sig = np.sqrt(np.outer(e, e)), 0.5 * (g[:, None] + g[None, :])
        out.append(dataclasses.replace(s, types=types, epsilon=eps, sigma=sig))
    return out


@pytest.mark.parametrize("checkpoint", [0, 5])
@pytest.mark.parametrize("n_types", [1, 2, 4])
def test_tiny_cotangents_give_tiny_parameter_gradients(n_types, checkpoint):
    specs = _specs(n_types)
    with Engine(specs) as eng:
        obs = eng.adjoint_forward(STEPS, RECORD, checkpoint)
        g = np.random.default_rng(3).standard_normal(obs.shape)
        full = eng.adjoint_backward(g)[:2]
        for scale in (1e-14, -1e-16, 1e-17, 1e-18, -1e-18):
            tiny = eng.adjoint_backward(scale * g)[:2]
            for r, s in enumerate(specs):
                # a contribution per particle and step: below one unit each,
                # and the total in float32 sums of the scaled terms
                bound = s.n * (STEPS + 1) * 2.0 ** -32
                for a, b in zip(full, tiny):
                    off = np.abs(b[r] - scale * a[r])
                    assert np.all(off <= bound + 1e-3 * np.abs(scale * a[r])), (scale, r, off.max())
