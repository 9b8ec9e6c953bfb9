"""What a signal's handler raises while execute_simulation runs reaches the
caller, whatever its type (the reference passes on the pending Python error,
native/src/bindings/module.cpp:29-34)."""

from __future__ import annotations

import signal
import time

import pytest

from beads_b200 import _native, workloads

pytestmark = pytest.mark.gpu


class _Stop(Exception):
    pass


@pytest.mark.parametrize("kind", [_Stop, KeyboardInterrupt, SystemExit])
def test_handler_exceptions_stop_the_run_and_reach_the_caller(kind, tmp_path, monkeypatch):
    from tests.golden.make_reference_fixtures import spec_for

    monkeypatch.chdir(tmp_path)
    spec = spec_for(workloads.lj_lattice(), 2_000_000, "long", forces=False, thermo_every=100_000)

    def on_alarm(signum, frame):
        raise kind("from the handler")

    old = signal.signal(signal.SIGALRM, on_alarm)
    try:
        signal.setitimer(signal.ITIMER_REAL, 0.7)
        t0 = time.perf_counter()
        with pytest.raises(kind, match="from the handler"):
            _native.execute_simulation(spec)
        elapsed = time.perf_counter() - t0
    finally:
        signal.setitimer(signal.ITIMER_REAL, 0.0)
        signal.signal(signal.SIGALRM, old)
    # the whole run would take some thirty seconds
    assert elapsed < 10.0, elapsed
