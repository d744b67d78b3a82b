"""qdfn_adjoint_run's timeout is a step's: a window in one long segment passes
with a limit of twenty steps' time, which the segment as a whole takes many times
over, and an expired limit ends the call with the timeout status."""
import time

import numpy as np
import pytest

from _systems import problem_for, small_network

pytestmark = pytest.mark.gpu


def _sim():
    from qdfn import assemble, simulate
    rec = small_network(seed=5, n_faults=3, patch=500.0)["records"]
    Ks, Kn = assemble.assemble_rect(rec, rec, 32e9, 0.25)
    sim = simulate.Simulation(problem_for(rec, Ks, seed=3))
    sim.set_dense(Ks, Kn, "fp64")
    return sim


def test_long_segments_have_their_steps_time(qdfn_mod):
    from qdfn import adjoint
    steps = 1000
    sim = _sim()
    start = sim.state(0)
    sim.run(20, timeout_s=60)
    t0 = time.perf_counter()
    sim.run(steps, timeout_s=60)
    step_s = (time.perf_counter() - t0) / steps
    sim.set_state(0, start)
    loss = np.ones(sim.N)
    ref = adjoint.gradient(sim, steps, dL_dD_final=loss, checkpoint_every=steps)
    sim.set_state(0, start)
    got = adjoint.gradient(sim, steps, dL_dD_final=loss, checkpoint_every=steps, timeout_s=20 * step_s)
    for k in ref:
        assert np.array_equal(ref[k], got[k]), k


def test_an_expired_limit_is_an_error(qdfn_mod):
    from qdfn import _lib, adjoint
    sim = _sim()
    with pytest.raises(_lib.QdfnError, match="TIMEOUT"):
        adjoint.gradient(sim, 400, dL_dD_final=np.ones(sim.N), checkpoint_every=400, timeout_s=1e-9)
