"""FP64 steps at the edges of the operator's row blocks (256 rows) and of the
blocks' own tiles: each instance against the oracle."""
import numpy as np
import pytest

from test_ensemble import _oracle_run, _rel
from _systems import problem_for

G, NU = 32e9, 0.25


@pytest.mark.gpu
@pytest.mark.parametrize("R", [1, 4])
@pytest.mark.parametrize("N", [1, 2, 33, 255, 256, 257, 513])
def test_solves_that_wait_for_their_row_block(qdfn_mod, oracle_mod, N, R):
    """Ten steps of N patches, R friction draws; 1e-9, as for other FP64 runs."""
    from qdfn import assemble, simulate, synth
    rec = synth.fault_network(seed=6, n_faults=8, patch=150.0, length=(1200.0, 2400.0))["records"]
    assert rec.shape[0] >= N
    rec = np.ascontiguousarray(rec[:N])
    Ks, Kn = assemble.assemble_rect(rec, rec, G, NU)
    prob = problem_for(rec, Ks)
    ext = synth.external_ramp(N, 1e6, 1e11)
    draws = synth.friction_draws(dict(prob, N=N), R, seed=6)
    p = dict(prob, **{k: draws[k] for k in ("a", "b", "Dc", "theta_i", "V_i", "f_i")})
    for k in ("sigma0", "V_const", "mass"):
        p[k] = np.tile(prob[k], R)
    sim = simulate.Simulation(p, n_inst=R)
    sim.set_dense(Ks, Kn, "fp64")
    sim.set_external_stress(ext["t"], ext["normal"], ext["shear"], ext["pressure"])
    sim.run(10, timeout_s=60)
    for r in range(R):
        o = _oracle_run(oracle_mod, (prob, ext, draws, Ks, Kn, N, R), r, 10)
        st = sim.state(r)
        assert st["step"] == o.step == 10
        assert abs(st["T"] / o.T - 1) < 1e-9
        assert _rel(st["D"], o.state["D"]) < 1e-9
    sim.close()
