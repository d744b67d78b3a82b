"""The high-velocity solve's short evaluations against the oracle's loop: patches
without coupling (a diagonal shear matrix), so that one step is one solve per
patch, with slip rates from the switch to 30 m/s, states off steady state, and
operands that the short path leaves to the reference loop (the slip law,
Alpha_Evo != 0).

Tolerance: both sides take the secant rule through the same points up to
rounding (1e-13) and stop at a step below 1e-9 V; where rounding decides
whether one more step is taken, the results differ by at most that step times
the rule's contraction: 2e-9 in V, and in theta and the slip, which carry it
scaled by at most one; the friction by a < 0.1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["usual", "alpha", "slip_law"])
@pytest.mark.parametrize("dt", [5e-4, 5e-3])
@pytest.mark.parametrize("n", [1, 40, 700])
def test_one_step_matches_the_secant_loop(qdfn_mod, oracle_mod, n, dt, kind):
    from qdfn import simulate
    rng = np.random.default_rng(31 * n + int(1e5 * dt))
    a = rng.uniform(0.008, 0.02, n)
    b = a + rng.uniform(-0.004, 0.004, n)
    Dc = 10.0 ** rng.uniform(-2, -0.5, n)
    V = 0.012 * 10.0 ** rng.uniform(0, 0.5 if kind == "slip_law" else 2, n)
    th = Dc / V * np.exp(0.3 * rng.standard_normal(n)) if kind == "slip_law" else Dc / 1e-9 * np.exp(
        -rng.uniform(0, 15, n))
    sig = rng.uniform(5e6, 1.2e8, n)
    f = 0.6 + a * np.log(V / 1e-6) + b * np.log(th * 1e-6 / Dc)
    K = 10.0 ** rng.uniform(7, 9, n)
    p = dict(N=n, Nload=0, a=a, b=b, Dc=Dc, theta_i=th, V_i=V, f_i=f, sigma0=sig, V_const=np.zeros(n),
             mass=np.full(n, 1.3e5), G=32e9, rho=2612.0, sigma_min=1e6, switch_v=1e-2, dt_cut=5.0, max_dt=1e7,
             alpha_evo=0.3 if kind == "alpha" else 0.0, evolution_dr=2 if kind == "slip_law" else 1,
             interp_at_told=0, rupture_dt=dt)
    st = dict(V=V, D=rng.uniform(0, 1e-3, n) * a * sig / K, theta=th, friction=f, accel=np.zeros(n), sigma_old=sig,
              T=0.0, dt=dt, step=0)
    Ks, Kn = np.diag(-K), np.zeros((n, n))
    sim = simulate.Simulation(p)
    sim.set_dense(Ks, Kn, "fp64")
    sim.set_state(0, st)
    sim.run(1, timeout_s=60)
    g = sim.state(0)
    assert sim.counters()["highv_solves"] >= n
    o = oracle_mod.Simulation(p, ("dense", Ks, Kn))
    for k, v in o.state.items():
        v[:] = st[k]
    o.set_scalars(0.0, dt, 0)
    o.run(1)
    assert abs(g["dt"] / o.dt - 1) < 1e-12, (g["dt"], o.dt)
    for k, tol in (("V", 2e-9), ("theta", 2e-9), ("friction", 2e-10), ("D", 2e-9)):
        ref = o.state[k]
        bad = np.abs(g[k] - ref) > tol * np.maximum(np.abs(ref), 1e-300)
        assert not bad.any(), (k, np.nonzero(bad)[0][:4], g[k][bad][:4], ref[bad][:4])
    sim.close()
