"""The low-velocity solve's Newton iteration against the oracle's secant loop.

Patches without coupling (a diagonal shear matrix), so that one step is one
solve per patch, over the operands the Newton iteration takes -- slip rates
from locked to near the switch, states off steady state, stresses that make V
change by orders of magnitude -- and over the ones it hands to the reference
loop: slip rates below its range, Alpha_Evo != 0, the slip law.

Tolerance: both iterations stop at a relative step below 1e-9 and leave at most
that step times the slope's relative error (below 1e-3 for the secant slope,
whose two residuals differ by 1e-10 V at a rounding noise of up to 1e-13), so
1e-12, plus the rounding of the residual, ulp(mu) / a ~ 1e-14: 1e-10 allows a
hundred times that.  Theta and the slip carry V's error scaled by at most one,
the friction by a < 0.1."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _patches(n, seed, dt, kind):
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.006, 0.02, n)
    b = a + rng.uniform(-0.004, 0.004, n)
    Dc = 10.0 ** rng.uniform(-4, -1, n)
    V = 10.0 ** rng.uniform(-14, -3, n) if dt < 1 else 1e-9 * np.exp(rng.standard_normal(n))
    if kind == "below_range":
        V[::7] = 10.0 ** rng.uniform(-40, -26, V[::7].size)
    th = Dc / 1e-9 * np.exp(0.3 * rng.standard_normal(n))
    sig = rng.uniform(5e6, 1.2e8, n)
    f = 0.6 + a * np.log(V / 1e-6) + b * np.log(th * 1e-6 / Dc)
    K = 10.0 ** rng.uniform(7, 10, n)
    D = rng.uniform(0, 1e-3, n)
    # slip that loads or unloads the patch by up to ~half a friction decade
    D += rng.uniform(-1, 1, n) * a * sig / K * min(1.0, dt / 1e3 if dt >= 1 else 1.0)
    p = dict(N=n, Nload=0, a=a, b=b, Dc=Dc, theta_i=th, V_i=V, f_i=f, sigma0=sig, V_const=np.zeros(n),
             mass=np.full(n, 1.3e5), G=32e9, rho=2612.0, sigma_min=1e6, switch_v=1e-2, dt_cut=5.0, max_dt=1e7,
             alpha_evo=0.3 if kind == "alpha" else 0.0, evolution_dr=2 if kind == "slip_law" else 1,
             interp_at_told=0, rupture_dt=1e-6)
    state = dict(V=V, D=D * 1e-3, theta=th, friction=f, accel=V / (5.0 * dt), sigma_old=sig, T=0.0, dt=dt, step=0)
    return p, K, state


@pytest.mark.parametrize("kind", ["usual", "below_range", "alpha", "slip_law"])
@pytest.mark.parametrize("dt", [5e-3, 10.0, 1e3])
@pytest.mark.parametrize("n", [1, 33, 771])
def test_one_step_matches_the_secant_loop(qdfn_mod, oracle_mod, n, dt, kind):
    from qdfn import simulate
    p, K, st = _patches(n, 17 * n + int(dt), dt, kind)
    Ks, Kn = np.diag(-K), np.zeros((n, n))
    sim = simulate.Simulation(p)
    sim.set_dense(Ks, Kn, "fp64")
    sim.set_state(0, st)
    sim.run(1, timeout_s=60)
    g = sim.state(0)
    o = oracle_mod.Simulation(p, ("dense", Ks, Kn))
    for k, v in o.state.items():
        v[:] = st[k]
    o.set_scalars(0.0, dt, 0)
    o.run(1)
    assert abs(g["dt"] / o.dt - 1) < 1e-12, (g["dt"], o.dt)   # the same halvings
    for k, tol in (("V", 1e-10), ("theta", 1e-10), ("friction", 1e-11), ("D", 1e-10)):
        ref = o.state[k]
        bad = np.abs(g[k] - ref) > tol * np.maximum(np.abs(ref), 1e-300)
        assert not bad.any(), (k, np.nonzero(bad)[0][:4], g[k][bad][:4], ref[bad][:4])
    sim.close()
