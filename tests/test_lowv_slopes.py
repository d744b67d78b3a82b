"""Low-velocity solves whose residual has a slope beyond FP32's safe range, which
the Newton iteration has to leave to the reference loop: a heavy patch, far
above its friction (friction inversion e^58.7 V0 at V = 1e-24 m/s).  With g/a =
4.8e21 the slope is 1.2e38, between __fdividef's 2^126 and FP32's largest, and the
solution is 1.7e-20 m/s, 84 secant steps away; with g/a = 1e40, beyond FP32, V
moves by 1e-40 m/s.

Tolerance: both sides run the secant loop of the reference, which stops at a
relative step below 1e-9; where rounding decides whether one more is taken, they
differ by at most that step: 2e-9 in V, and in theta and the slip, which carry it
scaled by at most one; the friction carries it times a (g/a)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ga", [4.8e21, 1e29, 1e31, 1e40])
@pytest.mark.parametrize("n", [1, 40])
def test_heavy_patches_match_the_secant_loop(qdfn_mod, oracle_mod, n, ga):
    from qdfn import simulate
    a, b, Dc, sig, dt = 0.01, 0.013, 1e-2, 5e7, 5e-4
    full = lambda v: np.full(n, v)
    th_i = full(1e2) * np.linspace(1.0, 1.5, n)
    p = dict(N=n, Nload=0, a=full(a), b=full(b), Dc=full(Dc), theta_i=th_i, V_i=full(1e10), f_i=full(0.6),
             sigma0=full(sig), V_const=np.zeros(n), mass=full(ga * dt * sig * a), G=32e9, rho=2612.0, sigma_min=1e6,
             switch_v=1e-2, dt_cut=5.0, max_dt=1e7, alpha_evo=0.0, evolution_dr=1, interp_at_told=0, rupture_dt=dt)
    st = dict(V=full(1e-24), D=np.zeros(n), theta=full(5e-4), friction=full(0.6), accel=full(1e-24 / (5.0 * dt)),
              sigma_old=full(sig), T=0.0, dt=dt, step=0)
    Ks, Kn = np.diag(full(-1e8)), np.zeros((n, n))
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
    assert abs(g["dt"] / o.dt - 1) < 1e-12, (g["dt"], o.dt)
    for k in ("V", "theta", "friction", "D"):
        ref = o.state[k]
        scale = np.abs(ref) + (a * ga * np.abs(o.state["V"]) if k == "friction" else 0.0)
        assert np.all(np.abs(g[k] - ref) <= 2e-9 * scale), (k, g[k][:3], ref[:3])
    sim.close()
