"""The patch solvers one by one (qdfn_check_solve), so that a test of one is a
test of it whatever the step loop would choose: the short solvers take every
ordinary patch and return what the reference's secant loops return, they leave
the slip law, Alpha_Evo != 0 and extreme operands alone, and the loops give the
same bits on a lane pair as on one lane, ordinary and failing solves alike.  In
the step loop, with the slip law and Alpha_Evo != 0, which always run the loops,
QDFN_PAIR_SOLVE changes no bit.

Tolerances: low velocity as in test_lowv_newton.py (1e-10; friction 1e-11), high
velocity as in test_highv_usual.py (2e-9; friction 2e-10)."""
import numpy as np
import pytest

from test_schedule_invariance import _run, _same, loaded_network  # noqa: F401

pytestmark = pytest.mark.gpu
LOW, HIGH = 0, 1
SHORT, ONE_LANE, PAIR = 0, 2, 4
FIELDS = ("taken", "V", "friction", "D", "theta", "dt", "instab", "flag", "iterations", "err")
ETA = 32e9 / 2 / np.sqrt(32e9 / 2612.0)


def _operands(n, seed, high, dt):
    rng = np.random.default_rng(seed)
    a = rng.uniform(0.006, 0.02, n)
    b = a + rng.uniform(-0.004, 0.004, n)
    Dc = 10.0 ** (rng.uniform(-2, -0.5, n) if high else rng.uniform(-4, -1, n))
    V = 0.012 * 10.0 ** rng.uniform(0, 2, n) if high else 1e-9 * np.exp(rng.standard_normal(n))
    th = Dc / 1e-9 * np.exp(-rng.uniform(0, 15, n) if high else 0.3 * rng.standard_normal(n))
    sig = rng.uniform(5e6, 1.2e8, n)
    K = 10.0 ** rng.uniform(7, 9, n)
    mass = np.full(n, 1.3e5)
    F0 = np.full(n, 0.6)
    f = F0 + a * np.log(V / 1e-9) + b * np.log(th * 1e-9 / Dc)
    D = rng.uniform(0, 1e-3, n)
    x = np.stack([D, f, th, V, F0, a, b, Dc, K, np.sqrt(K / mass), mass, sig, D,
                  rng.uniform(-0.3, 0.3, n) * a * sig, sig * rng.uniform(0.99, 1.01, n), f * sig, np.full(n, dt)], axis=1)
    return x


def _solve(which, x, alpha=0.0, dr=1):
    import torch
    from qdfn import _lib
    L = _lib.load()
    xt = torch.tensor(np.ascontiguousarray(x), device="cuda")
    y = torch.zeros((len(x), len(FIELDS)), dtype=torch.float64, device="cuda")
    _lib.check(L.qdfn_check_solve(which, len(x), xt.data_ptr(), ETA, alpha, dr, 1e-2, y.data_ptr(), None))
    return dict(zip(FIELDS, y.cpu().numpy().T))


@pytest.mark.parametrize("high,dt", [(LOW, 5e-3), (LOW, 10.0), (LOW, 1e3), (HIGH, 5e-4), (HIGH, 5e-3)])
@pytest.mark.parametrize("n", [1, 33, 4097])
def test_short_solvers_take_ordinary_patches(qdfn_mod, n, high, dt):
    x = _operands(n, 7 * n + high, high, dt)
    got, ref = _solve(SHORT + high, x), _solve(ONE_LANE + high, x)
    whole = ref["flag"] == 1   # (a solve that halves Dt is the loops' to end)
    assert np.mean(whole) > 0.99 or n == 1
    assert np.all(got["taken"][whole] == 1), np.nonzero(got["taken"][whole] == 0)
    for k, tol in (("V", 1e-10), ("friction", 1e-11), ("D", 1e-10), ("theta", 1e-10)):
        tol = tol if high == LOW else tol * 20
        off = np.abs(got[k] - ref[k])[whole]
        assert np.all(off <= tol * np.abs(ref[k])[whole]), (k, off.max())


@pytest.mark.parametrize("high", [LOW, HIGH])
def test_short_solvers_leave_the_rest(qdfn_mod, high):
    x = _operands(64, 3, high, 5e-3)
    assert not _solve(SHORT + high, x, alpha=0.3)["taken"].any()
    assert not _solve(SHORT + high, x, dr=2)["taken"].any()
    for field in (2, 3, 5, 6, 7, 11, 14, 16):          # theta, V, a, b, Dc, sigma, old sigma, Dt
        for bad in (np.nan, np.inf, 0.0, 1e-320):
            if field == 2 and high == LOW and bad != np.inf and not np.isnan(bad):
                continue                                # (theta + Dt counts there)
            y = x.copy()
            y[:, field] = bad
            assert not _solve(SHORT + high, y)["taken"].any(), (field, bad)


@pytest.mark.parametrize("high,dt", [(LOW, 5e-3), (LOW, 1e3), (LOW, 1e6), (HIGH, 5e-3), (HIGH, 1.0)])
@pytest.mark.parametrize("alpha,dr", [(0.0, 1), (0.2, 1), (0.0, 2)])
def test_lane_pairs_give_the_one_lane_loops_bits(qdfn_mod, alpha, dr, high, dt):
    """Ordinary patches, patches far off balance, and operands that end in every
    exit of the loops: locked, negative and NaN velocities, zero and infinite ages."""
    x = _operands(513, 11 + high, high, dt)
    x[::5, 13] *= 300.0
    for k, (field, value) in enumerate([(3, 0.0), (3, -1e-9), (3, np.nan), (2, 0.0), (2, np.inf), (11, np.nan), (8, 1e14)]):
        x[k * 7::61, field] = value
    one, two = _solve(ONE_LANE + high, x, alpha, dr), _solve(PAIR + high, x, alpha, dr)
    for k in FIELDS:
        assert np.array_equal(one[k], two[k], equal_nan=True), (k, np.nonzero(one[k] != two[k])[0][:5])


@pytest.mark.parametrize("change", [dict(evolution_dr=2), dict(alpha_evo=0.2)])
@pytest.mark.parametrize("precision", ["fp32", "bf16x2"])
def test_step_loop_on_lane_pairs(qdfn_mod, loaded_network, precision, change):  # noqa: F811
    prob, Ks, Kn, ext = loaded_network
    net = (dict(prob, **change), Ks, Kn, ext)
    ref, cnt = _run(net, {"QDFN_PAIR_SOLVE": 0}, 200, 100, precision)
    assert cnt["highv_solves"] > 0, cnt
    for pair in (1, 2):
        _same(ref, _run(net, {"QDFN_PAIR_SOLVE": pair}, 200, 100, precision)[0])
