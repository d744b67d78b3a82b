"""H-matrix products at the edges of the warp tasks: source ranges around the
batch lengths, ranks around the rows of a task, receiver ranges around the
64-row slices, and a matrix without low-rank blocks."""
import numpy as np
import pytest

from _systems import problem_for, small_network


def _system(low_rank, seed=0):
    from qdfn import hmatrix
    rng = np.random.default_rng(seed)
    rec = small_network(seed=5, n_faults=8, patch=100.0)["records"]
    N = rec.shape[0]
    ranges, dense, U, Vt = [], [], [], []
    for i in range(0, N, 40):   # diagonal blocks, the last one short
        e = min(i + 40, N)
        B = 1e6 * rng.normal(size=(e - i, e - i)) - 1e8 * np.eye(e - i)
        ranges.append((i, e - 1, i, e - 1)); dense.append(B); U.append(None); Vt.append(None)
    if low_rank:
        for k, ns in enumerate((1, 33, 64, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, N)):
            ns = min(ns, N)
            for rank in (0, 1, 2, 3, 4, 7, 8, 9):
                nr = (1, 32, 33, 63, 64, 65, 129)[(k + rank) % 7]
                r0 = (37 * k + 91 * rank) % (N - nr)
                ranges.append((N - ns, N - 1, r0, r0 + nr - 1))
                dense.append(None); U.append(1e3 * rng.normal(size=(nr, rank))); Vt.append(rng.normal(size=(rank, ns)))
    ranges = np.array(ranges, dtype=np.int64)
    H = hmatrix.HMatrix(ranges, dense, U, Vt, dense, U, Vt, None)
    return rec, H


@pytest.mark.gpu
@pytest.mark.parametrize("low_rank", [True, False])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("R", [1, 2, 4])
def test_products_at_the_edges_of_the_tasks(qdfn_mod, oracle_mod, R, precision, low_rank):
    """Against the oracle's product of the same blocks: 1e-12 in FP64, and FP32's
    rounding of entries, x and sums (64 terms of 2^-24 at most) otherwise."""
    from qdfn import hmatrix, simulate
    rec, H = _system(low_rank)
    N = rec.shape[0]
    assert N > 1025
    K = np.zeros((N, N))
    np.fill_diagonal(K, -1e8)
    prob = problem_for(rec, -K)
    prob["interp_at_told"] = 1
    p = dict(prob)
    for k in ("a", "b", "Dc", "theta_i", "V_i", "f_i", "sigma0", "V_const", "mass"):
        p[k] = np.tile(prob[k], R)
    sim = simulate.Simulation(p, n_inst=R)
    hmatrix.set_hmatrix(sim, H, precision)
    D = np.random.default_rng(4).uniform(0, 1, (R, N))
    tld, knd = sim.apply(D.ravel() if R > 1 else D[0])
    blocks = dict(range=H.ranges, sD=H.dense_s, sU=H.U_s, sVt=H.Vt_s, nD=H.dense_n, nU=H.U_n, nVt=H.Vt_n)
    o = oracle_mod.Simulation(dict(prob), ("hmat", blocks))
    tol = 1e-12 if precision == "fp64" else 64 * 2.0 ** -24
    for r in range(R):
        otld, oknd = o.apply(D[r])
        assert np.max(np.abs(tld[r] - otld)) <= tol * np.max(np.abs(otld))
        assert np.max(np.abs(knd[r] - oknd)) <= tol * np.max(np.abs(oknd))
    sim.close()
