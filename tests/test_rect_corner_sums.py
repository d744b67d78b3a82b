"""Rectangle stiffness by corner sums against the oracle, at the edges of the
kernel's tiling (one thread per receiver in blocks of 128, 1-8 sources a turn),
both layouts, vertical (cos dip = 0), shallow and ordinary dips, and with
receivers on the extensions of a source's edges, where the kernel evaluates
the general formulas.

Tolerance: each corner term is of the order of the self stiffness G / L and is
rounded to 2^-53 of itself times R / (R + xi), up to a few hundred for the
distances here; both sides share R + xi to the last bit, so 1e-11 G / L holds a
margin of ten over the 1e-12 of that estimate."""
import numpy as np
import pytest

from _systems import cols, mixed_rects

pytestmark = pytest.mark.gpu
G, NU = 32e9, 0.25


def _records(n, seed):
    rng = np.random.default_rng(seed)
    base = mixed_rects()
    rec = base[rng.integers(0, len(base), n)].copy()
    rec[:, 0] += rng.uniform(-6000, 6000, n)
    rec[:, 1] += rng.uniform(-6000, 6000, n)
    rec[:, 2] += rng.uniform(600, 3000, n)
    rec[:, 6] = np.where(rng.random(n) < 0.3, 90.0, rng.uniform(5, 89, n))
    rec[:, 7] = rng.uniform(-180, 180, n)
    return rec


def _check(src, recv, layout):
    from qdfn import assemble
    import oracle
    Ks, Kn = assemble.assemble_rect(src, recv, G, NU, layout=layout)
    Ks_o, Kn_o = oracle.assemble_rect(cols(src), cols(recv), G, NU)
    tol = 1e-11 * G / np.min(src[:, 3:5])
    for A, B in ((Ks, Ks_o), (Kn, Kn_o)):
        assert A.shape == B.shape == (len(recv), len(src))
        assert np.array_equal(np.isfinite(A), np.isfinite(B))
        m = np.isfinite(B)
        assert np.max(np.abs(A - B)[m], initial=0.0) <= tol


@pytest.mark.parametrize("layout", ["row", "col"])
@pytest.mark.parametrize("ns,nr", [(1, 1), (7, 128), (8, 129), (9, 127), (61, 64), (1300, 257), (2500, 130)])
def test_tile_edges(qdfn_mod, oracle_mod, ns, nr, layout):
    _check(_records(ns, ns + 1), _records(nr, 1000 + nr), layout)


def test_receivers_on_the_extensions_of_edges(qdfn_mod, oracle_mod):
    """Receivers in a vertical source's plane, level with its upper edge or
    below its end, at both sides (R + xi or R + eta rounds to zero there), and
    within and just outside the 1e-6 m that DCCON2 zeroes."""
    src = np.array([[0.0, 0.0, 2000.0, 400.0, 300.0, 0.0, 90.0, 30.0]])
    recv = []
    for along in (-5000.0, -700.0, 900.0, 4000.0):
        for off in (0.0, 5e-7, 3e-6, 1e-3):
            recv.append([along, off, 1850.0, 100.0, 100.0, 0.0, 90.0, 0.0])
            recv.append([200.0 + off, 0.0, 2000.0 + along / 4, 100.0, 100.0, 0.0, 90.0, 0.0])
    _check(src, np.array(recv), "row")
