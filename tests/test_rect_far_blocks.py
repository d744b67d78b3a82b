"""Rectangle stiffness of whole blocks against the published formulas term by
term (qdfn_check_rect, on the same device): steep and nearly vertical sources,
where the formulas multiply rounding by 1/cos^2(dip); receivers along and down a
source's own plane, by R/(R + xi) and R/(R + eta); ordinary and shallow dips;
blocks from next to the source to 60 patch lengths away.  A block is used by
itself (an H-matrix leaf), so its own size is the scale, and Ks and Kn have one
each.

Tolerance: a corner term is rounded about ten times to 2^-53 of itself, and what
is left of the amplification is at most 64: 7e-14.  At 60 patch lengths the four
corners cancel to (1/60)^2 of it: 2.6e-10 of an entry.  1e-9 of the block's
2-norm holds four times that; where the source's plane is the receivers', Kn
falls short of Ks by up to 1e-3, and Ks is its scale."""
import numpy as np
import pytest

from _systems import cols

pytestmark = pytest.mark.gpu
G, NU = 32e9, 0.25
TOL = 1e-9
DIPS = [90.0, 89.9998, 89.99, 89.9, 89.67, 89.0, 87.0, 85.0, 84.0, 96.0, 91.0, 75.0, 60.0, 30.0, 5.0, 110.0, 179.5]


def _fault(centre, strike, dip, rake, n=(7, 8), patch=100.0):
    from qdfn import synth
    return synth.grid_fault(*centre, n[0] * patch, n[1] * patch, strike, dip, rake, patch)


def _general(src, recv, layout):
    import torch
    from qdfn import _lib
    L = _lib.load()
    s, r = (torch.tensor(np.ascontiguousarray(x), device="cuda") for x in (src, recv))
    shape = (len(src), len(recv)) if layout == "col" else (len(recv), len(src))
    Ks, Kn = (torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(2))
    _lib.check(L.qdfn_check_rect(len(src), s.data_ptr(), len(recv), r.data_ptr(), G, NU, Ks.data_ptr(), Kn.data_ptr(),
                                 shape[1], _lib.LAYOUT_COL if layout == "col" else _lib.LAYOUT_ROW, None))
    K = [k.cpu().numpy() for k in (Ks, Kn)]
    return [k.T for k in K] if layout == "col" else K


def _check(src, recv, layout="row", same_plane=False):
    from qdfn import assemble
    got = assemble.assemble_rect(src, recv, G, NU, layout=layout)
    ref = _general(src, recv, layout)
    size = [np.linalg.norm(k) for k in ref]
    if same_plane:
        size = [max(size)] * 2
    for name, a, b, n in zip(("Ks", "Kn"), got, ref, size):
        assert np.all(np.isfinite(b))
        assert np.linalg.norm(a - b) <= TOL * n, (name, np.linalg.norm(a - b) / n)


@pytest.mark.parametrize("dip", DIPS)
def test_blocks_of_other_faults(qdfn_mod, dip):
    rng = np.random.default_rng(int(1e4 * dip))
    src = _fault((0.0, 0.0, 5000.0), rng.uniform(0, 180), dip, rng.uniform(-180, 180))
    for k, dist in enumerate((900.0, 2500.0, 6000.0)):
        az = rng.uniform(0, 2 * np.pi)
        recv = _fault((dist * np.cos(az), dist * np.sin(az), rng.uniform(1500, 6000)), rng.uniform(0, 180),
                      rng.uniform(60, 90), rng.uniform(-180, 180), n=(9, 4 + 3 * k))
        _check(src, recv, "col" if k % 2 else "row")


@pytest.mark.parametrize("dip", DIPS)
def test_blocks_in_the_sources_plane(qdfn_mod, dip):
    rng = np.random.default_rng(int(1e4 * dip) + 1)
    strike, rake = rng.uniform(0, 180), rng.uniform(-180, 180)
    src = _fault((0.0, 0.0, 5000.0), strike, dip, rake)
    along = np.array([np.sin(np.radians(strike)), np.cos(np.radians(strike))])
    for dist in (800.0, 2600.0, 6000.0):
        recv = src.copy()
        recv[:, :2] += dist * along
        _check(src, recv, same_plane=True)
        # down the plane: strike's right-hand side, and deeper
        down = src.copy()
        down[:, :2] += 0.4 * dist * np.cos(np.radians(dip)) * np.array([along[1], -along[0]])
        down[:, 2] += 0.4 * dist * np.sin(np.radians(dip))
        _check(src, down, same_plane=True)


def test_published_formulas_are_the_oracles(qdfn_mod, oracle_mod):
    """qdfn_check_rect against the oracle, on near blocks, where the formulas'
    rounding is small beside an entry (1e-12 of the block's largest)."""
    import oracle
    src = _fault((0.0, 0.0, 3000.0), 30.0, 70.0, 20.0)
    recv = _fault((300.0, 500.0, 3000.0), 75.0, 60.0, 20.0)
    for a, b in zip(_general(src, recv, "row"), oracle.assemble_rect(cols(src), cols(recv), G, NU)):
        assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
