"""Triangle stiffness against the oracle at the edges of the kernel's tiling (one
thread per receiver in blocks of 128, 1-8 sources a turn), both layouts, as
gathered pairs, and for the triangles whose local axes are special: horizontal
ones, one in the free surface, one with a vertical side, and receivers in a
triangle's plane inside, outside and on its edges (NaN there).

Tolerance: an ulp in one angle of the source moves an entry by up to 3e-10 of
the largest entry (the floor of any two libms' agreement); 1e-9 of it here."""
import numpy as np
import pytest

from _systems import bumpy_triangles

pytestmark = pytest.mark.gpu
G, NU = 32e9, 0.25


def _mesh(n, seed, shift):
    from qdfn import geometry
    rng = np.random.default_rng(seed)
    seg = bumpy_triangles(9, 8, seed=seed)
    seg = seg[rng.integers(0, len(seg), n)].copy()
    d = np.column_stack([rng.uniform(-3e3, 3e3, n), rng.uniform(-3e3, 3e3, n) + shift, -rng.uniform(0, 2e3, n)])
    for k in (0, 3, 6):
        seg[:, k:k + 3] += d
    seg[:, 9] = rng.uniform(-180, 180, n)
    P1, P2, P3, un, _, _, us = geometry.rot_verts_unit_vectors(seg, seg[:, 9])
    return P1, P2, P3, seg[:, 9].copy(), (P1 + P2 + P3) / 3, un, us


def _check(A, B, scale):
    assert A.shape == B.shape
    assert np.array_equal(np.isnan(A), np.isnan(B))
    m = ~np.isnan(B)
    assert np.max(np.abs(A - B)[m], initial=0.0) <= 1e-9 * scale


def _compare(src, recv, layout):
    import oracle
    from qdfn import assemble
    args = (*src[:4], *recv[4:], G, NU)
    Ks, Kn = assemble.assemble_tri(*args, layout=layout)
    Ks_o, Kn_o = oracle.assemble_tri(*args)
    scale = max(np.nanmax(np.abs(Ks_o)), np.nanmax(np.abs(Kn_o)))
    _check(Ks, Ks_o, scale)
    _check(Kn, Kn_o, scale)
    return Ks_o, Kn_o, scale


@pytest.mark.parametrize("layout", ["row", "col"])
@pytest.mark.parametrize("ns,nr", [(1, 1), (3, 128), (8, 129), (9, 127), (700, 130)])
def test_tile_edges_and_gathered_pairs(qdfn_mod, oracle_mod, ns, nr, layout):
    import torch
    from qdfn import assemble
    src, recv = _mesh(ns, 3, 0.0), _mesh(nr, 4, 900.0)
    Ks_o, Kn_o, scale = _compare(src, recv, layout)
    if layout == "row":   # the same entries from an index list over both meshes' triangles
        dv = [torch.tensor(np.concatenate([a, b]), device="cuda") for a, b in zip(src, recv)]
        n = min(ns * nr, 5000) - 1 if ns * nr > 1 else 1
        pick = np.random.default_rng(1).integers(0, ns * nr, n)
        r, s = pick // ns, pick % ns
        a, b = assemble.assemble_tri_pairs_dev(torch.tensor(r + ns, device="cuda"), torch.tensor(s, device="cuda"),
                                               *dv, G, NU)
        _check(a.cpu().numpy(), Ks_o[r, s], scale)
        _check(b.cpu().numpy(), Kn_o[r, s], scale)


def test_special_axes_and_points_in_the_plane(qdfn_mod, oracle_mod):
    tri = np.array([
        [[0, 0, -1000], [400, 0, -1000], [0, 300, -1000]],        # horizontal
        [[0, 0, -1000], [0, 300, -1000], [400, 0, -1000]],        # horizontal, other sense
        [[0, 0, 0], [400, 0, 0], [0, 300, 0]],                    # in the free surface
        [[0, 0, -500], [0, 0, -900], [350, 100, -700]],           # a vertical side
        [[100, 0, -600], [500, 0, -600], [300, 0, -950]],         # vertical, a horizontal side
    ], dtype=float)
    src = (tri[:, 0].copy(), tri[:, 1].copy(), tri[:, 2].copy(), np.array([0.0, 30.0, 60.0, 90.0, -45.0]))
    w = np.array([[1, 1, 1], [3, 1, 0.5], [-1, 2, 2], [2, -1, 2], [2, 2, -1], [1, 1, 0], [5, -1, -1.5]], dtype=float)
    w /= w.sum(axis=1, keepdims=True)
    X = np.concatenate([w @ t for t in tri] + [np.array([[250.0, 700.0, -300.0], [-800.0, 90.0, -2500.0]])])
    X = X[X[:, 2] <= 0]
    rng = np.random.default_rng(2)
    n = rng.standard_normal((len(X), 3))
    n /= np.linalg.norm(n, axis=1, keepdims=True)
    v = np.cross(n, rng.standard_normal((len(X), 3)))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    recv = (None, None, None, None, X, n, v)
    _compare(src, recv, "row")
