"""The kernels' own logarithm, exponential, reciprocals, square root, quotients
and conversions (friction_math.cuh, okada_sums.cuh) against CUDA's functions on
the same device, over every table interval and its edges, the ends of the stated
ranges and random arguments; and the tables against 60-digit values.

Bounds, with u = 2^-53 and CUDA's functions within 2 u of the value.  Logarithm:
the constant ln2 (2.3e-17 off), the table entry, its sum with k ln2 and the last
sum (u/2 of 0.69 or less each) on a result of at least 0.35 where k is not 0: 3 u;
the polynomial's FP32 part: five roundings to 2^-24 of r^4/4 <= 2^-34, below 2^-55;
against CUDA 5 u + 2^-55.  Exponential: the table entry and the last operation u/2
each, r 2^-53 of 2^-7.5, the FP32 part 2^-56 relative: 1.3 u; against CUDA 4 u.
Reciprocals: the last operation u/2 and e^3 < 2^-60, an ulp against IEEE division.
Corrected ones, quotients and the root differ from IEEE's by an ulp, and only
where the exact value lies within 2^-7 ulp of a rounding boundary or less: of
random arguments one in a thousand at most."""
import os
import re
from decimal import Decimal as D, getcontext

import numpy as np
import pytest

U = 2.0 ** -53
LOG, EXP, RCP, TO_FLOAT, FLOAT_TO, INT_TO, RECIP1, RECIP2, QUOTIENT, ROOT, RROOT = range(11)
OFF = 0x3fe6a09e    # upper word of the first interval's start


def _double(hi, lo=0):
    return ((np.asarray(hi, np.uint64) << np.uint64(32)) | np.asarray(lo, np.uint64)).view(np.float64)


def _near(x, ulps=2):
    b = np.asarray(x, np.float64).view(np.int64)
    return np.concatenate([(b + k).view(np.float64) for k in range(-ulps, ulps + 1)])


def _call(which, x, d=None):
    import torch
    from qdfn import _lib
    L = _lib.load()
    xt = torch.tensor(np.ascontiguousarray(x), dtype=torch.float64, device="cuda")
    dt = xt if d is None else torch.tensor(np.ascontiguousarray(d), dtype=torch.float64, device="cuda")
    y = torch.empty_like(xt)
    _lib.check(L.qdfn_check_math(which, xt.numel(), xt.data_ptr(), dt.data_ptr(), y.data_ptr(), None))
    return y.cpu().numpy(), xt, dt


def _log_arguments(lo, hi, n, seed):
    rng = np.random.default_rng(seed)
    edges = _near(_double(OFF + (np.arange(129) << 13)))       # interval edges of one octave
    centres = _double(OFF + (np.arange(128) << 13) + (1 << 12))
    octaves = np.concatenate([np.ldexp(np.concatenate([edges, centres]), k) for k in (-1000, -300, -83, -2, -1, 0, 1, 2, 93, 300, 1000)])
    ones = 1.0 + np.concatenate([s * 2.0 ** -np.arange(1, 53) for s in (1, -1)])
    x = np.concatenate([octaves, ones, [1.0, lo, hi], np.exp(rng.uniform(np.log(lo), np.log(hi), n)),
                        rng.uniform(0.98, 1.02, n)])
    return x[(x >= lo) & (x <= hi)]


@pytest.mark.gpu
def test_logarithm(qdfn_mod):
    import torch
    x = _log_arguments(np.finfo(float).tiny, np.finfo(float).max, 200000, 1)
    y, xt, _ = _call(LOG, x)
    ref = torch.log(xt).cpu().numpy()
    err = np.abs(y - ref) - (5 * U * np.abs(ref) + 2.0 ** -55)
    assert np.all(err <= 0), (x[np.argmax(err)], y[np.argmax(err)], ref[np.argmax(err)])


@pytest.mark.gpu
def test_exponential(qdfn_mod):
    import torch
    rng = np.random.default_rng(2)
    n = np.arange(-64600, 64601)
    x = np.concatenate([_near((n + 0.5) * (np.log(2.0) / 64), 1), n * (np.log(2.0) / 64), [0.0, 700.0, -700.0],
                        np.ldexp(1.0, -np.arange(1, 60)), -np.ldexp(1.0, -np.arange(1, 60)),
                        rng.uniform(-700, 700, 200000), rng.uniform(-1, 1, 100000)])
    x = x[np.abs(x) <= 700]
    y, xt, _ = _call(EXP, x)
    ref = torch.exp(xt).cpu().numpy()
    rel = np.abs(y / ref - 1)
    assert np.all(rel <= 4 * U), (x[np.argmax(rel)], rel.max() / U)


RANDOM = 300000   # the random ones of _positive, in front


def _positive(seed, lo, hi, n=RANDOM):
    rng = np.random.default_rng(seed)
    x = np.ldexp(rng.uniform(1, 2, n), rng.integers(lo, hi, n))
    edges = _near(np.ldexp(np.array([1.0, 1.5, np.nextafter(2.0, 0)])[:, None], np.arange(lo, hi)).ravel())
    return np.concatenate([x, edges])


def _ulps(a, b):
    return np.abs(a.view(np.int64) - b.view(np.int64))


@pytest.mark.gpu
@pytest.mark.parametrize("which,sign", [(RCP, 1), (RCP, -1), (RECIP1, 1), (RECIP2, 1), (RECIP2, -1)])
def test_reciprocals(qdfn_mod, which, sign):
    x = sign * _positive(3, -1000, 1000)
    y = _call(which, x)[0]
    off = _ulps(y, 1.0 / x)
    assert off.max() <= 1
    assert np.mean(off[:RANDOM] != 0) <= (1e-3 if which == RECIP2 else 0.05)


@pytest.mark.gpu
def test_quotients(qdfn_mod):
    rng = np.random.default_rng(4)
    d = _positive(4, -300, 300)
    x = np.ldexp(rng.uniform(-2, 2, d.size), rng.integers(-300, 300, d.size))
    x[:5] = 0.0
    y = _call(QUOTIENT, x, d)[0]
    off = _ulps(y, x / d)
    assert off.max() <= 1 and np.mean(off[:RANDOM] != 0) <= 1e-3


@pytest.mark.gpu
def test_square_root(qdfn_mod):
    x = np.concatenate([_positive(5, -400, 400), np.random.default_rng(5).uniform(0.25, 4, 200000) ** 2,
                        np.arange(1.0, 2000.0) ** 2])
    off = _ulps(_call(ROOT, x)[0], np.sqrt(x))
    assert off.max() <= 1 and np.mean(off[:RANDOM] != 0) <= 1e-3
    assert np.all(np.abs(_call(RROOT, x)[0] * np.sqrt(x) - 1) <= 4 * U)


@pytest.mark.gpu
def test_conversions(qdfn_mod):
    rng = np.random.default_rng(6)
    f = rng.integers(0x00800000, 0x7f000000, 200000).astype(np.uint32).view(np.float32)
    f = np.concatenate([f, -f, np.float32([0.0, -0.0, 2.0 ** -126, 1.0, -1.0, 2.0 ** 126])])
    half = (f.astype(np.float64).view(np.int64) | (1 << 28)).view(np.float64)   # halfway to the next FP32 number
    x = np.concatenate([f.astype(np.float64), _near(half, 1), rng.uniform(-1, 1, 200000),
                        np.ldexp(rng.uniform(1, 2, 1000), rng.integers(-300, -127, 1000))])
    y = _call(TO_FLOAT, x)[0]
    with np.errstate(under="ignore"):
        ref = x.astype(np.float32).astype(np.float64)
    tie = (x.view(np.int64) & 0x1fffffff) == 0x10000000
    away = ((x.view(np.int64) + 0x10000000) & ~np.int64(0x1fffffff)).view(np.float64)   # of a tie
    ref = np.where(tie, away, ref)
    ref = np.where(np.abs(x) < 2.0 ** -126, 0.0 * x, ref)
    assert np.array_equal(y, ref) and np.array_equal(np.signbit(y), np.signbit(ref))
    y = _call(FLOAT_TO, f.astype(np.float64))[0]
    assert np.array_equal(y, f.astype(np.float64)) and np.array_equal(np.signbit(y), np.signbit(f))
    k = np.concatenate([rng.integers(-2 ** 31, 2 ** 31, 100000), [0, 1, -1, 2 ** 31 - 1, -2 ** 31]]).astype(np.float64)
    assert np.array_equal(_call(INT_TO, k)[0], k)


def test_tables_are_the_60_digit_values():
    getcontext().prec = 60
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "quake-dfn_gb300", "csrc",
                        "friction_tables.cuh")
    text = open(path).read()
    pairs = [tuple(map(float.fromhex, m)) for m in re.findall(r"\{(-?0x\S+), (-?0x[^}]+)\}", text)]
    assert len(pairs) == 128
    for j, (c, t) in enumerate(pairs):
        lo, hi = OFF + (j << 13), OFF + ((j + 1) << 13)
        a, b = (float(v) for v in _double([lo, hi]))
        want = 1.0 if lo <= 0x3ff00000 < hi else float(1 / ((D(a) + D(b)) / 2))
        assert c == want and t == float(-D(c).ln())
        assert max(abs(a * c - 1), abs(b * c - 1)) <= 2.0 ** -8
    powers = [float.fromhex(v) for v in re.findall(r"0x\S+p[+-]\d+", text[text.index("kExpTab[64]"):])]
    assert powers == [float((D(2).ln() * D(j) / 64).exp()) for j in range(64)]
