"""The fast forms of the hot physics (csrc/mhd_fast.cuh), built for the host,
against the general ones: every value they vouch for is identical, bit for
bit, so no tolerance is involved.  The divisions and roots they are made of
are checked on the operands closest to a rounding boundary."""
from __future__ import annotations

import ctypes as C
import math
import subprocess
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent
CSRC = HERE.parent / "athena_cuda_b200" / "csrc"


@pytest.fixture(scope="module")
def fast(tmp_path_factory):
    so = tmp_path_factory.mktemp("fast") / "libfast_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-mfma", "-ffp-contract=off", "-frounding-math",
                    f"-I{CSRC}", "-o", str(so), str(HERE / "hostcheck" / "fast_host.cpp")], check=True)
    return C.CDLL(str(so))


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _ops(lib, op, x, y=None):
    x = np.ascontiguousarray(x, dtype=np.float64)
    y = np.ascontiguousarray(x if y is None else y, dtype=np.float64)
    f, g = np.empty_like(x), np.empty_like(x)
    lib.fast_ops(op, x.size, _p(x), _p(y), _p(f), _p(g))
    return f, g


def _hard_denominators():
    """Significands whose reciprocal, or a quotient by which, lies next to the
    middle of two doubles: near powers of two, and near 2^106 / M for
    midpoints M (the factors of 2^106 - k among them)."""
    D = {(1 << 53) - k for k in range(1, 600)} | {(1 << 52) + k for k in range(600)}
    rng = np.random.default_rng(5)
    for M in rng.integers(1 << 53, 1 << 54, 4000):
        D.add(min(max((1 << 106) // (int(M) | 1), 1 << 52), (1 << 53) - 1))
    for f in (3, 5, 7, 11, 107, 641, 6361, 69431):
        for k in range(1, 40):
            D.add((1 << 53) // f * 1 + k) if (1 << 52) <= (1 << 53) // f + k < (1 << 53) else None
    return np.array(sorted(D), dtype=np.float64)


def test_reciprocals_correctly_rounded(fast):
    d = _hard_denominators()
    d = np.concatenate([d * s for s in (1.0, 2.0 ** -52, 2.0 ** -500, 2.0 ** 447)])
    d = np.concatenate([d, 2.0 ** np.random.default_rng(1).uniform(-480, 480, 400000)])
    f, g = _ops(fast, 0, d)
    np.testing.assert_array_equal(f, g)


def test_quotients_correctly_rounded(fast):
    """a chosen so that a / d is as close to a midpoint as a 53-bit a allows:
    a 2^54 = +-k (mod d) for small k."""
    rng = np.random.default_rng(2)
    A, D = [], []
    dens = [int(x) | 1 for x in _hard_denominators()[::3]] + [int(x) | 1 for x in rng.integers(1 << 52, 1 << 53, 4000)]
    for d in dens:
        inv = pow(pow(2, 54, d), -1, d)
        for k in (1, -1, 2, -2, 3, -3):
            a = (k * inv) % d   # 2^54 a = k (mod d): a 2^54 / d is k/d off an integer
            while 0 < a < 1 << 52:
                a *= 2
            if 0 < a < 1 << 53:
                A.append(a)
                D.append(d)
    a, d = np.array(A, dtype=np.float64), np.array(D, dtype=np.float64)
    for sa, sd in ((1.0, 1.0), (2.0 ** -700, 2.0 ** 60), (2.0 ** 300, 2.0 ** -400)):
        f, g = _ops(fast, 2, d * sd, a * sa)
        np.testing.assert_array_equal(f, g)
    x = 2.0 ** rng.uniform(-200, 200, 400000)
    y = rng.choice([-1.0, 0.0, 1.0], x.size, p=[.45, .1, .45]) * 2.0 ** rng.uniform(-500, 200, x.size)
    f, g = _ops(fast, 2, x, y)
    np.testing.assert_array_equal(f, g)


def test_roots_correctly_rounded(fast):
    """x = m^2 -+ k 2^-106 for midpoints m: the roots nearest to a midpoint."""
    X = [float(1 + k * Fraction(1, 1 << 52)) for k in range(64)]
    X += [float(4 - k * Fraction(1, 1 << 51)) for k in range(64)]
    X += [float(2 - k * Fraction(1, 1 << 52)) for k in range(-64, 64)]
    rng = np.random.default_rng(3)
    for m in rng.integers(1 << 53, 1 << 54, 60000):
        m = int(m) | 1
        sq = m * m
        for shift in (54, 55):
            for a in (sq >> shift, (sq >> shift) + 1):
                if 1 << 52 <= a < 1 << 53:
                    X.append(math.ldexp(a, shift - 106))
    # m^2 = r (mod 2^54) with the smallest residues r
    for r in (1, 9, 17, 25, 33, 41, 49, (1 << 54) - 7, (1 << 54) - 15, (1 << 54) - 23, (1 << 54) - 31):
        s = 1
        for bit in range(3, 55):   # lift a square root of r modulo 2^bit
            if (s * s - r) % (1 << (bit + 1)):
                s += 1 << (bit - 1)
            if (s * s - r) % (1 << (bit + 1)):
                break
        for m in {s % (1 << 54), -s % (1 << 54), (s + (1 << 53)) % (1 << 54), (-s + (1 << 53)) % (1 << 54)}:
            m = m if m >= 1 << 53 else m + (1 << 53)
            for a in ((m * m) >> 54, ((m * m) >> 54) + 1):
                X.append(math.ldexp(a, -52) if a < 1 << 53 else math.ldexp(a // 2, -51))
    x = np.array(X)
    x = np.concatenate([x * 4.0 ** k for k in (0, -30, 200, -400)] + [2.0 ** rng.uniform(-900, 900, 400000), [0.0]])
    f, g = _ops(fast, 1, x)
    np.testing.assert_array_equal(f, g)
    f, g = _ops(fast, 3, x[x > 0])
    np.testing.assert_array_equal(f, g)


def _states(rng, n, kind):
    """n primitive states and normal fields: smooth O(1), strong jumps, exact
    zeros and equal components, or magnitudes spread over many decades."""
    w = np.empty((n, 7))
    w[:, 0] = np.exp(rng.normal(0, 1.0 if kind == "jumps" else 0.1, n))
    w[:, 4] = np.exp(rng.normal(0, 2.0 if kind == "jumps" else 0.1, n))
    w[:, 1:4] = rng.normal(0, 2.0 if kind == "jumps" else 0.7, (n, 3))
    w[:, 5:] = rng.normal(0, 1, (n, 2))
    bx = rng.normal(0, 1, n)
    if kind == "zeros":
        for c in (1, 2, 3, 5, 6):
            w[rng.random(n) < 0.4, c] = 0.0
        w[rng.random(n) < 0.5, 0] = 1.0 - 2.0 ** -53
        bx[rng.random(n) < 0.4] = 0.0
        bx[rng.random(n) < 0.1] = -0.0
    if kind == "wide":
        w *= 2.0 ** rng.uniform(-150, 30, (n, 7))
        w[rng.random((n, 7)) < 0.2] = 0.0
        w[:, 0], w[:, 4] = 2.0 ** rng.uniform(-40, 40, n), 2.0 ** rng.uniform(-60, 40, n)
        bx *= 2.0 ** rng.uniform(-158, 20, n)
    if kind == "extreme":
        w *= 2.0 ** rng.uniform(-1070, 500, (n, 7))
        w[:, 0], w[:, 4] = 2.0 ** rng.uniform(-150, 150, n), 2.0 ** rng.uniform(-150, 150, n)
        bx *= 2.0 ** rng.uniform(-1070, 200, n)
    if kind in ("edge", "still"):   # where a field fades out: all of it tiny, denormals included
        scale = 2.0 ** rng.uniform(-1072, -140, n)
        w[:, 5:] *= scale[:, None] * 2.0 ** rng.uniform(-30, 0, (n, 2))
        bx *= scale
        if kind == "still":         # in a uniform flow
            w[:, :5] = [1.0, 2.0, 1.0, 0.0, 1.0]
            w[:, 1] = rng.choice([2.0, 1.0, 0.0, -1.0], n)
    return w, bx


KINDS = ["smooth", "jumps", "zeros", "wide", "extreme", "edge", "still"]


@pytest.mark.parametrize("gamma", [5.0 / 3.0, 1.4, 2.5])
@pytest.mark.parametrize("kind", KINDS)
def test_plm_identical(fast, kind, gamma):
    n = 20000
    rng = np.random.default_rng(KINDS.index(kind))
    w0, b0 = _states(rng, 3 * n, kind)
    w, bx = w0.reshape(n, 3, 7), b0.reshape(n, 3)
    if kind in ("smooth", "zeros"):   # neighbours close, some components equal
        w[:, 1] = w[:, 0] * (1 + 1e-3 * rng.normal(size=(n, 7)))
        w[:, 2] = w[:, 1] * (1 + 1e-3 * rng.normal(size=(n, 7)))
        same = rng.random((n, 7)) < 0.2
        w[:, 2][same] = w[:, 1][same]
    w[rng.random(n) < 0.3, :, 1] += rng.choice([-8.0, 8.0])   # supersonic cells
    w, bx = np.ascontiguousarray(w), np.ascontiguousarray(bx)
    dtodx = np.ascontiguousarray(rng.uniform(0.05, 0.4, n))
    took = np.zeros(n, dtype=np.int32)
    f, g = np.empty((n, 14)), np.empty((n, 14))
    fast.fast_plm(n, _p(w), _p(bx), _p(dtodx), C.c_double(gamma), _p(took), _p(f), _p(g))
    ok = took.astype(bool)
    assert ok.mean() >= {"extreme": 0.0, "wide": 0.3, "edge": 0.8, "still": 0.8}.get(kind, 0.95)
    assert kind != "extreme" or not ok.all()
    np.testing.assert_array_equal(f[ok], g[ok])


@pytest.mark.parametrize("hlle", [0, 1])
@pytest.mark.parametrize("gamma", [5.0 / 3.0, 1.4, 2.5])
@pytest.mark.parametrize("kind", KINDS)
def test_flux_identical(fast, kind, gamma, hlle):
    n = 40000
    rng = np.random.default_rng(10 + KINDS.index(kind))
    w0, b0 = _states(rng, 2 * n, kind)
    w, bx = w0.reshape(n, 2, 7), np.ascontiguousarray(b0[:n])
    if kind in ("smooth", "zeros"):
        w[:, 1] = w[:, 0] * (1 + 10.0 ** rng.uniform(-16, -1, (n, 1)) * rng.normal(size=(n, 7)))
        same = rng.random((n, 7)) < 0.2
        w[:, 1][same] = w[:, 0][same]
    w[rng.random(n) < 0.2, :, 1] += rng.choice([-8.0, 8.0])
    w = np.ascontiguousarray(w)
    took = np.zeros(n, dtype=np.int32)
    f, g = np.empty((n, 7)), np.empty((n, 7))
    fast.fast_flux(hlle, n, _p(w), _p(bx), C.c_double(gamma), _p(took), _p(f), _p(g))
    ok = took.astype(bool)
    assert ok.mean() >= {"smooth": 0.99, "zeros": 0.9, "jumps": 0.5, "still": 0.7}.get(kind, 0.0)
    np.testing.assert_array_equal(f[ok], g[ok])


@pytest.mark.parametrize("kind", ["smooth", "jumps", "zeros"])
def test_plm_adjoint_agrees(fast, kind):
    """The adjoint's reverse is regrouped (fused multiply-adds, shared factors),
    so it agrees to rounding, not in bits: 23 outputs of ~1000 operations on
    terms up to 1/alpha times the result (alpha the smaller wave weight; 1e-3
    or more for all but 1 cell in 1000 here), hence 1000 eps / 1e-3 of the
    largest output, and no branch taken otherwise."""
    n = 20000
    rng = np.random.default_rng(20)
    w0, b0 = _states(rng, 3 * n, kind)
    w, bx = np.ascontiguousarray(w0.reshape(n, 3, 7)), np.ascontiguousarray(b0.reshape(n, 3))
    w[rng.random(n) < 0.3, :, 1] += rng.choice([-8.0, 8.0])
    dtodx, lam = rng.uniform(0.05, 0.4, n), rng.normal(size=(n, 14))
    took = np.zeros(n, dtype=np.int32)
    f, g = np.empty((n, 23)), np.empty((n, 23))
    fast.fast_plm_adj(n, _p(w), _p(bx), _p(dtodx), _p(lam), C.c_double(5.0 / 3.0), _p(took), _p(f), _p(g))
    ok = took.astype(bool)
    assert ok.mean() > 0.95
    err = np.abs(f - g)[ok].max(axis=1) / np.abs(g)[ok].max(axis=1)
    assert np.quantile(err, 0.999) <= 1000 * 2.0 ** -52 / 1e-3


@pytest.mark.parametrize("kind", ["smooth", "jumps", "zeros"])
def test_roe_adjoint_agrees(fast, kind):
    """The adjoint of the Roe flux, to rounding as above: ~1000 operations on
    terms up to 1/alpha (1e-3 or more for all but 1 face in 1000) times the
    largest output; subsonic faces of both signs, supersonic ones (the shift).
    It takes every face the fast flux takes (the others are the HLLE ones)."""
    n = 20000
    rng = np.random.default_rng(21)
    w0, b0 = _states(rng, 2 * n, kind)
    w, bx = np.ascontiguousarray(w0.reshape(n, 2, 7)), np.ascontiguousarray(b0[:n])
    w[rng.random(n) < 0.3, :, 1] += rng.choice([-8.0, 8.0])
    lam = rng.normal(size=(n, 7))
    took = np.zeros(n, dtype=np.int32)
    f, g = np.empty((n, 29)), np.empty((n, 29))
    fast.fast_roe_adj(n, _p(w), _p(bx), _p(lam), C.c_double(5.0 / 3.0), _p(took), _p(f), _p(g))
    ok = took.astype(bool)
    flux = np.zeros(n, dtype=np.int32)
    F, G = np.empty((n, 7)), np.empty((n, 7))
    fast.fast_flux(0, n, _p(w), _p(bx), C.c_double(5.0 / 3.0), _p(flux), _p(F), _p(G))
    assert ok.sum() > n // 4 and np.all(ok[flux.astype(bool)])
    err = np.abs(f - g)[ok].max(axis=1) / np.abs(g)[ok].max(axis=1)
    assert np.quantile(err, 0.999) <= 1000 * 2.0 ** -52 / 1e-3


def _fading(rng, n, sides, kind):
    """States where the field fades out (kind "edge" or "still"), every side of
    its own density, velocity and pressure, so that all jumps count."""
    w, b = _states(rng, sides * n, kind)
    w[:, 0] *= np.exp(0.1 * rng.normal(size=sides * n))
    w[:, 4] *= np.exp(0.1 * rng.normal(size=sides * n))
    w[:, 1:4] += 0.2 * rng.normal(size=(sides * n, 3))
    return np.ascontiguousarray(w.reshape(n, sides, 7)), b


def _worst(fast_values, general_values):
    return (np.abs(fast_values - general_values).max(axis=1) / np.abs(general_values).max(axis=1)).max()


# Fast and general adjoint of one face or cell where alpha_s = 0 (a field whose
# square does not show beside the pressure), so that nothing is divided by a small
# weight: ~1000 operations on terms no larger than the largest output.
FADING_TOL = 1000 * 2.0 ** -52


@pytest.mark.parametrize("kind", ["edge", "still"])
def test_roe_adjoint_where_fields_fade(fast, kind):
    """Wave speeds far below the flow speed do not show in the flux, but their
    derivatives do: every face the adjoint takes agrees with the general form."""
    n = 40000
    rng = np.random.default_rng(22)
    w, b = _fading(rng, n, 2, kind)
    bx, lam = np.ascontiguousarray(b[:n]), rng.normal(size=(n, 7))
    took = np.zeros(n, dtype=np.int32)
    f, g = np.empty((n, 29)), np.empty((n, 29))
    fast.fast_roe_adj(n, _p(w), _p(bx), _p(lam), C.c_double(5.0 / 3.0), _p(took), _p(f), _p(g))
    ok = took.astype(bool)
    assert ok.mean() > 0.5
    assert _worst(f[ok], g[ok]) <= FADING_TOL


def test_roe_adjoint_over_normal_fields(fast):
    """The normal field of one subsonic face from 1e-100 down to where it is zero."""
    bx = np.concatenate([10.0 ** np.linspace(-100, -170, 2801), [0.0]])
    bx = np.ascontiguousarray(np.concatenate([bx, -bx]))
    n = bx.size
    rng = np.random.default_rng(23)
    w = np.tile(np.array([[1.0, 0.5, 0.3, -0.2, 1.0, 0.0, 0.0], [1.1, 0.4, -0.1, 0.25, 0.9, 0.0, 0.0]]), (n, 1, 1))
    lam = rng.normal(size=(n, 7))
    took = np.zeros(n, dtype=np.int32)
    f, g = np.empty((n, 29)), np.empty((n, 29))
    fast.fast_roe_adj(n, _p(w), _p(bx), _p(lam), C.c_double(5.0 / 3.0), _p(took), _p(f), _p(g))
    ok = took.astype(bool)
    assert ok.mean() > 0.5
    assert _worst(f[ok], g[ok]) <= FADING_TOL


@pytest.mark.parametrize("kind", ["edge", "still"])
def test_plm_adjoint_where_fields_fade(fast, kind):
    n = 40000
    rng = np.random.default_rng(24)
    w, b = _fading(rng, n, 3, kind)
    bx = np.ascontiguousarray(b.reshape(n, 3))
    dtodx, lam = rng.uniform(0.05, 0.4, n), rng.normal(size=(n, 14))
    took = np.zeros(n, dtype=np.int32)
    f, g = np.empty((n, 23)), np.empty((n, 23))
    fast.fast_plm_adj(n, _p(w), _p(bx), _p(dtodx), _p(lam), C.c_double(5.0 / 3.0), _p(took), _p(f), _p(g))
    # the general form forms dl dr / (dl + dr) and has few bits of it where dl dr is denormal
    prod = np.abs((w[:, 1, 5:] - w[:, 0, 5:]) * (w[:, 2, 5:] - w[:, 1, 5:]))
    ok = took.astype(bool) & ~((prod > 0) & (prod < np.finfo(float).tiny)).any(axis=1)
    assert ok.mean() > 0.5
    assert _worst(f[ok], g[ok]) <= FADING_TOL


@pytest.mark.parametrize("spread", [1.0, 3.0, 8.0])
def test_roe_adjoint_branches_as_the_flux(fast, spread):
    """Faces on the path from a small jump to one that needs the HLLE fallback,
    bisected to the last pair of doubles where the flux still takes the fast
    form: the adjoint never goes on with Roe where the flux does not."""
    n = 20000
    rng = np.random.default_rng(int(spread))
    A = np.empty((n, 2, 7))
    A[:, :, 0], A[:, :, 4] = np.exp(spread * rng.normal(size=(2, n, 2)))
    A[:, :, 1:4], A[:, :, 5:] = 2.0 * rng.normal(size=(n, 2, 3)), rng.normal(size=(n, 2, 2))
    B = A.copy()
    B[:, 1] = B[:, 0] * (1 + 1e-3)
    bx, lam = rng.normal(size=n), np.ones((n, 7))

    def taken(t):
        t = t[:, None]
        w = (1 - t)[:, :, None] * B + t[:, :, None] * A
        for c in (0, 4):
            w[:, :, c] = np.exp((1 - t) * np.log(B[:, :, c]) + t * np.log(A[:, :, c]))
        w = np.ascontiguousarray(w)
        flux, adj = np.zeros((2, n), dtype=np.int32)
        f, g = np.empty((2, n, 29))
        fast.fast_flux(0, n, _p(w), _p(bx), C.c_double(5.0 / 3.0), _p(flux), _p(f), _p(g))
        fast.fast_roe_adj(n, _p(w), _p(bx), _p(lam), C.c_double(5.0 / 3.0), _p(adj), _p(f), _p(g))
        return flux.astype(bool), adj.astype(bool)

    lo, hi = np.zeros(n), np.ones(n)
    crossing = taken(lo)[0] & ~taken(hi)[0]
    assert crossing.sum() > n // 10
    for _ in range(54):
        mid = 0.5 * (lo + hi)
        flux, adj = taken(mid)
        assert not np.any(adj & ~flux)
        lo, hi = np.where(flux, mid, lo), np.where(flux, hi, mid)
    for k in range(-8, 9):
        flux, adj = taken(hi * (1 + k * 2.0 ** -52))
        assert not np.any(adj & ~flux)


@pytest.mark.parametrize("component,exponent", [(5, 0), (6, 0), (1, 115), (2, 115), (3, 115)])
def test_plm_slopes_of_denormal_size(fast, component, exponent):
    """The limiter's quotient 2 dl dr / (dl + dr) where it is a denormal: a jump of
    a few denormal ulps beside one of O(1) (of 2^115 where the fast form wants
    the product of the two above 2^-960), quotients on and next to a tie."""
    n = 40000
    rng = np.random.default_rng(30 + component)
    size = np.ldexp(rng.uniform(0.01, 1.0, n), exponent)
    size[::2] = np.ldexp(2.0 * rng.integers(1, 64, n // 2) / (rng.integers(1, 200, n // 2) + 0.5), exponent)
    w = np.zeros((n, 3, 7))
    w[:, :, 0], w[:, :, 4] = 2.0 ** -30, 1.0
    w[:, :, 1] = rng.choice([0.3, -0.2, 0.0], n)[:, None]
    w[:, :, component] = 0.0
    dl = np.ldexp(rng.integers(1 << 51 if exponent else 1, 1 << 52 if exponent else 2000, n).astype(float), -1074)
    if exponent == 0:   # such that 2 dl dr is a few denormal ulps
        dl[::2] = np.ldexp(np.round(rng.integers(1, 64, n // 2) / size[::2]), -1074)
    w[:, 0, component], w[:, 2, component] = -dl, size
    bx, dtodx = np.zeros((n, 3)), rng.uniform(0.05, 0.4, n)
    took = np.zeros(n, dtype=np.int32)
    f, g = np.empty((n, 14)), np.empty((n, 14))
    fast.fast_plm(n, _p(w), _p(bx), _p(dtodx), C.c_double(5.0 / 3.0), _p(took), _p(f), _p(g))
    ok = took.astype(bool)
    np.testing.assert_array_equal(f[ok], g[ok])


def test_operations_at_the_ends_of_their_ranges(fast):
    """Numerators and roots from 2^-960 on (the smallest the physics passes on as
    they are), denominators from 2^-540 (two jumps of a field whose product is
    not zero) to 2^500, and the root's by-product 1/(2 sqrt(x)), on which the
    adjoints rely: seeds of 20 bits and a cubic step leave 2.5 (2^-20)^3, and
    two roundings, below 2^-50."""
    rng = np.random.default_rng(40)
    n = 200000
    d = np.concatenate([2.0 ** rng.uniform(-540, -480, n), 2.0 ** rng.uniform(440, 500, n), 2.0 ** rng.uniform(-2, 2, n)])
    f, g = _ops(fast, 0, d)
    np.testing.assert_array_equal(f, g)
    a = rng.choice([-1.0, 1.0], 3 * n) * 2.0 ** np.concatenate([rng.uniform(-960, -870, 2 * n), rng.uniform(-960, 400, n)])
    # the quotient has to be normal
    ok = np.abs(np.log2(np.abs(a)) - np.log2(d)) < 1000
    f, g = _ops(fast, 2, d[ok], a[ok])
    np.testing.assert_array_equal(f, g)
    x = np.concatenate([2.0 ** rng.uniform(-960, -900, n), 2.0 ** rng.uniform(-60, 60, n), 2.0 ** rng.uniform(440, 950, n)])
    for op in (1, 3):
        f, g = _ops(fast, op, x)
        np.testing.assert_array_equal(f, g)
    f, g = _ops(fast, 4, x)
    assert np.max(np.abs(f / g - 1)) <= 2.0 ** -50


# 29 outputs of a face, 23 of a cell: fast and general adjoint differ by the
# rounding of ~1000 operations, each no worse than an ulp of some value on the
# way; what an ulp of the inputs changes in the general form says how much that
# is for each item, and no item is left out.
ITEM_TOL = 1000


def _every_item_agrees(adjoint, w, bx, lam, rng):
    took, f, g = adjoint(w, bx, lam)
    change = np.abs(g).max(axis=1) * 2.0 ** -52
    for _ in range(6):
        moved = [a * (1 + rng.choice([-1, 1], a.shape) * 2.0 ** -52) for a in (w, bx, lam)]
        again = adjoint(*(np.ascontiguousarray(a) for a in moved))[2]
        change = np.maximum(change, np.abs(again - g).max(axis=1))
    worst = np.abs(f - g).max(axis=1) / change
    assert took.mean() > 0.25
    assert worst[took].max() <= ITEM_TOL


@pytest.mark.parametrize("kind", ["smooth", "jumps", "zeros"])
def test_adjoints_agree_on_every_item(fast, kind):
    n = 20000
    rng = np.random.default_rng(50)
    dtodx, gamma = rng.uniform(0.05, 0.4, n), C.c_double(5.0 / 3.0)

    def roe(w, bx, lam):
        took, f, g = np.zeros(n, dtype=np.int32), np.empty((n, 29)), np.empty((n, 29))
        fast.fast_roe_adj(n, _p(w), _p(bx), _p(lam), gamma, _p(took), _p(f), _p(g))
        return took.astype(bool), f, g

    def plm(w, bx, lam):
        took, f, g = np.zeros(n, dtype=np.int32), np.empty((n, 23)), np.empty((n, 23))
        fast.fast_plm_adj(n, _p(w), _p(bx), _p(dtodx), _p(lam), gamma, _p(took), _p(f), _p(g))
        return took.astype(bool), f, g

    w, b = _states(rng, 2 * n, kind)
    _every_item_agrees(roe, np.ascontiguousarray(w.reshape(n, 2, 7)), np.ascontiguousarray(b[:n]),
                       rng.normal(size=(n, 7)), rng)
    w, b = _states(rng, 3 * n, kind)
    _every_item_agrees(plm, np.ascontiguousarray(w.reshape(n, 3, 7)), np.ascontiguousarray(b.reshape(n, 3)),
                       rng.normal(size=(n, 14)), rng)


def _faces(fast, hlle, w, bx, gamma=5.0 / 3.0):
    n = bx.size
    known, f, g = np.zeros(n, dtype=np.int32), np.empty((n, 7)), np.empty((n, 7))
    fast.fast_face(hlle, n, _p(w), _p(bx), C.c_double(gamma), _p(known), _p(f), _p(g))
    np.testing.assert_array_equal(f, g)
    return known.astype(bool)


@pytest.mark.parametrize("hlle", [0, 1])
@pytest.mark.parametrize("kind", KINDS)
def test_every_face_identical(fast, kind, hlle):
    """The flux of every face, whichever form it ends up in: fast, the HLLE
    fallback known to the fast Roe solver, or general."""
    n = 40000
    rng = np.random.default_rng(60 + KINDS.index(kind))
    w, b = _states(rng, 2 * n, kind)
    w = w.reshape(n, 2, 7)
    w[rng.random(n) < 0.2, :, 1] += rng.choice([-8.0, 8.0])
    known = _faces(fast, hlle, np.ascontiguousarray(w), np.ascontiguousarray(b[:n]))
    assert hlle or kind != "jumps" or known.mean() > 0.1


@pytest.mark.parametrize("spread", [1.0, 3.0, 8.0])
def test_fallback_known_only_where_taken(fast, spread):
    """Faces bisected to the last pair of doubles where the fallback is known."""
    n = 20000
    rng = np.random.default_rng(100 + int(spread))
    A = np.empty((n, 2, 7))
    A[:, :, 0], A[:, :, 4] = np.exp(spread * rng.normal(size=(2, n, 2)))
    A[:, :, 1:4], A[:, :, 5:] = 2.0 * rng.normal(size=(n, 2, 3)), rng.normal(size=(n, 2, 2))
    B = A.copy()
    B[:, 1] = B[:, 0] * (1 + 1e-3)
    bx = rng.normal(size=n)

    def known(t):
        w = (1 - t)[:, None, None] * B + t[:, None, None] * A
        for c in (0, 4):
            w[:, :, c] = np.exp((1 - t)[:, None] * np.log(B[:, :, c]) + t[:, None] * np.log(A[:, :, c]))
        return _faces(fast, 0, np.ascontiguousarray(w), bx)

    lo, hi = np.zeros(n), np.ones(n)
    assert (known(hi) & ~known(lo)).sum() > n // 20
    for _ in range(54):
        mid = 0.5 * (lo + hi)
        k = known(mid)
        lo, hi = np.where(k, lo, mid), np.where(k, mid, hi)
    for k in range(-8, 9):
        known(hi * (1 + k * 2.0 ** -52))


def test_adjoints_where_sound_and_alfven_speed_agree(fast):
    """The discriminant of the wave speeds is then the transverse field's alone:
    its root from O(1) down to denormals and zero, against the general forms."""
    n = 4000
    rng = np.random.default_rng(70)
    t = 10.0 ** np.linspace(-100, -170, n)
    gamma, lam = 1.5, rng.normal(size=(n, 14))
    w = np.zeros((n, 3, 7))
    w[:, 0, :5], w[:, 2, :5] = [0.9, 0.2, 0.1, -0.1, 5.5], [1.2, 0.45, -0.2, 0.3, 6.6]
    w[:, 1, :5] = [1.0, 0.25, 0.05, 0.02, 6.0]                          # a^2 = gamma p / d = 9
    w[:, :, 5], w[:, :, 6] = t[:, None], 0.5 * t[:, None]
    bx, dtodx = np.full((n, 3), 3.0), np.full(n, 0.2)                   # v_A^2 = 9
    took = np.zeros(n, dtype=np.int32)
    f, g = np.empty((n, 23)), np.empty((n, 23))
    fast.fast_plm_adj(n, _p(w), _p(bx), _p(dtodx), _p(lam), C.c_double(gamma), _p(took), _p(f), _p(g))
    ok = took.astype(bool)
    assert ok.mean() > 0.25
    assert _worst(f[ok], g[ok]) <= FADING_TOL
    w = np.zeros((n, 2, 7))
    w[:, :, :5] = [1.0, 0.25, 0.5, -0.5, 6.0]
    w[:, 1, 2:4] += [0.25, -0.5]
    w[:, :, 5], w[:, :, 6] = t[:, None] * [0.8, 1.0], 0.5 * t[:, None] * [1.1, 1.0]
    bx, lam = np.full(n, 3.0), np.ascontiguousarray(lam[:, :7])
    f, g = np.empty((n, 29)), np.empty((n, 29))
    fast.fast_roe_adj(n, _p(w), _p(bx), _p(lam), C.c_double(gamma), _p(took), _p(f), _p(g))
    ok = took.astype(bool)
    assert ok.mean() > 0.25
    assert _worst(f[ok], g[ok]) <= FADING_TOL


@pytest.mark.parametrize("side", [-1, 1])
def test_identical_at_the_edge_of_the_densities(fast, side):
    """States in units that put the density at 2^-120 or 2^120, where the fast
    forms end: what they take is the general forms', and they take most of it."""
    n = 30000
    rng = np.random.default_rng(80 + side)
    d0, p0 = 2.0 ** (side * rng.uniform(100, 122, n)), 2.0 ** rng.uniform(-100, 100, n)
    v0, b0 = np.sqrt(p0 / d0) * 2.0 ** rng.uniform(-6, 6, n), np.sqrt(p0) * 2.0 ** rng.choice([-400, -60, -3, 0, 3], n)

    def states(sides):
        r = rng.normal(size=(n, 1, 7)) + 10.0 ** rng.uniform(-12, 0, (n, 1, 1)) * rng.normal(size=(n, sides, 7))
        w = np.empty((n, sides, 7))
        w[:, :, 0], w[:, :, 4] = d0[:, None] * np.exp(0.3 * r[:, :, 0]), p0[:, None] * np.exp(0.3 * r[:, :, 4])
        w[:, :, 1:4], w[:, :, 5:] = v0[:, None, None] * r[:, :, 1:4], b0[:, None, None] * r[:, :, 5:]
        w[rng.random(n) < 0.2, :, 2] = 0.0
        return np.ascontiguousarray(w)

    w, bx, dtodx = states(3), b0[:, None] * rng.normal(size=(n, 3)), 2.0 ** rng.uniform(-8, 0, n)
    took = np.zeros(n, dtype=np.int32)
    f, g = np.empty((n, 14)), np.empty((n, 14))
    fast.fast_plm(n, _p(w), _p(bx), _p(dtodx), C.c_double(5.0 / 3.0), _p(took), _p(f), _p(g))
    ok = took.astype(bool)
    inside = np.abs(np.log2(w[:, :, 0])).max(axis=1) < 120
    assert ok[inside].mean() > 0.9 and not ok[np.abs(np.log2(w[:, 1, 0])) > 120.01].any()
    np.testing.assert_array_equal(f[ok], g[ok])
    _faces(fast, 0, states(2), np.ascontiguousarray(bx[:, 0]))
    _faces(fast, 1, states(2), np.ascontiguousarray(bx[:, 0]))
