"""The sm_100a step against the oracle restatement (oracle/mhd_oracle.cpp),
bit for bit, on states chosen for the branches of the fast physics: operands
inside and outside its ranges, faces that need the HLLE fallback or its
tests, supersonic faces, field-free and uniform regions, and grids at the
edges of the kernels' row segments and column marches."""
from __future__ import annotations

import numpy as np
import pytest

import oracle_cpu
import refutil
from athena_cuda_b200 import PLANES, Batch, Config, Grid

pytestmark = pytest.mark.gpu

NG = 4


def _state(kind: str, nx1: int, nx2: int, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    if kind in ("smooth", "noise"):
        return refutil.random_state(rng, nx1, nx2, kind == "smooth")
    S = np.zeros((11, nx2 + 2 * NG, nx1 + 2 * NG))
    i = S[:, NG:-NG, NG:-NG]
    shape = (nx2, nx1)
    x, y = np.meshgrid((np.arange(nx1) + 0.5) / nx1, (np.arange(nx2) + 0.5) / nx2)
    rho, p, v, A = np.ones(shape), np.ones(shape), np.zeros((3, *shape)), np.zeros((nx2 + 1, nx1 + 1))
    X, Y = np.meshgrid(np.arange(nx1 + 1) / nx1, np.arange(nx2 + 1) / nx2)
    b3 = np.zeros(shape)
    if kind == "strong":       # jumps that leave negative intermediate states
        rho, p = np.exp(rng.normal(0, 0.7, shape)), np.exp(rng.normal(0, 1.2, shape))
        v, A, b3 = rng.normal(0, 0.9, (3, *shape)), 0.01 * rng.normal(0, 1, X.shape), 0.3 * rng.normal(0, 1, shape)
    elif kind == "supersonic":
        v[0], v[1] = 6.0, -5.0 + 0.1 * rng.normal(0, 1, shape)
        A = 1e-3 * np.maximum(0.3 - np.hypot(X - 0.5, Y - 0.5), 0.0)
    elif kind == "fringe":     # fields that fall to denormals beside exact zeros
        A = 1e-3 * np.exp(-(np.hypot(X - 0.5, Y - 0.5) / 0.012) ** 2)
        v[0], v[1], v[2] = 1.0, 0.5, 1e-200 * rng.normal(0, 1, shape)
    elif kind == "tiny":       # densities close to the end of the fast ranges
        rho, p = 1e-35 * np.exp(rng.normal(0, 0.2, shape)), 1e-15 * np.exp(rng.normal(0, 0.2, shape))
        v = 1e9 * rng.normal(0, 1, (3, *shape))
    elif kind == "cgs":        # small but ordinary units
        rho, p = 1e-24 * np.exp(rng.normal(0, 0.3, shape)), 1e-12 * np.exp(rng.normal(0, 0.3, shape))
        v, b3 = 1e6 * rng.normal(0, 1, (3, *shape)), 1e-6 * rng.normal(0, 1, shape)
        A = 1e-8 * rng.normal(0, 1, X.shape)
    S[8, NG:NG + nx2, NG:NG + nx1 + 1] = (A[1:] - A[:-1]) * nx2
    S[9, NG:NG + nx2 + 1, NG:NG + nx1] = -(A[:, 1:] - A[:, :-1]) * nx1
    i[5] = 0.5 * (S[8, NG:NG + nx2, NG:NG + nx1] + S[8, NG:NG + nx2, NG + 1:NG + nx1 + 1])
    i[6] = 0.5 * (S[9, NG:NG + nx2, NG:NG + nx1] + S[9, NG + 1:NG + nx2 + 1, NG:NG + nx1])
    i[7], i[10] = b3, b3
    i[0], i[1], i[2], i[3] = rho, rho * v[0], rho * v[1], rho * v[2]
    i[4] = p / (5.0 / 3.0 - 1.0) + 0.5 * rho * (v ** 2).sum(0) + 0.5 * (i[5] ** 2 + i[6] ** 2 + i[7] ** 2)
    return S


def _config(nx1, nx2, bc, flux, gamma=1.6666666666666667):
    return Config(nx1=nx1, nx2=nx2, x1min=0.0, x1max=1.0, x2min=0.0, x2max=nx2 / nx1, bc_ix1=bc[0], bc_ox1=bc[1],
                  bc_ix2=bc[2], bc_ox2=bc[3], gamma=gamma, cour_no=0.8, tlim=1e30, nlim=-1, flux=flux, device=0)


def _oracle(cfg, S, bc, flux, steps):
    return oracle_cpu.run(S, 1.0 / cfg.nx1, (cfg.nx2 / cfg.nx1) / cfg.nx2, bc, cfg.gamma, 0.8, 1e30, flux=flux,
                          max_steps=steps)


def _check(ref, got):
    assert refutil.mismatch_report(ref[0], got[0], PLANES) == ""
    assert ref[1:] == got[1:]


@pytest.mark.parametrize("flux", [0, 1])
@pytest.mark.parametrize("kind", ["smooth", "noise", "strong", "supersonic", "fringe", "tiny", "cgs"])
def test_states_bit_exact(kind, flux):
    bc = (4, 4, 4, 4)
    cfg = _config(72, 50, bc, flux)
    S = _state(kind, 72, 50, 7)
    g = Grid.create(cfg)
    g.upload(S)
    g.set_bvals()
    g.new_dt()
    for _ in range(4):
        g.run_async(1)
    _check(_oracle(cfg, S, bc, flux, 4), g.download())


# widths around the 31 faces of a row segment, heights around a column march,
# the smallest grid, and sizes that leave partial blocks
@pytest.mark.parametrize("size", [(4, 4), (5, 33), (27, 6), (28, 9), (29, 31), (59, 40), (61, 13), (130, 5), (200, 3 + 64)])
@pytest.mark.parametrize("bc", [(4, 4, 4, 4), (1, 2, 2, 1)])
def test_sizes_bit_exact(size, bc):
    cfg = _config(*size, bc, 0)
    S = _state("smooth", *size, 11)
    g = Grid.create(cfg)
    g.upload(S)
    g.set_bvals()
    g.new_dt()
    g.run_async(3)
    _check(_oracle(cfg, S, bc, 0, 3), g.download())


@pytest.mark.parametrize("threads", [64, 128, 256])
def test_batch_bit_exact(threads):
    bc = (4, 4, 4, 4)
    sizes = [(40, 33), (64, 20), (33, 95)]
    kinds = ["strong", "fringe", "supersonic"]
    cfgs = [_config(*s, bc, 0) for s in sizes]
    states = [_state(k, *s, 3) for k, s in zip(kinds, sizes)]
    b = Batch(cfgs)
    b.threads = threads
    for k, S in enumerate(states):
        b.upload(k, S)
    b.prepare()
    b.run_async(3)
    b.synchronize()
    for k, (cfg, S) in enumerate(zip(cfgs, states)):
        _check(_oracle(cfg, S, bc, 0, 3), b.download(k))


@pytest.mark.parametrize("flux", [0, 1])
@pytest.mark.parametrize("unit", [2.0 ** -10, 2.0 ** 235])
def test_densities_outside_the_ranges_bit_exact(unit, flux):
    """The density of "tiny" (1e-35, 2^-116) in other units: below 2^-120 and
    just short of 2^120, on both sides of it."""
    bc = (4, 4, 4, 4)
    cfg = _config(72, 50, bc, flux)
    S = _state("tiny", 72, 50, 7)
    S[[0, 1, 2, 3, 4]] *= unit
    g = Grid.create(cfg)
    g.upload(S)
    g.set_bvals()
    g.new_dt()
    g.run_async(4)
    _check(_oracle(cfg, S, bc, flux, 4), g.download())
