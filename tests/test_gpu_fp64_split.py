"""pairFP64Split (csrc/pair_fp64.cu) on plans that take it -- the context's plan line says so -- against sums in
extended precision.

A pair's velocity term x cross y s, s = W / (1 - x.y + eps^2), is off by at most
  2^-45 of itself                       the split's operations, about 2^-48 each,
  2^-50 (1 + |x|) / |1 - x.y + eps^2|   the rounding of 1 - x.y in the reference's operations, and
  2^-51 (1 + |x|) |s|                   that of the cross product;
the bound of a target is the sum over its pairs.
"""
import re

import numpy as np
import pytest
import torch

import lpmkokkos_gb300 as P
from lpmkokkos_gb300 import bve

pytestmark = pytest.mark.gpu
L = np.longdouble


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _unit(x):
    return x / np.linalg.norm(x, axis=1, keepdims=True)


def _split_items(capfd):
    """Work items that the last plan gave pairFP64Split."""
    return int(re.findall(r"split=(\d+)", capfd.readouterr().err)[-1])


def _cube5():
    """6,144 sources on which every target of the sphere takes the split at eps = 0."""
    m = bve.build_mesh(P.SEED_CUBED, 5)
    leaf = m["fmask"] == 0
    return m["fx"][leaf], bve.rh54_gaussians(3, 2)(m["fx"][leaf]), m["farea"][leaf]


def _sums(tgt, src, w, eps=0.0):
    """Velocity, stream function and the velocity's bound at every target (w = -zeta area)."""
    u, p, bound = np.zeros((len(tgt), 3), L), np.zeros(len(tgt), L), np.zeros(len(tgt))
    y, w4 = src.astype(L), w.astype(L) / (4 * L("3.14159265358979323846264338327950288"))
    for i, x in enumerate(tgt.astype(L)):
        omd = 1 - (y[:, 0] * x[0] + y[:, 1] * x[1] + y[:, 2] * x[2]) + L(eps) * L(eps)
        s = w4 / omd
        c = np.stack([x[1] * y[:, 2] - x[2] * y[:, 1], x[2] * y[:, 0] - x[0] * y[:, 2], x[0] * y[:, 1] - x[1] * y[:, 0]], 1)
        u[i] = (s[:, None] * c).sum(0)
        p[i] = (np.log(omd) * w4).sum()
        r, s64, cn = 1 + float(np.sqrt((x * x).sum())), np.abs(s).astype(float), np.linalg.norm(c.astype(float), axis=1)
        bound[i] = (s64 * (cn * (2.0**-45 + 2.0**-50 * r / np.abs(omd).astype(float)) + 2.0**-51 * r)).sum()
    return u, p, bound


def _call(c, x, src, zeta, area, mask, psi, eps=0.0):
    u, p = c.velocity(x, src, zeta, area, mask, eps=eps, flags=P.FP64 | (P.PSI if psi else 0))
    torch.cuda.synchronize()
    return u.cpu().numpy(), p.cpu().numpy() if psi else None


RADII = (0.25, 0.99, 0.9999, 1.0, 1.0001, 1.001, 1.01, 1.2, 1.9, 2.1, 1000.0)


@pytest.mark.parametrize("psi", [False, True])
@pytest.mark.parametrize("off", [0.0, 0.01])
def test_points_off_the_sphere(oracle, capfd, psi, off):
    """A plan of points on the sphere keeps its kernel when the points move (a time loop does so): on, beside
    and off the sphere, sources up to `off` off it.  At 1 - x.y < 0 the logarithm is NaN, as in the reference."""
    src, zeta, area = _cube5()
    rng = np.random.default_rng(11)
    n = 24 * len(RADII)
    x = _dev(_unit(rng.normal(size=(n, 3))))
    y, z, a, k = _dev(src), _dev(zeta), _dev(area), torch.zeros(len(src), dtype=torch.uint8, device="cuda")
    near = _unit(src[rng.choice(len(src), n, False)] + rng.normal(size=(n, 3)) * 10.0 ** rng.uniform(-7, -1.5, size=(n, 1)))
    far = _unit(rng.normal(size=(n, 3)))
    tgt = np.where(np.arange(n)[:, None] % 2 == 0, near, far) * np.repeat(RADII, 24)[:, None]
    moved = src * (1 + off * rng.uniform(-1, 1, size=(len(src), 1)))
    with bve.Context(verbose=True) as c:
        _call(c, x, y, z, a, k, psi)
        assert _split_items(capfd) > 0
        x.copy_(_dev(tgt))
        y.copy_(_dev(moved))
        u, p = _call(c, x, y, z, a, k, psi)
        assert "plan:" not in capfd.readouterr().err
    with np.errstate(all="ignore"):
        want, wp, bound = _sums(tgt, moved, -zeta * area)
        ref, rp = oracle.velocity_distinct(tgt, moved, zeta, area, np.zeros(len(src), np.uint8), psi=True)
    err = np.linalg.norm((u - want).astype(float), axis=1)
    assert (err <= bound).all(), (err / bound).reshape(len(RADII), 24).max(1)
    if psi:
        assert np.array_equal(np.isnan(p), np.isnan(rp))
        ok = ~np.isnan(rp)
        scale = np.abs(wp[ok]).max()
        assert np.abs((p - wp)[ok]).max() <= 10 * np.abs((rp - wp)[ok]).max() + 1e-14 * scale


def test_a_plan_with_a_point_off_the_sphere_takes_the_exact_kernel(oracle, capfd):
    src, zeta, area = _cube5()
    tgt = _unit(np.random.default_rng(2).normal(size=(300, 3)))
    y, z, a, k = _dev(src), _dev(zeta), _dev(area), torch.zeros(len(src), dtype=torch.uint8, device="cuda")
    for scale, split in ((1.0, True), (1.002, False), (0.5, False), (np.nan, False)):
        tgt[7] *= scale
        with bve.Context(verbose=True) as c:
            u, _ = _call(c, _dev(tgt), y, z, a, k, False)
            assert (_split_items(capfd) > 0) == split, scale
        with np.errstate(all="ignore"):
            ref = oracle.velocity_distinct(tgt, src, zeta, area, np.zeros(len(src), np.uint8))
        assert np.array_equal(np.isnan(u), np.isnan(ref))
        assert np.nanmax(np.abs(u - ref)) <= 1e-12 * np.nanmax(np.abs(ref))


@pytest.mark.parametrize("psi", [False, True])
def test_near_pairs_and_what_is_not_finite(oracle, capfd, psi):
    """Targets on a source, 1e-7 and 2^-6 beside one, NaN and infinite, on a plan that keeps the split; then a
    source that is NaN and one that is infinite."""
    src, zeta, area = _cube5()
    rng = np.random.default_rng(4)
    n = 300
    x = _dev(_unit(rng.normal(size=(n, 3))))
    y, z, a, k = _dev(src), _dev(zeta), _dev(area), torch.zeros(len(src), dtype=torch.uint8, device="cuda")
    tgt = _unit(rng.normal(size=(n, 3)))
    tgt[:100] = src[:100]
    tgt[100:130] = _unit(src[200:230] + 1e-7 * rng.normal(size=(30, 3)))
    tgt[130:200] = _unit(src[300:370] + 2.0**-6 * _unit(rng.normal(size=(70, 3))) * rng.uniform(0.99, 1.01, size=(70, 1)))
    tgt[200] = np.nan
    tgt[201] = (np.inf, 0.3, 0.2)
    tgt[202] = (0.1, -np.inf, np.nan)
    tgt[203] = 0.0
    with bve.Context(verbose=True) as c:
        _call(c, x, y, z, a, k, psi)
        assert _split_items(capfd) > 0
        x.copy_(_dev(tgt))
        u, p = _call(c, x, y, z, a, k, psi)
        for row in ((np.nan, 0.0, 0.0), (np.inf, 0.0, 0.0)):
            bad = src.copy()
            bad[40] = row
            y.copy_(_dev(bad))
            v, _ = _call(c, x, y, z, a, k, psi)
            with np.errstate(all="ignore"):
                rv = oracle.velocity_distinct(tgt, bad, zeta, area, np.zeros(len(src), np.uint8))
            assert np.array_equal(np.isnan(v), np.isnan(rv))
    with np.errstate(all="ignore"):
        ref, rp = oracle.velocity_distinct(tgt, src, zeta, area, np.zeros(len(src), np.uint8), psi=True)
        want, _, bound = _sums(tgt[100:200], src, -zeta * area)
    for got, r in ((u, ref), (p, rp)):
        if got is not None:
            assert np.array_equal(np.isnan(got), np.isnan(r)) and np.array_equal(np.isinf(got), np.isinf(r))
    err = np.linalg.norm((u[100:200] - want).astype(float), axis=1)
    assert (err <= bound).all()
    assert np.abs(u[204:] - ref[204:]).max() <= 1e-12 * np.abs(ref[204:]).max()


@pytest.mark.parametrize("psi", [False, True])
def test_weights_of_any_size(capfd, psi):
    """Weights times a power of two give the same digits, also where FP32 does not hold them; weights 80 orders of
    magnitude apart, zero and near the ends of FP64's range stay within the bound."""
    src, zeta, area = _cube5()
    rng = np.random.default_rng(8)
    tgt = _unit(rng.normal(size=(500, 3)))
    tgt[:50] = _unit(src[:50] + 1e-3 * rng.normal(size=(50, 3)))  # near pairs
    x, y, a, k = _dev(tgt), _dev(src), _dev(area), torch.zeros(len(src), dtype=torch.uint8, device="cuda")
    with bve.Context(verbose=True) as c:
        u, p = _call(c, x, y, _dev(zeta), a, k, psi)
        assert _split_items(capfd) > 0
        for e in (-900, -160, -130, -100, 40, 130, 900):
            v, q = _call(c, x, y, _dev(np.ldexp(zeta, e)), a, k, psi)
            assert np.array_equal(v, np.ldexp(u, e)), e
            assert not psi or np.array_equal(q, np.ldexp(p, e)), e
        mixed = zeta * np.where(rng.uniform(size=len(src)) < 0.5, 1e-42, 1e40)
        mixed[:2000] = 0.0
        tail = zeta * np.exp(-((np.arccos(np.clip(src @ src[17], -1, 1)) / 0.1) ** 2))
        for z in (mixed, tail, zeta * 1e-290):
            v, _ = _call(c, x, y, _dev(z), a, k, psi)
            want, _, bound = _sums(tgt, src, -z * area)
            assert (np.linalg.norm((v - want).astype(float), axis=1) <= bound).all()


@pytest.mark.parametrize("seed,level,eps,velocity,rk4", [
    (P.SEED_CUBED, 4, 0.0, False, False),      # 1,536 sources
    (P.SEED_CUBED, 5, 0.0, True, True),        # 6,144
    (P.SEED_CUBED, 5, 1e-6, False, True),
    (P.SEED_CUBED, 5, 0.03, False, True),
    (P.SEED_CUBED, 5, 0.031, False, False),
    (P.SEED_ICOS_TRI, 5, 0.0, False, False),   # 20,480, parents on their children
    (P.SEED_ICOS_TRI, 5, 0.01, True, True),
    (P.SEED_ICOS_TRI, 5, 1.0, True, True),
    (P.SEED_ICOS_TRI, 5, 1.01, False, False),
    (P.SEED_ICOS_TRI, 5, 1e30, False, False),
])
def test_which_solves_take_the_split(oracle, capfd, seed, level, eps, velocity, rk4):
    """The sizes and regularisations at which its error is no larger than the reference's (csrc/engine.hpp)."""
    s = bve.BVESphere(seed, level)
    with bve.Context(verbose=True) as c:
        s.init_vorticity(bve.rh54_gaussians(3, 2), c, flags=P.FP64, eps=eps)
        torch.cuda.synchronize()
        assert (_split_items(capfd) > 0) == velocity
        c.rk4_step(s.state(), 0.0, 0.0, 1, flags=P.FP64, eps=eps)
        torch.cuda.synchronize()
        assert (_split_items(capfd) > 0) == rk4
    m = s.mesh
    ref = oracle.velocity_distinct(m["vx"][:40], m["fx"], s.relVortFaces.cpu().numpy(), m["farea"], m["fmask"], eps=eps)
    assert np.abs(s.velocityVerts[:40].cpu().numpy() - ref).max() <= 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("nt,chunks", [(1, 48), (6146, 48), (16000, 48), (96000, 8), (400000, 8)])
def test_partial_sums_stay_few_with_many_targets(capfd, nt, chunks):
    """Small solves spread their sources over 48 chunks; sets of many targets have items enough and keep the 8
    chunks of the other kernels, whose partial sums bound the workspace (32 bytes per target and chunk)."""
    src, zeta, area = _cube5()
    x = _unit(np.random.default_rng(6).normal(size=(nt, 3)))
    mask = torch.zeros(len(src), dtype=torch.uint8, device="cuda")
    with bve.Context(verbose=True) as c:
        u, _ = _call(c, _dev(x), _dev(src), _dev(zeta), _dev(area), mask, False)
        line = capfd.readouterr().err
        v, _ = _call(c, _dev(x[:1000]), _dev(src), _dev(zeta), _dev(area), mask, False)
    assert int(re.findall(r"split=(\d+)", line)[0]) > 0 and int(re.findall(r"chunks=(\d+)", line)[0]) == chunks
    assert np.abs(u[:1000] - v).max() <= 1e-12 * np.abs(v).max()
