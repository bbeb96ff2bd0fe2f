"""The forms a solve takes by its size give the same bits: a batch that fills a fraction of the GPU
(pairFP32CSub: targets in items of 256, sources in sub-blocks of 64, 128 x 2 or 64 x 4 threads and targets)
against the same solve beside a large one (pairFP32C), a request alone in the server against several at
once, and a plan sorted by keys from the device (32,768 points and more) against one sorted by the host's."""
import re

import numpy as np
import pytest
import torch

import lpmkokkos_gb300 as P
from lpmkokkos_gb300 import bve

pytestmark = pytest.mark.gpu

KEYS = ("vx", "vzeta", "vvel", "fx", "fzeta", "fvel")


def _points(n, rng):
    x = rng.normal(size=(n, 3))
    return x / np.linalg.norm(x, axis=1, keepdims=True)


def _velocity(ctx, tgt, src, zeta, area, mask, flags, psi):
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    u, p = ctx.velocity(dev(tgt), dev(src), dev(zeta), dev(area), dev(mask), flags=P.FP32C | flags | (P.PSI if psi else 0))
    torch.cuda.synchronize()
    ctx.invalidate()
    return u.cpu().numpy(), p.cpu().numpy() if psi else None


@pytest.mark.parametrize("ns", [1, 63, 64, 65, 1000])
@pytest.mark.parametrize("flags,psi", [(0, False), (0, True), (P.RCP_APPROX, False)])
def test_few_targets_have_the_bits_of_many(ctx, ns, flags, psi):
    rng = np.random.default_rng(ns)
    src, zeta, area = _points(ns, rng), rng.normal(size=ns), np.full(ns, 4 * np.pi / ns)
    mask = (rng.uniform(size=ns) < 0.1).astype(np.uint8) if ns > 100 else np.zeros(ns, np.uint8)
    many = _points(262144, rng)
    u, p = _velocity(ctx, many, src, zeta, area, mask, flags, psi)
    for nt in (1, 31, 255, 256, 257, 700):
        su, sp = _velocity(ctx, many[:nt], src, zeta, area, mask, flags, psi)
        assert np.array_equal(su, u[:nt])
        assert sp is None or np.array_equal(sp, p[:nt])


@pytest.mark.parametrize("seed,level", [(0, 2), (0, 3), (0, 4), (1, 4), (1, 5)])
def test_small_step_has_the_bits_of_the_ensemble(ctx, seed, level):
    a, b, big = bve.BVESphere(seed, level), bve.BVESphere(seed, level), bve.BVESphere(0, 6)
    for s in (a, b, big):
        s.init_vorticity(bve.rh54_gaussians(3, 2), ctx, flags=P.FP32C)
        ctx.invalidate()
    ctx.rk4_step(a.state(), 0.005, 2 * np.pi, 2, flags=P.FP32C)
    ens = ctx.ensemble([b.state(), big.state()], flags=P.FP32C)
    ens.step(np.array([0.005, 0.0025]), 2 * np.pi, 2)
    torch.cuda.synchronize()
    ens.close()
    for k in ("physFaces", "physVerts", "relVortFaces", "relVortVerts", "velocityFaces", "velocityVerts"):
        assert np.array_equal(getattr(a, k).cpu().numpy(), getattr(b, k).cpu().numpy(), equal_nan=True), k


def test_requests_at_once_have_the_bits_of_one_alone():
    specs = [dict(seed=int(k % 3 == 2), level=2 + k % 3, dt=0.005, nsteps=3, ic_seed=k, n_gaussians=1 + k % 4) for k in range(6)]
    alone = []
    for s in specs:
        with bve.Server(0, flags=P.FP32C) as srv:
            rid = srv.submit(**s)
            assert srv.wait(rid, 600.0)
            alone.append(srv.result(rid))
    with bve.Server(0, flags=P.FP32C) as srv:
        ids = [srv.submit(**s) for s in specs]
        for rid, want in zip(ids, alone):
            assert srv.wait(rid, 600.0)
            got = srv.result(rid)
            for k in KEYS:
                assert np.array_equal(got[k], want[k], equal_nan=True), (rid, k)


def test_device_keys_sort_as_the_hosts(ctx):
    rng = np.random.default_rng(3)
    src, zeta, area, mask = _points(2000, rng), rng.normal(size=2000), np.full(2000, 0.006), np.zeros(2000, np.uint8)
    tgt = np.concatenate([_points(20000, rng), rng.uniform(-1.2, 1.2, size=(11000, 3))])
    step = 2.1 / 1024  # cell boundaries, points outside the cube, points on a source, not finite
    tgt[:3000] = np.rint(tgt[:3000] / step) * step
    tgt[3000:3100] = src[:100]
    tgt[3100] = np.nan
    tgt[3101] = (np.inf, 0.0, -np.inf)
    src[:50] = np.rint(src[:50] / step) * step
    host, _ = _velocity(ctx, tgt[:20000], src, zeta, area, mask, 0, False)  # 22,000 points
    dev, _ = _velocity(ctx, tgt, src, zeta, area, mask, 0, False)           # 33,000 points
    assert np.array_equal(host, dev[:20000], equal_nan=True)


def test_stream_function_on_a_plan_made_without_it(ctx):
    """A small plan's sub-block sums have room for what its first call asked; either order gives the same bits."""
    rng = np.random.default_rng(9)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    src, tgt = dev(_points(1500, rng)), dev(_points(900, rng))
    zeta, area, mask = dev(rng.normal(size=1500)), dev(np.full(1500, 0.008)), dev(np.zeros(1500, np.uint8))
    out = []
    for order in ((0, P.PSI), (P.PSI, 0)):
        for psi in order:
            u, p = ctx.velocity(tgt, src, zeta, area, mask, flags=P.FP32C | psi)
            torch.cuda.synchronize()
            out.append((u.cpu().numpy(), p.cpu().numpy() if psi else None))
        ctx.invalidate()
    assert all(np.array_equal(o[0], out[0][0]) for o in out)
    assert np.array_equal(out[1][1], out[2][1])


@pytest.mark.parametrize("ns", [1, 63, 64, 65, 1000])
@pytest.mark.parametrize("flags,psi", [(0, False), (0, True), (P.RCP_APPROX, False)])
def test_sub_blocks_have_the_bits_of_the_plain_kernel(native, capfd, ns, flags, psi):
    """Few targets against a million, whose plan takes the plain kernel: the plan lines say so."""
    rng = np.random.default_rng(ns)
    src, zeta, area = _points(ns, rng), rng.normal(size=ns), np.full(ns, 4 * np.pi / ns)
    mask = np.zeros(ns, np.uint8)
    many = _points(1 << 20, rng)
    subs = lambda: int(re.findall(r"sub=(\d+)", capfd.readouterr().err)[-1])  # noqa: E731
    with bve.Context(verbose=True) as c:
        u, p = _velocity(c, many, src, zeta, area, mask, flags, psi)
        assert subs() == 0
        for nt in (1, 31, 255, 256, 257, 700, 200000):
            su, sp = _velocity(c, many[:nt], src, zeta, area, mask, flags, psi)
            assert subs() > 0
            assert np.array_equal(su, u[:nt])
            assert sp is None or np.array_equal(sp, p[:nt])
