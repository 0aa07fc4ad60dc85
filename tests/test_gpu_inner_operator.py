"""The FP32 operator of the refined solves' inner cycles (its own kernels: k_p2m_points and
k_p2m_chunks, k_m2l_f32w and k_m2l_f32p, the packed k_near32 and k_far32, the direct sums) at the
sizes where its work splits change: expansion orders around the 32 of a warp, boxes of one chunk
of 64 points and of several, tiles of 16 and 17 targets, odd source counts, leaves of one point
and of several tiles, trees on both sides of the 8,192 boxes where the M2L changes, with and without
the wall. The FP64 operator at the same order and M2L tolerance has the same truncation, so the
two differ by FP32 rounding: 1e-5 of the largest value, the bar of the other FP32 parity tests."""
import ctypes

import numpy as np
import pytest

from electricbubbles_gb300 import configs

pytestmark = pytest.mark.gpu
OPS = ["fasmvp", "fasmvp_lap", "fasmvp_adjoint", "fasmvp_lap_adjoint"]


def check_all(ctx, rng, ops=OPS):
    import torch

    inner = ctx._lib.eb_inner_matvec
    inner.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p]
    for name in ops:
        x = torch.from_numpy(rng.standard_normal(ctx.nbk * (1 if "lap" in name else 2))).cuda()
        got = torch.empty_like(x)
        torch.cuda.synchronize()
        ref = getattr(ctx, name)(x, "fp64")
        assert inner(ctx._h, OPS.index(name), x.data_ptr(), got.data_ptr()) == 0
        ctx.sync()
        assert float((got - ref).abs().max() / ref.abs().max()) < 1e-5, name


def scattered(ctx, n, rng, decades):
    """One 'drop' of n points of several scales, its charges of random directions and large enough
    that the sums, not the identity, make up the result."""
    z = (rng.uniform(-1, 1, n) + 1j * rng.uniform(0, 1, n)) * 10.0 ** -rng.uniform(0, decades, n)
    dz = 10.0 * np.sqrt(n) * (rng.standard_normal(n) + 1j * rng.standard_normal(n))
    ctx.set_geometry([n], z, dz, np.ones(n), np.zeros(n), np.array([50.0 + 50.0j]))


@pytest.mark.parametrize("p", [2, 7, 20, 31, 32, 33, 60])
@pytest.mark.parametrize("n", [63, 65, 130, 2001])
def test_orders(gpu_ctx_factory, p, n):
    rng = np.random.default_rng(p * n)
    ctx = gpu_ctx_factory(p64=p, p32=p, tol64=1e-7, tol32=1e-7, leaf64=17, leaf_cap=33)
    scattered(ctx, n, rng, 1.5)
    check_all(ctx, rng)


def drops_of(ctx, oracle, cfg):
    ex = oracle.extractdat(cfg.nd, cfg.rku())
    ctx.set_geometry(cfg.nd, ex["z"], ex["dz"], ex["dsda"], ex["kappa"], ex["zk"])


@pytest.mark.parametrize("leaf", [(1, 1), (3, 7), (15, 16), (17, 17), (30, 64), (90, 200)])
@pytest.mark.parametrize("p", [20, 33])
def test_leaves(gpu_ctx_factory, oracle, p, leaf):
    cfg = configs.small_drops(7, 320, box=6.0)
    rng = np.random.default_rng(p)
    ctx = gpu_ctx_factory(p64=p, p32=p, tol64=1e-7, tol32=1e-7, leaf64=leaf[0], leaf_cap=leaf[1])
    drops_of(ctx, oracle, cfg)
    check_all(ctx, rng)


@pytest.mark.parametrize("n,wide", [(6000, False), (60001, True)])
def test_wide_m2l(gpu_ctx_factory, n, wide):
    rng = np.random.default_rng(n)
    ctx = gpu_ctx_factory(p64=20, p32=20, tol64=1e-7, tol32=1e-7, leaf64=4, leaf_cap=9)
    scattered(ctx, n, rng, 0.0)
    first = ctx.tree_info()["nboxes"] - 5  # boxes of the levels from 2 on
    assert (first >= 8192) == wide
    check_all(ctx, rng)


@pytest.mark.parametrize("leaf,wide", [((32, 96), False), ((4, 6), True)])
def test_wall(gpu_ctx_factory, leaf, wide):
    cfg = configs.wall_drops(k=64, n=512, seed=12, box=24.0)
    rng = np.random.default_rng(1)
    ctx = gpu_ctx_factory(p64=20, p32=20, tol64=1e-7, tol32=1e-7, leaf64=leaf[0], leaf_cap=leaf[1])
    ctx.set_wall(1)
    ctx.extractdat(cfg.nd, cfg.rku())
    assert (ctx.tree_info()["nboxes"] >= 8300) == wide
    check_all(ctx, rng, OPS[:1])


@pytest.mark.parametrize("drops,nodes", [(1, 64), (3, 100), (1, 450), (7, 130)])
def test_direct_sums(gpu_ctx_factory, oracle, drops, nodes):
    cfg = configs.small_drops(drops, nodes, box=6.0)
    rng = np.random.default_rng(nodes)
    ctx = gpu_ctx_factory(direct_max=1024)
    drops_of(ctx, oracle, cfg)
    check_all(ctx, rng)
