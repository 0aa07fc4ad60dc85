"""The fixed-point M2L where the boxes of one list have very different exponents: regions whose
charges differ by up to 2^600 stand beside each other, so that a target box adds entries of which some
are shifted out of sight. Each point's error is held to the sum of its terms' moduli (1e-12): where
the near charges are the large ones the far ones' errors are small beside them, and the other way
round. Stokes sums of both signs (two expansions, each with its own exponent, psi moved to the
target's centre), with and without the wall's images, and Cauchy sums; orders up to the last that
it takes and the first that the CUDA-core kernel keeps; zeros and non-finite densities."""
import numpy as np
import pytest

from electricbubbles_gb300 import configs

pytestmark = pytest.mark.gpu


def scales(rng, k, df64):
    """A power of two per region (double-float charges have a float's range)."""
    return 2.0 ** rng.integers(*((-25, 26) if df64 > 0 else (-300, 301)), k)


@pytest.mark.parametrize("df64", [-1, 1])
def test_cauchy_regions(gpu_ctx_factory, oracle, df64):
    rng = np.random.default_rng(1)
    n, side = 12000, 12
    cell = rng.integers(0, side * side, n)
    z = (cell % side + rng.uniform(0, 1, n)) + 1j * (cell // side + rng.uniform(0, 1, n))
    q = (rng.standard_normal(n) + 1j * rng.standard_normal(n)) * scales(rng, side * side, df64)[cell]
    ctx = gpu_ctx_factory(leaf64=4, leaf_cap=8, df64=df64)
    got, ref = ctx.dapif2(z, q), oracle.cauchy_direct(z, z, q, True)
    for i in np.array_split(np.arange(n), 8):
        d = np.abs(z[i][:, None] - z[None, :])
        d[np.arange(i.size), i] = np.inf
        assert (np.abs(got[i] - ref[i]) / (np.abs(q)[None, :] / d).sum(1)).max() < 1e-12


def setup(oracle, wall):
    cfg = configs.wall_drops(16, 256) if wall else configs.many_drops(16, 256, seed=3, box=8.0)
    return cfg, oracle.extractdat(cfg.nd, cfg.rku()), oracle.point_h(cfg.nd)


def context(factory, cfg, ex, wall, **kw):
    ctx = factory(leaf64=8, leaf_cap=16, **kw)
    if wall:
        ctx.set_wall(1)
    ctx.set_geometry(cfg.nd, ex["z"], ex["dz"], ex["dsda"], ex["kappa"], ex["zk"])
    return ctx


@pytest.mark.parametrize("wall", [False, True])
@pytest.mark.parametrize("df64", [-1, 1])
@pytest.mark.parametrize("p64", [44, 46, 47, 48])
def test_stokes_regions(gpu_ctx_factory, oracle, p64, df64, wall):
    cfg, ex, h = setup(oracle, wall)
    rng = np.random.default_rng(p64)
    u = rng.standard_normal(cfg.nbk) + 1j * rng.standard_normal(cfg.nbk)
    u = u * np.repeat(scales(rng, cfg.k, df64), cfg.nd)
    z, w = ex["z"], np.abs(u * ex["dz"]) * h / (2 * np.pi)  # |qa|; |qb| is at most twice that
    d = np.abs(z[:, None] - z[None, :])
    np.fill_diagonal(d, np.inf)
    size = (4 * w[None, :] / d).sum(1)  # qa / D, conj(qb / D) and D conj(qa / D^2)
    if wall:  # 12 |qa| + 3 |qb| bound an image's terms (the source is nearer than its image)
        size = size + (18 * w[None, :] / np.abs(z.conj()[None, :] - z[:, None])).sum(1)
    ctx = context(gpu_ctx_factory, cfg, ex, wall, p64=p64, df64=df64)
    for sign in (-1, 1):
        ref = oracle.stokes_direct(z, ex["dz"], h, u, sign)
        if wall:
            ref = ref + oracle.stokes_image_direct(z, ex["dz"], h, u, sign)
        assert (np.abs(ctx.stokes_sum(u, sign) - ref) / size).max() < 1e-12


@pytest.mark.parametrize("wall", [False, True])
@pytest.mark.parametrize("df64", [-1, 1])
def test_stokes_zero_and_non_finite(gpu_ctx_factory, oracle, df64, wall):
    cfg, ex, _ = setup(oracle, wall)
    ctx = context(gpu_ctx_factory, cfg, ex, wall, df64=df64)
    u = np.zeros(cfg.nbk, complex)
    assert np.abs(ctx.stokes_sum(u, -1)).max() == 0.0
    for bad in (np.inf, np.nan):
        u = np.random.default_rng(1).standard_normal(cfg.nbk) + 0j
        u[7] = bad
        assert not np.isfinite(np.delete(ctx.stokes_sum(u, -1), 7)).any()
