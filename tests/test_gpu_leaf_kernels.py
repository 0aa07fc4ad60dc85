"""The near- and far-field kernels at the sizes where their work splits change: leaves of one
point, of a part of a tile, of several tiles, and U lists longer than one round of boxes,
for the three pair forms (FASMVP's charges of both signs, the transposed operator's
complex charges, the Cauchy sum) in the three arithmetics, against the oracle's direct
sums. Bars as in the other parity tests: 1e-12 for the FP64-class sums, 1e-5 for FP32, of
the largest value."""
import numpy as np
import pytest

from electricbubbles_gb300 import configs

pytestmark = pytest.mark.gpu
LEAVES = [(1, 1), (3, 7), (16, 17), (32, 33), (40, 80), (90, 200)]
ARITH = [("fp64", -1, 1e-12), ("fp64", 1, 1e-12), ("fp32", -1, 1e-5)]


def relmax(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("leaf", LEAVES)
@pytest.mark.parametrize("prec,df64,bar", ARITH)
def test_pairs(gpu_ctx_factory, oracle, leaf, prec, df64, bar):
    cfg = configs.small_drops(5, 256, box=5.0)
    ex = oracle.extractdat(cfg.nd, cfg.rku())
    h = oracle.point_h(cfg.nd)
    rng = np.random.default_rng(3)
    u = rng.standard_normal(cfg.nbk) + 1j * rng.standard_normal(cfg.nbk)
    v = rng.standard_normal(2 * cfg.nbk)
    ctx = gpu_ctx_factory(leaf64=leaf[0], leaf_cap=leaf[1], df64=df64)
    ctx.set_geometry(cfg.nd, ex["z"], ex["dz"], ex["dsda"], ex["kappa"], ex["zk"])
    for sign in (-1, 1):
        ref = oracle.stokes_direct(ex["z"], ex["dz"], h, u, sign)
        assert relmax(ctx.stokes_sum(u, sign, prec), ref) < bar
    # the transpose of FASMVP and of FASMVP_LAP: <A^T v, w> = <v, A w> with the exact A w
    g = oracle.Geometry.from_extract(cfg.nd, ex)
    w = rng.standard_normal(2 * cfg.nbk)
    aw = oracle.fasmvp(g, w, 0)
    scale = np.linalg.norm(v) * np.linalg.norm(aw)
    assert abs(ctx.fasmvp_adjoint(v, prec) @ w - v @ aw) < bar * scale
    assert relmax(ctx.fasmvp_lap(w[:cfg.nbk], prec), np.asarray(oracle.fasmvp_lap(g, w[:cfg.nbk]))[:cfg.nbk]) < bar


@pytest.mark.parametrize("n", [2, 3, 31, 129, 1500])
@pytest.mark.parametrize("prec,df64,bar", ARITH)
def test_cauchy_scales(gpu_ctx_factory, oracle, n, prec, df64, bar):
    """Points of scales from 1 down to 1e-4 (long U lists, W lists), odd counts."""
    rng = np.random.default_rng(n)
    z = (rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)) * 10.0 ** -rng.uniform(0, 4, n)
    q = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    ctx = gpu_ctx_factory(leaf64=8, leaf_cap=8, df64=df64)
    assert relmax(ctx.dapif2(z, q, prec), oracle.cauchy_direct(z, z, q, True)) < bar


@pytest.mark.parametrize("n", [300, 3000, 30000])
@pytest.mark.parametrize("p64", [5, 44])
def test_level_passes(gpu_ctx_factory, oracle, n, p64):
    """M2M and L2L on levels of a few, some hundred and thousands of boxes (their outputs are
    dealt to four, two or one blocks per box), and the far field's two lane layouts: at 1e-12
    against direct sums, at a low order against the double-float kernels (1e-11)."""
    rng = np.random.default_rng(n)
    z = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)
    q = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    got = gpu_ctx_factory(p64=p64, leaf64=8, leaf_cap=8).dapif2(z, q)
    if p64 == 44:
        i = rng.integers(0, n, 200)
        d = z[i][:, None] - z[None, :]
        d[np.arange(200), i] = np.inf
        assert relmax(got[i], (q[None, :] / d).sum(1)) < 1e-12
    else:
        ref = gpu_ctx_factory(p64=p64, leaf64=8, leaf_cap=8, df64=1).dapif2(z, q)
        assert relmax(got, ref) < 1e-11
