"""The FP32 operator's kernels at the sizes where their work splits change: expansion orders
around the 32 of a warp, boxes of one chunk of 64 points and of several, tiles of 16 and 17
targets, odd source counts. The FP64 operator at the same order and M2L tolerance has the same
truncation, so the two differ by FP32 rounding: 1e-5 of the largest value, the bar of the other
FP32 parity tests."""
import numpy as np
import pytest

from electricbubbles_gb300 import configs

pytestmark = pytest.mark.gpu


def relmax(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("p", [2, 7, 20, 31, 32, 33, 60])
@pytest.mark.parametrize("n", [63, 65, 130, 2001])
def test_orders(gpu_ctx_factory, p, n):
    rng = np.random.default_rng(p * n)
    z = (rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)) * 10.0 ** -rng.uniform(0, 1.5, n)
    q = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    ctx = gpu_ctx_factory(p64=p, p32=p, tol64=1e-7, tol32=1e-7, leaf64=17, leaf_cap=33, direct_max=-1)
    assert relmax(ctx.dapif2(z, q, "fp32"), ctx.dapif2(z, q, "fp64")) < 1e-5


@pytest.mark.parametrize("p", [5, 20, 33])
@pytest.mark.parametrize("leaf", [(15, 16), (17, 17), (30, 64)])
def test_stokes_orders(gpu_ctx_factory, oracle, p, leaf):
    cfg = configs.small_drops(7, 320, box=6.0)
    ex = oracle.extractdat(cfg.nd, cfg.rku())
    rng = np.random.default_rng(p)
    u = rng.standard_normal(cfg.nbk) + 1j * rng.standard_normal(cfg.nbk)
    ctx = gpu_ctx_factory(p64=p, p32=p, tol64=1e-7, tol32=1e-7, leaf64=leaf[0], leaf_cap=leaf[1])
    ctx.set_geometry(cfg.nd, ex["z"], ex["dz"], ex["dsda"], ex["kappa"], ex["zk"])
    for sign in (-1, 1):
        assert relmax(ctx.stokes_sum(u, sign, "fp32"), ctx.stokes_sum(u, sign, "fp64")) < 1e-5
