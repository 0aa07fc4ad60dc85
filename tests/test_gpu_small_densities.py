"""Sums over densities near the ends of the double range: the operators are linear, so that
charges scaled by a power of two give the scaled sums, to the FP64 parity tests' 1e-12 of the largest
value (the fixed-point M2L takes each box by its own exponent)."""
import numpy as np
import pytest

from electricbubbles_gb300 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("e", [-965, -930, -500, 500, 960])
def test_scaled_charges(gpu_ctx_factory, e):
    rng = np.random.default_rng(1)
    n = 3000
    z = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)
    q = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    ctx = gpu_ctx_factory(leaf64=8, leaf_cap=16)
    ref = ctx.dapif2(z, q)
    got = ctx.dapif2(z, q * 2.0 ** e) / 2.0 ** e
    assert np.abs(got - ref).max() < 1e-12 * np.abs(ref).max()


@pytest.mark.parametrize("e", [-965, -930, -500, 500, 960])
@pytest.mark.parametrize("sign", [-1, 1])
def test_scaled_density(gpu_ctx_factory, oracle, e, sign):
    cfg = configs.many_drops(16, 256, seed=3, box=8.0)
    ex = oracle.extractdat(cfg.nd, cfg.rku())
    rng = np.random.default_rng(2)
    u = rng.standard_normal(cfg.nbk) + 1j * rng.standard_normal(cfg.nbk)
    ctx = gpu_ctx_factory()
    ctx.set_geometry(cfg.nd, ex["z"], ex["dz"], ex["dsda"], ex["kappa"], ex["zk"])
    ref = ctx.stokes_sum(u, sign)
    got = ctx.stokes_sum(u * 2.0 ** e, sign) / 2.0 ** e
    assert np.abs(got - ref).max() < 1e-12 * np.abs(ref).max()
