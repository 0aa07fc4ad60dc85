"""The double-float M2L's two kernels: the CUDA-core one below order 36 (one launch), the fixed-point
one from there on (two: the conversion and the M2L), for two expansions on trees of any size, with
the wall's images and without. Both against the native FP64 operator at the same order, which
truncates the same: 1e-11 of the largest value."""
import numpy as np
import pytest

from electricbubbles_gb300 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wall", [False, True])
def test_orders(gpu_ctx_factory, oracle, wall):
    cfg = configs.wall_drops(16, 256) if wall else configs.many_drops(16, 256, seed=3, box=8.0)
    ex = oracle.extractdat(cfg.nd, cfg.rku())
    rng = np.random.default_rng(1)
    u = rng.standard_normal(cfg.nbk) + 1j * rng.standard_normal(cfg.nbk)
    launches = {}
    for p in (12, 35, 36, 44):
        got = []
        for df64 in (-1, 1):
            ctx = gpu_ctx_factory(p64=p, df64=df64)
            if wall:
                ctx.set_wall(1)
            ctx.set_geometry(cfg.nd, ex["z"], ex["dz"], ex["dsda"], ex["kappa"], ex["zk"])
            n0 = ctx.launch_count()
            got.append(ctx.stokes_sum(u, -1))
            launches[p] = ctx.launch_count() - n0
        assert np.abs(got[0] - got[1]).max() < 1e-11 * np.abs(got[0]).max()
    m2l = 2 if wall else 1  # M2L passes
    assert launches[12] == launches[35] == launches[36] - m2l == launches[44] - m2l
