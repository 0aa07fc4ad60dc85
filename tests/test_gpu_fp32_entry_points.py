"""The FP32 operator of the entry points and that of the refined solves' inner cycles: the one
keeps its order of additions, the other is faster; both approximate the FP64 operator. Sizes:
direct sums, a tree without far levels, several levels.
"""
import numpy as np
import pytest

from electricbubbles_gb300 import configs
from electricbubbles_gb300.api import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("drops,nodes,direct", [(1, 64, -1), (1, 256, 0), (3, 128, -1), (16, 256, 0), (64, 512, 0)])
def test_fp32_entry_points(drops, nodes, direct):
    cfg = configs.small_drops(drops, nodes) if drops < 16 else configs.many_drops(drops, nodes)
    rng = np.random.default_rng(7)
    u, v = rng.standard_normal(2 * cfg.nbk), rng.standard_normal(cfg.nbk)
    with Context(device=0, direct_max=direct) as ctx:
        ctx.extractdat(cfg.nd, cfg.rku())
        for op, x in ((ctx.fasmvp, u), (ctx.fasmvp_lap, v)):
            ref, got = op(x, "fp64"), op(x, "fp32")
            # FP32 sums of smooth terms: 1e-5 of the largest entry, the bound of the smoke test
            assert np.abs(got - ref).max() < 1e-5 * np.abs(ref).max()
            assert np.array_equal(got, op(x, "fp32"))


@pytest.mark.parametrize("p", [20, 31, 33])
@pytest.mark.parametrize("drops,nodes,direct", [(3, 128, -1), (5, 64, 0), (16, 256, 0)])
def test_inner_operator(drops, nodes, direct, p):
    cfg = configs.small_drops(drops, nodes, box=6.0) if drops < 16 else configs.many_drops(drops, nodes)
    with Context(device=0, direct_max=direct, p32=p) as ctx:
        g = ctx.extractdat(cfg.nd, cfg.rku())
        rhs = np.ascontiguousarray(-0.5 * g["dz"] / g["dsda"]).view(np.float64).copy()
        x, info = ctx.solvei(rhs, "fp32_refined")[:2]
        # the residual that the solve reports is that of the FP64 operator; its own limit is 1e-10
        res = np.linalg.norm(rhs - ctx.fasmvp(x, "fp64")) / np.linalg.norm(rhs)
        assert res < 2e-10
