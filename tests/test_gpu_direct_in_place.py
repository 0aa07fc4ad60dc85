"""Direct sums that form their charges in place (small problems) against the oracle, at the
sizes where that ends and with one and several drops, and with the result written over the
density, where the charges' kernels run first. 1e-12 of the largest value, as in the other FP64
parity tests."""
import numpy as np
import pytest

from electricbubbles_gb300 import configs

pytestmark = pytest.mark.gpu


def relmax(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("drops,nodes", [(1, 4), (1, 128), (2, 128), (1, 256), (5, 64), (11, 32), (12, 32), (4, 128), (5, 128), (1, 1024)])
@pytest.mark.parametrize("over", [False, True])
def test_operators(gpu_ctx_factory, oracle, drops, nodes, over):
    torch = pytest.importorskip("torch")
    cfg = configs.small_drops(drops, nodes, box=8.0) if drops > 1 else configs.single_drop(nodes)
    ex = oracle.extractdat(cfg.nd, cfg.rku())
    g = oracle.Geometry.from_extract(cfg.nd, ex)
    rng = np.random.default_rng(nodes)
    w = rng.standard_normal(2 * cfg.nbk)
    ctx = gpu_ctx_factory(direct_max=0)  # (the default: direct sums up to 1,024 points)
    ctx.set_geometry(cfg.nd, ex["z"], ex["dz"], ex["dsda"], ex["kappa"], ex["zk"])
    for op, x, ref in ((ctx.fasmvp, w, oracle.fasmvp(g, w, 0)),
                       (ctx.fasmvp_lap, w[:cfg.nbk], np.asarray(oracle.fasmvp_lap(g, w[:cfg.nbk]))[:cfg.nbk])):
        t = torch.from_numpy(x.copy()).cuda()
        y = op(t, "fp64", out=t if over else torch.empty_like(t))
        torch.cuda.synchronize()
        assert relmax((t if over else y).cpu().numpy(), ref) < 1e-12
