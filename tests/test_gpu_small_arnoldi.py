"""The one-launch Arnoldi step of small systems (k_gm_step: a cluster of 16 blocks, a row per
thread, up to 8,192 rows) at its edges: fewer rows than blocks, odd counts, the last size it
takes and the first that the separate kernels keep, for both solves and modes, in the graphs
and in the host-driven loop. The true residual, recomputed with the FP64 operator, meets the
tolerance (1e-10, with 1e-12 for the estimate's own rounding), and the graph and the host loop
agree as in test_gpu_graph.py (1e-13 FP64, 1e-11 refined, of the largest value)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ellipse(n):
    t = 2 * np.pi * np.arange(n) / n
    z, z1, z2 = np.cos(t) + 0.8j * np.sin(t), -np.sin(t) + 0.8j * np.cos(t), -np.cos(t) - 0.8j * np.sin(t)
    s = np.abs(z1)
    return z, -z1, s, -(z1.conj() * z2).imag / s ** 3, np.array([0j])


def relmax(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


@pytest.mark.parametrize("n", [4, 9, 100, 513, 4095, 4096, 4097])
@pytest.mark.parametrize("mode", ["fp64", "fp32_refined"])
def test_sizes(gpu_ctx_factory, n, mode):
    z, dz, s, ka, zk = ellipse(n)
    got = []
    for graphs in (1, -1):
        ctx = gpu_ctx_factory(graphs=graphs, direct_max=0)
        ctx.set_geometry([n], z, dz, s, ka, zk)
        for b, solve, op in ((np.ascontiguousarray(-0.5 * dz / s).view(np.float64).copy(), ctx.solvei, ctx.fasmvp),
                             (-2.0 * z.real, ctx.solve_lapl, ctx.fasmvp_lap)):
            x, info = solve(b, mode)
            assert info["ierr"] == 0 and info["graph"] == (graphs == 1)
            assert np.linalg.norm(b - op(x)) <= (1e-10 + 1e-12) * np.linalg.norm(b)
            got.append((x, info["iters"]))
    for (xg, ig), (xe, ie) in zip(got[:2], got[2:]):
        assert ig == ie and relmax(xg, xe) < (1e-13 if mode == "fp64" else 1e-11)
