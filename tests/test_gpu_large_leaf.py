"""A leaf of more than 262,144 points: a cluster inside one box of the finest level, with two
points far away. Its points go through one P2M block (the far points' field) and pair with each
other. Fields at some points against direct sums, 1e-12 of the sum of the terms' moduli."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_cluster_in_one_box(gpu_ctx_factory):
    import torch

    n, rng = 262400, np.random.default_rng(1)
    side = 2.0 * (1.0 + 1e-9) / 2 ** 20  # of a box of level 20; one starts at the middle, 1 + i
    z = 1.0 + 1.0j + side * (rng.uniform(0.3, 0.7, n + 2) + 1j * rng.uniform(0.3, 0.7, n + 2))
    z[0], z[n + 1] = 0.0, 2.0 + 2.0j
    q = rng.standard_normal(n + 2) + 1j * rng.standard_normal(n + 2)
    zt, qt = torch.from_numpy(z).cuda(), torch.from_numpy(q).cuda()
    got = gpu_ctx_factory().dapif2(zt, qt)
    i = torch.tensor([0, 1, 2, n // 2, n, n + 1], device="cuda")
    d = zt[i][:, None] - zt[None, :]
    d[torch.arange(len(i)), i] = float("inf")
    ref, scale = (qt[None, :] / d).sum(1), (qt.abs()[None, :] / d.abs()).sum(1)
    assert float(((got[i] - ref).abs() / scale).max()) < 1e-12
