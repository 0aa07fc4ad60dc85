"""The tree build at the sizes where its kernels change: blocks of 256 points, the sort of one
cluster (up to 65,536 points, 1 to 4 rounds of 16 x 1,024) and the one above, levels of one
box and of many, coincident points. Every pair is covered exactly once whatever the
tree, so the sums are those over all pairs: 1e-12 of the largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 17, 255, 256, 257, 1025, 4096, 16384, 16385, 32769, 65535, 65536, 65537])
@pytest.mark.parametrize("spread", ["even", "scales", "two_spots"])
def test_all_pairs_once(gpu_ctx_factory, n, spread):
    rng = np.random.default_rng(n)
    z = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)
    if spread == "scales":
        z = z * 10.0 ** -rng.uniform(0, 4, n)
    if spread == "two_spots":
        z = 1e-3 * z + np.where(np.arange(n) % 2, 1.0, -1.0 - 0.5j)
    q = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    ctx = gpu_ctx_factory(leaf64=8, leaf_cap=24) if n < 4096 else gpu_ctx_factory()
    got = ctx.dapif2(z, q)
    i = np.unique(np.concatenate([[0, n - 1], rng.integers(0, n, 64)]))
    d = z[i][:, None] - z[None, :]
    d[np.arange(len(i)), i] = np.inf
    ref = (q[None, :] / d).sum(1)
    assert np.abs(got[i] - ref).max() < 1e-12 * np.abs(got).max()


def test_sort_is_stable(gpu_ctx_factory):
    """Many equal keys (points closer than the finest cells): the same results on each call."""
    rng = np.random.default_rng(1)
    n = 20000
    z = np.round(rng.uniform(-1, 1, n), 2) + 1e-12 * rng.standard_normal(n) + 1j * np.round(rng.uniform(-1, 1, n), 2)
    q = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    a = [gpu_ctx_factory().dapif2(z, q) for _ in range(2)]
    assert np.isfinite(a[0]).all() and np.array_equal(a[0], a[1])
