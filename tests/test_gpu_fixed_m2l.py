"""The fixed-point M2L of the FP64-class operators at the edges of its work split: expansion
orders up to the last it takes (47) and the first that the CUDA-core kernel keeps (48),
lists of 0 to 27 entries (a few boxes, a dense cloud, a ring), multipoles of very different
sizes, zeros and non-finite ones. Against the oracle's direct sums, 1e-12 of the largest
value where the order truncates below it; the cut orders against the same order in
double-float with the CUDA-core kernel (its truncation, its arithmetic within 1e-11)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def relmax(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


CLOUDS = {
    "cloud": lambda rng: rng.uniform(-1, 1, 3000) + 1j * rng.uniform(-1, 1, 3000),
    "ring": lambda rng: np.exp(2j * np.pi * rng.uniform(0, 1, 2000)),
    "corners": lambda rng: np.concatenate([c + 1e-3 * (rng.uniform(-1, 1, 40) + 1j * rng.uniform(-1, 1, 40))
                                           for c in (0, 1, 1j, 1 + 1j)]),
}


@pytest.mark.parametrize("cloud", list(CLOUDS))
@pytest.mark.parametrize("p64", [44, 46, 47, 48])
def test_orders(gpu_ctx_factory, oracle, cloud, p64):
    rng = np.random.default_rng(1)
    z = CLOUDS[cloud](rng)
    q = rng.standard_normal(z.size) + 1j * rng.standard_normal(z.size)
    ctx = gpu_ctx_factory(p64=p64, leaf64=8, leaf_cap=16)
    assert relmax(ctx.dapif2(z, q), oracle.cauchy_direct(z, z, q, True)) < 1e-12


@pytest.mark.parametrize("p64", [2, 9, 24])
def test_low_orders(gpu_ctx_factory, p64):
    rng = np.random.default_rng(2)
    z = CLOUDS["cloud"](rng)
    q = rng.standard_normal(z.size) + 1j * rng.standard_normal(z.size)
    got = [gpu_ctx_factory(p64=p64, leaf64=8, leaf_cap=16, df64=df).dapif2(z, q) for df in (-1, 1)]
    assert relmax(got[0], got[1]) < 1e-11


def test_scales(gpu_ctx_factory, oracle):
    """Charges from 1e-150 to 1e150 next to each other: each region's field is held to its
    own size (the regions are far apart, so the large ones' error must stay theirs)."""
    rng = np.random.default_rng(3)
    n = 600
    z = np.concatenate([50.0 * c + rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n) for c in range(3)])
    q = rng.standard_normal(3 * n) + 1j * rng.standard_normal(3 * n)
    for scale in (1e-150, 1e150):
        got = gpu_ctx_factory(leaf64=8, leaf_cap=16).dapif2(z, scale * q)
        assert relmax(got, scale * oracle.cauchy_direct(z, z, q, True)) < 1e-12
    zero = gpu_ctx_factory(leaf64=8, leaf_cap=16).dapif2(z, 0 * q)
    assert np.abs(zero).max() == 0.0


def test_non_finite(gpu_ctx_factory):
    rng = np.random.default_rng(4)
    z = CLOUDS["cloud"](rng)
    q = rng.standard_normal(z.size) + 0j
    q[5] = np.inf
    got = gpu_ctx_factory(leaf64=8, leaf_cap=16).dapif2(z, q)
    assert not np.isfinite(np.delete(got, 5)).any()
