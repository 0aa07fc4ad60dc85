"""The FP64 near field on trees with many W lists, where a block takes half a tile: leaves of one
point (an empty half), of odd and even sizes around half a tile, and of several tiles, for the four
pair forms (FASMVP, FASMVP_LAP and their transposes). Against the direct sums of the same
operators, 1e-12 of the largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf", [(8, 1), (8, 3), (40, 17), (60, 33), (90, 64)])
@pytest.mark.parametrize("n", [400, 1999])
def test_halves(gpu_ctx_factory, n, leaf):
    rng = np.random.default_rng(n)
    z = (rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)) * 10.0 ** -rng.uniform(0, 3, n)
    dz = np.sqrt(n) * (rng.standard_normal(n) + 1j * rng.standard_normal(n))
    geometry = ([n], z, dz, np.ones(n), np.zeros(n), np.array([50.0 + 50.0j]))
    fmm = gpu_ctx_factory(leaf64=leaf[0], leaf_cap=leaf[1])
    direct = gpu_ctx_factory(direct_max=4096)
    for c in (fmm, direct):
        c.set_geometry(*geometry)
    assert fmm.tree_info()["w_pairs"] > n // 8
    for name in ("fasmvp", "fasmvp_lap", "fasmvp_adjoint", "fasmvp_lap_adjoint"):
        x = rng.standard_normal(n if "lap" in name else 2 * n)
        a, b = getattr(fmm, name)(x), getattr(direct, name)(x)
        assert np.abs(a - b).max() < 1e-12 * np.abs(b).max(), name
