"""The fixed-point M2L's bounded wait for the tensor memory, run out in one team of a block, in the
other and in both: the call ends, its expansions are not finite, and the context works on. A
team that has issued products waits for them as ever (no products are issued without the wait)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("teams", [(0,), (1,), (0, 1)])
@pytest.mark.parametrize("df64", [-1, 1])
def test_wait_runs_out(gpu_ctx_factory, teams, df64):
    rng = np.random.default_rng(1)
    n = 30000  # more boxes than one round of the blocks; 3,072 are needed in double-float
    z = rng.uniform(-1, 1, n) + 1j * rng.uniform(-1, 1, n)
    q = rng.standard_normal(n) + 1j * rng.standard_normal(n)
    ctx = gpu_ctx_factory(leaf64=4, leaf_cap=8, df64=df64)
    limit = ctx._lib.eb_fx_lock_limit
    limit.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_longlong]
    good = ctx.dapif2(z, q)
    assert np.isfinite(good).all()
    for t in teams:
        assert limit(ctx._h, t, 0) == 0
    assert not np.isfinite(ctx.dapif2(z, q)).any()
    for t in teams:
        assert limit(ctx._h, t, 1 << 22) == 0
    assert np.array_equal(ctx.dapif2(z, q), good)
