"""The double-float near field's offsets across a leaf boundary. Two nodes D = 2^-14 leaf sides apart
in neighbouring leaves sit near +1/2 and -1/2 of theirs: their offsets, each within 2^-54 of a
side, differ by D after the index offset of the leaves, so that 1 / D is within 2^-53 / D = 2^-39
(and the pair's double-float arithmetic, 2^-43). The square's side is one whose rounded
reciprocal is almost 2^-53 off: an offset formed with it alone misses the bound."""
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def side():
    """The nodes' extent s in [1, 2) and the square's side W for it, the worst of some."""
    rng = np.random.default_rng(1)
    best = (0.0, None, None)
    for s in rng.uniform(1, 2, 2000):
        W = s * (1.0 + 1e-9)
        off = abs(float(Fraction(1.0 / W) * Fraction(W) - 1))
        best = max(best, (off, s, W))
    assert best[0] > 0.9 * 2.0 ** -53
    return best[1:]


@pytest.mark.parametrize("along", ["x", "y"])
def test_pairs_across_boundaries(gpu_ctx_factory, along):
    s, W = side()
    rng = np.random.default_rng(2)
    x0, r, D, m = 0.5 * s - 0.5 * W, W / 32, 2.0 ** -14, 32
    col, row = (a.ravel() for a in np.meshgrid(np.arange(1, m), np.arange(m)))
    a = rng.uniform(0.05, 0.95, col.size)
    x = x0 + np.concatenate([(col - a * D) * r, (col + (1 - a) * D) * r])
    y = np.tile(x0 + (row + rng.uniform(0.1, 0.9, row.size)) * r, 2)
    z = np.concatenate([[0.0, s * (1 + 1j)], x + 1j * y])
    if along == "y":
        z = z.imag + 1j * z.real
    q = np.ones(z.size, complex)
    ctx = gpu_ctx_factory(leaf64=2, leaf_cap=4, df64=1)
    got = ctx.dapif2(z, q)
    d = z[:, None] - z[None, :]
    np.fill_diagonal(d, np.inf)
    ref = (1.0 / d).sum(1)
    err = np.abs(got - ref)[2:] / np.abs(ref)[2:]
    assert np.abs(ref[2:]).min() > 0.9 / (D * r)  # the pair's term carries the sum
    assert err.max() < 2.0 ** -39 + 2.0 ** -43
