"""The FTLE kernel cell by cell against the same 32-bit Jacobian and Cauchy-Green
tensor formed by numpy, its eigenvalues taken in 64 bits. Tolerance: one rounding
to 32 bits (6e-8 relative) beside the closed form's 4e-12 in the eigenvalue, which
the logarithm halves and the horizon divides."""
import numpy as np
import pytest

import dpa_b200
from dpa_b200 import Particles, estimate_ftle
from bitwise import assert_same

pytestmark = pytest.mark.gpu


def _final(kind, x, rng):
    if kind == "identity":  # C = I: a triple eigenvalue
        return x.copy()
    if kind == "double":    # two equal largest eigenvalues
        return (x * np.float32([3.0, 3.0, 0.5])).astype(np.float32)
    if kind == "nearly":    # two largest eigenvalues 1e-9 to 1e-3 apart, turned in space
        turn = np.linalg.qr(rng.standard_normal((3, 3)))[0]
        near = 1.0 + 10.0 ** -rng.uniform(3, 9)
        return (x @ (turn * [2.0, 2.0 * near, 0.25])).astype(np.float32)
    if kind == "zero":      # every particle in one place
        return np.ones_like(x)
    out = (x + rng.standard_normal(x.shape) * rng.choice([1e-3, 1.0, 30.0])).astype(np.float32)
    if kind == "not finite":
        bad = rng.integers(0, len(x), max(1, len(x) // 9))
        out[bad, rng.integers(0, 3, len(bad))] = rng.choice([np.inf, -np.inf, np.nan, 3e38],
                                                            len(bad))
    return out


@pytest.mark.parametrize("spacing", [(0.7, 1.0, 0.3), (1e-9, 0.7, 1e9)])
@pytest.mark.parametrize("shape", [(1, 1, 1), (2, 1, 5), (7, 3, 33), (16, 13, 129)])
@pytest.mark.parametrize("kind", ["identity", "double", "nearly", "zero", "noise", "not finite"])
def test_ftle_cells(ctx, kind, shape, spacing):
    rng = np.random.default_rng(sum(shape))
    grid = dpa_b200.RegularGrid.from_data(np.zeros(shape + (3,), np.float32), spacing)
    field = ctx.field(grid)
    i = np.stack(np.meshgrid(*map(np.arange, shape), indexing="ij"), -1).reshape(-1, 3)
    x = (i.astype(np.float32) * grid.spacing).astype(np.float32)
    final = _final(kind, x, rng)
    got = estimate_ftle(ctx, field, 50, (1, 1, 1), 0.1,
                        Particles(final, np.zeros(len(x), np.uint64), x), "lattice").data
    field.close()
    flow = final.reshape(shape + (3,))
    with np.errstate(all="ignore"):
        J = np.empty(shape + (3, 3), np.float32)
        for d in range(3):
            at = np.arange(shape[d])
            J[..., d] = (np.take(flow, np.minimum(at + 1, shape[d] - 1), d)
                         - np.take(flow, np.maximum(at - 1, 0), d)) \
                / (np.float32(2) * grid.spacing[d])
        C = np.empty_like(J)
        for r in range(3):
            for c in range(3):
                p = [J[..., k, r] * J[..., k, c] for k in range(3)]
                C[..., r, c] = p[0] + (p[1] + p[2])
        plain = np.isfinite(C).all((-1, -2))
        top = np.linalg.eigvalsh(np.where(plain[..., None, None], C, 0).astype(np.float64))[..., 2]
        top = np.maximum(top, 0.0)
        T = float(abs(np.float32(0.1) * np.float32(50)))
        want = np.log(np.sqrt(top)) / T
    if kind != "not finite":
        assert plain.all()
    assert_same(np.isneginf(got[plain]), np.isneginf(want[plain]))
    fine = plain & np.isfinite(want)
    np.testing.assert_allclose(got[fine], want[fine], rtol=1.2e-7, atol=4e-12)
    assert not np.isfinite(got[~plain]).any()  # infinite or NaN, never a plain number
