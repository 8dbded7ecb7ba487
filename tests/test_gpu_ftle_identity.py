"""FTLE of flow maps near the identity (short horizons, weak stretching), where the
logarithm takes the digits of the eigenvalue's distance from 1, with the two largest
eigenvalues apart and close together: one rounding of the exact value.

The Jacobian of every third cell of a 3 m x 3 x 3 lattice is set through its six
neighbours; its Cauchy-Green tensor in 32 bits is then known, and its eigenvalues
come from Jacobi rotations in 80 bits. Tolerance: half a unit in the last place of 32
bits (at most 2^-24 of the value); 2^-35 of it for the cells whose eigenvalue comes
from the closed form; and 16 roundings of 64 bits in an eigenvalue near 1, divided by
its logarithm."""
import numpy as np
import pytest

import dpa_b200
from dpa_b200 import Particles, estimate_ftle

pytestmark = pytest.mark.gpu


def _largest(C):
    """Largest eigenvalues of symmetric 3x3 matrices, cyclic Jacobi in 80 bits."""
    a = C.astype(np.longdouble)
    for _ in range(12):
        for p, q in ((0, 1), (0, 2), (1, 2)):
            apq = a[:, p, q]
            some = apq != 0
            with np.errstate(over="ignore"):  # nothing left to turn
                theta = (a[:, q, q] - a[:, p, p]) / np.where(some, 2 * apq, 1)
                t = np.where(theta >= 0, 1, -1) / (abs(theta) + np.sqrt(theta * theta + 1))
            t = np.where(some, t, 0)
            c = 1 / np.sqrt(t * t + 1)
            turn = np.zeros_like(a)
            turn[:, (0, 1, 2), (0, 1, 2)] = 1
            turn[:, p, p] = turn[:, q, q] = c
            turn[:, p, q], turn[:, q, p] = t * c, -t * c
            a = np.einsum("nji,njk,nkl->nil", turn, a, turn)
    return a[:, (0, 1, 2), (0, 1, 2)].max(1)


@pytest.mark.parametrize("close", [True, False])
@pytest.mark.parametrize("s", [1.0, 1e-2, 1e-3, 1e-4, 1e-5, 1e-6])
def test_ftle_near_the_identity(ctx, s, close):
    rng = np.random.default_rng(3)
    m = 4000
    turn = np.linalg.qr(rng.standard_normal((m, 3, 3)))[0]
    e = s * rng.standard_normal((m, 3))
    if close:
        e = s * np.stack([np.ones(m), 1 - 10.0 ** -rng.uniform(0, 4, m),
                          -rng.uniform(0.1, 2, m)], 1)
    J = (np.eye(3) + np.einsum("nij,nj,nkj->nik", turn, e, turn)).astype(np.float32)
    flow = np.zeros((m, 3, 3, 3, 3), np.float32)  # cell 3 k + i, j, l as [k, i, j, l]
    flow[:, 2, 1, 1], flow[:, 1, 2, 1], flow[:, 1, 1, 2] = J[..., 0], J[..., 1], J[..., 2]
    # A spacing of one half: the differences are divided by 1.
    grid = dpa_b200.RegularGrid.from_data(np.zeros((3 * m, 3, 3, 3), np.float32), (0.5, 0.5, 0.5))
    field = ctx.field(grid)
    n = 27 * m
    got = estimate_ftle(ctx, field, 50, (1, 1, 1), 0.1,
                        Particles(flow.reshape(n, 3), np.zeros(n, np.uint64),
                                  np.zeros((n, 3), np.float32)), "lattice").data
    field.close()
    got = got.reshape(m, 3, 3, 3)[:, 1, 1, 1]
    C = np.empty((m, 3, 3), np.float32)
    for r in range(3):
        for c in range(3):
            p = [J[:, k, r] * J[:, k, c] for k in range(3)]
            C[:, r, c] = p[0] + (p[1] + p[2])
    log = np.log(_largest(C))
    want = log / (2 * np.longdouble(abs(np.float32(0.1) * np.float32(50))))
    some = log != 0
    error = abs(got[some] / want[some] - 1)
    assert (error <= 2.0 ** -24 + 2.0 ** -35 + 16 * 2.0 ** -53 / abs(log[some])).all(), error.max()
    assert (got[~some] == 0).all()
