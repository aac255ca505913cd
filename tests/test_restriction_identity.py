"""What the V-cycle restricts: after red columns are solved from x = 0 and black
ones with the red x beside them, the full residual b - (A + C/dt) x is zero at the
black cells and the lateral terms of the black x at the red ones (mg_dev.cuh,
restrict_sum). In FP64, against the full residual, one-column grids to odd ones."""
import numpy as np
import pytest


@pytest.mark.parametrize("nx,ny,nz", [(1, 1, 3), (2, 1, 3), (1, 5, 2), (4, 4, 1), (5, 4, 6), (7, 9, 10)])
def test_residual_after_red_and_black(nx, ny, nz):
    rng = np.random.default_rng(nx * 100 + ny * 10 + nz)
    gE, gN, gU = (rng.uniform(0.1, 1.0, (nz, ny, nx)) for _ in range(3))
    gU *= 1e4
    gE[:, :, -1] = 0.0
    gN[:, -1, :] = 0.0
    cap = rng.uniform(0.0, 2.0, (nz, ny, nx))
    b = rng.standard_normal((nz, ny, nx))

    def lateral(x):
        s = np.zeros_like(x)
        s[:, :, 1:] += gE[:, :, :-1] * x[:, :, :-1]
        s[:, :, :-1] += gE[:, :, :-1] * x[:, :, 1:]
        s[:, 1:, :] += gN[:, :-1, :] * x[:, :-1, :]
        s[:, :-1, :] += gN[:, :-1, :] * x[:, 1:, :]
        return s

    one = np.ones_like(b)
    diag = lateral(one) + gU + cap  # the last gU is the sink's
    diag[1:] += gU[:-1]

    def vertical(x):
        s = np.zeros_like(x)
        s[1:] += gU[:-1] * x[:-1]
        s[:-1] += gU[:-1] * x[1:]
        return s

    colour = (np.arange(nx)[None, :] + np.arange(ny)[:, None]) % 2
    x = np.zeros_like(b)
    for c in (0, 1):
        rhs = b + lateral(x)
        for j, i in zip(*np.nonzero(colour == c)):
            m = np.diag(diag[:, j, i]) - np.diag(gU[:-1, j, i], 1) - np.diag(gU[:-1, j, i], -1)
            x[:, j, i] = np.linalg.solve(m, rhs[:, j, i])
    full = b - (diag * x - vertical(x) - lateral(x))
    red = np.broadcast_to(colour == 0, full.shape)
    black_only = np.where(red, 0.0, x)
    # rounding of the solves and of the sum: 1e-16 of the largest term, tens of times
    tol = 1e-14 * np.abs(diag * x).max()
    assert np.abs(full[~red]).max(initial=0.0) <= tol
    assert np.abs(full - lateral(black_only))[red].max() <= tol
