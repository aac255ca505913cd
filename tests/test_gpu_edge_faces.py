"""gE of the last column and gN of the last row are no faces of the grid: whatever a
caller's arrays hold there, every field is bit for bit the one with zeros there. Grids
that one cluster's shared memory holds from the finest level on, with half-rows that
fill their slots (a multiple of 8 columns: the next slot is another row's) and that
do not, and one whose finest level runs outside it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(8, 8), (16, 16), (17, 13), (64, 64), (40, 33), (130, 66)])
@pytest.mark.parametrize("prec", ["MG_FP32_FLEX", "MG_FP32", "MG_FP32_FLEX_DW", "MG_FP64", "batch"])
def test_edge_faces_are_not_read(ct, nx, ny, prec):
    layers = [ct.Layer("Si", 50e-6, 130.0, 1.66e6, 3, True), ct.Layer("bond", 10e-6, 2.0, 1.70e6, 1, False),
              ct.Layer("Cu", 1e-3, 400.0, 3.45e6, 4, False)]
    m = ct.build_model(layers, nx, ny, 10e-3, 10e-3 * ny / nx, 2e4, 0.0)
    m.P[:] = 1e-3 * np.random.default_rng(nx + ny).random(m.ncells())
    ct.finalize(m)

    def field():
        if prec == "batch":
            with ct.GpuBatch([m], precision=ct.Precision.MG_FP32_FLEX) as b:
                b.set_x_zero()
                b.set_rhs_steady()
                return b.solve(1e-10, 300)[0].iters, b.get_x(0)
        with ct.GpuPcg(m, ct.Precond.Multigrid, getattr(ct.Precision, prec)) as s:
            s.set_x_zero()
            s.set_rhs_steady()
            return s.solve(1e-10, 300).iters, s.get_x()

    it, T = field()
    for junk in (7.0, np.nan):
        m.gE.reshape(-1, ny, nx)[:, :, -1] = junk
        m.gN.reshape(-1, ny, nx)[:, -1, :] = junk
        jt, U = field()
        assert jt == it and np.array_equal(T, U)
