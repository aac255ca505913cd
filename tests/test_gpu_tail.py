"""The coarse end of the FP32 V-cycle in one thread-block cluster (k_tail.cu)
against the same levels as grid launches (CT_SMALL_BYTES=0), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stack(ct, nx, ny, cu_planes):
    """Si / bond / Si / TIM / Cu of 4 + cu_planes + 1 planes (1 and 2: Cu and Si
    alone), a TSV block, uneven power."""
    layers = [ct.Layer("Cu", 1e-3, 400.0, 3.45e6, max(1, cu_planes), False)]
    if cu_planes != 1:
        layers = [ct.Layer("Si", 50e-6, 130.0, 1.66e6, 1, True)] + layers
    if cu_planes > 1:
        layers = [ct.Layer("Si 2", 50e-6, 130.0, 1.66e6, 2, True),
                  ct.Layer("bond", 10e-6, 2.0, 1.70e6, 1, False)] + layers
    m = ct.build_model(layers, nx, ny, 10e-3, 10e-3 * ny / nx, 2e4, 0.0)
    rng = np.random.default_rng(nx * 1000 + ny)
    m.P[:] = 1e-3 * rng.uniform(0.0, 1.0, m.ncells()) * (rng.random(m.ncells()) < 0.3)
    if cu_planes > 1:
        ct.add_tsv_region(m, 1, 2e-3, 2e-3 * ny / nx, 3e-3, 3e-3 * ny / nx, 0.5)
    ct.finalize(m)
    return m


# one CTA alone; rows of one parent a CTA (odd first coarse rows); a bottom CTA
# of its own and one with rows; long and flat levels; every column-register
# form (4, 8, 10, 12, 14, 16, 24, 32 planes) at and below its size
@pytest.mark.parametrize("nx,ny,cu", [(1, 1, 6), (16, 16, 6), (17, 13, 6), (64, 64, 6), (50, 49, 6), (33, 63, 3),
                                      (65, 64, 8), (3, 200, 6), (200, 3, 6), (40, 37, 1), (37, 41, 0), (96, 43, 12),
                                      (60, 46, 9), (130, 66, 10), (48, 48, 16), (45, 30, 20), (64, 64, 28)])
@pytest.mark.parametrize("prec", ["MG_FP32_FLEX", "MG_FP32_FLEX_DW"])
def test_cluster_tail_bitwise(ct, nx, ny, cu, prec, monkeypatch):
    m = stack(ct, nx, ny, cu)
    out = []
    for flag in ("0", None):
        if flag is None:
            monkeypatch.delenv("CT_SMALL_BYTES", raising=False)
        else:
            monkeypatch.setenv("CT_SMALL_BYTES", flag)
        with ct.GpuPcg(m, ct.Precond.Multigrid, getattr(ct.Precision, prec)) as s:
            s.set_x_zero()
            s.set_rhs_steady()
            res = [s.solve(1e-10, 300).iters, s.get_x()]
            s.set_dt(1e-4)
            for _ in range(2):
                s.set_rhs_transient()
                res += [s.solve(1e-9, 300).iters, s.get_x()]
        out.append(res)
    for a, b in zip(*out):
        assert np.array_equal(a, b)
