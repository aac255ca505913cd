"""The batch's grid sweeps with a thread a column and plane (kb_sweep_split, forced on
every depth by CT_BATCH_SPLIT=1; the tuner takes it where it is the fastest) against
those with a thread a column (CT_BATCH_TILE=512), bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stack(ct, nx, ny, planes):
    layers = [ct.Layer("Si", 50e-6, 130.0, 1.66e6, 1, True), ct.Layer("bond", 10e-6, 2.0, 1.70e6, 1, False),
              ct.Layer("Cu", 1e-3, 400.0, 3.45e6, planes - 2, False)]
    m = ct.build_model(layers, nx, ny, 10e-3, 10e-3 * ny / nx, 2e4, 0.0)
    m.P[:] = 1e-3 * np.random.default_rng(nx * ny + planes).random(m.ncells())
    ct.finalize(m)
    return m


# odd rows and columns, half-rows that fill their slots and that do not, tasks whose
# last blocks are empty (a tile is eight blocks of 32 columns), stacks of fewer planes
# than the bucket's deepest beside it, each plane-count form (8, 12, 16, 32) below and
# at its size
@pytest.mark.parametrize("planes", [7, 8, 11, 12, 15, 16, 21, 32])
@pytest.mark.parametrize("prec", ["MG_FP32_FLEX", "MG_FP32_FLEX_DW"])
def test_split_sweeps_bitwise(ct, planes, prec, monkeypatch):
    ms = [stack(ct, nx, ny, p) for nx, ny, p in ((45, 34, planes), (130, 66, planes - 3), (128, 65, 3), (61, 203, planes),
                                                 (97, 96, planes - 1), (17, 150, planes))]
    monkeypatch.setenv("CT_SWEEP_TMA", "0")
    out = []
    for name, value, other in (("CT_BATCH_TILE", "512", "CT_BATCH_SPLIT"), ("CT_BATCH_SPLIT", "1", "CT_BATCH_TILE")):
        monkeypatch.setenv(name, value)
        monkeypatch.delenv(other, raising=False)
        with ct.GpuBatch(ms, precision=getattr(ct.Precision, prec)) as b:
            tiles = {t for k in b.buckets() for t in k["sweep_tiles"]}
            assert tiles == {512 if name == "CT_BATCH_TILE" else 256}
            b.set_x_zero()
            b.set_rhs_steady()
            res = [s.iters for s in b.solve(1e-10, 300)] + [b.get_x(i) for i in range(len(ms))]
            b.step_transient([1e-4] * len(ms), 1e-9, 300)
            out.append(res + [b.get_x(i) for i in range(len(ms))])
    for a, c in zip(*out):
        assert np.array_equal(a, c)


def test_split_sweeps_early_loads(ct, monkeypatch):
    """The loads ahead of the wait, as test_gpu_early_loads has them, with the form
    that has them on every depth."""
    import test_gpu_early_loads
    monkeypatch.setenv("CT_BATCH_SPLIT", "1")
    monkeypatch.setenv("CT_SWEEP_TMA", "0")
    test_gpu_early_loads.test_early_loads_bitwise(ct, "batch")
