"""Tensor maps (the coarse end of the V-cycle, k_tail.cu; in device memory the batch's
staged sweeps', k_sweep_tma.cu) where solvers are built, solved and freed one after
another: stacks of several shapes with the same number of cells, so that arrays and
maps lie where another shape's lay. Every field is bit for bit the one that launches
without tensor maps give."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def stack(ct, nx, ny):
    layers = [ct.Layer("Si", 50e-6, 130.0, 1.66e6, 2, True), ct.Layer("bond", 10e-6, 2.0, 1.70e6, 1, False),
              ct.Layer("Cu", 1e-3, 400.0, 3.45e6, 3, False)]
    m = ct.build_model(layers, nx, ny, 10e-3, 10e-3 * ny / nx, 2e4, 0.0)
    m.P[:] = 1e-3 * np.random.default_rng(nx).random(m.ncells())
    ct.finalize(m)
    return m


SHAPES = [(64, 48), (48, 64), (96, 32)]


def test_single_solvers(ct, monkeypatch):
    ms = [stack(ct, nx, ny) for nx, ny in SHAPES]

    def field(m):
        with ct.GpuPcg(m, ct.Precond.Multigrid, ct.Precision.MG_FP32_FLEX) as s:
            s.set_x_zero()
            s.set_rhs_steady()
            assert s.solve(1e-10, 300).converged
            return s.get_x()

    monkeypatch.setenv("CT_SMALL_BYTES", "0")
    ref = [field(m) for m in ms]
    monkeypatch.delenv("CT_SMALL_BYTES")
    for _ in range(12):
        for m, T in zip(ms, ref):
            assert np.array_equal(field(m), T)


def test_batches(ct, monkeypatch):
    shapes = [(128, 64), (64, 128), (256, 32)]
    ms = [stack(ct, nx, ny) for nx, ny in shapes]

    def fields(k):
        three = [ms[(k + i) % 3] for i in range(3)]
        with ct.GpuBatch(three, precision=ct.Precision.MG_FP32_FLEX) as b:
            b.set_x_zero()
            b.set_rhs_steady()
            assert all(s.converged for s in b.solve(1e-10, 300))
            return [b.get_x(i) for i in range(3)]

    monkeypatch.setenv("CT_SWEEP_TMA", "0")
    ref = [fields(k) for k in range(3)]
    monkeypatch.delenv("CT_SWEEP_TMA")
    monkeypatch.setenv("CT_BATCH_TMA_TILES", "1")
    for _ in range(6):
        for k in range(3):
            for T, R in zip(fields(k), ref[k]):
                assert np.array_equal(T, R)
