"""The double-word batch's residual replacement where a block walks several tasks
(more tasks of rows than one wave of blocks, k_batch.cu): instances whose first phases
end in the same body, the last task of each shorter than the others,
bit for bit as in batches of one task a block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NX, NY, COUNT, PART = 12, 250, 24, 6  # 2 x 250 x 10 rows: 79 tasks of 64, the last of 8


def test_more_tasks_than_a_wave(ct):
    layers = [ct.Layer("Si", 50e-6, 130.0, 1.66e6, 4, True), ct.Layer("bond", 10e-6, 2.0, 1.70e6, 1, False),
              ct.Layer("Cu", 1e-3, 400.0, 3.45e6, 5, False)]
    m = ct.build_model(layers, NX, NY, 1e-3, 20e-3, 2e4, 0.0)
    ct.finalize(m)
    rng = np.random.default_rng(5)
    maps = [1e-3 * rng.random(m.ncells()) for _ in range(COUNT)]

    def fields(which):
        with ct.GpuBatch([m] * len(which)) as b:
            for i, k in enumerate(which):
                b.set_power(i, maps[k])
            b.set_x_zero()
            b.set_rhs_steady()
            st = b.solve(1e-10, 300)
            assert all(s.converged and not s.breakdown for s in st)
            return [(s.iters, s.relres, b.get_x(i)) for i, s in enumerate(st)]

    whole = fields(range(COUNT))
    parts = [f for k in range(0, COUNT, PART) for f in fields(range(k, k + PART))]
    for (it, rel, T), (jt, rrel, U) in zip(whole, parts):
        assert (it, rel) == (jt, rrel) and np.array_equal(T, U)
