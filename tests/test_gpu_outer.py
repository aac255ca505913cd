"""The FP64 outer iteration on the V-cycle's z (k_az64, kb_az64): sums of float
products outside the fixed-point range take the plain FP64 chain."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def tsv_stack(ct, nx, ny):
    layers = [ct.Layer("Si", 50e-6, 130.0, 1.66e6, 2, True), ct.Layer("bond", 10e-6, 2.0, 1.70e6, 1, False),
              ct.Layer("Si 2", 50e-6, 130.0, 1.66e6, 1, True), ct.Layer("Cu", 1e-3, 400.0, 3.45e6, 3, False)]
    m = ct.build_model(layers, nx, ny, 10e-3, 10e-3 * ny / nx, 2e4, 0.0)
    ct.add_uniform_power(m, 0, 20.0)
    ct.add_power_block(m, 2, 1e-3, 1e-3, 2e-3, 3e-3, 10.0)
    ct.add_tsv_region(m, 1, 2e-3, 2e-3, 3e-3, 2e-3, 0.7)
    ct.finalize(m)
    return m


# Powers scaled by 2^k scale every field exactly, so only the FP64 sums' path
# differs (products under 2^-91 or over 2^122: the FP64 chain): the answers agree
# to rounding, here 1e-12 against 1e-16 times some tens of iterations' growth.
@pytest.mark.parametrize("k", [-104, -60, 60, 104])
@pytest.mark.parametrize("prec", ["MG_FP32_FLEX", "MG_FP32"])
@pytest.mark.parametrize("batch", [False, True])
def test_scaled_power(ct, k, prec, batch):
    if batch and prec != "MG_FP32_FLEX":
        pytest.skip("the batch solves in FLEX or double words")
    m = tsv_stack(ct, 45, 34)
    P, out = m.P.copy(), []
    for s in (1.0, 2.0 ** k):
        m.P[:] = P * s
        if batch:
            with ct.GpuBatch([m], precision=ct.Precision.MG_FP32_FLEX) as b:
                b.set_x_zero()
                b.set_rhs_steady()
                it, T = b.solve(1e-10, 200)[0].iters, b.get_x(0)
        else:
            with ct.GpuPcg(m, ct.Precond.Multigrid, getattr(ct.Precision, prec)) as g:
                g.set_x_zero()
                g.set_rhs_steady()
                it, T = g.solve(1e-10, 200).iters, g.get_x()
        out.append((it, T / s))
    assert out[0][0] == out[1][0]
    assert np.abs(out[1][1] - out[0][1]).max() <= 1e-12 * np.abs(out[0][1]).max()



# On a layered stack the six products of a cell often add up to a tie of the
# rounding to double, and A z is a small difference of large sums: a rounding
# that leans one way shows as 1e-12 in the field. Both modes solved to 1e-13 agree
# to the rounding of sums that do not lean: 1e-16 times the 1e3 of diagonal over
# row sum at the sink.
@pytest.mark.parametrize("batch", [False, True])
def test_layered_field_equals_fp64(ct, batch):
    import workloads
    m = workloads.steady_hotspot(96, seed=2)
    out = []
    for prec in ("MG_FP64", "MG_FP32_FLEX"):
        P = getattr(ct.Precision, prec)
        with ct.GpuBatch([m], precision=P) if batch and out else ct.GpuPcg(m, ct.Precond.Multigrid, P) as s:
            s.set_x_zero()
            s.set_rhs_steady()
            s.solve(1e-13, 300)
            out.append(s.get_x(0) if batch and out else s.get_x())
    assert np.abs(out[1] - out[0]).max() <= 2e-13 * np.abs(out[0]).max()


# A z in pairs of slots (FP64 V-cycle, double words) against the float form's cell
# a lane: one column to rows of a few slots, odd and even widths and heights of
# either parity, the third neighbour at both ends. Solved to 1e-12 the fields agree
# to rounding (1e-16 times the 1e3 of diagonal over row sum), ten times over for
# the iterations' sums.
@pytest.mark.parametrize("nx,ny", [(1, 1), (2, 3), (3, 2), (7, 5), (8, 4), (9, 6), (15, 16), (16, 15), (17, 18), (66, 33)])
def test_pairs_equal_cells(ct, nx, ny):
    m = tsv_stack(ct, nx, ny)
    out = []
    for prec in ("MG_FP32_FLEX", "MG_FP64", "MG_FP32_FLEX_DW", "batch"):
        if prec == "batch":
            with ct.GpuBatch([m], precision=ct.Precision.MG_FP32_FLEX_DW) as b:
                b.set_x_zero()
                b.set_rhs_steady()
                b.solve(1e-12, 200)
                out.append(b.get_x(0))
            continue
        with ct.GpuPcg(m, ct.Precond.Multigrid, getattr(ct.Precision, prec)) as s:
            s.set_x_zero()
            s.set_rhs_steady()
            s.solve(1e-12, 200)
            out.append(s.get_x())
    for T in out[1:]:
        assert np.abs(T - out[0]).max() <= 1e-12 * np.abs(out[0]).max()
