"""Kernels that load ahead of the wait for the preceding kernel give the bits of
kernels that each start after the one before (CT_PDL=0), which is read once a
process: fields of cold and warm solves, with new operators between them, hashed in a
child process for each setting."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CHILD = """
import sys, hashlib
sys.path[:0] = [sys.argv[1]]
import numpy as np
import cthermal as ct, workloads
h = hashlib.sha1()
if sys.argv[2] == "batch":
    sp = workloads.batch_instance_specs(6, 7)
    for prec in (ct.Precision.MG_FP32_FLEX, ct.Precision.MG_FP32_FLEX_DW):
        with ct.GpuBatch.from_specs([c for c, _, _ in sp], [a for _, a, _ in sp], [a for _, _, a in sp],
                                    precision=prec) as b:
            for _ in range(2):
                b.set_x_zero()
                b.set_rhs_steady()
                b.solve(1e-10, 300)
            for i in range(len(b)):
                h.update(np.ascontiguousarray(b.get_x(i)).tobytes())
else:
    for n in (66, 129, 203, 300):
        with ct.GpuPcg(workloads.steady_hotspot(n, seed=n), ct.Precond.Multigrid,
                       getattr(ct.Precision, sys.argv[2])) as s:
            for k in range(4):
                s.set_dt(0.0)
                s.set_x_zero()
                s.set_rhs_steady()
                s.solve(1e-10, 300)
                h.update(np.ascontiguousarray(s.get_x()).tobytes())
                s.set_dt(1e-5 * 3.0 ** k)
                s.set_rhs_transient()
                s.solve(1e-9, 300)
                h.update(np.ascontiguousarray(s.get_x()).tobytes())
print(h.hexdigest())
"""


@pytest.mark.parametrize("what", ["MG_FP32_FLEX", "MG_FP64", "MG_FP32_FLEX_DW", "batch"])
def test_early_loads_bitwise(ct, what):
    pkg = os.path.dirname(ct.__file__)
    out = []
    for pdl in ("0", "1"):
        r = subprocess.run([sys.executable, "-c", CHILD, pkg, what], env=dict(os.environ, CT_PDL=pdl),
                           capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        out.append(r.stdout.split()[-1])
    assert out[0] == out[1]
