"""The admission estimate of a member covers the device memory that it takes, and
not much more."""
import ctypes

import pytest

from atmospheric_flows_gb300.hill import HillParams, build_case, mg_hierarchy
from atmospheric_flows_gb300.serving import member_bytes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("nx,nz,degree,mapping_degree", [(160, 80, 4, 2), (128, 64, 5, 2),
                                                         (160, 80, 3, 3)])
def test_estimate_covers_what_a_member_takes(cuda_ok, nx, nz, degree, mapping_degree, precision):
    from atmospheric_flows_gb300 import _lib
    from atmospheric_flows_gb300.euler_solver import EulerSolver

    def free():
        f, t = ctypes.c_double(), ctypes.c_double()
        torch.cuda.synchronize()
        assert _lib.load().atm_device_memory(ctypes.byref(f), ctypes.byref(t)) == 0
        return f.value

    p = HillParams(nx=nx, nz=nz, degree=degree, mapping_degree=mapping_degree, cfl=5.0)
    case = build_case(p)
    levels = mg_hierarchy(p, max_levels=3) if precision else None
    kw = dict(levels=levels, precision=precision) if precision else {}
    EulerSolver(case, eps=1e-8, **kw).run(1)  # modules and graphs are loaded
    before = free()
    s = EulerSolver(case, eps=1e-8, **kw)
    s.run(1)
    used = before - free()
    estimate = member_bytes(p, precision)
    assert used <= estimate < 1.4 * used + (32 << 20), (used, estimate)
    s.close()
