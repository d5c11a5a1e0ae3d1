"""Kernels that read a tuned block shape differently have their own entries in the
autotuner's table: the general kernels (mapping degree >= 3) beside those of
degree <= 2, and C/D of large meshes (face integrals from a kernel of its own)."""
import numpy as np
import pytest

from atmospheric_flows_gb300 import _lib
from atmospheric_flows_gb300.hill import HillParams, build_case

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def families(nx, nz, degree, mapping_degree):
    from atmospheric_flows_gb300.euler_operator import EULEROperator, MatrixFreeStorage

    case = build_case(HillParams(nx=nx, nz=nz, degree=degree, cfl=3.0,
                                 mapping_degree=mapping_degree))
    op = EULEROperator(MatrixFreeStorage.from_case(case), case.dt, case.Ma, case.Fr)
    rho, u, p = (torch.tensor(np.ascontiguousarray(a), device="cuda")
                 for a in (case.rho, case.u, case.p))
    op.set_rho_for_fixed(rho)
    op.set_pres_fixed(p)
    op.set_NS_stage(2)
    s = torch.empty_like(p)
    op.vmult(s, p)
    op.vmult_rhs_rho_update(s, [rho, u])
    torch.cuda.synchronize()
    op.close()
    log2 = int(np.log2(nx * nz))
    return {r["family"] for r in _lib.autotune_table()
            if r["degree"] == degree and r["log2_cells"] == log2 and r["bytes"] == 8}


def test_families(cuda_ok):
    assert {"B", "CD", "rhs_rho"} <= families(52, 41, 2, 2)
    assert {"B_general", "CD_general", "rhs_rho_general"} <= families(52, 41, 2, 3)
    assert {"B", "CD_faces"} <= families(75, 52, 5, 2)  # 140,400 unknowns
