"""Explicit right-hand sides on both sides of the cell count where the face
kernels change from a point to a face per thread (6000 cells, conforming
meshes), with a last block that is not full.  Single-operator bar: 1e-12 in the
max norm against the oracle."""
import numpy as np
import pytest

from atmospheric_flows_gb300.hill import HillParams, build_case
from oracle.oracle import OracleOperator

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,degree,periodic", [(103, 58, 1, True), (109, 55, 2, False),
                                                   (100, 60, 1, False), (97, 62, 2, True),
                                                   (101, 60, 3, False), (5, 3, 4, False)])
def test_rhs_on_both_routes(cuda_ok, nx, nz, degree, periodic):
    from atmospheric_flows_gb300.euler_operator import EULEROperator, MatrixFreeStorage

    case = build_case(HillParams(nx=nx, nz=nz, degree=degree, cfl=3.0, periodic=periodic))
    g = EULEROperator(MatrixFreeStorage.from_case(case), case.dt, case.Ma, case.Fr)
    o = OracleOperator(case)
    rng = np.random.default_rng(4)
    st = [(case.rho * (1 + 0.01 * rng.standard_normal(case.rho.shape)),
           case.u + 2.0 * rng.standard_normal(case.u.shape),
           case.p * (1 + 0.01 * rng.standard_normal(case.p.shape))) for _ in range(4)]
    for stage in (1, 2, 3):
        g.set_HYPERBOLIC_stage(stage)
        o.set_stage(stage, 1)
        for kind, (fn, ref) in enumerate([
                (g.vmult_rhs_rho_update, o.vmult_rhs_rho_update),
                (g.vmult_rhs_velocity_fixed, o.vmult_rhs_velocity_fixed),
                (g.vmult_rhs_pressure, o.vmult_rhs_pressure)]):
            src = []
            for j in range(stage):
                src += [st[j][0], st[j][1]] if kind == 0 else list(st[j])
            if kind == 1 and stage < 3:
                src.append(st[3][0])
            if kind == 2:
                src += [st[3][0], st[3][1]]
            dst = torch.full((g.n_scalar * (2 if kind == 1 else 1),), np.nan,
                             dtype=torch.float64, device="cuda")
            fn(dst, [torch.tensor(s, device="cuda") for s in src])
            r = ref(src)
            err = np.max(np.abs(dst.cpu().numpy() - r)) / np.max(np.abs(r))
            assert err < 1e-12, (stage, kind, err)
