"""Explicit right-hand sides on the routes of large meshes: a face per thread
at k = 4 and 5 (6000 cells and more) and with hanging faces (12,000 cells and
more), and the sizes just below.  1e-12 in the max norm against the oracle."""
import numpy as np
import pytest

from atmospheric_flows_gb300.hill import HillParams, build_case
from oracle.oracle import OracleOperator

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,degree,adaptive", [
    (101, 60, 4, False), (97, 62, 5, False), (107, 57, 4, False), (24, 12, 4, True),
    (110, 81, 3, True), (110, 81, 2, True), (111, 81, 4, True)])
def test_rhs_of_large_meshes(cuda_ok, nx, nz, degree, adaptive):
    from atmospheric_flows_gb300 import amr
    from atmospheric_flows_gb300.euler_operator import EULEROperator, MatrixFreeStorage

    p = HillParams(nx=nx, nz=nz, degree=degree, cfl=3.0, periodic=(nx + nz) % 2 == 1)
    if adaptive:
        tree = amr.example_tree(nx, nz, p.periodic)
        if nx > 100:
            tree.refine([(0, i, j) for i in range(30, 70) for j in range(10, 40)])
            tree.balance()
        case = amr.adaptive_case(p, tree)
        assert nx < 100 or case.n_cells > 12000
        assert np.any(case.inner_faces[:, 4] > 0)
    else:
        case = build_case(p)
    g = EULEROperator(MatrixFreeStorage.from_case(case), case.dt, case.Ma, case.Fr)
    o = OracleOperator(case)
    rng = np.random.default_rng(9)
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
    g.close()
