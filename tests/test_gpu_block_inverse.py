"""The cell-wise inverses on both sides of the cell counts from which a warp
takes several cells (4096; 6000 at k = 5), with a last warp and a last block
that are not full, and their FP32 form on the multigrid levels."""
import numpy as np
import pytest
from test_gpu_levels import dev, vcycles

from atmospheric_flows_gb300.hill import HillParams, build_case
from oracle.oracle import OracleOperator

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,degree", [(65, 63, 1), (241, 17, 1), (241, 17, 2), (65, 63, 3),
                                          (241, 17, 3), (241, 17, 4), (241, 17, 5), (353, 17, 5)])
def test_inverse_of_many_cells(cuda_ok, nx, nz, degree):
    """A^{-1} b times A, applied by the operator that the oracle pins: b again,
    to the rounding of a solve (the condition of A is below 1e3)."""
    from atmospheric_flows_gb300.euler_operator import EULEROperator, MatrixFreeStorage

    case = build_case(HillParams(nx=nx, nz=nz, degree=degree, cfl=3.0))
    g = EULEROperator(MatrixFreeStorage.from_case(case), case.dt, case.Ma, case.Fr)
    rng = np.random.default_rng(6)
    rho = case.rho * (1 + 0.01 * rng.standard_normal(case.rho.shape))
    g.set_rho_for_fixed(dev(rho))
    for stage, n in ((3, 2), (1, 1)):  # A with rho_fix, the mass matrix
        g.set_NS_stage(stage)
        b = dev(rng.standard_normal(n * g.n_scalar))
        x, c = torch.full_like(b, float("nan")), torch.full_like(b, float("nan"))
        g.solve(x, b, 0.0)
        g.vmult(c, x)
        assert ((c - b).abs().max() / b.abs().max()).item() < 1e-11
    # and S, which holds A^{-1}, against the oracle
    pf = case.p * (1 + 0.01 * rng.standard_normal(case.p.shape))
    g.set_pres_fixed(dev(pf))
    g.set_NS_stage(2)
    o = OracleOperator(case)
    o.set_stage(1, 2)
    o.set_rho_for_fixed(rho)
    o.set_pres_fixed(pf)
    s = torch.full((g.n_scalar,), np.nan, dtype=torch.float64, device="cuda")
    g.vmult(s, dev(case.p))
    r = o.vmult(case.p)
    assert np.max(np.abs(s.cpu().numpy() - r)) < 1e-11 * np.max(np.abs(r))
    g.close()


@pytest.mark.parametrize("nx,nz,degree", [(68, 64, 1), (68, 64, 2), (68, 64, 3), (68, 64, 4),
                                          (100, 64, 5)])
def test_fp32_inverse_of_many_cells(cuda_ok, nx, nz, degree):
    """The FP32 V-cycle follows the FP64 one to FP32 rounding."""
    f, d = vcycles(nx, nz, degree)
    assert np.linalg.norm(f - d) < 1e-4 * np.linalg.norm(d)


@pytest.mark.parametrize("nx,nz,degree", [(188, 187, 1), (125, 125, 2), (75, 75, 4)])
def test_schur_with_face_integrals_of_their_own(cuda_ok, nx, nz, degree):
    """S just above 140,000 unknowns at the orders that no other test takes there."""
    from atmospheric_flows_gb300.euler_operator import EULEROperator, MatrixFreeStorage

    case = build_case(HillParams(nx=nx, nz=nz, degree=degree, cfl=3.0, periodic=nz != nx))
    assert 140000 <= case.rho.size < 142000
    g = EULEROperator(MatrixFreeStorage.from_case(case), case.dt, case.Ma, case.Fr)
    o = OracleOperator(case)
    rng = np.random.default_rng(7)
    rho, pf, p = (a * (1 + 0.01 * rng.standard_normal(a.shape)) for a in (case.rho, case.p, case.p))
    g.set_rho_for_fixed(dev(rho))
    g.set_pres_fixed(dev(pf))
    g.set_NS_stage(2)
    o.set_stage(1, 2)
    o.set_rho_for_fixed(rho)
    o.set_pres_fixed(pf)
    s = torch.full((g.n_scalar,), np.nan, dtype=torch.float64, device="cuda")
    g.vmult(s, dev(p))
    r = o.vmult(p)
    assert np.max(np.abs(s.cpu().numpy() - r)) < 1e-11 * np.max(np.abs(r))
    g.close()
