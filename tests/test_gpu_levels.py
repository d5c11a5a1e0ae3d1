"""FP32 multigrid levels against FP64 ones where a kernel or a layout changes:
mapping degree 3 (the general kernels, A^{-1} as packed triangles) for every k."""
import numpy as np
import pytest

from atmospheric_flows_gb300.hill import HillParams, build_case, mg_hierarchy

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def vcycles(nx, nz, degree, mapping_degree=2):
    """The FP32 and the FP64 V-cycle of one right-hand side, as arrays."""
    from atmospheric_flows_gb300.euler_operator import EULEROperator, MatrixFreeStorage

    case = build_case(HillParams(nx=nx, nz=nz, degree=degree, cfl=5.0,
                                 mapping_degree=mapping_degree))
    op = EULEROperator(MatrixFreeStorage.from_case(case), case.dt, case.Ma, case.Fr)
    for level in mg_hierarchy(case.params, max_levels=3):
        op.add_mg_level(level)
    rng = np.random.default_rng(2)
    op.set_rho_for_fixed(dev(case.rho * (1 + 0.01 * rng.standard_normal(case.rho.shape))))
    op.set_pres_fixed(dev(case.p * (1 + 0.01 * rng.standard_normal(case.p.shape))))
    op.set_NS_stage(2)
    b = dev(rng.standard_normal(op.n_scalar))
    z = [torch.empty_like(b), torch.empty_like(b)]
    for i in (0, 1):
        op.mg_vcycle(z[i], b, i + 1)
    torch.cuda.synchronize()
    out = [a.cpu().numpy() for a in z]
    op.close()
    return out


@pytest.mark.parametrize("degree", [1, 2, 3, 5])
def test_general_fp32_levels(cuda_ok, degree):
    """The FP32 levels of a mapping of degree 3 see its degree-2 interpolant: a
    change of the preconditioner of up to a percent (the bar of k = 4)."""
    f, d = vcycles(32, 16, degree, mapping_degree=3)
    assert np.linalg.norm(f - d) < 1e-2 * np.linalg.norm(d)
