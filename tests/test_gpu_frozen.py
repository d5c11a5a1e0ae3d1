"""Setting p_fix and rho_fix copies them: what the caller does with its vectors
afterwards changes nothing.  Bars of the single operators against the oracle."""
import numpy as np
import pytest

from atmospheric_flows_gb300.hill import HillParams, build_case
from oracle.oracle import OracleOperator

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("adaptive,mapping_degree", [(False, 2), (True, 2), (False, 3)])
@pytest.mark.parametrize("degree", [1, 2, 3, 4, 5])
def test_frozen_fields_are_copies(cuda_ok, degree, adaptive, mapping_degree):
    from atmospheric_flows_gb300 import amr
    from atmospheric_flows_gb300.euler_operator import EULEROperator, MatrixFreeStorage

    p = HillParams(nx=9, nz=5, degree=degree, cfl=3.0, mapping_degree=mapping_degree)
    case = amr.adaptive_case(p, amr.example_tree(9, 5, True)) if adaptive else build_case(p)
    rng = np.random.default_rng(8)
    rho = case.rho * (1 + 0.01 * rng.standard_normal(case.rho.shape))
    pf = case.p * (1 + 0.01 * rng.standard_normal(case.p.shape))
    w = case.u + rng.standard_normal(case.u.shape)
    g = EULEROperator(MatrixFreeStorage.from_case(case), case.dt, case.Ma, case.Fr)
    o = OracleOperator(case)
    a, b = dev(rho), dev(pf)
    g.set_rho_for_fixed(a)
    g.set_pres_fixed(b)
    a.fill_(float("nan"))
    b.fill_(float("nan"))
    o.set_stage(1, 2)
    o.set_rho_for_fixed(rho)
    o.set_pres_fixed(pf)
    g.set_NS_stage(2)
    s = torch.empty(g.n_scalar, dtype=torch.float64, device="cuda")
    for fn, ref, x, bar in ((g.vmult_enthalpy, o.vmult_enthalpy, w, 1e-12),
                            (g.vmult, o.vmult, case.p, 1e-11)):
        fn(s, dev(x))
        r = ref(x)
        assert np.max(np.abs(s.cpu().numpy() - r)) < bar * np.max(np.abs(r))
    g.close()


@pytest.mark.parametrize("nx,nz,degree", [(40, 20, 2), (96, 50, 4), (160, 80, 3)])
def test_apply_directly_behind_a_rebuild(cuda_ok, nx, nz, degree):
    """S launched right behind new frozen fields, and behind each other, gives
    the bits of the same calls with the device idle in between."""
    from atmospheric_flows_gb300.euler_operator import EULEROperator, MatrixFreeStorage

    case = build_case(HillParams(nx=nx, nz=nz, degree=degree, cfl=3.0))
    g = EULEROperator(MatrixFreeStorage.from_case(case), case.dt, case.Ma, case.Fr)
    g.set_NS_stage(2)
    rng = np.random.default_rng(12)
    field = lambda a: dev(a * (1 + 0.01 * rng.standard_normal(a.shape)))  # noqa: E731
    sets = [(field(case.rho), field(case.p), field(case.p)) for _ in range(3)]
    out = [torch.empty(2, g.n_scalar, dtype=torch.float64, device="cuda") for _ in sets]

    def run(wait):
        for (rho, p, x), s in zip(sets, out):
            g.set_rho_for_fixed(rho)
            wait()
            g.set_pres_fixed(p)
            wait()
            g.vmult(s[0], x)
            wait()
            g.vmult(s[1], s[0])
            wait()

    run(torch.cuda.synchronize)
    ref = [s.clone() for s in out]
    for _ in range(20):
        for s in out:
            s.fill_(float("nan"))
        run(lambda: None)
        torch.cuda.synchronize()
        for s, r in zip(out, ref):
            assert torch.equal(s, r)
    g.close()
