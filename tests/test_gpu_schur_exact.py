"""The Schur kernels at the points where their launch or their route changes:
cell counts around the blocks' multiples of eight, every degree, mappings of
degree 1 and 2 (the kernels with exact point sets) and 3 (the general ones).

Oracle comparisons use the single-operator bar of 1e-12 in the max norm; S
compounds B, an exact inverse and C, and takes 1e-11."""
import numpy as np
import pytest

from atmospheric_flows_gb300.hill import HillParams, build_case
from oracle.oracle import OracleOperator

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def rel(a, b):
    return np.max(np.abs(a.cpu().numpy() - b)) / np.max(np.abs(b))


def operators(case, seed=5):
    from atmospheric_flows_gb300.euler_operator import EULEROperator, MatrixFreeStorage

    rng = np.random.default_rng(seed)
    g = EULEROperator(MatrixFreeStorage.from_case(case), case.dt, case.Ma, case.Fr)
    o = OracleOperator(case)
    rho = case.rho * (1 + 0.01 * rng.standard_normal(case.rho.shape))
    pf = case.p * (1 + 0.01 * rng.standard_normal(case.p.shape))
    g.set_rho_for_fixed(dev(rho))
    g.set_pres_fixed(dev(pf))
    g.set_NS_stage(2)
    o.set_stage(1, 2)
    o.set_rho_for_fixed(rho)
    o.set_pres_fixed(pf)
    return g, o, rng


@pytest.mark.parametrize("mapping_degree", [1, 2, 3])
@pytest.mark.parametrize("nx,nz,degree", [(3, 1, 1), (7, 1, 2), (3, 3, 3), (11, 3, 4), (5, 5, 5)])
def test_operators_at_block_edges(cuda_ok, nx, nz, degree, mapping_degree):
    case = build_case(HillParams(nx=nx, nz=nz, degree=degree, cfl=3.0,
                                 mapping_degree=mapping_degree, periodic=nx > 3))
    g, o, rng = operators(case)
    p = case.p * (1 + 0.01 * rng.standard_normal(case.p.shape))
    w = case.u + rng.standard_normal(case.u.shape)
    b = torch.full((2 * g.n_scalar,), np.nan, dtype=torch.float64, device="cuda")
    s = torch.full((g.n_scalar,), np.nan, dtype=torch.float64, device="cuda")
    g.vmult_pressure(b, dev(p))
    assert rel(b, o.vmult_pressure(p)) < 1e-12
    g.vmult_enthalpy(s, dev(w))
    assert rel(s, o.vmult_enthalpy(w)) < 1e-12
    g.vmult(s, dev(p))
    assert rel(s, o.vmult(p)) < 1e-11


@pytest.mark.parametrize("nx,nz,degree,adaptive", [(74, 52, 5, False), (75, 52, 5, False),
                                                   (98, 90, 3, True)])
def test_face_integrals_of_their_own(cuda_ok, nx, nz, degree, adaptive):
    """Just below and above the size from which C/D reads its face integrals
    from k_exact_face_C (140,000 unknowns), walls, and hanging faces above it."""
    p = HillParams(nx=nx, nz=nz, degree=degree, cfl=3.0, periodic=adaptive)
    case = build_case(p)
    if adaptive:
        from atmospheric_flows_gb300 import amr

        case = amr.adaptive_case(p, amr.example_tree(nx, nz, True))
        assert case.n_cells * (degree + 1) ** 2 > 140000
    g, o, rng = operators(case)
    w = case.u + rng.standard_normal(case.u.shape)
    s = torch.full((g.n_scalar,), np.nan, dtype=torch.float64, device="cuda")
    g.vmult_enthalpy(s, dev(w))
    assert rel(s, o.vmult_enthalpy(w)) < 1e-12
    q = case.p * (1 + 0.01 * rng.standard_normal(case.p.shape))
    g.vmult(s, dev(q))
    assert rel(s, o.vmult(q)) < 1e-11


def test_upload_mesh_changes_the_route(cuda_ok):
    """A mapping of degree 2, then 3, then 2 in one context: p_fix set once."""
    from atmospheric_flows_gb300 import _lib
    from atmospheric_flows_gb300.euler_operator import _np_d, _np_i

    cases = [build_case(HillParams(nx=6, nz=4, degree=3, cfl=3.0, mapping_degree=m))
             for m in (2, 3, 2)]
    g, o, rng = operators(cases[0])
    p = dev(cases[0].p * (1 + 0.01 * rng.standard_normal(cases[0].p.shape)))
    w = dev(cases[0].u + rng.standard_normal(cases[0].u.shape))
    out = []
    for i, c in enumerate(cases):
        if i:
            keep = [_np_d(c.mapping_nodes), _np_i(c.inner_faces), _np_i(c.boundary_faces)]
            _lib.call("atm_upload_mesh", g.handle, c.params.mapping_degree, keep[0][1],
                      len(c.inner_faces), keep[1][1], len(c.boundary_faces), keep[2][1])
        s = torch.empty(g.n_scalar, dtype=torch.float64, device="cuda")
        g.vmult_enthalpy(s, w)
        out.append(s)
    assert torch.equal(out[0], out[2])
    assert rel(out[0], o.vmult_enthalpy(w.cpu().numpy())) < 1e-12
    assert not torch.equal(out[0], out[1])  # another geometry


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_nonfinite_values_stay_visible(cuda_ok, bad):
    """A non-finite pressure value makes its cell's B and S non-finite and
    leaves cells that share no face with it (or its neighbours) alone."""
    case = build_case(HillParams(nx=16, nz=8, degree=4, cfl=3.0))
    g, o, rng = operators(case)
    p = case.p.copy()
    q = p.copy()
    cell, nn2 = 3 * 16 + 7, 25
    q[cell * nn2 + 12] = bad  # the middle node: inside, on no face
    s, t = (torch.empty(g.n_scalar, dtype=torch.float64, device="cuda") for _ in range(2))
    g.vmult(s, dev(p))
    g.vmult(t, dev(q))
    s, t = (a.cpu().numpy().reshape(-1, nn2) for a in (s, t))
    assert not np.isfinite(t[cell]).any()
    near = {cell, cell - 1, cell + 1, cell - 16, cell + 16}
    far = [c for c in range(case.n_cells) if c not in near]
    assert np.array_equal(s[far], t[far])
