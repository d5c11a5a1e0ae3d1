"""Shell kernels at the cell counts where their blocks end: the face kernels
take 32 faces per block, B and C/D eight cells, the right-hand sides four (below
1500 cells) or fourteen.  Oracle bars as in test_gpu_shell.py: 1e-12 for one
operator in the max norm, 1e-11 for S."""
import numpy as np
import pytest

from atmospheric_flows_gb300.shell import ShellSolver, build_shell
from oracle.oracle import OracleShell

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), device="cuda")


def state(case, seed):
    rng = np.random.default_rng(seed)
    return (case.rho * (1 + 0.01 * rng.standard_normal(case.rho.shape)),
            case.u + rng.standard_normal(case.u.shape),
            case.p * (1 + 0.01 * rng.standard_normal(case.p.shape)))


def rel(a, b):
    return np.max(np.abs(a.cpu().numpy() - b)) / np.max(np.abs(b))


@pytest.mark.parametrize("n,nr,rotate", [(1, 1, 0), (1, 3, 2), (3, 1, 4), (5, 2, 3), (16, 1, 7)])
def test_operators_at_block_edges(cuda_ok, n, nr, rotate):
    case = build_shell(n=n, nr=nr, r_in=6.36122e6, r_out=6.37122e6, rotate_every=rotate)
    g, o = ShellSolver(case), OracleShell(case, inner_tol=1e-15)
    st = [state(case, 3 + k) for k in range(4)]
    ns = case.n_cells * 8
    for stage in (1, 2, 3):
        g.set_stage(stage, 2)
        o.set_stage(stage, 2)
        for which in (0, 1, 2):
            src = []
            for j in range(stage):
                src += [st[j][0], st[j][1]] if which == 0 else list(st[j])
            if which == 1 and stage < 3:
                src.append(st[3][0])
            if which == 2:
                src += [st[3][0], st[3][1]]
            out = torch.full((3 * ns if which == 1 else ns,), np.nan, dtype=torch.float64,
                             device="cuda")
            g.rhs(which, out, [dev(s) for s in src])
            assert rel(out, o.rhs(which, src)) < 1e-12, (which, stage)
    g.set_frozen(rho=dev(st[0][0]), pres=dev(st[0][2]))
    o.set_frozen(rho=st[0][0], p=st[0][2])
    out = torch.full((ns,), np.nan, dtype=torch.float64, device="cuda")
    g.apply(2, out, dev(st[1][2]))
    assert rel(out, o.apply(2, st[1][2], ns)) < 1e-11
    g.close()
