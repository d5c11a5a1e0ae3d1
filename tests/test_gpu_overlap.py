"""Operator calls of one handle that overlap on the GPU, or whose launches
interleave: with their own inputs and outputs they give the bits of the same
calls made one after the other.  The operators that need the handle's
workspace (S, the solves) are the caller's to order and are not among them."""
import ctypes
import threading

import numpy as np
import pytest

from atmospheric_flows_gb300.hill import HillParams, build_case

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def dev(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def setup(nx, nz, degree, adaptive, stage=2):
    from atmospheric_flows_gb300 import amr
    from atmospheric_flows_gb300.euler_operator import EULEROperator, MatrixFreeStorage

    p = HillParams(nx=nx, nz=nz, degree=degree, cfl=3.0)
    case = amr.adaptive_case(p, amr.example_tree(nx, nz, True)) if adaptive else build_case(p)
    op = EULEROperator(MatrixFreeStorage.from_case(case), case.dt, case.Ma, case.Fr)
    op.set_HYPERBOLIC_stage(stage)
    return op, case, np.random.default_rng(11)


def state(case, rng):
    return [dev(case.rho * (1 + 0.01 * rng.standard_normal(case.rho.shape))),
            dev(case.u + 2.0 * rng.standard_normal(case.u.shape)),
            dev(case.p * (1 + 0.01 * rng.standard_normal(case.p.shape)))]


def rhs_calls(op, case, rng):
    """The three right-hand sides of stage 2, and the density's once more on
    other inputs: (function, sources, destination, its serial result)."""
    calls = []
    for kind in (0, 1, 2, 0):
        a, b = state(case, rng), state(case, rng)
        src = a[:2] + b[:2] if kind == 0 else a + b
        src += [[], [a[0]], [b[0], b[1]]][kind]
        fn = (op.vmult_rhs_rho_update, op.vmult_rhs_velocity_fixed, op.vmult_rhs_pressure)[kind]
        dst = torch.empty(op.n_scalar * (2 if kind == 1 else 1), dtype=torch.float64, device="cuda")
        calls.append((fn, src, dst))
    out = []
    for fn, src, dst in calls:
        fn(dst, src)
        torch.cuda.synchronize()
        out.append((fn, src, dst, dst.clone()))
    return out


def set_stream(op, s):
    from atmospheric_flows_gb300 import _lib

    _lib.call("atm_set_stream", op.handle, ctypes.c_void_p(s.cuda_stream if s else 0))


MESHES = [(60, 40, 4, False), (103, 61, 4, False), (50, 30, 2, False), (24, 12, 3, True)]


@pytest.mark.parametrize("nx,nz,degree,adaptive", MESHES)
def test_right_hand_sides_on_streams_of_one_handle(cuda_ok, nx, nz, degree, adaptive):
    op, case, rng = setup(nx, nz, degree, adaptive)
    calls = rhs_calls(op, case, rng)
    streams = [torch.cuda.Stream() for _ in calls]
    for _ in range(40):
        for _, _, dst, _ in calls:
            dst.fill_(float("nan"))
        torch.cuda.synchronize()
        for s, (fn, src, dst, _) in zip(streams, calls):
            set_stream(op, s)
            fn(dst, src)
        torch.cuda.synchronize()
        for _, _, dst, ref in calls:
            assert torch.equal(dst, ref)
    set_stream(op, None)
    op.close()


@pytest.mark.parametrize("nx,nz,degree,adaptive", MESHES)
def test_right_hand_sides_in_branches_of_a_graph(cuda_ok, nx, nz, degree, adaptive):
    op, case, rng = setup(nx, nz, degree, adaptive)
    calls = rhs_calls(op, case, rng)  # tuned here, outside the capture
    main = torch.cuda.Stream()
    side = [torch.cuda.Stream() for _ in calls]
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=main):
        for s, (fn, src, dst, _) in zip(side, calls):
            s.wait_stream(main)
            set_stream(op, s)
            fn(dst, src)
        for s in side:
            main.wait_stream(s)
    set_stream(op, None)
    for _ in range(20):
        for _, _, dst, _ in calls:
            dst.fill_(float("nan"))
        g.replay()
        torch.cuda.synchronize()
        for _, _, dst, ref in calls:
            assert torch.equal(dst, ref)
    op.close()


def test_threads_share_a_handle_and_its_stream(cuda_ok):
    op, case, rng = setup(40, 24, 4, False)
    calls = rhs_calls(op, case, rng)
    bad = []

    def work(fn, src, dst, ref):
        for _ in range(40):
            fn(dst, src)
            torch.cuda.synchronize()
            if not torch.equal(dst, ref):
                bad.append(1)

    threads = [threading.Thread(target=work, args=c) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    op.close()


@pytest.mark.parametrize("nx,nz,degree,adaptive", MESHES)
def test_energy_rhs_into_its_density(cuda_ok, nx, nz, degree, adaptive):
    """dst may be a source that is read cell by cell only (the density of the
    kinetic term).  The faces are then added in another order: the
    single-operator bar of 1e-12 in the max norm."""
    op, case, rng = setup(nx, nz, degree, adaptive)
    fn, src, dst, ref = rhs_calls(op, case, rng)[2]
    own = src[6].clone()
    fn(own, src[:6] + [own, src[7]])
    torch.cuda.synchronize()
    err = (own - ref).abs().max().item() / ref.abs().max().item()
    assert err < 1e-12, err
    op.close()


@pytest.mark.parametrize("nx,nz,degree,adaptive", [(101, 60, 4, False), (60, 40, 4, False),
                                                   (94, 96, 3, True)])
def test_operators_beside_the_schur_apply(cuda_ok, nx, nz, degree, adaptive):
    """B, C, the static-scratch S and a right-hand side, each on a stream of its
    own, beside the one call that uses the handle's workspace: S (with a face
    buffer from 140,000 unknowns on, first and last mesh)."""
    from atmospheric_flows_gb300 import _lib

    op, case, rng = setup(nx, nz, degree, adaptive)
    rho, _, p = state(case, rng)
    op.set_rho_for_fixed(rho)
    op.set_pres_fixed(p)
    op.set_NS_stage(2)
    q, w = state(case, rng)[2], state(case, rng)[1]
    rhs, src, mom, _ = rhs_calls(op, case, rng)[1]
    out = [torch.empty_like(q), torch.empty_like(w), torch.empty_like(q), torch.empty_like(q), mom]
    static = lambda d, s: _lib.call("atm_schur_vmult_static_scratch", op.handle,  # noqa: E731
                                    ctypes.c_void_p(d.data_ptr()), ctypes.c_void_p(s.data_ptr()))
    calls = [(op.vmult, q), (op.vmult_pressure, q), (op.vmult_enthalpy, w), (static, q), (rhs, src)]
    for (fn, s), d in zip(calls, out):
        fn(d, s)
        torch.cuda.synchronize()
    ref = [d.clone() for d in out]
    streams = [torch.cuda.Stream() for _ in calls]
    for _ in range(40):
        for d in out:
            d.fill_(float("nan"))
        torch.cuda.synchronize()
        for st, (fn, s), d in zip(streams, calls, out):
            set_stream(op, st)
            fn(d, s)
        torch.cuda.synchronize()
        for d, r in zip(out, ref):
            assert torch.equal(d, r)
    set_stream(op, None)
    op.close()


def test_threads_share_a_shell(cuda_ok):
    """Host threads that call the right-hand sides and C of one shell handle."""
    from atmospheric_flows_gb300.shell import ShellSolver, build_shell

    case = build_shell(n=4, nr=2, r_in=6.36122e6, r_out=6.37122e6, rotate_every=5)
    op, rng = ShellSolver(case), np.random.default_rng(3)
    op.set_stage(1, 2)
    op.set_frozen(dev(case.rho), dev(case.p))
    calls = []
    for which in (0, 1, 2, 0, 3):
        rho, u, p = state(case, rng)
        src = [[rho, u], [rho, u, p, rho], [rho, u, p, rho, u]][which] if which < 3 else u
        dst = torch.empty_like(u if which == 1 else rho)
        fn = (lambda d, s, w=which: op.rhs(w, d, s)) if which < 3 else (
            lambda d, s: op.apply(1, d, s))
        fn(dst, src)
        calls.append((fn, src, dst, dst.clone()))
    bad = []

    def work(fn, src, dst, ref):
        for _ in range(60):
            fn(dst, src)
            torch.cuda.synchronize()
            if not torch.equal(dst, ref):
                bad.append(1)

    threads = [threading.Thread(target=work, args=c) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
