"""Error statuses of the C ABI on the GPU, each failure made on the host (a NaN in the
input, an iteration cap of 1, device memory already held by the caller, a bisection
cap): no kernel is made to fault, and the library stays usable after each."""
import ctypes as C

import numpy as np
import pytest

from conftest import cantilever_load

pytestmark = pytest.mark.gpu


def _solve_status(P, F, **kw):
    from topologyoptimization_b200 import _native as N
    P.set_load(F)
    o = N.default_solve_opts(**kw)
    U = np.zeros(P.ndof)
    info = N.SolveInfo()
    st = N.lib().tpo_solve(P.h, C.byref(o), N.ptr(U), C.byref(info))
    return st, info, U


@pytest.mark.parametrize("precond", ["jacobi", "mg"])
def test_nan_load_is_nonfinite(native, precond):
    from topologyoptimization_b200 import Problem, mesh
    dims = (8, 4, 4)
    fixed = mesh.fixed_mask(*dims, "left")
    F = cantilever_load(*dims)
    with Problem(*dims, fixed) as P:
        P.set_densities(np.full(128, 0.5, np.float32), 3.0)
        bad = F.copy()
        bad[np.flatnonzero(fixed == 0)[7]] = np.nan
        pc = native.PREC_MG if precond == "mg" else native.PREC_JACOBI
        st, _, _ = _solve_status(P, bad, precond=pc, max_iter=200, tol=1e-8)
        assert st == native.TPO_NONFINITE, native.status_string(st)
        st, info, _ = _solve_status(P, F, precond=pc, max_iter=2000, tol=1e-8)
        assert st == native.TPO_OK and info.converged == 1


def test_nan_load_ebe_pcg(native, oracle):
    from topologyoptimization_b200 import _native as N
    dims = (4, 3, 3)
    fixed = oracle.fixed_mask(*dims, "left")
    free = np.flatnonzero(fixed == 0).astype(np.int32)
    F = cantilever_load(*dims)
    F[free[3]] = np.nan
    U = np.zeros(len(F))
    it = C.c_int32()
    st = N.lib().tpo_ebe_pcg(N.ptr(np.ones(36)), N.ptr(oracle.lk(0.3)), N.ptr(oracle.edofs3d(*dims)), N.ptr(F),
                             N.ptr(U), N.ptr(free), 36, 24, len(F), len(free), 1e-9, 1.0, 3.0, 100, 1e-8, C.byref(it))
    assert st == N.TPO_NONFINITE


def test_iteration_cap_is_not_converged(native):
    from topologyoptimization_b200 import Problem, mesh
    dims = (8, 4, 4)
    fixed = mesh.fixed_mask(*dims, "left")
    with Problem(*dims, fixed) as P:
        P.set_densities(np.full(128, 0.5, np.float32), 3.0)
        for pc in (native.PREC_JACOBI, native.PREC_MG):
            st, info, U = _solve_status(P, cantilever_load(*dims), precond=pc, max_iter=1, tol=1e-8)
            assert st == native.TPO_NOT_CONVERGED and info.converged == 0 and info.iterations == 1
            assert np.isfinite(U).all() and np.any(U)  # the iterate is still written


def test_device_memory_exhausted_is_oom(native):
    """The caller holds all but 256 MB of the device; creating a 12.8M-DOF problem (whose
    hierarchy needs several GB) returns TPO_OOM and frees what it had taken, and the same
    creation succeeds once the memory is released."""
    import torch
    from topologyoptimization_b200 import Problem, mesh
    from topologyoptimization_b200 import _native as N
    dims = (256, 128, 128)
    fixed = mesh.fixed_mask(*dims, "left")
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    hold = torch.empty(max(free - (256 << 20), 0), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(N.TpoError) as e:
            Problem(*dims, fixed)
        assert e.value.status == N.TPO_OOM
    finally:
        del hold
        torch.cuda.empty_cache()
    with Problem(*dims, fixed) as P:
        assert P.levels >= 2


def test_bisection_cap_is_timeout(native):
    """An OC bisection cap below the steps the bracket needs returns TPO_TIMEOUT; the same
    call with the default cap succeeds."""
    import torch
    from topologyoptimization_b200 import Problem, mesh
    from topologyoptimization_b200 import _native as N
    dims = (8, 4, 4)
    rng = np.random.default_rng(3)
    x = torch.from_numpy(rng.uniform(0.1, 1, 128).astype(np.float32)).cuda()
    dc = torch.from_numpy((-rng.uniform(0.5, 2, 128) * 1e2).astype(np.float32)).cuda()
    xn = torch.empty_like(x)
    with Problem(*dims, mesh.fixed_mask(*dims, "left")) as P:
        with pytest.raises(N.TpoError) as e:
            P.oc_update_dev(x, dc, xn, 0.3, max_bisections=5)
        assert e.value.status == N.TPO_TIMEOUT
        ch, lm, nb = P.oc_update_dev(x, dc, xn, 0.3)
        assert nb > 5 and ch > 0


def _jacobi(P, F, n=60):
    from topologyoptimization_b200 import _native as N
    P.set_load(F)
    return P.solve(None, precond=N.PREC_JACOBI, max_iter=n, tol=0.0, warm_start=0, ref_epsilon=0)


def test_barrier_wait_is_timeout_and_leaves_the_handle_usable(native):
    """Barrier waits of a single poll run out (some 140 blocks do not all arrive within one):
    TPO_TIMEOUT from the Jacobi solve and from the OC update, and with the limit back both
    give what a handle gives that never saw one."""
    import torch
    from topologyoptimization_b200 import Problem, mesh
    from topologyoptimization_b200 import _native as N
    dims = (60, 20, 20)
    fixed = mesh.fixed_mask(*dims, "left")
    rng = np.random.default_rng(4)
    x = rng.uniform(0.2, 1, 24000).astype(np.float32)
    F = rng.standard_normal(len(fixed)) * (fixed == 0)
    d_x = torch.from_numpy(x).cuda()
    d_dc = torch.from_numpy((-rng.uniform(0.5, 2, 24000)).astype(np.float32)).cuda()
    d_xn, d_ref = torch.empty_like(d_x), torch.empty_like(d_x)
    with Problem(*dims, fixed) as P, Problem(*dims, fixed) as Q:
        for A in (P, Q):
            A.set_densities(x, 3.0)
        P.set_launch_limits(polls=1)
        for call in (lambda: _jacobi(P, F), lambda: P.oc_update_dev(d_x, d_dc, d_xn, 0.3)):
            with pytest.raises(N.TpoError) as e:
                call()
            assert e.value.status == N.TPO_TIMEOUT
        P.set_launch_limits()
        U, info = _jacobi(P, F)
        Ur, infor = _jacobi(Q, F)
        assert info.iterations == infor.iterations == 60 and np.array_equal(U, Ur)
        assert P.oc_update_dev(d_x, d_dc, d_xn, 0.3) == Q.oc_update_dev(d_x, d_dc, d_ref, 0.3)
        assert torch.equal(d_xn, d_ref)


@pytest.mark.parametrize("dims", [(4, 4, 4), (40, 22, 20)])
def test_jacobi_solve_split_over_launches(native, dims):
    """The one-launch Jacobi solve handed over between launches of 2, 8 and 64 iterations: bit for
    bit the solve in one (19,803 nodes: five a lane), at a count that is no multiple of them."""
    from topologyoptimization_b200 import Problem, mesh
    from topologyoptimization_b200 import _native as N
    fixed = mesh.fixed_mask(*dims, "left")
    rng = np.random.default_rng(6)
    F = rng.standard_normal(len(fixed)) * (fixed == 0)
    with Problem(*dims, fixed) as P:
        P.set_densities(rng.uniform(0.2, 1, int(np.prod(dims))).astype(np.float32), 3.0)
        U, info = _jacobi(P, F, 77)
        for iterations in (2, 8, 64):
            P.set_launch_limits(iterations=iterations)
            V, infov = _jacobi(P, F, 77)
            assert infov.iterations == info.iterations and np.array_equal(U, V)
        for bad in (dict(iterations=3), dict(iterations=0), dict(polls=0)):
            with pytest.raises(N.TpoError) as e:
                P.set_launch_limits(**bad)
            assert e.value.status == N.TPO_BAD_ARG
