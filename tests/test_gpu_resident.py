"""Small grids (16..128) advance whole steps in one launch (the resident
kernel): against the oracle over integrators, dealiasing rules and states with
and without content in the columns that the 2/3 rule empties, and across the
launch boundaries of a long run.

Tolerances: those of the parity tests, 1e-12 of max|w_hat| for a few FP64
steps and 1e-4 in FP32 (rounding of a few steps: 1e-15 and 1e-6 times the
number of evaluations, with room for growth)."""
import numpy as np
import pytest

from _util import rel_err
from ns2d import Solver, abi, initial
from pyoracle import Oracle

pytestmark = pytest.mark.gpu

TOL = {abi.FP64: 1e-12, abi.FP32: 1e-4}


def _state(n, wide, seed):
    """Wide: energy in every mode, the columns past the 2/3 circle included."""
    w = initial.decaying(n, seed=seed, k0=n / 8.0, dealias=None if wide else "2/3")
    return w + 1e-3 * initial.hermitian(np.full_like(w, np.abs(w).max())) if wide else w


def _run(obj, p, w0, steps, dt, one_call):
    obj.set_w_hat(w0)
    if one_call:
        obj.step_n(steps, dt)
    else:
        for k in range(steps):
            obj.ab4_step(dt, k + 1) if p.integrator == abi.AB4 else obj.rk4_step(dt)
    return obj.get_w_hat()


@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("dealias", [abi.DEALIAS_23, abi.DEALIAS_HOU_LI])
@pytest.mark.parametrize("integ", [abi.RK4CN, abi.RK4, abi.AB4])
@pytest.mark.parametrize("n", [16, 32, 64, 128])
def test_steps_match_oracle(n, integ, dealias, wide, precision):
    dt, steps = 2e-4, 7
    p = abi.default_params(nx=n, ny=n, nu=1e-3, ekmn_drag_flag=1, integrator=integ, dealias=dealias, dt=dt,
                           precision=precision)
    w0 = _state(n, wide, 40 + n)
    s = Solver(p)
    l0 = s.launch_count
    got = _run(s, p, w0, steps, dt, True)
    assert s.launch_count - l0 < 9 * steps  # not the nine pass launches per step
    s.close()
    assert rel_err(got, _run(Oracle(p), p, w0, steps, dt, False)) <= TOL[precision]


@pytest.mark.parametrize("integ", [abi.RK4CN, abi.AB4])
def test_long_run_equals_single_calls(integ):
    """More steps than one launch takes; AB4 rotates its history in the kernel
    and on the host between launches."""
    n, dt, steps = 32, 1e-3, 261
    p = abi.default_params(nx=n, ny=n, nu=1e-3, integrator=integ, dt=dt)
    w0 = _state(n, False, 5)
    a, b = Solver(p), Solver(p)
    got = _run(a, p, w0, steps, dt, True)
    assert np.array_equal(got, _run(b, p, w0, steps, dt, False))


@pytest.mark.parametrize("integ", [abi.RK4CN, abi.AB4])
def test_forced_modes_past_the_circle(integ):
    """Listed-mode forcing of a mode that dealiasing empties, switched on and
    off again: the state (and AB4's history) then hold content the transforms
    must not leave out."""
    n, dt = 64, 1e-3
    p = abi.default_params(nx=n, ny=n, nu=1e-3, integrator=integ, dt=dt)
    w0 = _state(n, False, 9)
    idx = np.array([3 * (n // 2 + 1) + n // 2 - 2, 2 * (n // 2 + 1) + 1], np.int32)
    val = np.array([30.0 + 10.0j, 5.0 - 2.0j]) * n
    s, ref = Solver(p), Solver(p)
    ref.set_kernel_timing(True)  # per-pass timing: the pass kernels
    for obj in (s, ref):
        obj.set_w_hat(w0)
        obj.step_n(4, dt)
        obj.set_forcing_modes(idx, val)
        obj.step_n(3, dt)
        obj.set_forcing_modes([], [])
        obj.step_n(6, dt)
    assert rel_err(s.get_w_hat(), ref.get_w_hat()) <= 1e-12
    assert rel_err(s.nonlinear_rhs(None), ref.nonlinear_rhs(None)) <= 1e-12


def test_blowup_stops_the_launch():
    n = 32
    s = Solver(abi.default_params(nx=n, ny=n, nu=1e-3))
    w = _state(n, False, 3)
    w[2, 2] = np.nan
    s.set_w_hat(w)
    with pytest.raises(Exception, match="BLOWUP"):
        s.step_n(200, 1e-3)
    s.set_w_hat(_state(n, False, 3))
    s.step_n(3, 1e-3)
    assert np.all(np.isfinite(s.get_w_hat()))


@pytest.mark.parametrize("n", [64, 256])
def test_rhs_after_a_blowup(n):
    """The RHS of a given field does not depend on the handle's state: after a
    failed step it is still that of a new handle."""
    p = abi.default_params(nx=n, ny=n, nu=1e-3)
    w = initial.decaying(n, seed=3, k0=n / 16.0, dealias="2/3")
    fresh, s = Solver(p), Solver(p)
    other = initial.decaying(n, seed=4, k0=n / 16.0, dealias="2/3")
    s.nonlinear_rhs(other)
    s.rk4_step_host(other, 1e-3)
    bad = w.copy()
    bad[2, 2] = np.nan
    s.set_w_hat(bad)
    with pytest.raises(Exception, match="BLOWUP"):
        s.step_n(3, 1e-3)
    assert np.array_equal(s.nonlinear_rhs(w), fresh.nonlinear_rhs(w))
    assert not np.all(np.isfinite(s.nonlinear_rhs()))  # the failed state's own


@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32])
def test_device_memory_in_the_place_of_host_arrays(precision):
    """Arrays that CUDA knows are copied by the driver, wherever they are."""
    import ctypes as C

    import torch

    n = 64
    p = abi.default_params(nx=n, ny=n, nu=1e-3, precision=precision)
    w = initial.decaying(n, seed=3, k0=4.0, dealias="2/3")
    s = Solver(p)
    d_in = torch.from_numpy(w.view(np.float64).copy()).cuda()
    d_out = torch.zeros_like(d_in)
    ptr = [C.cast(t.data_ptr(), C.POINTER(C.c_double)) for t in (d_in, d_out)]
    torch.cuda.synchronize()
    s._ck(s.L.ns2d_nonlinear_rhs(s.h, ptr[0], ptr[1]))
    assert np.array_equal(d_out.cpu().numpy().view(np.complex128), s.nonlinear_rhs(w))
    s._ck(s.L.ns2d_rk4_step_host(s.h, ptr[0], 1e-3))
    s.rk4_step_host(w, 1e-3)
    assert np.array_equal(d_in.cpu().numpy().view(np.complex128), w)


@pytest.mark.parametrize("integ", [abi.RK4CN, abi.RK4])
@pytest.mark.parametrize("n", [16, 32, 64, 128])
def test_passes_give_the_same_states(n, integ):
    """Per-pass timing takes the pass kernels: the same bits, except at 64, whose
    row pass transforms each row by itself in half the length."""
    p = abi.default_params(nx=n, ny=n, nu=1e-3, integrator=integ)
    w0 = _state(n, False, 8)
    a, b = Solver(p), Solver(p)
    b.set_kernel_timing(True)
    for s in (a, b):
        s.set_w_hat(w0)
        s.step_n(5, 1e-3)
    if n == 64:
        assert rel_err(a.get_w_hat(), b.get_w_hat()) <= TOL[abi.FP64]
    else:
        assert np.array_equal(a.get_w_hat(), b.get_w_hat())
