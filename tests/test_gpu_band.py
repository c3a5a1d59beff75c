"""The pass kernels leave out the columns that the 2/3 rule empties when the
state holds nothing there, and must take them back in when it does: states set
from outside with content past the circle (a whole spectrum, or one mode in the
first emptied column), a forced mode there, changes from one kind to the other
on one handle, ensembles of both kinds, and a reverse sweep after the state was
replaced.  Against the oracle, FP64, to the parity tests' 1e-12 of max|w_hat|."""
import numpy as np
import pytest

from _util import rel_err
from ns2d import Ensemble, Solver, abi, initial
from pyoracle import Oracle

pytestmark = pytest.mark.gpu


def _state(n, kind, seed=3):
    w = initial.decaying(n, seed=seed, k0=n / 16.0, dealias="2/3")
    top = np.abs(w).max()
    if kind == "wide":
        w = w + initial.hermitian(np.full_like(w, 1e-3 * top))
    elif kind == "edge":  # ky = int(n/3), the first column with no kept mode
        w[5, int(n / 3.0)] = 0.05 * top * (1 + 2j)
    return w


def _oracle(p, w0, steps, dt):
    o = Oracle(p, threads=8)
    o.set_w_hat(w0)
    for k in range(steps):
        if p.integrator == abi.AB4:
            o.ab4_step(dt, k + 1)
        else:
            o.compute_forcing(dt)
            o.rk4_step(dt)
    return o.get_w_hat()


@pytest.mark.parametrize("kind", ["narrow", "edge", "wide"])
@pytest.mark.parametrize("integ", [abi.RK4CN, abi.RK4, abi.AB4])
@pytest.mark.parametrize("n", [256, 512, 1024])
def test_steps_match_oracle(n, integ, kind):
    dt, steps = 1e-4, 5
    p = abi.default_params(nx=n, ny=n, nu=1e-3, ekmn_drag_flag=1, integrator=integ, dt=dt)
    w0 = _state(n, kind)
    s = Solver(p)
    s.set_w_hat(w0)
    s.step_n(steps, dt)
    assert rel_err(s.get_w_hat(), _oracle(p, w0, steps, dt)) <= 1e-12
    assert rel_err(s.nonlinear_rhs(w0), _rhs(p, w0)) <= 1e-12
    s.close()


def _rhs(p, w):
    o = Oracle(p, threads=8)
    o.set_w_hat(w)
    return o.nonlinear_rhs(w)


def test_one_handle_changes_kind():
    n, dt = 256, 2e-4
    p = abi.default_params(nx=n, ny=n, nu=1e-3, ekmn_drag_flag=1, dt=dt)
    s = Solver(p)
    for k, kind in enumerate(["narrow", "edge", "narrow", "wide", "narrow"]):
        w0 = _state(n, kind, seed=20 + k)
        s.set_w_hat(w0)
        s.step_n(4, dt)  # the step graph stays captured across the changes
        assert rel_err(s.get_w_hat(), _oracle(p, w0, 4, dt)) <= 1e-12, (k, kind)
    for k, kind in enumerate(["edge", "narrow", "wide"]):
        w0 = _state(n, kind, seed=30 + k)
        w = w0.copy()
        for _ in range(3):
            s.rk4_step_host(w, dt)
        assert rel_err(w, _oracle(p, w0, 3, dt)) <= 1e-12, (k, kind)
    s.close()


def test_forced_mode_past_the_circle():
    n, dt = 256, 1e-3
    p = abi.default_params(nx=n, ny=n, nu=1e-3, ekmn_drag_flag=1, dt=dt, forcing=abi.FORCING_KOLM, force_k=n // 2 - 3,
                           force_scale=50.0)
    w0 = _state(n, "narrow")
    s = Solver(p)
    s.set_w_hat(w0)
    s.step_n(6, dt)
    assert rel_err(s.get_w_hat(), _oracle(p, w0, 6, dt)) <= 1e-12


def test_ensemble_of_both_kinds():
    sizes, kinds, dt = [256, 512, 64, 256, 128], ["edge", "narrow", "wide", "narrow", "edge"], 2e-4
    p = abi.default_params(nu=1e-3, ekmn_drag_flag=1, dt=dt)
    w0 = [_state(n, k, seed=m) for m, (n, k) in enumerate(zip(sizes, kinds))]
    e = Ensemble(p, sizes)
    for stage_launch in (0, 1):
        e.set_shape(stage_launch=stage_launch)
        for m, w in enumerate(w0):
            e.set_w_hat(m, w)
        e.step_n(4, dt)
        for m, n in enumerate(sizes):
            q = p.copy()
            q.nx = q.ny = n
            assert rel_err(e.get_w_hat(m), _oracle(q, w0[m], 4, dt)) <= 1e-12, (stage_launch, m)
    e.close()


def test_reverse_sweep_after_the_state_was_replaced():
    n, dt = 256, 1e-3
    p = abi.default_params(nx=n, ny=n, nu=1e-3, quirks=0, dt=dt)
    lam = initial.decaying(n, 8, k0=5.0, dealias="2/3")
    grads = []
    for replace in (False, True):
        s = Solver(p)
        s.set_w_hat(_state(n, "edge"))
        s.adjoint_record(6, dt, 3)
        if replace:
            s.set_w_hat(_state(n, "narrow"))
            s.step_n(2, dt)
        grads.append(s.adjoint_backward(lam))
        s.close()
    assert np.array_equal(grads[0], grads[1])


@pytest.mark.parametrize("quirks", [abi.QUIRKS_REFERENCE, abi.QUIRKS_REFERENCE & ~abi.QUIRK_HOU_LI_INT & ~abi.QUIRK_RK4_LINEAR])
@pytest.mark.parametrize("integ", [abi.RK4CN, abi.RK4, abi.AB4])
@pytest.mark.parametrize("n", [256, 512])
def test_houli_steps_match_oracle(n, integ, quirks):
    """Hou-Li dealiasing empties no column; its factors (integer or real ratios)
    and the explicit linear term's brackets come from per-mode tables."""
    dt = 1e-4
    p = abi.default_params(nx=n, ny=n, nu=1e-3, ekmn_drag_flag=1, integrator=integ, dealias=abi.DEALIAS_HOU_LI,
                           quirks=quirks, dt=dt)
    w0 = initial.decaying(n, seed=6, k0=n / 10.0)
    s = Solver(p)
    s.set_w_hat(w0)
    s.step_n(3, dt)
    s.step_n(2, 0.5 * dt)  # another table
    o = Oracle(p, threads=8)
    o.set_w_hat(w0)
    for k in range(5):
        d = dt if k < 3 else 0.5 * dt
        o.ab4_step(d, k + 1) if integ == abi.AB4 else o.rk4_step(d)
    assert rel_err(s.get_w_hat(), o.get_w_hat()) <= 1e-12
    s.close()


@pytest.mark.parametrize("precision", [abi.FP64, abi.FP32])
@pytest.mark.parametrize("integ", [abi.RK4CN, abi.RK4, abi.AB4])
@pytest.mark.parametrize("dealias", [abi.DEALIAS_23, abi.DEALIAS_HOU_LI])
@pytest.mark.parametrize("n", [256, 1024])
def test_runs_equal_single_steps(n, dealias, integ, precision):
    """In a run of steps the final pass goes on to the next step's first; the
    states are those of single steps, bit for bit, over run lengths and changes
    of dt, and so are the column 0 snapshots AB4's conjugacy takes."""
    p = abi.default_params(nx=n, ny=n, nu=1e-3, integrator=integ, dealias=dealias, precision=precision)
    w0 = initial.decaying(n, seed=12, k0=n / 16.0, dealias="2/3")
    a, b = Solver(p), Solver(p)
    a.set_w_hat(w0)
    b.set_w_hat(w0)
    k = 0
    for run, dt in ((5, 1e-4), (2, 1e-4), (1, 1e-4), (3, 5e-5), (4, 1e-4)):
        a.step_n(run, dt)
        for _ in range(run):
            k += 1
            b.ab4_step(dt, k) if integ == abi.AB4 else b.rk4_step(dt)
        assert np.array_equal(a.get_w_hat(), b.get_w_hat()), k
    a.close()
    b.close()


@pytest.mark.parametrize("run", [True, False])
@pytest.mark.parametrize("ky", [341, 342, 343])
def test_forcing_of_an_earlier_state_leaves_nothing_behind(ky, run):
    """1024^2 FP64, where the stage pass takes two columns a block and the others
    four, and the emptied columns begin at 341, in the middle of a tile: after
    steps with a mode forced there, a state set anew steps as on a new handle."""
    n, dt = 1024, 1e-4
    p = abi.default_params(nx=n, ny=n, nu=1e-3, dt=dt)
    w0 = _state(n, "narrow")
    s, fresh = Solver(p), Solver(p)
    s.set_w_hat(w0)
    s.set_forcing_modes([3 * (n // 2 + 1) + ky], [np.abs(w0).max() * (1 + 2j)])
    s.step_n(2, dt)
    s.set_forcing_modes([], [])
    for obj in (s, fresh):
        obj.set_w_hat(w0)
        if run:
            obj.step_n(4, dt)
        else:
            obj.rk4_step(dt)
    assert np.array_equal(s.get_w_hat(), fresh.get_w_hat())
    s.close()
    fresh.close()


def test_forcing_set_before_the_reverse_sweep():
    """A mode in the emptied columns, forced from after the recorded run on: the
    steps that follow the sweep take it up."""
    n, dt = 256, 1e-3
    p = abi.default_params(nx=n, ny=n, nu=1e-3, quirks=0, dt=dt)
    idx, val = [3 * (n // 2 + 1) + n // 2 - 9, 2 * (n // 2 + 1) + 1], [30.0 * n, 5.0 * n]
    s, ref = Solver(p), Solver(p)
    s.set_w_hat(_state(n, "narrow"))
    s.adjoint_record(6, dt, 3)
    w6 = s.get_w_hat()
    s.set_forcing_modes(idx, val)
    s.adjoint_backward(initial.decaying(n, 8, k0=5.0, dealias="2/3"))
    assert np.array_equal(s.get_w_hat(), w6)
    ref.set_w_hat(w6)
    ref.set_forcing_modes(idx, val)
    for obj in (s, ref):
        obj.step_n(4, dt)
    assert np.abs(ref.get_w_hat()[3, n // 2 - 9]) > 0
    assert rel_err(s.get_w_hat(), ref.get_w_hat()) <= 1e-12
    s.close()
    ref.close()


def test_history_of_forced_steps_after_a_host_step():
    """The host-resident step replaces the state and keeps AB4's history, whose
    right-hand sides hold an earlier forcing of the emptied columns.  Reference:
    the same calls with 1e-280 in an emptied column of the host's array, which
    keeps those columns in use whatever the history holds."""
    n, dt = 256, 1e-3
    p = abi.default_params(nx=n, ny=n, nu=1e-3, integrator=abi.AB4, dt=dt)
    out = []
    for trace in (0.0, 1e-280):
        s = Solver(p)
        s.set_w_hat(_state(n, "narrow"))
        s.set_forcing_modes([3 * (n // 2 + 1) + n // 2 - 9], [30.0 * n])
        s.step_n(5, dt)
        s.set_forcing_modes([], [])
        w = _state(n, "narrow", seed=5)
        w[7, n // 2 - 4] = trace
        s.rk4_step_host(w, dt)
        s.ab4_step(dt, 6)
        out.append(s.get_w_hat())
        s.close()
    assert np.abs(out[1][3, n // 2 - 9]) > 0
    assert rel_err(out[0], out[1]) <= 1e-12


@pytest.mark.parametrize("integ", [abi.RK4CN, abi.RK4])
@pytest.mark.parametrize("steps", [64, 83])
def test_long_runs_equal_single_steps(steps, integ):
    """Long runs replay graphs of several steps and end with single ones."""
    n, dt = 256, 1e-4
    p = abi.default_params(nx=n, ny=n, nu=1e-3, integrator=integ)
    w0 = initial.decaying(n, seed=12, k0=n / 16.0, dealias="2/3")
    a, b = Solver(p), Solver(p)
    for s in (a, b):
        s.set_w_hat(w0)
    for run in (steps, 21, 9):
        a.step_n(run, dt)
        for _ in range(run):
            b.rk4_step(dt)
        assert np.array_equal(a.get_w_hat(), b.get_w_hat()), run
    a.close()
    b.close()
