"""Row transforms in FP32, whose shared-memory padding differs from FP64's at 128
to 512 (teams of 16 lanes and more with radix 8): against the FP64 oracle, to
the parity tests' FP32 bounds, 5e-5 of max for one RHS and 1e-4 for a state."""
import pytest

from _util import rel_err
from ns2d import Ensemble, Solver, abi, initial
from pyoracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dealias", [abi.DEALIAS_23, abi.DEALIAS_HOU_LI])
@pytest.mark.parametrize("n", [64, 128, 256, 512])
def test_fp32_rhs_and_ensemble_steps(n, dealias):
    p = abi.default_params(nx=n, ny=n, nu=1e-3, dt=1e-3, dealias=dealias)
    p32 = abi.default_params(nx=n, ny=n, nu=1e-3, dt=1e-3, dealias=dealias, precision=abi.FP32)
    w0 = initial.decaying(n, seed=n + 1, k0=6.0, dealias="2/3")
    o = Oracle(p, threads=8)
    o.set_w_hat(w0)
    s = Solver(p32)
    s.set_w_hat(w0)
    assert rel_err(s.nonlinear_rhs(w0), o.nonlinear_rhs(w0)) <= 5e-5
    s.close()
    e = Ensemble(p32, [n, n])
    for m in range(2):
        e.set_w_hat(m, w0)
    e.step_n(5, 1e-3)
    o.set_w_hat(w0)
    for _ in range(5):
        o.rk4_step(1e-3)
    for m in range(2):
        assert rel_err(e.get_w_hat(m), o.get_w_hat()) <= 1e-4
    e.close()
