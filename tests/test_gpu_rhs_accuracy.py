"""Accuracy of one FP32 evaluation of the nonlinear term, and of its adjoint."""
import numpy as np
import pytest

from ns2d import Solver, abi, initial

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,k0,seeds,bound", [(16, 2.0, 8, 2.61e-7), (64, 4.0, 8, 3.35e-7), (1024, 6.0, 2, 6.48e-7)])
def test_fp32_rhs_error_against_fp64(n, k0, seeds, bound):
    """Root-mean-square error of an FP32 RHS relative to the FP64 one, mean over
    seeded decaying spectra: no more than where U, V, w_x and w_y went through
    the x-transforms one by one with every twiddle a power of one table entry
    (the bounds are that form's errors)."""
    a, b = (Solver(abi.default_params(nx=n, ny=n, nu=1e-3, precision=q)) for q in (abi.FP32, abi.FP64))
    err = []
    for seed in range(seeds):
        w = initial.decaying(n, seed=100 + seed, k0=k0, dealias="2/3")
        w = w.astype(np.complex64).astype(np.complex128)
        want = b.nonlinear_rhs(w)
        err.append(np.linalg.norm(a.nonlinear_rhs(w) - want) / np.linalg.norm(want))
    a.close()
    b.close()
    assert np.mean(err) <= bound


@pytest.mark.parametrize("n,k0,bound", [(32, 2.0, 5.85e-8), (64, 4.0, 6.1e-8), (256, 6.0, 1.18e-7)])
def test_fp32_gradient_error_against_fp64(n, k0, bound):
    """The same for a reverse sweep over one step whose nonlinear part is as large
    as the linear one: the bounds are the errors with every multiplier (kx/k^2,
    ky/k^2) formed in FP64 and rounded once, term by term."""
    err = []
    for seed in range(6):
        w, lam = (initial.decaying(n, seed=s0 + seed, k0=k, dealias="2/3").astype(np.complex64).astype(np.complex128)
                  for s0, k in ((50, k0), (90, n / 8.0)))
        g = []
        for q in (abi.FP32, abi.FP64):
            s = Solver(abi.default_params(nx=n, ny=n, nu=1e-3, quirks=0, precision=q))
            s.set_w_hat(w)
            s.adjoint_record(1, 0.02, 1)
            g.append(s.adjoint_backward(lam))
            s.close()
        err.append(np.linalg.norm(g[0] - g[1]) / np.linalg.norm(g[1]))
    assert np.mean(err) <= bound
