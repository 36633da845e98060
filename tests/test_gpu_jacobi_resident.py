"""The resident Jacobi kernel (many sweeps in one cooperative launch, T in shared memory) against
one sweep per launch (jacobi_block = 1), through the C ABI: the same bits, for every grid side it
is built for, tiles of one plane to several groups of planes with remainders, both boundary
models, odd and even sweep counts.  No tolerance is involved."""
import numpy as np
import pytest

from cushg_b200 import params as P
from cushg_b200 import shg

pytestmark = pytest.mark.gpu


def setup(n, nz, precision, boundary):
    import torch
    p = P.workload(n, nz, 9000.0, 30.0, 40.0, 4500.0, 40.0, precision=precision, thermal=1)
    p.boundary, p.ly, p.h_conv, p.t_inf = boundary, p.lx * 0.9, 3e-8, 22.0
    dt = torch.float64 if precision == 64 else torch.float32
    g = torch.Generator(device="cuda").manual_seed(n + nz)
    T = 40.0 + torch.rand((nz, n, n), dtype=dt, device="cuda", generator=g)
    Q = torch.rand((nz, n, n), dtype=dt, device="cuda", generator=g) * 60.0 * p.kappa / p.lx ** 2
    return p, T, Q


@pytest.mark.parametrize("boundary", [0, 1])
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("n,nz,sweeps", [(32, 3, 8), (32, 149, 9), (64, 40, 11), (64, 201, 8), (128, 9, 8), (128, 46, 9),
                                         (128, 200, 30), (256, 5, 9), (256, 52, 8), (256, 60, 9)])
def test_resident_equals_one_sweep_per_launch(n, nz, sweeps, precision, boundary):
    import torch
    p, T, Q = setup(n, nz, precision, boundary)
    A, B = T.clone(), T.clone()
    shg.heat_sweeps_device(p, A, Q, sweeps)
    shg.heat_sweeps_device(p.replace(jacobi_block=1), B, Q, sweeps)
    assert torch.equal(A, B)
    assert not torch.equal(A, T)


@pytest.mark.parametrize("n,precision", [(64, 32), (128, 64)])
def test_thermal_run_equals_one_sweep_per_launch(n, precision):
    p = P.workload(n, 21, 6000.0, 25.0, 30.0, 3000.0, 31.0, precision=precision, thermal=1)
    p.alpha_p, p.alpha_s, p.beta_s = 2e-5, 1e-4, 1e-3
    p.max_outer, p.conv_rule, p.check_every, p.jacobi_tol = 3, P.SHG_CONV_MAXABS, 50, 2e-4
    a, b = shg.solve(p, want_temperature=True), shg.solve(p.replace(jacobi_block=1), want_temperature=True)
    assert a.stats.jacobi_sweeps == b.stats.jacobi_sweeps > 50
    assert a.stats.outer_iterations == b.stats.outer_iterations
    assert np.array_equal(a.temperature, b.temperature) and np.array_equal(a.signal, b.signal)


def test_tangent_sweeps_without_a_source():
    """The tangent's first sweeps have no heat source (its own instantiation)."""
    p = P.workload(256, 9, 4000.0, 30.0, 25.0, 2000.0, 34.0, precision=64, thermal=1)
    p.alpha_p, p.alpha_s, p.beta_s = 2e-5, 1e-4, 1e-3
    p.conv_rule, p.max_sweeps, p.max_outer = P.SHG_CONV_FIXED, 40, 2
    a, b = shg.thermal_grad(p), shg.thermal_grad(p.replace(jacobi_block=1))
    assert a["d_temp"] == b["d_temp"] and a["sh_power"] == b["sh_power"]
