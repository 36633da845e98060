"""The direct heat solve at grids that pick each tile of its transform products (32, 64 and 128
wide), each depth of its finishing pass, and either transformed direction beside x (y, or z with
its closed-form modes), with odd and even slice counts, both boundary models and heat transfer
from none to far above a Dirichlet face's, through the C ABI.

Reference: the solution is a fixed point of the pinned Jacobi sweep (one FP64 sweep moves it by
rounding only, <= 1e-10 K, as in test_gpu_heat_direct), and the returned residual says the same."""
import numpy as np
import pytest

from cushg_b200 import params as P
from cushg_b200 import shg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nz,boundary", [(16, 3, 0), (32, 9, 1), (48, 21, 0), (64, 50, 1), (96, 37, 1), (98, 11, 0),
                                           (128, 100, 0), (192, 61, 1), (256, 33, 0), (512, 5, 1)])
def test_steady_is_a_fixed_point(n, nz, boundary, h_conv=None):
    import torch
    p = P.workload(n, nz, 8000.0, 20.0, 30.0, 4000.0, 40.0, precision=64, thermal=1)
    p.boundary = boundary
    p.h_conv = p.h_conv if h_conv is None else h_conv
    g = torch.Generator(device="cuda").manual_seed(n + nz)
    T = torch.full((nz, n, n), 40.0, dtype=torch.float64, device="cuda")
    Q = torch.rand((nz, n, n), dtype=torch.float64, device="cuda", generator=g) * 60.0 * p.kappa / p.lx ** 2
    resid = shg.heat_steady_device(p, T, Q)
    after = T.clone()
    shg.heat_sweeps_device(p, after, Q, 1)
    moved = float((after - T).abs().max())
    assert np.isfinite(moved) and moved <= 1e-10 and resid <= 1e-10
    assert float((T - 40.0).abs().max()) > 1e-6  # the source did heat it


@pytest.mark.parametrize("n,nz,boundary,h_conv", [(64, nz, 0, h) for nz in (3, 4, 5) for h in (0.0, 1e-14, 1e-6, 1e-2)]
                         + [(64, 4, 1, 0.0), (64, 5, 1, 1e-2), (256, 101, 0, 1e-9), (512, 12, 1, 1e-2)])
def test_z_modes_over_heat_transfer(n, nz, boundary, h_conv):
    """Biot numbers of the z faces from 0 to far above 1 (theta of the modes from the Neumann to
    nearly the Dirichlet values, and the mode that turns hyperbolic)."""
    test_steady_is_a_fixed_point(n, nz, boundary, h_conv)
