"""Powers against the output fields they are sums of, through the C ABI: for every march of single
runs and small batches, each power over its field's sum of |.|^2 is one constant of the parameter
set (0.5 eps0 c n dx dy), whatever the step count.

Tolerance: the device and numpy add N^2 <= 6.6e4 FP64 terms of one sign in different orders; each of
the at most 16 roundings of a pairwise or row-wise sum is below 1.2e-16, and of the 256 additions of a
sequential part 3e-14: 1e-13."""
import numpy as np
import pytest

from cushg_b200 import params as P
from cushg_b200 import shg

pytestmark = pytest.mark.gpu


def case(n, precision, nz):
    p = P.workload(n, nz, 6000.0, 20.0, 30.0, 3000.0, 30.0, precision=precision)
    p.lz = 500.0 * (nz - 1)  # the same dz
    return p


def ratio(power, field):
    return power / np.sum(np.abs(np.asarray(field, np.complex128)) ** 2)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("n", [32, 48, 64, 96, 128, 192, 256])
def test_powers_are_the_sums_of_the_fields(n, precision):
    import torch
    ref = shg.solve(case(n, precision, 4).replace(march=P.SHG_MARCH_FUSED))
    rs, rp = ratio(ref.sh_power, ref.signal), ratio(ref.stats.pump_power, ref.pump)
    for nz in (2, 3, 5, 8) * 4:
        a = shg.solve(case(n, precision, nz))
        assert abs(ratio(a.sh_power, a.signal) / rs - 1) <= 1e-13, nz
        assert abs(ratio(a.stats.pump_power, a.pump) / rp - 1) <= 1e-13, nz
    dt = torch.complex128 if precision == 64 else torch.complex64
    for count in (2, 7, 14, 15, 40):
        ps = [case(n, precision, 2 + i % 5) for i in range(count)]
        sig = [torch.empty((n, n), dtype=dt, device="cuda") for _ in ps]
        power = shg.solve_batch_device(ps, None, sig)
        for i in range(count):
            assert abs(ratio(power[i], sig[i].cpu().numpy()) / rs - 1) <= 1e-13, (count, i)
