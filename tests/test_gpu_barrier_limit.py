"""The bounded waits of the cooperative launches (wide march, resident Jacobi sweeps): a wait that
runs out ends the kernel, every call that waits for its results returns SHG_ERR_CUDA, with or
without statistics, and the device stays usable.  The wait is made to run out by a barrier target
one above the number of arriving CTAs (shg_selftest_withhold_arrival)."""
import ctypes

import numpy as np
import pytest

from cushg_b200 import params as P
from cushg_b200 import shg

pytestmark = pytest.mark.gpu

WAIT_US = 300.0


@pytest.fixture
def withheld():
    """Calls made inside `with withheld:` wait in vain."""
    class Withheld:
        def __enter__(self):
            shg.selftest_withhold_arrival(WAIT_US)

        def __exit__(self, *exc):
            shg.selftest_withhold_arrival(0.0)

    yield Withheld()
    shg.selftest_withhold_arrival(0.0)


def plain(n=128, precision=32):
    return P.workload(n, 6, 6000.0, 20.0, 30.0, 3000.0, 30.0, precision=precision)


def thermal(n, precision, heat=P.SHG_HEAT_DIRECT):
    p = P.workload(n, 7, 6000.0, 20.0, 30.0, 3000.0, 30.0, precision=precision, thermal=1)
    p.alpha_p, p.alpha_s, p.beta_s = 2e-5, 1e-4, 1e-3
    p.conv_rule, p.max_sweeps, p.max_outer, p.heat_solver = P.SHG_CONV_FIXED, 20, 2, heat
    p.lx = p.ly = 300.0
    return p


def expect_ran_out(call):
    with pytest.raises(shg.ShgError) as e:
        call()
    assert e.value.status == P.SHG_ERR_CUDA and "ran out" in str(e.value)


def buffers(p):
    dt = np.complex128 if p.precision == 64 else np.complex64
    return np.empty((p.ny, p.nx), dt), np.empty((p.ny, p.nx), dt)


@pytest.mark.parametrize("n,precision", [(128, 32), (256, 64), (512, 32)])
def test_single_runs(n, precision, withheld):
    p = plain(n, precision)
    before = shg.solve(p)
    L = shg.lib()
    a, b = buffers(p)
    sl = np.empty((p.nz, n, n), a.dtype)
    ptr = lambda x: ctypes.c_void_p(x.ctypes.data)  # noqa: E731
    with withheld:
        expect_ran_out(lambda: shg.solve(p))
        expect_ran_out(lambda: shg.sh_power(p, None))
        # host buffers without statistics
        assert L.shg_solve(ctypes.byref(p), None, ptr(a), ptr(b), None, None) == P.SHG_ERR_CUDA
        assert L.shg_solve_slices(ctypes.byref(p), None, ptr(sl), None, None, None) == P.SHG_ERR_CUDA
    after = shg.solve(p)
    assert np.array_equal(after.signal, before.signal) and after.sh_power == before.sh_power
    assert L.shg_solve(ctypes.byref(p), None, ptr(a), ptr(b), None, None) == P.SHG_OK
    assert np.array_equal(b, before.signal)


def test_batches_and_plans(withheld):
    import torch
    ps = [plain(256, 32), plain(192, 32).replace(power=11.0)]
    outs = [[torch.empty((p.ny, p.nx), dtype=torch.complex64, device="cuda") for p in ps] for _ in range(2)]
    power = shg.solve_batch_device(ps, *outs)
    L = shg.lib()
    arr = (shg.ShgParams * 2)(*ps)
    host = [buffers(p) for p in ps]
    vp = ctypes.c_void_p
    hp, hs = ((vp * 2)(*[vp(h[k].ctypes.data) for h in host]) for k in range(2))
    with withheld:
        expect_ran_out(lambda: shg.solve_batch_device(ps, *outs))
        assert L.shg_solve_batch(arr, 2, hp, hs, None) == P.SHG_ERR_CUDA
        plan = shg.BatchPlan(ps, *outs)
    try:
        plan.launch()
        expect_ran_out(plan.powers)
    finally:
        plan.close()
    assert L.shg_solve_batch(arr, 2, hp, hs, None) == P.SHG_OK
    assert np.array_equal(shg.solve_batch_device(ps, *outs), power)
    for i in range(2):
        assert np.array_equal(host[i][1], outs[1][i].cpu().numpy())


@pytest.mark.parametrize("n,precision", [(64, 64), (128, 32), (512, 32)])
def test_thermal_optical_passes(n, precision, withheld):
    import torch
    p = thermal(n, precision)
    before = shg.solve(p)
    L = shg.lib()
    a, b = buffers(p)
    ptr = lambda x: ctypes.c_void_p(x.ctypes.data)  # noqa: E731
    dt = torch.complex128 if precision == 64 else torch.complex64
    sig = torch.empty((n, n), dtype=dt, device="cuda")
    arr = (shg.ShgParams * 1)(p)
    ds = (ctypes.c_void_p * 1)(ctypes.c_void_p(sig.data_ptr()))
    with withheld:
        expect_ran_out(lambda: shg.solve(p))
        assert L.shg_solve(ctypes.byref(p), None, ptr(a), ptr(b), None, None) == P.SHG_ERR_CUDA
        assert L.shg_thermal_batch(arr, 1, None, ds, None, None, None, None) == P.SHG_ERR_CUDA
    after = shg.solve(p)
    assert np.array_equal(after.signal, before.signal) and after.sh_power == before.sh_power
    assert after.stats.pump_power == before.stats.pump_power


@pytest.mark.parametrize("precision", [64, 32])
def test_resident_sweeps(precision, withheld):
    import torch
    p = thermal(64, precision, heat=P.SHG_HEAT_JACOBI).replace(nz=40)
    dt = torch.float64 if precision == 64 else torch.float32
    T = torch.full((40, 64, 64), 30.0, dtype=dt, device="cuda")
    Q = torch.zeros_like(T)
    with withheld:
        expect_ran_out(lambda: shg.heat_sweeps_device(p, T, Q, 50))
        expect_ran_out(lambda: shg.solve(p))
    a, b = torch.full_like(T, 30.0), torch.full_like(T, 30.0)
    shg.heat_sweeps_device(p, a, Q, 50)
    shg.heat_sweeps_device(p.replace(jacobi_block=1), b, Q, 50)
    assert torch.equal(a, b)


def test_argument_is_checked():
    for bad in (-1.0, float("nan"), 1e9):
        with pytest.raises(shg.ShgError) as e:
            shg.selftest_withhold_arrival(bad)
        assert e.value.status == P.SHG_ERR_INVALID
