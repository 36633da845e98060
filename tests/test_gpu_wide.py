"""The marches of single runs and small batches (one instance over the whole GPU, or for small sides
over a 16-CTA cluster with a thread per field) against the fused and multi-pass marches of the same instance, through the C ABI.

All marches write every operation a field value passes through with explicit rounding, so the
fields and powers must be the same bits; no tolerance is involved."""
import numpy as np
import pytest

from cushg_b200 import params as P
from cushg_b200 import shg

pytestmark = pytest.mark.gpu

SIDES = [32, 48, 64, 96, 128, 192, 256, 512]


def case(n, precision, nz, seed, thermal=0):
    rng = np.random.default_rng(seed)
    p = P.workload(n, nz, 6000.0, float(rng.uniform(5, 40)), float(rng.uniform(20, 45)), float(rng.uniform(0, 6000.0)),
                   float(rng.uniform(25, 45)), precision=precision, thermal=thermal)
    if not thermal:
        p.rho_p, p.rho_s = float(rng.uniform(0, 0.01)), float(rng.uniform(0, 0.01))
    p.ly = p.lx * 0.9
    return p


def other(p):
    """The same run on the march a large batch takes."""
    multi = p.nx == 512 or (p.thermal and p.nx >= 128)
    return p.replace(march=P.SHG_MARCH_MULTIPASS if multi else P.SHG_MARCH_FUSED)


@pytest.mark.parametrize("nz", [2, 3, 12])
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("n", SIDES)
def test_single_run_equals_batch_march(n, precision, nz):
    p = case(n, precision, nz, seed=n + nz)
    a, b = shg.solve(p), shg.solve(other(p))
    assert np.array_equal(a.pump, b.pump) and np.array_equal(a.signal, b.signal)
    assert a.sh_power == b.sh_power and a.stats.pump_power == b.stats.pump_power


@pytest.mark.parametrize("n,precision", [(48, 32), (96, 64), (256, 32)])
def test_signal_in_and_slices(n, precision):
    p = case(n, precision, 5, seed=3)
    rng = np.random.default_rng(0)
    s0 = (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))) * 1e-6
    a, b = shg.solve(p, signal_in=s0), shg.solve(other(p), signal_in=s0)
    assert np.array_equal(a.signal, b.signal) and np.array_equal(a.pump, b.pump)
    sa, sb = shg.solve_slices(p, signal_in=s0), shg.solve_slices(other(p), signal_in=s0)
    assert np.array_equal(sa[0], sb[0]) and np.array_equal(sa[1], sb[1])


def test_poling_and_guard():
    p = case(128, 64, 9, seed=5)
    pol = np.random.default_rng(1).normal(0.0, 0.3, p.nz - 1)
    assert shg.sh_power(p, pol) == shg.sh_power(other(p), pol)
    q = case(64, 32, 9, seed=6)
    q.fp32_guard = 1e-12  # marches in FP64, writes FP32
    a, b = shg.solve(q), shg.solve(other(q))
    assert a.signal.dtype == np.complex64 and np.array_equal(a.signal, b.signal) and a.sh_power == b.sh_power


@pytest.mark.parametrize("sides", [[256, 256], [64, 96, 128, 32], [512], [64] * 40, [128, 256, 256, 256]])
@pytest.mark.parametrize("precision", [64, 32])
def test_batches_on_either_side_of_the_rule(precision, sides):
    """Batches that fit the device side by side take the wide march, larger ones do not; the
    instances are those of single runs either way, and a plan replays the direct call."""
    import torch
    ps = [case(n, precision, 5 + i % 3, seed=i) for i, n in enumerate(sides)]
    dt = torch.complex128 if precision == 64 else torch.complex64
    outs = [[torch.empty((p.ny, p.nx), dtype=dt, device="cuda") for p in ps] for _ in range(2)]
    power = shg.solve_batch_device(ps, *outs)
    for i, p in enumerate(ps):
        r = shg.solve(p)
        assert np.array_equal(outs[1][i].cpu().numpy(), r.signal) and np.array_equal(outs[0][i].cpu().numpy(), r.pump), i
        assert power[i] == r.sh_power, i
    plan = shg.BatchPlan(ps, *outs)
    try:
        plan.launch()
        assert np.array_equal(plan.powers(), power)
    finally:
        plan.close()


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("n", [32, 48, 64, 96, 128, 192])
def test_every_split_for_few_runs(n, precision):
    """Batches of every size range that has a variant of its own, against the default variant."""
    import torch
    dt = torch.complex128 if precision == 64 else torch.complex64
    for count in [1, 3, 8, 15, 29, 49, 73, 105] if n < 192 else [1, 10, 20, 40]:
        ps = [case(n, precision, 3 + i % 2, seed=i) for i in range(count)]
        res = []
        for qs in (ps, [other(p) for p in ps]):
            o = [[torch.empty((n, n), dtype=dt, device="cuda") for _ in qs] for _ in range(2)]
            res.append((shg.solve_batch_device(qs, *o), o))
        (pa, a), (pb, b) = res
        assert np.array_equal(pa, pb), count
        assert all(torch.equal(u, v) for f in range(2) for u, v in zip(a[f], b[f])), count


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("n", [32, 64, 128])
def test_gradient_splits(n, precision):
    """Gradients of one instance in batches of every size range that has a split of its own.  The
    fields and per-job terms are the same bits; up to 1e6 of them are added in FP64 in another order
    (1e-16 each, times a cancellation of up to 1e4 near an optimum: 1e-10 with room)."""
    p = case(n, precision, 11, seed=2).replace(rho_p=0.0, rho_s=0.0)
    p.ly = p.lx
    ref = shg.grad(p, checkpoint_every=4)
    for count in (8, 15, 33, 37):
        g = shg.grad_batch([p] + [p.replace(power=5.0 + i) for i in range(count - 1)], checkpoint_every=4)[0]
        for key in ("sh_power", "d_waist", "d_focus", "d_temp"):
            assert abs(g[key] - ref[key]) <= 1e-10 * abs(ref[key]), (count, key)
        assert np.abs(g["d_poling"] - ref["d_poling"]).max() <= 1e-10 * np.abs(ref["d_poling"]).max(), count


@pytest.mark.parametrize("n,precision,count", [(32, 64, 1), (64, 32, 1), (128, 64, 1), (128, 32, 9), (256, 32, 1),
                                               (256, 64, 5), (512, 32, 2), (512, 64, 1)])
def test_thermal_equals_batch_march(n, precision, count):
    """A thermal batch's optical passes on the wide march (few instances) and on
    the march of large batches."""
    import torch
    ps = []
    for i in range(count):
        p = case(n, precision, 7, seed=i, thermal=1)
        p.alpha_p, p.alpha_s, p.beta_s = 2e-5, 1e-4, 1e-3
        p.conv_rule, p.max_sweeps, p.max_outer = P.SHG_CONV_FIXED, 20, 2
        p.lx = p.ly = 300.0
        ps.append(p)
    cdt, rdt = (torch.complex128, torch.float64) if precision == 64 else (torch.complex64, torch.float32)

    def run(qs):
        pump = [torch.empty((n, n), dtype=cdt, device="cuda") for _ in qs]
        sig = [torch.empty((n, n), dtype=cdt, device="cuda") for _ in qs]
        T = [torch.empty((7, n, n), dtype=rdt, device="cuda") for _ in qs]
        st, _ = shg.thermal_batch(qs, pump, sig, T)
        return pump, sig, T, [(s.sh_power, s.pump_power) for s in st]

    a, b = run(ps), run([other(p) for p in ps])
    for x, y in zip(a[:3], b[:3]):
        assert all(torch.equal(u, v) for u, v in zip(x, y))
    assert a[3] == b[3] and all(s > 0 for s, _ in a[3])
