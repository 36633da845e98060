"""What the library's calls hold of the device's memory, and what they do when little is left."""
import numpy as np
import pytest

from cushg_b200 import params as P
from cushg_b200 import shg

pytestmark = pytest.mark.gpu


def free_bytes():
    import torch
    return torch.cuda.mem_get_info()[0]


def test_release_gives_the_pool_back():
    """A gradient with every step kept takes 0.8 GB (256 x 256 FP64, 401 slices); the pool keeps it
    between calls until it is released, and the next call gives the same numbers."""
    import torch
    torch.cuda.synchronize()
    p = P.workload(256, 401, 6000.0, 20.0, 30.0, 3000.0, 30.0, precision=64)
    a = shg.grad(p, checkpoint_every=p.nz)
    held = free_bytes()
    shg.release_device_memory()
    assert free_bytes() - held >= 600 << 20
    b = shg.grad(p, checkpoint_every=p.nz)
    for key in ("sh_power", "d_waist", "d_focus", "d_temp"):
        assert a[key] == b[key]
    assert np.array_equal(a["d_poling"], b["d_poling"])
    held = free_bytes()
    shg.release_device_memory(1 << 40)  # keeps what is there
    assert free_bytes() == held


def small(i, precision=32, n=256):
    return P.workload(n, 2 + i % 2, 6000.0, 5.0 + i % 7, 30.0, 3000.0, 30.0, precision=precision)


def test_a_batch_of_more_runs_than_a_grid_dimension_holds():
    """66 000 powers-only 256 x 256 runs: two planes for each would take 69 GB, and 65 535 is the
    largest y and z of a grid.  Each equals its run alone."""
    count = 66000
    kinds = [small(i) for i in range(14)]
    alone = [shg.solve(p).sh_power for p in kinds]
    shg.release_device_memory()
    before = free_bytes()
    power = shg.solve_batch_device([kinds[i % 14] for i in range(count)])
    assert np.array_equal(power, np.array([alone[i % 14] for i in range(count)]))
    assert before - free_bytes() <= 1 << 30


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("count", [7, 257, 300])
def test_rounds_of_the_multipass_march(count, precision):
    """Automatic batches of 256 x 256 runs (the multi-pass march, in rounds) against the fused
    march: the same bits."""
    import torch
    dt = torch.complex128 if precision == 64 else torch.complex64
    res = []
    for march in (P.SHG_MARCH_AUTO, P.SHG_MARCH_FUSED):
        ps = [small(i, precision).replace(march=march) for i in range(count)]
        o = [[torch.empty((256, 256), dtype=dt, device="cuda") for _ in ps] for _ in range(2)]
        res.append((shg.solve_batch_device(ps, *o), o))
    (pa, a), (pb, b) = res
    assert np.array_equal(pa, pb)
    assert all(torch.equal(u, v) for f in range(2) for u, v in zip(a[f], b[f]))


def test_little_memory_left():
    """100 FP64 256 x 256 runs want 210 MB of planes; with 64 MB left they take the fused march,
    which wants none."""
    import torch
    ps = [small(i, 64) for i in range(100)]
    ref = shg.solve_batch_device(ps)                                         # both marches loaded
    assert np.array_equal(shg.solve_batch_device([p.replace(march=P.SHG_MARCH_FUSED) for p in ps]), ref)
    torch.cuda.synchronize()
    shg.release_device_memory()
    torch.cuda.empty_cache()
    hold = []
    try:
        while free_bytes() > 80 << 20:
            hold.append(torch.empty(min(free_bytes() - (64 << 20), 16 << 30), dtype=torch.uint8, device="cuda"))
        with pytest.raises(shg.ShgError) as e:                               # the 512 side has no other march
            shg.solve_batch_device([small(i, 64, 512) for i in range(20)])
        assert e.value.status == P.SHG_ERR_NOMEM
        assert np.array_equal(shg.solve_batch_device(ps), ref)
    finally:
        hold.clear()
        torch.cuda.empty_cache()
    assert np.array_equal(shg.solve_batch_device(ps), ref)
