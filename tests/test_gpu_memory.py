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
