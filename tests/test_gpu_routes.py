"""Which march and split plain calls take, from the names of the kernels they launch (the profiler's
records): the rule by the number of runs, and what tuned and pinned schedules do to it."""
import re

import pytest

from cushg_b200 import params as P
from cushg_b200 import shg

pytestmark = pytest.mark.gpu


def marches(call):
    """The march kernels that `call` launches: 'plain<float, 64, 4, 128>', 'wide<float, 128>',
    'multipass<float, 256>'."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    call()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    out = set()
    for e in prof.events():
        m = re.search(r"ssfm_plain_kernel<(\w+), (\d+), (\d+), (\d+)", e.name)
        if m:
            out.add("plain<%s, %s, %s, %s>" % m.groups())
        m = re.search(r"(ssfm_wide|mp_row)_kernel<(\w+), (\d+)", e.name)
        if m:
            out.add("%s<%s, %s>" % ("wide" if m.group(1) == "ssfm_wide" else "multipass", m.group(2), m.group(3)))
    return out


def run(n, precision=32, nz=4):
    return P.workload(n, nz, 6000.0, 20.0, 30.0, 3000.0, 30.0, precision=precision)


def batch(*classes):
    ps = [run(n) for n, count in classes for _ in range(count)]
    return lambda: shg.solve_batch_device(ps)


def test_rule_by_the_number_of_runs():
    assert marches(lambda: shg.solve(run(128))) == {"wide<float, 128>"}
    assert marches(lambda: shg.solve(run(48, 64))) == {"plain<double, 48, 16, 160>"}
    assert marches(batch((256, 20))) == {"multipass<float, 256>"}
    assert marches(batch((64, 160))) == {"plain<float, 64, 4, 128>"}
    assert marches(batch((128, 200))) == {"plain<float, 128, 2, 512>"}


def test_ends_of_the_rows_for_few_runs():
    """Where a variant's clusters no longer fit at once the next one is as fast or faster, and not a
    run later (16 runs of 192 x 192 FP32: 39.8 us per step on 8-CTA clusters, 37.4 on the default)."""
    assert marches(batch((192, 15))) == {"plain<float, 192, 8, 192>"}
    assert marches(batch((192, 16))) == {"plain<float, 192, 4, 384>"}
    assert marches(batch((192, 48))) == {"plain<float, 192, 8, 192>"}
    assert marches(batch((192, 51))) == {"plain<float, 192, 4, 384>"}
    assert marches(batch((256, 7))) == {"plain<float, 256, 16, 256>"}
    assert marches(batch((256, 8))) == {"multipass<float, 256>"}
    for count, march in [(4, "wide<double, 256>"), (7, "plain<double, 256, 16, 256>"), (8, "multipass<double, 256>")]:
        ps = [run(256, 64)] * count
        assert marches(lambda: shg.solve_batch_device(ps)) == {march}


def test_many_small_runs_beside_others():
    """Four-CTA clusters of 64 x 64 FP32 runs hold up clusters that need a whole SM: they are for
    batches of small sides, with at most three runs of 96 or 128 beside them."""
    for others in [(), ((32, 40),), ((48, 8),), ((96, 3),), ((128, 3),)]:
        assert "plain<float, 64, 4, 128>" in marches(batch((64, 160), *others)), others
    for others in [((96, 8),), ((128, 4),), ((96, 2), (128, 2)), ((256, 2),), ((192, 1),)]:
        assert "plain<float, 64, 1, 512>" in marches(batch((64, 160), *others)), others
    assert marches(batch((64, 140))) == {"plain<float, 64, 1, 512>"}


def test_many_small_runs_by_their_lengths():
    """One CTA per run is the faster split where the runs fill the device's waves (two full waves of
    equal runs) or where the longest bounds the batch."""
    assert marches(batch((64, 230))) == {"plain<float, 64, 4, 128>"}
    assert marches(batch((64, 296))) == {"plain<float, 64, 1, 512>"}
    assert marches(batch((64, 330))) == {"plain<float, 64, 4, 128>"}
    assert marches(batch((64, 444))) == {"plain<float, 64, 1, 512>"}
    ps = [run(64, nz=20 + i % 60) for i in range(200)]
    assert marches(lambda: shg.solve_batch_device(ps)) == {"plain<float, 64, 1, 512>"}
    ps = [run(64, nz=40 + i % 3) for i in range(200)]
    assert marches(lambda: shg.solve_batch_device(ps)) == {"plain<float, 64, 4, 128>"}



def test_256_fp32_runs_beside_smaller_ones():
    """While the batch's clusters do not fill the device the 256 x 256 FP32 runs of a mixed batch stay on
    clusters of their own; alone, in larger batches and beside 64 x 64 runs only they take the multi-pass march."""
    fused, multi = "plain<float, 256, 16, 256>", "multipass<float, 256>"
    for classes in [((256, 9), (192, 8), (128, 8), (64, 8)), ((256, 7), (192, 6), (128, 8)), ((256, 12), (192, 12), (64, 12))]:
        got = marches(batch(*classes))
        assert fused in got and multi not in got, classes
    for classes in [((256, 9),), ((256, 9), (64, 100)), ((256, 30), (192, 30)), ((256, 13), (128, 1)), ((256, 8), (192, 40)),
                    ((256, 9), (512, 2), (192, 8))]:
        got = marches(batch(*classes))
        assert multi in got and fused not in got, classes



def test_wide_march_in_a_mixed_batch():
    """A cooperative launch has the device to itself, so the classes beside it wait: a mixed batch takes it
    where its class bounds the batch, and clusters side by side where another class does."""
    def got(n_large, n_small):
        ps = [run(192, 64, nz=n_large)] + [run(64, 64, nz=n_small)] * 3
        return marches(lambda: shg.solve_batch_device(ps))
    assert got(60, 5) == {"wide<double, 192>", "plain<double, 64, 16, 256>"}
    assert got(6, 60) == {"plain<double, 192, 16, 192>", "plain<double, 64, 16, 256>"}


@pytest.fixture
def no_choices():
    shg.autotune_reset()
    yield
    shg.autotune_reset()


def test_the_class_tuner_starts_from_the_automatic_choice(no_choices):
    """256 x 256 batches are automatically on the multi-pass march, 1.4 times as fast as the fused
    splits on a full device: the tuner's reference rate is that march's, and it stays automatic."""
    r = shg.autotune(32, 256)
    assert r["automatic"] and r["cluster"] == 0
    assert r["pt_steps_per_s"] == r["default_pt_steps_per_s"]
    assert marches(batch((256, 60))) == {"multipass<float, 256>"}


def test_tuning_a_sweep_leaves_single_runs_alone(no_choices):
    """Whatever the tuners choose for large batches, single runs and small batches of the classes keep
    the variants they have of their own."""
    ps = [run(n, nz=30) for n in (64, 128, 192, 256) for _ in range(24)]
    res = shg.autotune_batch(ps)
    assert sorted(r["n"] for r in res) == [64, 128, 192, 256]
    shg.autotune(32, 128)
    assert marches(lambda: shg.solve(run(128))) == {"wide<float, 128>"}
    assert marches(lambda: shg.solve(run(64))) == {"plain<float, 64, 16, 128>"}
    assert marches(batch((128, 5))) == {"plain<float, 128, 16, 256>"}
    for r in res:  # and each result can be set again
        if not r["automatic"]:
            shg.set_schedule(r["precision"], r["n"], r["cluster"], r["threads"])


def test_tuning_a_small_batch_keeps_the_faster_march(no_choices):
    """Two 128 x 128 FP32 runs take 6.5 us per step on the wide march and 30 on the fused one."""
    ps = [run(128, nz=60), run(128, nz=60)]
    r = shg.autotune_batch(ps)[0]
    assert r["automatic"] and r["pt_steps_per_s"] == r["default_pt_steps_per_s"]
    assert marches(lambda: shg.solve_batch_device(ps)) == {"wide<float, 128>"}


def test_a_pinned_schedule_holds_for_single_runs_too(no_choices):
    shg.set_schedule(32, 128, 2, 256)
    assert marches(lambda: shg.solve(run(128))) == {"plain<float, 128, 2, 256>"}
    assert marches(batch((128, 5))) == {"plain<float, 128, 2, 256>"}
