"""bench.py's roofline speaks of the kernels that the timed solves ran: the step kernels, or a small LP's
cluster kernel, whose profiled solves run other kernels."""
from types import SimpleNamespace

import pytest

import bench

BM = {"primal_commit": 300_000, "primal_plain": 200_000, "dual": 180_000, "dual_commit_extra": 30_000}


def _result(kernels, accepted=760, rejected=8):
    return SimpleNamespace(kernels_launched=kernels, accepted_steps=accepted, rejected_steps=rejected,
                           primal_spmv_launches=760, step_loop_device_sec=6e-3, primal_kernel_launches=768,
                           primal_kernel_sec=4e-3, dual_kernel_sec=5e-3)


def test_route_from_the_launches():
    assert bench.on_cluster([_result(160)] * 3)
    assert not bench.on_cluster([_result(1700)] * 3)


def test_cluster_kernel_from_its_own_time():
    r = bench.cluster_roofline([_result(160)] * 2, BM, 6790.0, "file")
    moved = 2 * (760 * 300_000 + 8 * 200_000 + 768 * 180_000 + 760 * 30_000)
    assert (r["kernel"], r["bound"]) == ("cluster_kernel", "latency")
    assert r["achieved"] == pytest.approx(moved / 12e-3 / 1e9)
    assert r["us_per_attempt"] == pytest.approx(6e-3 / 768 * 1e6)


def test_step_kernels_from_their_events():
    r = bench.step_roofline([_result(1700)], BM, 6790.0, "file", "plain", "FP64")
    assert (r["kernel"], r["bound"]) == ("dual_step_kernel", "hbm")
    assert r["achieved"] == pytest.approx((768 * 180_000 + 760 * 30_000) / 5e-3 / 1e9)
