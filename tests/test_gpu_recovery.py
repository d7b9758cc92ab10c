"""Runs after one that failed: the failure is reported once and leaves nothing behind."""
import numpy as np
import pytest

import feyntrop_gb300 as ft
from feyntrop_gb300 import workloads

pytestmark = pytest.mark.gpu


def test_a_refused_allocation_fails_one_run_only():
    """1e13 mixed samples want a hand-off queue of 25 TB, which the host refuses; the plan and the
    others go on as if it had not been asked."""
    p, fresh = ft.Plan(workloads.k4_euclidean()), ft.Plan(workloads.k4_euclidean())
    want = [fresh.integrate(50_001, seed=4, precision=prec)["moments"] for prec in (ft.MIXED, ft.FP64)]
    with pytest.raises(ft.FeyntropError):
        p.integrate(10**13, seed=4, precision=ft.MIXED)
    assert p.integrate(50_001, seed=4, precision=ft.MIXED)["moments"] == want[0]
    with pytest.raises(ft.FeyntropError):
        p.integrate(10**13, seed=4, precision=ft.MIXED)
    assert fresh.integrate(50_001, seed=4, precision=ft.FP64)["moments"] == want[1]
    b = ft.Batch([fresh], ft.FP64)
    r = b.run([50_001], seeds=[4])[0]
    assert r["kept"] == 50_001 and np.isfinite(r["integral"]).all()
    b.close()
    p.close()
    fresh.close()


def test_a_run_after_a_failed_one_on_another_stream():
    """The failed run has launched its stride matrices and stopped before the sampling kernel; the next
    ones, on other streams, with its stride and others, give a fresh plan's values."""
    import torch
    p, fresh = ft.Plan(workloads.double_box()), ft.Plan(workloads.double_box())
    streams = [torch.cuda.Stream() for _ in range(3)]
    for n, s in ((70_001, 0), (500, 1), (2_000_003, 2), (70_001, 1)):
        with pytest.raises(ft.FeyntropError):
            p.integrate(10**13, seed=1, precision=ft.MIXED, stream=streams[(s + 1) % 3].cuda_stream)
        got = p.integrate(n, seed=2, precision=ft.MIXED, stream=streams[s].cuda_stream)
        want = fresh.integrate(n, seed=2, precision=ft.MIXED)
        assert got["moments"] == want["moments"] and got["kept"] == want["kept"]
    p.close()
    fresh.close()
