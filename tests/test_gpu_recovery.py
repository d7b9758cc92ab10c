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
