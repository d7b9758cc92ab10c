"""Scratch that closed plans leave to later ones can be given back."""
import pytest

import feyntrop_gb300 as ft
from feyntrop_gb300 import workloads

pytestmark = pytest.mark.gpu


def test_idle_scratch_is_given_back():
    import torch

    def use():
        plans = [ft.Plan(workloads.k4_euclidean()) for _ in range(6)]
        out = [p.integrate(1_000_001, seed=k, precision=ft.MIXED)["moments"] for k, p in enumerate(plans)]
        for p in plans:
            p.close()
        return out

    want = use()   # the kernels are loaded, the driver's own pools grown
    ft.release_scratch()
    free = torch.cuda.mem_get_info()[0]
    assert use() == want
    assert torch.cuda.mem_get_info()[0] <= free - 6 * 2**20   # 1.3 MB of matrices and 5 MB of queue each
    ft.release_scratch()
    assert torch.cuda.mem_get_info()[0] >= free
    ft.release_scratch()   # nothing left to free
    assert use() == want


def test_idle_scratch_makes_room_for_a_run():
    """A refused allocation is tried once more without the idle sets, which are gone afterwards."""
    import torch
    p = ft.Plan(workloads.k4_euclidean())

    def scenario():
        others = [ft.Plan(workloads.k4_euclidean()) for _ in range(4)]
        for q in others:
            q.integrate(1_000_001, precision=ft.MIXED)
        for q in others:
            q.close()
        held = torch.cuda.mem_get_info()[0]
        with pytest.raises(ft.FeyntropError):
            p.integrate(10**13, precision=ft.MIXED)
        return held, torch.cuda.mem_get_info()[0]

    for _ in range(5):   # a refused run leaves its plan one stride's matrices more, up to four
        free = scenario()[1]
    held, after = scenario()
    assert held < free and after >= free
    p.close()
