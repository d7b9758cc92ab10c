"""Plans whose table goes to the device through pinned staging and ones whose table is too large for that, in
turn, on their own streams and on the caller's."""
import random

import pytest

import feyntrop_gb300 as ft

pytestmark = pytest.mark.gpu


def ladder(loops):
    """Two-point ladder of 3 loops + 1 edges, Euclidean, unit-order masses."""
    n = loops + 1
    g = [[[i, n + i], 1] for i in range(n)] + [[[i, i + 1], 1] for i in range(loops)]
    g += [[[n + i, n + i + 1], 1] for i in range(loops)]
    top = {0: 0, 2 * n - 1: 1}   # the external vertices first
    for v in range(1, 2 * n - 1):
        top[v] = v + 1
    P = [[0.0] * (2 * n) for _ in range(2 * n)]
    P[0][0] = P[1][1] = -1.0
    P[0][1] = P[1][0] = 1.0
    rng = random.Random(loops)
    return {"graph": [[[top[a], top[b]], w] for (a, b), w in g], "dimension": 4, "scalarproducts": P,
            "masses_sqr": [rng.uniform(0.5, 3) for _ in g], "num_eps_terms": 1, "lambda": 0, "N": 1000, "seed": 0}


def test_staged_and_unstaged_tables_in_turn():
    import torch
    stream = torch.cuda.Stream()
    inputs = {E: ladder((E - 1) // 3) for E in (4, 16, 19)}   # 1 KB, 2.9 MB and 23 MB
    want = {}
    for E in (19, 4, 16, 19, 4, 19, 16):
        p = ft.Plan(inputs[E])
        got = p.integrate(20_001, seed=3, precision=ft.MIXED, stream=stream.cuda_stream)["moments"]
        assert got == want.setdefault(E, got)
        assert p.integrate(20_001, seed=3, precision=ft.MIXED)["moments"] == got
        # a batch copies the table by itself; positive terms, 100-bit sums in another order
        (one, _), _ = p.integrate(20_001, seed=3, precision=ft.FP64)["integral"][0]
        b = ft.Batch([p], ft.FP64)
        (two, _), _ = b.run([20_001], seeds=[3])[0]["integral"][0]
        assert abs(one - two) <= 1e-12 * abs(one)
        b.close()
        p.close()
