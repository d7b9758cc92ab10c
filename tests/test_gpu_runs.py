"""What surrounds the samples: the FP64 form's functions at extreme edge weights, its sums over few
and many threads and blocks, work items sized by a run's counts, samples whose derivatives are
taken by the general route, and scratch that passes from plan to plan."""
import random
import threading

import numpy as np
import pytest

import feyntrop_gb300 as ft
import oracle_lib as ol
from feyntrop_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nu", [0.02, 0.3, 7.5, 60.0])
def test_fp64_powers_at_extreme_weights(nu):
    """1/r from 1/120 to 50: X = prod (1 - u)^(1/r) within 50 |log(1 - u)| 2^-52 < 1e-12, and the
    positive one-loop integrand moves by at most its degree (below 200) times that."""
    inp = {"graph": [[[0, 1], nu], [[0, 1], nu]], "dimension": 1 if nu < 0.1 else 2, "scalarproducts": [[-1.0, 1.0], [1.0, -1.0]],
           "masses_sqr": [1.0, 2.0], "num_eps_terms": 2, "lambda": 0, "N": 1000, "seed": 0}
    if nu < 0.1:
        inp["graph"] = [[[0, 1], 1], [[0, 1], nu]]
    p = ft.Plan(inp)
    ref = ol.Prepared(inp).samples(3, 0, 4096)
    rec = p.records(4096, seed=3, precision=ft.FP64)
    p.close()
    assert (rec["order"] == ref["order"]).all()
    ok = ref["X"] > 1e-290
    assert (np.abs(rec["X"] - ref["X"])[ok] <= 1e-12 * ref["X"][ok]).all()
    fin = np.isfinite(ref["R"]).all(axis=1) & ok.all(axis=1)
    assert fin.sum() > 4000
    assert (np.abs(rec["R"] - ref["R"])[fin].max(axis=1) <= 2e-10 * np.abs(ref["R"][fin]).max(axis=1)).all()


@pytest.mark.parametrize("n", [1, 31, 400, 5003, 200_001])
def test_fp64_sums(n):
    """The launch's sums against the records' (the sums keep 100 bits; the mean is rounded once)."""
    for inp in (workloads.k4_euclidean(), workloads.box_pentagon(random.Random(2))):
        p = ft.Plan(inp)
        r = p.integrate(n, seed=4, precision=ft.FP64)
        R = p.records(n, seed=4, precision=ft.FP64)["R"]
        R = R[np.isfinite(R).all(axis=1)]
        assert r["kept"] == len(R)
        for j, ((re, _), (im, _)) in enumerate(r["integral"]):
            for got, x in ((re, R[:, j].real), (im, R[:, j].imag)):
                assert abs(got - x.mean()) <= 1e-13 * np.abs(x).mean(), (n, j)
        p.close()


def test_fp64_batch_items_follow_the_counts():
    """Counts for which every chunk from the smallest to the largest is taken, in one batch that
    keeps its buffers and graph: the single integrals' values (1e-12 of the mean magnitude, sums in
    another order), the same bits when a run is repeated after others."""
    plans = [ft.Plan(workloads.box_pentagon(random.Random(k))) for k in range(3)] + [ft.Plan(workloads.k4_euclidean())]
    b = ft.Batch(plans, ft.FP64)
    seen = {}
    for Ns in ([7, 1, 0, 3], [900_001, 300, 70_000, 2_000_003], [60_000, 60_001, 59_999, 250_000],
               [200_000, 150_000, 111_111, 600_000], [7, 1, 0, 3], [900_001, 300, 70_000, 2_000_003]):
        out = b.run(Ns, seeds=[5, 6, 7, 8])
        key = tuple(Ns)
        if key in seen:
            assert [r["moments"] for r in out] == [r["moments"] for r in seen[key]]
            continue
        seen[key] = out
        for p, n, s, r in zip(plans, Ns, [5, 6, 7, 8], out):
            if n == 0:
                assert r["kept"] == 0
                continue
            one = p.integrate(n, seed=s, precision=ft.FP64)
            assert r["kept"] == one["kept"]
            for x, y in zip(r["moments"], one["moments"]):
                size = (abs(y[3] + y[4]) * n) ** 0.5   # at least the sum of the magnitudes
                assert abs((x[1] + x[2]) - (y[1] + y[2])) <= 1e-12 * size
                assert abs((x[3] + x[4]) - (y[3] + y[4])) <= 1e-12 * abs(y[3] + y[4])
    b.close()
    for p in plans:
        p.close()


def test_samples_with_floating_edges_are_drawn_again():
    """A double-box sample with x_e = 9.9e-8 takes the reference's route to the derivatives, from
    the generator's state behind it, in whatever thread and order: always the same value, and
    the oracle's within that route's own loss, 8 eps / x_e^2 = 0.18 (any other X is far off)."""
    inp = workloads.double_box(seed=68180207)
    i = 2532781
    ref = ol.Prepared(inp).samples(2011, i, 1)
    p = ft.Plan(inp)
    got = []
    for first in (i, i - 7, i - 8, i - 31):
        rec = p.records(40, seed=2011, first_sample=first, precision=ft.FP64)
        assert rec["flags"][i - first] & 8
        got.append(rec["R"][i - first])
    for g in got[1:]:
        assert (g == got[0]).all()
    assert np.abs(got[0] - ref["R"][0]).max() <= 0.18 * np.abs(ref["R"][0]).max()
    p.close()


def test_scratch_passes_between_plans_and_threads():
    """Plans of different sizes made, run and closed in turn and in eight threads: each run's
    values are those of a plan of its own."""
    inputs = [workloads.triangle(random.Random(1)), workloads.k4_euclidean(), workloads.double_box(),
              workloads.cube_propagator()]

    def one(k):
        p = ft.Plan(inputs[k % 4])
        prec = ft.MIXED if k % 3 else ft.FP64
        r = [p.integrate(n, seed=k, precision=prec)["moments"] for n in (1000 + k, 40_001)]
        p.close()
        return r

    want = [one(k) for k in range(16)]
    assert [one(k) for k in reversed(range(16))][::-1] == want
    got = [None] * 16
    errors = []

    def work(t):
        try:
            for k in range(t, 16, 8):
                got[k] = one(k)
        except Exception as e:   # reported below
            errors.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    assert got == want
