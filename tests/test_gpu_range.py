"""Samples at the ends of FP64's range: a power that overflows by itself drops its sample, whatever the product
with the other one, as in the reference (srcs/feynman_integral.hpp:201-262, 305-345)."""
import numpy as np
import pytest

import feyntrop_gb300 as ft
import oracle_lib as ol

pytestmark = pytest.mark.gpu


def sunrise(deformed):
    """A two-loop sunrise whose subdivergence is nearly logarithmic (r = 0.02): X = (1 - u)^50, so that
    psi_tr^(-D/2) passes 1e308 in one sample of a hundred."""
    s = 9.0 if deformed else -1.0
    return {"graph": [[[0, 1], 1.51], [[0, 1], 1.51], [[0, 1], 4]], "dimension": 6,
            "scalarproducts": [[s, -s], [-s, s]], "masses_sqr": [0.3, 0.2, 0.1] if deformed else [1.0, 2.0, 1.5],
            "num_eps_terms": 2, "lambda": 0.3 if deformed else 0, "N": 1000, "seed": 0}


@pytest.mark.parametrize("deformed", [False, True])
def test_overflowing_powers_drop_their_samples(deformed):
    inp, n = sunrise(deformed), 4096
    ref = ol.Prepared(inp).samples(3, 0, n)
    assert 20 < ref["dropped"].sum() < 100
    p = ft.Plan(inp)
    rec = p.records(n, seed=3, precision=ft.FP64)
    assert ((rec["flags"] & 1 != 0) == ref["dropped"]).all()
    if not deformed:   # positive: its condition is its degree, below 20, over a dozen rounded steps
        ok = ~ref["dropped"]
        assert (np.abs(rec["R"] - ref["R"])[ok, 0] <= 1e-12 * np.abs(ref["R"][ok, 0])).all()
    batches = {prec: ft.Batch([p], prec) for prec in (ft.FP64, ft.MIXED)}
    for prec, b in batches.items():
        for r in (p.integrate(n, seed=3, precision=prec), b.run([n], seeds=[3])[0]):
            assert (r["kept"], r["dropped"]) == ((~ref["dropped"]).sum(), ref["dropped"].sum())
        b.close()
    p.close()
