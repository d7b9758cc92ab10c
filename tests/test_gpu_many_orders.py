"""A deformed 12-edge graph with many eps orders: its sums leave room for blocks of two warps and of one."""
import pytest

import feyntrop_gb300 as ft
import oracle_lib as ol
from feyntrop_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [14, 21])
def test_small_blocks(K):
    inp = workloads.cube_propagator()
    s = 14.0
    inp["scalarproducts"][0][0] = inp["scalarproducts"][1][1] = s
    inp["scalarproducts"][0][1] = inp["scalarproducts"][1][0] = -s
    inp.update(masses_sqr=[0.3 + 0.05 * k for k in range(12)], num_eps_terms=K, **{"lambda": 0.3})
    n = 3001
    cpu, _, _ = ol.Prepared(inp).integrate(n, 2, 4)
    p = ft.Plan(inp)
    assert p.info["deformed"]
    r = p.integrate(n, seed=2, precision=ft.FP64)
    assert r["kept"] == n
    for j in range(K):   # the same samples: the comparison of the smoke check
        re, dre = r["integral"][j][0]
        assert abs(re - cpu[j, 0]) <= 1e-6 * max(abs(cpu[j, 0]), dre), j
    b = ft.Batch([p], ft.FP64)
    for (re, _), (one, dre) in zip((x[0] for x in b.run([n], seeds=[2])[0]["integral"]),
                                   (x[0] for x in r["integral"])):
        assert abs(re - one) <= 1e-9 * max(abs(one), dre)
    b.close()
    p.close()
