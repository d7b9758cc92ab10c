"""What the framework's speed is measured on: the calls its users make, over the sizes they make them at.

A case is one call: `ft.run_json` (the drop-in JSON contract, which plans, uploads and integrates in every
call), `Plan.integrate` (one integral, the plan kept) or `Batch.run` (many integrals, the batch kept).  The
graphs are the repository's own workloads (feyntrop_gb300/workloads.py), from one loop and three edges to
five loops and twelve edges, undeformed (Euclidean) and deformed (Minkowski), in both arithmetic forms.

Outputs are the eps-expansion coefficients with their standard errors, [order][re, im][average, error], and
the number of samples kept; the counters and times a result also carries say how a run went, not what it
computed.  The FP64 form's averages are FP64 numbers.  The mixed form evaluates its samples in FP32 and
two-float arithmetic (documented per-sample error 1e-5), so its averages are numbers of FP32's precision
and are handed on in that type.
"""
import random

import numpy as np
import torch

import feyntrop_gb300 as ft
from feyntrop_gb300 import workloads

# Floating-point operations a sample cannot do without, counted on the plain algorithm (one real add,
# subtract, multiply, divide, square root or transcendental each): profiles/flop_counts.txt.
FLOPS = {"triangle": 95.0, "k4": 214.9, "wheel": 360.1, "ladder_euclidean": 1137.6, "cube": 1197.9,
         "double_box": 4550.5, "box_pentagon": 7035.5, "ladder_minkowski": 11390.9}
EDGES = {"triangle": 3, "k4": 6, "wheel": 8, "ladder_euclidean": 10, "cube": 12, "double_box": 7,
         "box_pentagon": 8, "ladder_minkowski": 10}
ORDERS = {"triangle": 3, "k4": 3, "wheel": 2, "ladder_euclidean": 3, "cube": 4, "double_box": 2,
          "box_pentagon": 3, "ladder_minkowski": 3}
DEFORMED = ("double_box", "box_pentagon", "ladder_minkowski")
MIX = ("triangle", "ladder_euclidean", "ladder_minkowski", "wheel", "box_pentagon")


def listed():
    return [
        # The smallest use: the JSON contract on a one-loop triangle, plan and all, as a script that
        # evaluates a phase-space point per call does it; launches, allocations and latency.
        {"name": "json_triangle", "call": "json", "graph": "triangle", "precision": "fp64", "N": 50_000},
        # A kept plan called again and again with few samples (an integrator's inner loop): latency.
        {"name": "triangle_small", "call": "integrate", "graph": "triangle", "precision": "mixed", "N": 100_000},
        # A pilot run on one Minkowski point, as the choice of the deformation parameter makes it.
        {"name": "box_pentagon_pilot", "call": "integrate", "graph": "box_pentagon", "precision": "mixed", "N": 200_001},
        # The reference's own low-level example in its own arithmetic (FP64, the default), at its size.
        {"name": "k4_fp64", "call": "integrate", "graph": "k4", "precision": "fp64", "N": 10_000_000},
        # A Minkowski integral in the default arithmetic, an ordinary size, ragged.
        {"name": "double_box_fp64", "call": "integrate", "graph": "double_box", "precision": "fp64", "N": 3_000_017},
        # The headline workload: the double box in the mixed form.
        {"name": "double_box_mixed", "call": "integrate", "graph": "double_box", "precision": "mixed", "N": 50_000_000},
        # The largest deformed class: three loops, ten edges.
        {"name": "ladder_minkowski_mixed", "call": "integrate", "graph": "ladder_minkowski", "precision": "mixed", "N": 10_000_000},
        # The deepest Euclidean class, both forms: five loops, twelve edges, a table of 4096 subgraphs.
        {"name": "cube_mixed", "call": "integrate", "graph": "cube", "precision": "mixed", "N": 50_000_000},
        {"name": "cube_fp64", "call": "integrate", "graph": "cube", "precision": "fp64", "N": 2_000_003},
        # A kinematic scan: many points of one topology in one launch, uneven sample counts.
        {"name": "scan_mixed", "call": "batch", "graph": "box_pentagon", "precision": "mixed", "count": 24, "nmin": 100_000, "nmax": 3_000_000},
        {"name": "scan_fp64", "call": "batch", "graph": "box_pentagon", "precision": "fp64", "count": 12, "nmin": 10_000, "nmax": 300_000},
        # A batch of every kind of integral, Euclidean and Minkowski side by side, uneven sample counts.
        {"name": "mixed_batch", "call": "batch", "graph": "all", "precision": "mixed", "count": 20, "nmin": 100_000, "nmax": 10_000_000},
    ]


# Largest sample count drawn for one integral: about as long a pass as the longest listed ones.
LARGEST = {"mixed": {"triangle": 10**8, "k4": 10**8, "wheel": 10**8, "ladder_euclidean": 4 * 10**7, "cube": 5 * 10**7,
                     "double_box": 3 * 10**7, "box_pentagon": 2 * 10**7, "ladder_minkowski": 10**7},
           "fp64": {"triangle": 10**7, "k4": 10**7, "wheel": 5 * 10**6, "ladder_euclidean": 3 * 10**6, "cube": 3 * 10**6,
                    "double_box": 3 * 10**6, "box_pentagon": 2 * 10**6, "ladder_minkowski": 10**6}}


def _log_uniform(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    call = rng.choice(("json", "integrate", "integrate", "integrate", "batch"))
    precision = rng.choice(("mixed", "mixed", "fp64"))
    if call == "batch":
        graph = rng.choice(("box_pentagon", "double_box", "all"))
        most = (2_000_000 if graph == "all" else 1_000_000) if precision == "mixed" else 100_000
        nmin = _log_uniform(rng, 10_000, most / 4)
        return {"call": call, "graph": graph, "precision": precision, "count": rng.randint(3, 24), "nmin": nmin,
                "nmax": _log_uniform(rng, 2 * nmin, most)}
    graph = rng.choice(tuple(FLOPS))
    most = LARGEST[precision][graph]
    if call == "json":   # the whole contract's smaller calls
        most = min(most, 1_000_000)
    return {"call": call, "graph": graph, "precision": precision, "N": _log_uniform(rng, 20_000, most)}


def _input(graph, seed):
    """The low-level JSON input of a graph at kinematics drawn from the seed."""
    rng = random.Random("%s %d" % (graph, seed))
    if graph == "k4":
        inp = workloads.k4_euclidean(masses=[rng.uniform(0, 5) for _ in range(6)])
    elif graph == "double_box":
        inp = workloads.double_box(seed=rng.randrange(1 << 30))
    elif graph == "box_pentagon":
        inp = workloads.box_pentagon(rng)
    elif graph == "cube":
        inp = workloads.cube_propagator()
    elif graph == "wheel":
        inp = workloads.wheel4_vacuum()
    elif graph == "triangle":
        inp = workloads.triangle(rng)
    else:
        inp = workloads.ladder3(rng, euclidean=graph == "ladder_euclidean")
    return inp


def _counts(case):
    """Sample counts of a batch's integrals, spread over the case's range."""
    n, lo, hi = case["count"], case["nmin"], case["nmax"]
    return [int(lo * (hi / lo) ** ((i + 0.5) / n)) | 1 for i in range(n)]


def _graphs(case):
    return [case["graph"] if case["graph"] != "all" else MIX[i % len(MIX)] for i in range(case["count"])]


def _integrals(case, seed):
    """(graph, input, samples, stream seed) of every integral of the case."""
    if case["call"] == "batch":
        return [(g, _input(g, seed * 1000 + i), n, seed * 1000 + i)
                for i, (g, n) in enumerate(zip(_graphs(case), _counts(case)))]
    return [(case["graph"], _input(case["graph"], seed), case["N"], seed)]


def prepare(case, seed):
    work = _integrals(case, seed)
    precision = ft.MIXED if case["precision"] == "mixed" else ft.FP64
    state = {"call": case["call"], "precision": precision, "graphs": [w[0] for w in work],
             "dtype": np.float32 if precision == ft.MIXED else np.float64}
    if case["call"] == "json":
        state["input"] = dict(work[0][1], N=case["N"], seed=seed, precision=case["precision"])
    elif case["call"] == "integrate":
        state.update(plan=ft.Plan(work[0][1]), N=case["N"], seed=seed)
    else:
        state["plans"] = ft.create_plans([w[1] for w in work])
        state.update(batch=ft.Batch(state["plans"], precision), N=[w[2] for w in work], seeds=[w[3] for w in work])
    return state


def run(state):
    dtype = state["dtype"]
    if state["call"] == "json":
        return {"integral": np.array(ft.run_json(state["input"])["integral"], dtype=dtype)}
    if state["call"] == "integrate":
        r = state["plan"].integrate(state["N"], seed=state["seed"], precision=state["precision"])
        return {"integral": np.array(r["integral"], dtype=dtype), "kept": r["kept"]}
    rs = state["batch"].run(state["N"], seeds=state["seeds"])
    out = {"kept": np.array([r["kept"] for r in rs], dtype=np.int64)}
    for g in dict.fromkeys(state["graphs"]):
        out[g] = np.array([r["integral"] for r, h in zip(rs, state["graphs"]) if h == g], dtype=dtype)
    return out


def work(case):
    """Flops of the samples; bytes of each integral's subgraph table (Jr/r, Jr, 1/r and a byte per subgraph)
    and parameters read once and its sums written once."""
    if case["call"] == "batch":
        parts = list(zip(_graphs(case), _counts(case)))
    else:
        parts = [(case["graph"], case["N"])]
    return {"bytes": float(sum(25 * 2 ** EDGES[g] + 1024 + 64 * ORDERS[g] for g, _ in parts)),
            "flops": float(sum(FLOPS[g] * n for g, n in parts))}


# ------------------------------------------------------------------ the same integrals in plain FP64 torch

def _subgraph_table(inp):
    """The tropical sampling table of Borinsky, Munch and Tellander (arXiv:2302.08955): J(gamma), r(gamma), loop
    numbers and mass-momentum-spanning flags of every edge subset, and whether the contour is deformed."""
    ends = [(max(e[0]), min(e[0])) for e in inp["graph"]]
    nu = [float(e[1]) for e in inp["graph"]]
    E, D, m2 = len(ends), float(inp["dimension"]), [float(m) for m in inp["masses_sqr"]]
    V = max(k for k, _ in ends) + 1
    P = np.array(inp["scalarproducts"], dtype=np.float64)
    deform = not all(x <= 1e-12 * max(1.0, np.abs(P).max()) for x in np.linalg.eigvalsh(P))
    full, loops, pseudo = (1 << E) - 1, E - V + 1, True
    W = sum(nu) - D / 2.0 * loops
    ref = float(np.linalg.norm(P[:-1, :-1])) + float(np.linalg.norm(m2))
    probes = 1.0 + 2.0 * np.random.RandomState(1).random_sample((4, E))
    L, mm = [0] * (full + 1), [False] * (full + 1)
    for sub in range(full + 1):
        part = list(range(V))
        for e in range(E):
            if sub >> e & 1:
                a, b = part[ends[e][0]], part[ends[e][1]]
                part = [b if p == a else p for p in part]
        names = {p: i for i, p in enumerate(dict.fromkeys(part))}
        part = [names[p] for p in part]
        n = len(names) - 1
        L[sub] = bin(sub).count("1") - V + n + 1
        pick = np.zeros((n + 1, V))
        pick[part, range(V)] = 1.0
        Q = (pick @ P @ pick.T)[:n, :n]
        if n == 1 and Q[0, 0] > 1e-12 * ref:
            pseudo = False
        rest = [e for e in range(E) if not sub >> e & 1]
        inc = np.zeros((n + 1, len(rest)))
        for i, e in enumerate(rest):
            inc[part[ends[e][0]], i] += 1.0
            inc[part[ends[e][1]], i] -= 1.0
        size = 0.0
        for x in probes[:, rest]:
            lap = (inc[:n] / x) @ inc[:n].T
            size += abs(sum(m2[e] * t for e, t in zip(rest, x)) - (np.trace(np.linalg.solve(lap, Q)) if n else 0.0))
        mm[sub] = size < 1e-11 * ref
    J, r = [1.0] * (full + 1), [1.0] * (full + 1)
    for sub in sorted(range(1, full + 1), key=lambda s: bin(s).count("1")):
        J[sub] = 0.0
        for e in range(E):
            if sub >> e & 1:
                J[sub] += J[sub ^ 1 << e] / r[sub ^ 1 << e]
        r[sub] = sum(nu[e] for e in range(E) if sub >> e & 1) - D / 2.0 * L[sub] - (W if mm[sub] else 0.0)
    return dict(E=E, V=V, ends=ends, nu=nu, D=D, m2=m2, P=P, W=W, loops=loops, J=J, r=r, L=L, mm=mm,
                kappa=0.0 if pseudo or not deform else -float(inp["lambda"]))


MASK = (1 << 64) - 1


def _seed_state(seed):
    """splitmix64's four words of the seed (Blackman and Vigna, prng.di.unimi.it)."""
    s, x = [], seed
    for _ in range(4):
        x = (x + 0x9E3779B97F4A7C15) & MASK
        z = x
        z = ((z ^ z >> 30) * 0xBF58476D1CE4E5B9) & MASK
        z = ((z ^ z >> 27) * 0x94D049BB133111EB) & MASK
        s.append(z ^ z >> 31)
    return s


def _signed(x):
    return x - (1 << 64) if x >> 63 else x


def _shift(x, k):
    return (x >> k) & ((1 << 64 - k) - 1)


def _next(s):
    """One xoshiro256+ step on int64 tensors: the output, the state replaced in place."""
    out = s[0] + s[3]
    t = s[1] << 17
    s[2] = s[2] ^ s[0]
    s[3] = s[3] ^ s[1]
    s[1] = s[1] ^ s[2]
    s[0] = s[0] ^ s[3]
    s[2] = s[2] ^ t
    s[3] = (s[3] << 45) | _shift(s[3], 19)
    return out


def _lanes(seed, steps, lanes):
    """States of `lanes` generators, `steps` outputs of the seed's stream apart."""
    bit = torch.arange(256, device="cuda")
    def words(b):   # bits [256, n] -> four int64 words
        return [sum(b[64 * w + i].long() << i for i in range(64)) for w in range(4)]
    def bits(s):
        return torch.stack([s[int(i) >> 6] >> (int(i) & 63) & 1 for i in bit.tolist()]).float()
    step = words((bit[:, None] == bit[None]).float())   # columns: the unit states
    _next(step)
    square, jump = bits(step), None
    while steps:
        if steps & 1:
            jump = square if jump is None else (square @ jump) % 2
        square, steps = (square @ square) % 2, steps >> 1
    states = bits([torch.tensor([_signed(w)], device="cuda") for w in _seed_state(seed)])
    while states.shape[1] < lanes:
        states, jump = torch.cat([states, (jump @ states) % 2], 1), (jump @ jump) % 2
    return words(states[:, :lanes])


def _uniform(s):
    return _shift(_next(s), 11).double() * 2.0**-53


def _eliminate(t, y):
    """Pivots and multipliers of the reduced Laplacian with conductances y, vertex V-1 deleted."""
    n = t["V"] - 1
    zero = torch.zeros_like(y[0])
    c = [[zero] * (n + 1) for _ in range(n + 1)]
    for e, (k, l) in enumerate(t["ends"]):
        c[l][k] = c[l][k] + y[e]
    d, a = [], [[None] * n for _ in range(n)]
    for k in range(n):
        d.append(sum(c[k][k + 2:], c[k][k + 1]))
        for i in range(k + 1, n):
            a[k][i] = c[k][i] / d[k]
        for i in range(k + 1, n):
            for j in range(i + 1, n + 1):
                c[i][j] = c[i][j] + a[k][i] * c[k][j]
    return d, a


def _inverse(d, a):
    """The inverse of the matrix with those pivots and multipliers."""
    n = len(d)
    m = [[None] * n for _ in range(n)]
    for i in reversed(range(n)):
        m[i][i] = torch.ones_like(d[0])
        for j in range(i + 1, n):
            m[i][j] = sum(a[i][k] * m[k][j] for k in range(i + 1, j + 1))
    g = [[None] * n for _ in range(n)]
    for i in range(n):
        for j in range(i, n):
            g[i][j] = g[j][i] = sum(m[i][k] * m[j][k] / d[k] for k in range(j, n))
    return g


def _product(v):
    p = v[0]
    for x in v[1:]:
        p = p * x
    return p


def _values(t, s, K):
    """The integrand's eps orders (arXiv:2302.08955, section 5) at the next sample of every lane."""
    E, D, W, n, P, dev = t["E"], t["D"], t["W"], t["V"] - 1, t["P"], "cuda"
    J = torch.tensor(t["J"], dtype=torch.float64, device=dev)
    r = torch.tensor(t["r"], dtype=torch.float64, device=dev)
    w, inv = J / r, 1.0 / r
    L, mm = torch.tensor(t["L"], device=dev), torch.tensor(t["mm"], device=dev)
    sub = torch.full_like(s[0], (1 << E) - 1)
    x = torch.ones(sub.shape, dtype=torch.float64, device=dev)
    X = [x] * E
    psi_tr, v_tr, loops, span = x, x, torch.full_like(sub, t["loops"]), torch.ones_like(sub, dtype=torch.bool)
    for step in range(E):
        R, T = _uniform(s) * J[sub], torch.zeros_like(x)
        cut, found = torch.zeros_like(sub), torch.zeros_like(span)
        for e in range(E):
            here = (sub >> e & 1).bool() & ~found
            T = torch.where(here, T + w[sub ^ 1 << e], T)
            cut = torch.where(here, e, cut)
            found = found | here & (T > R)
        sub = sub ^ (torch.ones_like(sub) << cut)
        X = [torch.where(cut == e, x, X[e]) for e in range(E)]
        v_tr = torch.where(span & ~mm[sub], x, v_tr)
        span = mm[sub]
        psi_tr = torch.where(L[sub] < loops, psi_tr * x, psi_tr)
        loops = torch.minimum(loops, L[sub])
        if step < E - 1:
            x = x * (1.0 - _uniform(s)) ** inv[sub]
    scale = (psi_tr ** (-D / 2) * v_tr ** -W) ** (1.0 / (D / 2 * t["loops"] + W)) if D / 2 * t["loops"] + W else 1.0
    X = [v * scale for v in X]
    Y = [1.0 / v for v in X]
    d, a = _eliminate(t, Y)
    if not t["kappa"]:
        psi = _product(d) * _product(X)
        G = _inverse(d, a)
        V = sum(m * v for m, v in zip(t["m2"], X)) - sum(P[i, j] * G[i][j] for i in range(n) for j in range(n) if P[i, j])
        R, log = t["J"][-1] * psi ** (-D / 2) * V ** -W, psi.log() - t["loops"] * V.log()
    else:
        G = _inverse(d, a)
        F = [[sum(G[i][k] * P[k, j] for k in range(n)) for j in range(n)] for i in range(n)]
        S = [[None] * n for _ in range(n)]
        for i in range(n):
            for j in range(i, n):
                S[i][j] = S[j][i] = sum(F[i][k] * G[k][j] for k in range(n))
        def drop(M, e, f):
            (k, l), (p, q) = t["ends"][e], t["ends"][f]
            at = lambda i, j: 0.0 if i == n or j == n else M[i][j]  # noqa: E731
            return at(k, p) + at(l, q) - at(k, q) - at(l, p)
        kappa = t["kappa"]
        theta = [kappa * (t["m2"][e] - Y[e] ** 2 * drop(S, e, e)) for e in range(E)]
        A = [[None] * E for _ in range(E)]
        for e in range(E):
            for f in range(e, E):
                h = -2.0 * Y[e] ** 2 * Y[f] ** 2 * drop(S, e, f) * drop(G, e, f)
                if e == f:
                    h = h + 2.0 * Y[e] ** 3 * drop(S, e, e)
                A[e][f] = torch.complex(torch.full_like(x, float(e == f)), kappa * h * (X[e] * X[f]).sqrt())
        jac = None
        for k in range(E):
            jac = A[k][k] if jac is None else jac * A[k][k]
            for i in range(k + 1, E):
                f = A[k][i] / A[k][k]
                for j in range(i, E):
                    A[i][j] = A[i][j] - f * A[k][j]
        turn = [torch.polar(torch.ones_like(x), th) for th in theta]
        Z = [v * u for v, u in zip(X, turn)]
        d, a = _eliminate(t, [y * u.conj() for y, u in zip(Y, turn)])
        psi = _product(d) * _product(Z)
        G = _inverse(d, a)
        V = sum(m * v for m, v in zip(t["m2"], Z)) - sum(P[i, j] * G[i][j] for i in range(n) for j in range(n) if P[i, j])
        R = t["J"][-1] * jac * (-D / 2 * psi.log() - W * V.log() + 1j * sum(u * th for u, th in zip(t["nu"], theta))).exp()
        log = psi.log() - t["loops"] * V.log()
    out = [R]
    for j in range(1, K):
        out.append(out[-1] * log / j)
    return out


def _exact_integral(inp, N, seed):
    """[order][re, im][average, standard error] and the samples kept, of the first N samples of the seed's stream."""
    t, K = _subgraph_table(inp), int(inp["num_eps_terms"])
    per = 2 * t["E"] - 1
    each = max(1, -(-N // 500_000))   # samples of a lane
    s = _lanes(seed, per * each, -(-N // each))
    sums, kept = torch.zeros(K, 2, 2, dtype=torch.float64, device="cuda"), 0
    lane = torch.arange(s[0].numel(), device="cuda")
    for i in range(each):
        R = _values(t, s, K)
        ok = (lane * each + i < N) & torch.isfinite(torch.view_as_real(R[0]).sum(-1) if R[0].is_complex() else R[0])
        kept += int(ok.sum())
        for j in range(K):
            for p, v in enumerate((R[j].real, R[j].imag) if R[j].is_complex() else (R[j],)):
                v = torch.where(ok, v, 0.0)
                sums[j, p, 0] += v.sum()
                sums[j, p, 1] += v.square().sum()
    mean, square = sums[..., 0] / kept, sums[..., 1] / kept
    error = ((square - mean ** 2) / (kept - 1)).clamp(min=0).sqrt()
    return torch.stack([mean, error], -1).cpu().numpy(), kept


def exact(case, seed):
    """run()'s outputs from the textbook formulas in FP64 (up to the sizes where that takes seconds)."""
    work = _integrals(case, seed)
    if sum(n * FLOPS[g] for g, _, n, _ in work) > 1.5e11:
        return None
    got = [(g,) + _exact_integral(inp, n, s) for g, inp, n, s in work]
    if case["call"] != "batch":
        out = {"integral": got[0][1]}
        return out if case["call"] == "json" else dict(out, kept=got[0][2])
    out = {"kept": np.array([k for _, _, k in got], dtype=np.int64)}
    for g in dict.fromkeys(h for h, _, _ in got):
        out[g] = np.array([v for h, v, _ in got if h == g])
    return out
