"""The work that this engine does for its users, as cases that can be timed and compared.

A case is a dict of plain values; ``kind`` says which public entry points one pass goes through:

* ``solve``: the allocation-free Option-B Newton solve on device buffers (the smallest call).
* ``fed``: training from resident client data: initial shifts, ``rounds`` FedNL rounds, read-back of
  the iterate, the gradient and the master's Hessian estimate (FP64 engine, every compressor, plain
  and partial participation, fixed and reference arithmetic order, {0,1} and dense features).
* ``job``: the same from the caller's arrays: create, upload, train, read back, destroy.
* ``mixed``: further rounds of the mixed-precision engine on a resident problem.
* ``serve``: one tick of the serving loop over a set of live problems of different dimension
  (every problem's client phase, one batched solve, every problem's statistics).

Sizes are those of the benchmark workloads (a9a-, w8a- and phishing-like sets, the dense d = 1024
set with fewer clients) and of the request stream that the serving loop draws.
"""
import ctypes as C
import math

import numpy as np
import torch

from ufednl_gb300 import datagen, fednl

LAM = 1e-3


def listed():
    return [
        # the Newton step of the phishing-like problem: the smallest call, launch and latency bound
        {"name": "solve_d69", "kind": "solve", "d": 69},
        # the Newton step of the w8a-like problem (odd dimension, the whole GPU in one cooperative launch)
        {"name": "solve_d301", "kind": "solve", "d": 301},
        # plain FedNL on an a9a-like set: TopK k = 8d, even clients, small d
        fed("fed_a9a_topk", 124, 80, 407, 407, 0.11, "topk", 8, 20),
        # the headline workload: w8a-like, uneven clients, TopLEK k = 8d, 16 rounds to ||g|| <= 1e-9
        fed("fed_w8a_toplek", 301, 142, 200, 600, 0.039, "toplek", 8, 16),
        # the same set with the randomised compressor that needs no sorting (k = 8d, alpha = k / U)
        fed("fed_w8a_randk", 301, 142, 200, 600, 0.039, "randk", 8, 16),
        # partial participation: 2048 clients of 6 samples, 128 sampled per round, RandSeqK k = d
        fed("pp_phishing_randseqk", 69, 2048, 6, 6, 0.45, "randseqk", 1, 40, tau=128),
        # real-valued features in FP64, backtracking line search off
        fed("fed_dense_topk", 512, 24, 300, 900, 0.0, "topk", 8, 4),
        # the local driver's default arithmetic: the reference's operation order, bit for bit
        fed("ref_w8a_toplek", 301, 142, 200, 600, 0.039, "toplek", 8, 6, order="reference"),
        # the whole job a caller pays for, from host arrays to the minimiser
        dict(fed("job_w8a_toplek", 301, 142, 200, 600, 0.039, "toplek", 8, 16), kind="job"),
        # mixed precision on the headline workload (TF32 client Hessians, refined FP32 solve)
        mixed("mixed_w8a_toplek", 301, 142, 200, 600, 0.039, "toplek", 8, 16),
        # mixed precision on dense FP32 features: the tensor-core Gram matrices dominate
        mixed("mixed_dense_randk", 1024, 32, 512, 4096, 0.0, "randk_philox", 4, 8),
        # a serving tick: live problems of d 69, 124, 301 and 1024, two of each, on the mixed engine
        {"name": "serve_tick", "kind": "serve", "problems": 8, "d_max": 1024, "clients": 24, "n_lo": 50,
         "n_hi": 800, "layout": 4},
    ]


def fed(name, d, clients, n_lo, n_hi, density, comp, kmul, rounds, tau=0, order="fixed", line_search=False):
    c = {"name": name, "kind": "fed", "d": d, "clients": clients, "n_lo": n_lo, "n_hi": n_hi, "layout": 1,
         "density": density, "comp": comp, "kmul": kmul, "rounds": rounds, "tau": tau, "order": order,
         "line_search": line_search}
    if not name:
        del c["name"]
    return c


def mixed(name, d, clients, n_lo, n_hi, density, comp, kmul, rounds):
    c = {"name": name, "kind": "mixed", "d": d, "clients": clients, "n_lo": n_lo, "n_hi": n_hi, "layout": 2,
         "density": density, "comp": comp, "kmul": kmul, "rounds": rounds}
    if not name:
        del c["name"]
    return c


def _spread(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    what = rng.choice(["solve", "fed", "fed", "fed", "pp", "dense", "ref", "job", "mixed", "mixed", "serve"])
    layout = rng.randrange(1 << 16)
    if what == "solve":
        return {"kind": "solve", "d": _spread(rng, 16, 512)}
    if what == "serve":
        return {"kind": "serve", "problems": rng.randint(2, 8), "d_max": rng.choice([124, 301, 1024]),
                "clients": _spread(rng, 16, 24), "n_lo": 50, "n_hi": _spread(rng, 100, 800), "layout": layout}
    if what == "pp":
        clients = _spread(rng, 128, 2048)
        n = _spread(rng, 4, 40)
        c = fed("", _spread(rng, 24, 124), clients, n, n + rng.randint(0, 8), rng.uniform(0.05, 0.5),
                rng.choice(["randseqk", "natural", "topk"]), 1, rng.randint(8, 40), tau=max(8, clients // 16))
    elif what == "dense":
        c = fed("", _spread(rng, 24, 512), _spread(rng, 4, 24), 50, _spread(rng, 100, 800), 0.0,
                rng.choice(["topk", "toplek", "randk", "identity"]), 4, rng.randint(2, 4))
    elif what == "ref":
        c = fed("", _spread(rng, 24, 301), _spread(rng, 8, 142), 50, _spread(rng, 100, 600),
                rng.uniform(0.03, 0.2), rng.choice(["topk", "toplek", "randk", "natural"]), rng.choice([1, 4, 8]),
                rng.randint(3, 6), order="reference")
    elif what == "mixed":
        d = _spread(rng, 64, 1024)
        comp = rng.choice(["topk", "toplek", "randk_philox"])
        return dict(mixed("", d, _spread(rng, 8, 32 if d > 301 else 142), 50, _spread(rng, 100, 2000),
                          rng.choice([0.0, rng.uniform(0.03, 0.5)]), comp, 4 if comp == "randk_philox" else 8,
                          rng.randint(4, 8)), layout=layout)
    else:
        c = fed("", _spread(rng, 24, 400), _spread(rng, 8, 142), 50, _spread(rng, 100, 700),
                math.exp(rng.uniform(math.log(0.02), math.log(0.4))),
                rng.choice(["topk", "toplek", "randk", "randseqk", "natural", "identity"]), rng.choice([1, 4, 8]),
                rng.randint(6, 16), line_search=what == "fed" and rng.random() < 0.25)
        if what == "job":
            c["kind"] = "job"
    c["layout"] = layout
    return c


# ---- inputs -----------------------------------------------------------------------------------

def _samples(case):
    """The clients' sample counts: part of the case, not of the seed."""
    return np.random.default_rng(case["layout"]).integers(case["n_lo"], case["n_hi"] + 1, size=case["clients"])


def _draw_data(rng, d, S, density):
    """Features [S, d] and labels [S]: Bernoulli(density) attributes plus an intercept column of ones,
    or N(0, 1) attributes (density 0) as FP32 values; labels from a planted w* ~ N(0, I / d)."""
    if density > 0.0:
        a = np.empty((S, d), dtype=np.float32)
        a[:, :-1] = rng.random((S, d - 1), dtype=np.float32) < density
        a[:, -1] = 1.0
    else:
        a = rng.standard_normal((S, d), dtype=np.float32)
    w = rng.normal(0.0, 1.0 / np.sqrt(d), size=d).astype(np.float32)
    p = 1.0 / (1.0 + np.exp(-(a @ w).astype(np.float64)))
    return a, np.where(rng.random(S) < p, 1.0, -1.0)


def _data(case, seed):
    ns = _samples(case)
    a, y = _draw_data(np.random.default_rng(seed), case["d"], int(ns.sum()), case["density"])
    return ns, a, y


def _problem(case, seed, dtype):
    ns, a, y = _data(case, seed)
    return datagen.Problem(case["d"], ns.astype(np.int32), np.ascontiguousarray(a, dtype=dtype), y, LAM)


def _k_alpha(case):
    d = case["d"]
    U = d * (d + 1) // 2
    k = min(case["kmul"] * d, U)
    comp = case["comp"]
    if comp in ("randk", "randseqk", "randk_philox"):
        return k, k / U
    return k, 1.0 / (1.0 + 1.0 / 8.0) if comp == "natural" else 1.0


def _system(case, seed):
    """H = A^T D A + lambda I of a logistic problem, the Option-B shift l and a gradient, in FP64."""
    d = case["d"]
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(4 * d, d, generator=g, device="cuda", dtype=torch.float64)
    s = torch.sigmoid(torch.randn(4 * d, generator=g, device="cuda", dtype=torch.float64))
    H = (a * (s * (1 - s) / (4 * d))[:, None]).T @ a + LAM * torch.eye(d, device="cuda", dtype=torch.float64)
    H = ((H + H.T) / 2).contiguous()
    return H, 0.05, torch.randn(d, generator=g, device="cuda", dtype=torch.float64)


def _engine(case, prob):
    k, alpha = _k_alpha(case)
    return fednl.FedNL(prob, case["comp"], k, alpha, workers=16, clients_per_round=case["tau"], order=case["order"],
                       line_search=(0.5, 0.5, 5) if case["line_search"] else None)


def _serve_cases(case):
    """The live problems of a serving tick: d, clients, samples, features and compressor of each."""
    rng = np.random.default_rng(case["layout"])
    ds = [d for d in (69, 124, 301, 1024) if d <= case["d_max"]]
    out = []
    for i in range(case["problems"]):
        out.append({"d": ds[i % len(ds)], "clients": int(rng.integers(16, case["clients"] + 1)),
                    "n_lo": case["n_lo"], "n_hi": case["n_hi"], "layout": case["layout"] + 1 + i,
                    "density": float(rng.uniform(0.05, 0.5)) if rng.random() < 0.5 else 0.0,
                    "comp": str(rng.choice(["topk", "toplek", "randk_philox"])), "kmul": 8})
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "solve":
        H, l, g = _system(case, seed)
        return {"kind": kind, "d": case["d"], "H": H, "l": l, "g": g, "dx": torch.empty_like(g)}
    if kind == "serve":
        ps = []
        for i, c in enumerate(_serve_cases(case)):
            k, alpha = _k_alpha(c)
            ps.append(fednl.MixedFedNL(_problem(c, seed + 1000 * i, np.float32), k, alpha, compressor=c["comp"]))
        return {"kind": kind, "problems": ps}
    if kind == "mixed":
        k, alpha = _k_alpha(case)
        m = fednl.MixedFedNL(_problem(case, seed, np.float32), k, alpha, compressor=case["comp"], solver="fp32_coop")
        return {"kind": kind, "engine": m, "rounds": case["rounds"]}
    prob = _problem(case, seed, np.float64)
    if kind == "job":
        return {"kind": kind, "case": case, "prob": prob}
    return {"kind": kind, "engine": _engine(case, prob), "rounds": case["rounds"]}


# ---- one pass ---------------------------------------------------------------------------------

def _check(rc):
    if rc != 0:
        raise RuntimeError(fednl.load().fednl_gpu_last_error().decode())


def run(state):
    kind = state["kind"]
    if kind == "solve":
        d, H, g, dx = state["d"], state["H"], state["g"], state["dx"]
        _check(fednl.load().fednl_gpu_optionb_solve_noalloc(H.data_ptr(), d, d, state["l"], g.data_ptr(),
                                                            dx.data_ptr(), None))
        return dx
    if kind == "serve":
        ps = state["problems"]
        for p in ps:
            p.client_phase()
        fednl.solve_batch(ps)
        return {"norms": np.array([p.round_result() for p in ps]), "x": [p.x() for p in ps],
                "grad": [p.grad() for p in ps], "l": np.array([p.l() for p in ps])}
    if kind == "mixed":
        m = state["engine"]
        norms = m.run(state["rounds"])
        return {"norms": norms, "first": norms[0], "x": m.x(), "grad": m.grad(), "l": m.l()}
    if kind == "job":
        f = _engine(state["case"], state["prob"])
        norms = f.run(state["case"]["rounds"])
        out = {"norms": norms, "first": norms[0], "x": f.x(), "grad": f.grad()}
        f.close()
        return out
    f = state["engine"]
    _check(fednl.load().fednl_gpu_init_shifts(f._h, None))       # a fresh run on the resident data, x0 = 0
    norms = f.run(state["rounds"])
    return {"norms": norms, "first": norms[0], "x": f.x(), "grad": f.grad(), "H": f.H(), "l": f.l()}


# ---- what a pass cannot do without ---------------------------------------------------------------

def _round_work(c, features_bytes, state_bytes):
    """Bytes and operations of one round: the features and the clients' shifts read once, the sent
    entries and the master's system written; margins, gradients, Hessians and the solve."""
    ns = _samples(c)
    d, nc = c["d"], len(ns)
    n_act = c.get("tau") or nc
    S = float(ns.sum())
    U = d * (d + 1) / 2
    k = _k_alpha(c)[0] if c["comp"] not in ("natural", "identity") else U
    part = n_act / nc
    if c["density"] > 0:
        fb, nnz = S * d / 8, S * (c["density"] * (d - 1) + 1)
        pairs = S * (c["density"] * (d - 1) + 1) ** 2 / 2
        hess = part * pairs
    else:
        fb, nnz = S * d * features_bytes, S * d
        hess = part * S * d * (d + 1)
    by = fb + n_act * (U + k) * state_bytes + 2 * U * 8 + nc * d * 8
    fl = 4 * nnz + hess + n_act * U + d ** 3 / 3 + 2 * d * d
    return by, fl


def work(case):
    kind = case["kind"]
    if kind == "solve":
        d = case["d"]
        return {"bytes": d * (d + 1) / 2 * 8 + 16 * d, "flops": d ** 3 / 3 + 2 * d * d}
    if kind == "serve":
        ws = [_round_work(c, 4, 4) for c in _serve_cases(case)]
        return {"bytes": sum(w[0] for w in ws), "flops": sum(w[1] for w in ws)}
    by, fl = _round_work(case, 4 if kind == "mixed" else 8, 4 if kind == "mixed" else 8)
    R = case["rounds"] + (0 if kind == "mixed" else 1)       # the initial shifts cost a round's Hessians
    host = float(_samples(case).sum()) * case["d"] * 8 if kind == "job" else 0.0
    return {"bytes": R * by + host, "flops": R * fl}


# ---- the same in 64 bits ------------------------------------------------------------------------

def _first_gradient(ns, a, y):
    """Mean of the clients' gradients at x = 0 (labels folded in), in FP64."""
    g, o = np.zeros(a.shape[1]), 0
    for n in ns:
        g -= 0.5 / n * (a[o:o + n].astype(np.float64) * y[o:o + n, None]).sum(axis=0)
        o += n
    return g / len(ns)


def _minimiser(ns, a, y):
    """Newton's method on the clients' mean objective, on the GPU in FP64."""
    A = torch.from_numpy(a).cuda().double() * torch.from_numpy(y).cuda()[:, None]
    w = torch.from_numpy(np.repeat(1.0 / (len(ns) * ns.astype(np.float64)), ns)).cuda()
    x = torch.zeros(a.shape[1], dtype=torch.float64, device="cuda")
    for _ in range(12):
        s = torch.sigmoid(A @ x)
        g = LAM * x - A.T @ (w * (1 - s))
        H = A.T @ (A * (w * s * (1 - s))[:, None]) + LAM * torch.eye(len(x), dtype=torch.float64, device="cuda")
        x = x - torch.linalg.solve(H, g)
    return x.cpu().numpy()


#: listed runs that end at the minimiser (||g|| of 1e-9 or so)
_CONVERGES = ("fed_a9a_topk", "fed_w8a_toplek", "job_w8a_toplek", "mixed_w8a_toplek")


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve":
        H, l, g = _system(case, seed)
        return torch.linalg.solve(H + l * torch.eye(case["d"], device="cuda", dtype=torch.float64), g)
    if kind == "serve":
        first = []
        for i, c in enumerate(_serve_cases(case)):
            first.append(_first_gradient(*_data(c, seed + 1000 * i)))
        return {"norms": np.array([np.linalg.norm(g) for g in first]), "x": None, "grad": first, "l": None}
    ns, a, y = _data(case, seed)
    x = _minimiser(ns, a, y) if case.get("name") in _CONVERGES else None
    # the first round's ||g|| belongs to x = 0 (a mixed case's first pass starts there)
    out = {"norms": None, "first": np.linalg.norm(_first_gradient(ns, a, y)), "x": x, "grad": None}
    return out if kind == "job" else dict(out, l=None) if kind == "mixed" else dict(out, H=None, l=None)
