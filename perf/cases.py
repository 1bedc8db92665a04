"""Calls that a program built on this library makes, for timing them and comparing their results.

Three kinds of work: searches (a block of queries against a block of
references through the handle's process_packed, or gtb_process_resident on
blocks kept on the device), clustering runs (all against all, then the
linkage), and the TM-score adjoint on fixed alignments (gradients, autograd,
polishing).  Structures come from gtalign_alpha_b200.synth, with the length
distributions of the benchmark's workloads; alignments for the adjoint are
random walks of 3.8 A steps against rigidly moved copies with 1.5 A noise.

A search ends in the local optimum that its FP32 comparisons choose, and the
library promises the same bits for the same inputs, so its records, transforms,
numeric errors and alignment rows are compared exactly; records are returned as
the 32-bit words they are (two of their fields are packed coordinates).
"""
import ctypes
import math

import numpy as np
import torch

from gtalign_alpha_b200 import adjoint, api, synth


def listed():
    return [
        # the smallest call: one structure against one other at the command
        # line's default options, as a viewer or a notebook makes it; latency
        {"name": "pair_150", "kind": "search", "speed": 9, "nq": 1, "qlen": 150, "nr": 1, "lo": 150,
         "hi": 150, "homologs": 1.0, "rows": True, "resident": False},
        # one query against a small library, default options (detailed search on)
        {"name": "query_1000_default", "kind": "search", "speed": 9, "nq": 1, "qlen": 150, "nr": 1000,
         "lo": 50, "hi": 500, "homologs": 0.2, "rows": True, "resident": False},
        # the same at the fastest preset
        {"name": "query_1000_fast", "kind": "search", "speed": 13, "nq": 1, "qlen": 150, "nr": 1000,
         "lo": 50, "hi": 500, "homologs": 0.2, "rows": True, "resident": False},
        # a block of queries from host buffers, detailed search off, alignment
        # rows back: what a query server does per batch; ragged lengths
        {"name": "block_16x500", "kind": "search", "speed": -1, "nq": 16, "qlen": 0, "nr": 500,
         "lo": 0, "hi": 0, "homologs": 0.05, "rows": True, "resident": False},
        # a database chunk kept on the device, two queries per call (the
        # benchmark's shape, a tenth of its references)
        {"name": "chunk_2x20000", "kind": "search", "speed": -1, "nq": 2, "qlen": 0, "nr": 20000,
         "lo": 0, "hi": 0, "homologs": 0.05, "rows": False, "resident": True},
        # the same with the detailed search on
        {"name": "chunk_2x8000_default", "kind": "search", "speed": 9, "nq": 2, "qlen": 0, "nr": 8000,
         "lo": 0, "hi": 0, "homologs": 0.05, "rows": False, "resident": True},
        # two large assemblies superposed
        {"name": "pair_5000", "kind": "long", "speed": -1, "len": 5000},
        # a clustering run: all against all under the coverage filter, then
        # complete linkage
        {"name": "cluster_400", "kind": "cluster", "n": 400},
        # gradients of a few alignments (the inner loop of an optimiser)
        {"name": "adjoint_64", "kind": "adjoint", "pairs": 64, "lo": 60, "hi": 600},
        # gradients of many alignments
        {"name": "adjoint_50000", "kind": "adjoint", "pairs": 50000, "lo": 60, "hi": 600},
        # the TM-score as a differentiable function: forward and backward
        {"name": "tmscore_20000", "kind": "tmscore", "pairs": 20000, "lo": 60, "hi": 600},
        # polishing the transforms of many fixed alignments, 10 steps
        {"name": "polish_100000", "kind": "polish", "pairs": 100000, "lo": 60, "hi": 600, "steps": 10},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["pair", "query", "block", "chunk", "long", "cluster", "adjoint", "tmscore", "polish"])
    speed = rng.choice([9, 13, -1])
    if what == "pair":
        return {"kind": "search", "speed": speed, "nq": 1, "qlen": _log(rng, 40, 800), "nr": 1,
                "lo": 40, "hi": 800, "homologs": rng.choice([0.0, 1.0]), "rows": rng.random() < 0.5, "resident": False}
    if what == "query":
        return {"kind": "search", "speed": speed, "nq": 1, "qlen": _log(rng, 50, 500), "nr": _log(rng, 10, 2000),
                "lo": 50, "hi": 500, "homologs": 0.2, "rows": rng.random() < 0.5, "resident": False}
    if what == "block":
        return {"kind": "search", "speed": speed, "nq": rng.randint(2, 16), "qlen": 0, "nr": _log(rng, 20, 500),
                "lo": 0, "hi": 0, "homologs": 0.05, "rows": rng.random() < 0.5, "resident": False}
    if what == "chunk":
        return {"kind": "search", "speed": speed, "nq": rng.randint(1, 2), "qlen": 0, "nr": _log(rng, 1000, 12000),
                "lo": 0, "hi": 0, "homologs": 0.05, "rows": False, "resident": True}
    if what == "long":
        return {"kind": "long", "speed": rng.choice([13, -1]), "len": _log(rng, 1200, 5000)}
    if what == "cluster":
        return {"kind": "cluster", "n": _log(rng, 40, 400)}
    lo = rng.randint(20, 100)
    hi = lo + rng.randint(20, 600)
    if what == "adjoint":
        return {"kind": "adjoint", "pairs": _log(rng, 1, 50000), "lo": lo, "hi": hi}
    if what == "tmscore":
        return {"kind": "tmscore", "pairs": _log(rng, 1, 20000), "lo": lo, "hi": hi}
    return {"kind": "polish", "pairs": _log(rng, 1, 80000), "lo": lo, "hi": hi, "steps": rng.randint(1, 12)}


# -------------------------------------------------------------------------
# searches

def _options(case, **kw):
    if case["speed"] < 0:
        return api.Options(**kw)            # the defaults with the detailed search off
    return api.Options.speed(case["speed"], **kw)


def _lengths(case):
    """Query and reference lengths, the same for every seed.  qlen 0: those of
    the benchmark's large workload (queries U(80,800), references log-normal,
    median 250); else one query of qlen residues against targets U(lo,hi)."""
    rng = np.random.default_rng([case["nq"], case["nr"], case["qlen"]])
    if case["qlen"] == 0:
        ql = rng.integers(80, 801, size=case["nq"])
        rl = np.clip(np.round(rng.lognormal(math.log(250.0), 0.6, size=case["nr"])), 30, 2000).astype(int)
    else:
        ql = np.full(case["nq"], case["qlen"])
        rl = rng.integers(case["lo"], case["hi"] + 1, size=case["nr"])
    return ql, rl, rng


def _workload(case, seed):
    """(queries, references): random chains of these lengths; a share of the
    references are homologs of the queries (0.5-4 A of noise, up to 15% of
    indels, the same indels for every seed)."""
    ql, rl, shape = _lengths(case)
    rng = np.random.default_rng(seed)
    queries = synth.random_chains(rng, ql, "q")
    refs = synth.random_chains(rng, rl, "r")
    for i in np.nonzero(shape.random(len(refs)) < case["homologs"])[0]:
        refs[i] = synth.homolog(shape, queries[int(shape.integers(len(queries)))], float(shape.uniform(0.5, 4.0)),
                                float(shape.uniform(0.0, 0.15)), "h")
    return synth.pack(queries), synth.pack(refs)


class _Host:
    """Blocks in host memory and the handle a program keeps."""

    def __init__(self, q, r, options, rows):
        self.q, self.r, self.rows = api.pack_fields(q), api.pack_fields(r), rows
        self.g = api.GTalignB200(0, 0, options)

    def run(self):
        res = self.g.process_packed(self.q, self.r, scorethld=0.5, alignments=self.rows)
        out = [res.alndata.view(np.int32), res.tfm, res.numerr]
        return out + [res.alns_raw] if self.rows else out


class _Resident:
    """Blocks and result buffers on the device."""

    def __init__(self, q, r, options):
        self.g = api.GTalignB200(0, 0, options)
        self.q = self.g.upload(api.pack_fields(q))
        self.r = self.g.upload(api.pack_fields(r))
        n = q.n * r.n
        self.rec = torch.zeros((n, api.NOUT), dtype=torch.float32, device="cuda")
        self.tfm = torch.zeros((n, 12), dtype=torch.float32, device="cuda")
        self.err = torch.zeros((n, api.NERR), dtype=torch.float32, device="cuda")

    def run(self):
        p = [ctypes.c_void_p(t.data_ptr()) for t in (self.rec, self.tfm, self.err)]
        st = self.g.lib.gtb_process_resident(self.g.handle, 0.5, self.q.h, self.r.h, *p)
        if st != 0:
            raise api.GTBError(st, self.g.lib.gtb_last_error(self.g.handle).decode())
        return [self.rec.view(torch.int32), self.tfm, self.err]

    def __del__(self):
        for b in ("q", "r"):
            if hasattr(self, b):
                getattr(self, b).free()
        if hasattr(self, "g"):
            self.g.close()


class _Cluster:
    def __init__(self, s):
        self.s = s
        idx = np.arange(s.n, dtype=np.int32)
        self.q, self.r = api.pack_fields(s, idx), api.pack_fields(s, idx)
        self.g = api.GTalignB200(0, 0, api.Options.speed(13, clsfilter=1))

    def run(self):
        res = self.g.process_packed(self.q, self.r, scorethld=0.5, alignments=False, numerr=False)
        c = api.cluster(res.alndata, self.s.lens)
        return [res.alndata.view(np.int32), res.tfm, c.pi, c.lam]


# -------------------------------------------------------------------------
# fixed alignments

def _lens(case):
    return np.random.default_rng([case["pairs"], case["lo"], case["hi"]]).integers(
        case["lo"], case["hi"] + 1, size=case["pairs"])


def _alignments(case, seed):
    """q, r (N, 3), off, n, tfm (P, 12), d0 (P,) on the device: a chain, its
    rigidly moved copy with 1.5 A noise, and a transform 0.05 rad and 0.5 A
    off the true one."""
    n = torch.from_numpy(_lens(case)).cuda()
    P, L = case["pairs"], case["hi"]
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)

    off = torch.cumsum(n, 0) - n
    # padded to the longest: sums along a row have one order, so that a seed
    # gives the same bits each time
    there = torch.arange(L, device="cuda")[None, :] < n[:, None]
    x = torch.cumsum(torch.nn.functional.normalize(normal(P, L, 3), dim=2) * 3.8, 1)
    x = x - (x * there[:, :, None]).sum(1, keepdim=True) / n[:, None, None]
    x = x[there]
    N = x.shape[0]
    pid = torch.repeat_interleave(torch.arange(P, device="cuda"), n, output_size=N)
    R = _rotation(normal(P, 4))
    E = _rotation(torch.cat([torch.ones(P, 1, dtype=torch.float64, device="cuda"), 0.025 * normal(P, 3)], 1))
    t = 10.0 * normal(P, 3)
    y = _apply(R, pid, x) + t[pid] + 1.5 * normal(N, 3)
    R0 = (E[:, :, :, None] * R[:, None, :, :]).sum(2)
    tfm = torch.cat([R0.reshape(P, 9), t + 0.5 * normal(P, 3)], 1)
    d0 = torch.clamp(1.24 * torch.sign(n - 15.0) * torch.abs(n - 15.0).double() ** (1 / 3) - 1.8, min=0.5)
    return {"q": x.float(), "r": y.float(), "off": off, "n": n.int(), "tfm": tfm.float(), "d0": d0.float(),
            "pid": pid}


def _apply(M, pid, x):
    """Each row of x by its pair's matrix."""
    return (M[pid] * x[:, None, :]).sum(2)


def _rotation(q):
    a, b, c, d = torch.nn.functional.normalize(q, dim=1).unbind(1)
    return torch.stack([a * a + b * b - c * c - d * d, 2 * (b * c - a * d), 2 * (b * d + a * c),
                        2 * (b * c + a * d), a * a - b * b + c * c - d * d, 2 * (c * d - a * b),
                        2 * (b * d - a * c), 2 * (c * d + a * b), a * a - b * b - c * c + d * d],
                       1).reshape(-1, 3, 3)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "search":
        q, r = _workload(case, seed)
        return _Resident(q, r, _options(case)) if case["resident"] else _Host(q, r, _options(case), case["rows"])
    if kind == "long":
        wl = synth.config2(seed=seed, lengths=(case["len"],))
        return _Host(synth.pack(wl.queries), synth.pack(wl.refs), _options(case), True)
    if kind == "cluster":
        return _Cluster(synth.pack(synth.config4(seed=seed, n=case["n"]).queries))
    s = _alignments(case, seed)
    del s["pid"]
    if kind == "tmscore":
        s["gout"] = torch.rand(case["pairs"], generator=torch.Generator(device="cuda").manual_seed(seed + 1),
                               device="cuda")
        s["q"].requires_grad_(True)
        s["tfm"].requires_grad_(True)
    s["case"] = case
    return s


def run(state):
    if not isinstance(state, dict):
        return state.run()
    q, r, off, n, tfm, d0 = (state[k] for k in ("q", "r", "off", "n", "tfm", "d0"))
    kind = state["case"]["kind"]
    if kind == "adjoint":
        return list(adjoint.tm_adjoint(q, r, off, n, tfm, d0, want_gq=True))
    if kind == "tmscore":
        tm = adjoint.TMScore.apply(q, tfm, r, off, n, d0)
        gq, gt = torch.autograd.grad(tm, (q, tfm), state["gout"])
        return [tm.detach(), gq, gt]
    t = tfm.clone()                            # polishing works in place
    before, after = adjoint.polish(q, r, off, n, t, d0, steps=state["case"]["steps"])
    return [before, after, t]


# -------------------------------------------------------------------------

def _search_work(ql, rl):
    """Least work of a search over every pair: the seed (each diagonal with at
    least half the shorter chain: a covariance and three scored passes), the
    refinement of each alignment's fragments (three rounds of three passes)
    and the two DP matrices before the score filter; 48 operations per scored
    position, 12 per DP cell.  What the filter leaves is not counted."""
    q = np.asarray(ql, np.float64)[:, None]
    r = np.asarray(rl, np.float64)[None, :]
    m = np.minimum(q, r)
    visits = q * r - (m / 2) ** 2
    variants = 6.0 * (m / 40 + 1)
    flops = (visits * 105 + variants * 9 * m * 48 + 24 * q * r).sum()
    nbytes = 13.0 * (q.sum() + r.sum()) + 4.0 * (16 + 12 + 4) * q.size * r.size
    return {"bytes": float(nbytes), "flops": float(flops)}


def work(case):
    kind = case["kind"]
    if kind == "search":
        ql, rl, _ = _lengths(case)
        return _search_work(ql, rl)
    if kind == "long":
        return _search_work([case["len"]], [case["len"]])
    if kind == "cluster":
        rl = np.clip(np.random.default_rng(0).lognormal(math.log(220.0), 0.6, size=case["n"]), 40, 1200)
        # the triangle, and of it the pairs the coverage filter lets through
        keep = np.minimum(rl[:, None], rl) >= 0.7 * np.maximum(rl[:, None], rl)
        w = _search_work(rl, rl)
        return {"bytes": w["bytes"], "flops": w["flops"] * float(np.tril(keep, -1).mean())}
    N, P = float(_lens(case).sum()), case["pairs"]
    if kind == "adjoint":
        return {"bytes": N * 36 + P * 96, "flops": N * 75}
    if kind == "tmscore":
        return {"bytes": N * 36 + P * 130, "flops": N * 110}
    # polishing: a step needs the centroid, the gradient with its curvature,
    # and a trial score, and the pass before the first step
    return {"bytes": N * 24 + P * 120, "flops": N * (25 + case["steps"] * 120)}


def tolerance(case):
    # FP32 sums over an alignment in another order
    if case["kind"] == "adjoint":
        return {"rel": 4e-6}
    if case["kind"] == "tmscore":
        return {"rel": 4e-6}
    if case["kind"] == "polish":
        # a step near the optimum is kept or halved on the last bits of the score
        return {"rel": 1e-5, "max": 0.05}
    return "exact"


# -------------------------------------------------------------------------
# the adjoint's outputs in 64 bits

def _segment(v, pid, P):
    return torch.zeros((P,) + v.shape[1:], dtype=torch.float64, device="cuda").index_add_(0, pid, v)


def _terms(q, r, pid, T, d0):
    p = _apply(T[:, :9].reshape(-1, 3, 3), pid, q)
    e = p + T[pid, 9:] - r
    u = d0[pid] ** 2 + (e * e).sum(1)
    return p, e, u


def _polish64(q, r, pid, n, T, d0, steps):
    P = T.shape[0]

    def score(X):
        return _segment(d0[pid] ** 2 / _terms(q, r, pid, X, d0)[2], pid, P)

    before = cur = score(T)
    live = torch.ones(P, dtype=torch.bool, device="cuda")
    for _ in range(steps):
        p, e, u = _terms(q, r, pid, T, d0)
        c = _segment(p + T[pid, 9:], pid, P) / n[:, None]
        k = d0[pid] ** 2 / (u * u)
        ge = -2.0 * k[:, None] * e
        a = p + T[pid, 9:] - c[pid]
        ht = _segment(2.0 * k, pid, P)
        hw = _segment(2.0 * k * (a * a).sum(1), pid, P)
        w = _segment(torch.linalg.cross(a, ge), pid, P) / hw[:, None]
        dt = _segment(ge, pid, P) / ht[:, None]
        todo = live.clone()
        for _ in range(10):
            if not bool(todo.any()):
                break
            K = torch.zeros(P, 3, 3, dtype=torch.float64, device="cuda")
            K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -w[:, 2], w[:, 1], -w[:, 0]
            E = torch.linalg.matrix_exp(K - K.transpose(1, 2))
            X = torch.cat([torch.bmm(E, T[:, :9].reshape(-1, 3, 3)).reshape(-1, 9),
                           torch.bmm(E, (T[:, 9:] - c)[:, :, None])[:, :, 0] + c + dt], 1)
            s = score(X)
            up = todo & (s > cur)
            T = torch.where(up[:, None], X, T)
            cur = torch.where(up, s, cur)
            todo = todo & ~up
            w, dt = 0.5 * w, 0.5 * dt
        live = live & ~todo
    return [before, cur, T]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("search", "long", "cluster"):
        # the end point of a search over local optima that FP32 scores choose:
        # there is no 64-bit value of it apart from the search itself
        return None
    s = _alignments(case, seed)
    pid, P, n = s["pid"], case["pairs"], s["n"].double()
    q, r, T, d0 = (s[k].double() for k in ("q", "r", "tfm", "d0"))
    if kind == "polish":
        return _polish64(q, r, pid, n, T, d0, case["steps"])
    p, e, u = _terms(q, r, pid, T, d0)
    d02 = d0[pid] ** 2
    tm = _segment(d02 / u, pid, P)
    ge = -2.0 * (d02 / (u * u))[:, None] * e
    gq = _apply(T[:, :9].reshape(-1, 3, 3).transpose(1, 2), pid, ge)
    gt = _segment(ge, pid, P)
    if kind == "adjoint":
        return [tm, torch.cat([_segment(torch.linalg.cross(p, ge), pid, P), gt], 1), gq]
    gout = torch.rand(P, generator=torch.Generator(device="cuda").manual_seed(seed + 1), device="cuda").double()
    gR = _segment(ge[:, :, None] * q[:, None, :], pid, P)
    return [tm, gq * gout[pid, None], torch.cat([gR.reshape(P, 9), gt], 1) * gout[:, None]]
