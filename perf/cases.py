"""What the performance of this solver is measured on.

Every case is one pass through an entry point that a user's program calls:
``mrrr`` and ``dsyeig`` on host arrays, ``mr3_batched`` with page-locked host
buffers, batched solves on device arrays and the serving handle.  Inputs come
from a seed alone (``mr3smp_b200.workloads``; families whose entries are fixed
are multiplied by a factor drawn from the seed, a change of units).  The
solver overwrites D and E, so a pass on device arrays starts with their copy.
"""
import ctypes as C
import math

import numpy as np
import torch

import mr3smp_b200 as M
from mr3smp_b200 import workloads as wl

# sizes and shares of the serving mix up to 4096
SERVE_MIX = ((64, 0.4), (256, 0.3), (1024, 0.2), (4096, 0.1))


def listed():
    return [
        # one small problem per call from host arrays: latency of a call
        dict(name="call_tiny", kind="call", family="uniform", n=33, jobz="V", range="A"),
        # the drop-in call at an ordinary size, eigenpairs, relative accuracy asked for
        dict(name="call_1000", kind="call", family="uniform", n=1000, jobz="V", range="A", tryrac=1),
        # eigenvalues only, to full precision
        dict(name="values_3001", kind="call", family="uniform", n=3001, jobz="N", range="A"),
        # eigenpairs of a value interval of a matrix with structured spectrum
        dict(name="interval_2000", kind="device", family="121", n=2000, jobz="V", range="V",
             lo=0.3, hi=0.65),
        # graded matrix whose eigenvalues keep high relative accuracy (dlarrj)
        dict(name="graded_1500", kind="device", family="graded", n=1500, jobz="V", range="A",
             tryrac=1),
        # many small problems at once, arrays in device memory
        dict(name="batch_small", kind="batch", count=1000, nmin=20, nmax=200),
        # the mixed batch (n log-uniform in [32, 4096], 25 % 1-2-1), a quarter of its count
        dict(name="batch_mixed", kind="batch", count=1024, nmin=32, nmax=4096),
        # a batch from and to host memory, copies of the eigenvectors included
        dict(name="host_batch", kind="host_batch", count=200, nmin=32, nmax=2048),
        # the lower half of 30 glued Wilkinson blocks: deep clusters, one large problem
        dict(name="glued_20010", kind="device", family="glued", n=20010, jobz="V", range="I",
             lo=0.0, hi=0.5),
        # half random, half glued Wilkinson blocks, all eigenpairs
        dict(name="mixed_9000", kind="device", family="mixed", n=9000, jobz="V", range="A"),
        # a burst of requests of the serving mix, ranges A and I alternating
        dict(name="serve_burst", kind="serve", count=60),
        # the dense symmetric driver from and to host arrays
        dict(name="dense_700", kind="dense", n=700, jobz="V", range="A", uplo="L"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("call", "call", "device", "device", "batch", "batch", "host_batch",
                       "serve", "dense"))
    if kind == "batch":
        nmax = _log_int(rng, 100, 4096)
        return dict(kind=kind, count=min(1024, _log_int(rng, 24, 1500)),
                    nmin=_log_int(rng, 10, nmax // 4), nmax=nmax)
    if kind == "host_batch":
        return dict(kind=kind, count=_log_int(rng, 8, 200), nmin=_log_int(rng, 16, 64),
                    nmax=_log_int(rng, 100, 2048))
    if kind == "serve":
        return dict(kind=kind, count=_log_int(rng, 20, 120))
    rg = rng.choice("AAIV")
    c = dict(kind=kind, jobz=rng.choice("VVVN"), range=rg)
    if rg != "A":
        c["lo"] = round(rng.uniform(0.0, 0.6), 3)
        c["hi"] = round(min(1.0, c["lo"] + rng.uniform(0.05, 0.5)), 3)
    if kind == "dense":
        return dict(c, n=_log_int(rng, 50, 700), uplo=rng.choice("LU"))
    if kind == "call":
        c.update(family=rng.choice(("uniform", "uniform", "121")), n=_log_int(rng, 20, 2000))
        if rng.random() < 0.3:
            c["tryrac"] = 1
        return c
    c.update(family=rng.choice(("uniform", "121", "glued", "mixed")), n=_log_int(rng, 500, 12000))
    return c


def _matrix(family, n, seed):
    if family == "uniform":
        return wl.uniform(n, seed)
    s = 1.0 + 0.5 * float(np.random.default_rng(seed).random())
    if family == "121":
        D, E = wl.one_two_one(n)
    elif family == "glued":
        D, E = wl.glued_wilkinson(-(-n // 667), 667, 1e-12)
        D, E = D[:n].copy(), E[:n].copy()
        E[-1] = 0.0
    elif family == "mixed":
        D, E = wl.large_mixed(n, seed)
    elif family == "graded":
        g = 10.0 ** (-np.arange(n) * (280.0 / n))
        D, E = 3.0 * g, np.r_[np.sqrt(g[:-1] * g[1:]), 0.0]
    else:
        raise ValueError(family)
    return s * D, s * E


def _span(D, E):
    """Gershgorin bounds of the spectrum."""
    r = np.abs(E) + np.r_[0.0, np.abs(E[:-1])]
    return float((D - r).min()), float((D + r).max())


def _bounds(case, n, gl, gu):
    """The range arguments of a case: il, iu (range I) or vl, vu (range V)."""
    if case["range"] == "I":
        il = 1 + int(case["lo"] * (n - 1))
        return dict(il=il, iu=max(il, int(case["hi"] * n)))
    if case["range"] == "V":
        return dict(vl=gl + case["lo"] * (gu - gl), vu=gl + case["hi"] * (gu - gl))
    return {}


def _cols(case, n, kw):
    return kw["iu"] - kw["il"] + 1 if "il" in kw else n


def _symmetric(n, seed):
    A = np.random.default_rng(seed).uniform(-1.0, 1.0, (n, n))
    return np.tril(A) + np.tril(A, -1).T


def _batch(case, seed):
    """(D, E) of a batch: sizes log-uniform in [nmin, nmax], a quarter 1-2-1;
    the sizes are the distribution's quantiles, in an order from the seed."""
    k, a, b = case["count"], case["nmin"], case["nmax"]
    rng = np.random.default_rng(seed)
    ns = rng.permutation(np.rint(a * (b / a) ** ((np.arange(k) + 0.5) / k)).astype(int))
    return [wl.one_two_one(int(n)) if rng.random() < 0.25 else
            wl.uniform(int(n), int(rng.integers(1 << 30))) for n in ns]


def _serve_requests(count):
    """(n, wanted) of the serving mix: per size alternately all eigenpairs
    and the lowest tenth."""
    return [(n, n if k % 2 == 0 else -(-n // 10)) for n, p in SERVE_MIX
            for k in range(max(1, round(p * count)))]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "dense":
        A = _symmetric(case["n"], seed)
        r = math.sqrt(case["n"] * 4 / 3)   # the semicircle's radius
        return dict(case=case, A=A, kw=_bounds(case, case["n"], -r, r))
    if kind == "call":
        D, E = _matrix(case["family"], case["n"], seed)
        return dict(case=case, D=D, E=E, kw=dict(_bounds(case, case["n"], *_span(D, E)),
                                                 tryrac=case.get("tryrac", 0)))
    if kind == "device":
        n = case["n"]
        Dh, Eh = _matrix(case["family"], n, seed)
        kw = _bounds(case, n, *_span(Dh, Eh))
        cols = _cols(case, n, kw)
        D0, E0 = torch.from_numpy(Dh).cuda(), torch.from_numpy(Eh).cuda()
        pb = dict(jobz=case["jobz"], range=case["range"], D=D0.clone(), E=E0.clone(),
                  W=torch.zeros(n, dtype=torch.float64, device="cuda"),
                  tryrac=case.get("tryrac", 0), **kw)
        if case["jobz"] == "V":
            pb["Z"] = torch.zeros(n * cols, dtype=torch.float64, device="cuda")
            pb["Zsupp"] = torch.zeros(2 * cols, dtype=torch.int32, device="cuda")
        return dict(case=case, D0=D0, E0=E0, pb=pb, stream=torch.cuda.Stream())
    if kind == "batch":
        recs, T = M.device_batch(_batch(case, seed))
        return dict(case=case, recs=recs, T=T, solver=M.Solver(0), stream=torch.cuda.Stream())
    if kind == "host_batch":
        probs = _batch(case, seed)
        ns = [len(D) for D, _ in probs]
        N, NZ = sum(ns), sum(n * n for n in ns)

        def pinned(k, dtype=torch.float64):
            return torch.zeros(k, dtype=dtype, pin_memory=True).numpy()
        s = dict(case=case, D0=np.concatenate([p[0] for p in probs]),
                 E0=np.concatenate([p[1] for p in probs]), D=pinned(N), E=pinned(N), W=pinned(N),
                 Z=pinned(NZ), Zsupp=pinned(2 * N, torch.int32))
        recs = (M.HostProb * len(ns))()
        o = oz = 0
        for h, n in zip(recs, ns):
            h.jobz, h.range, h.n, h.il, h.iu, h.ldz = b"V", b"A", n, 1, 1, n
            for name, at in (("D", o), ("E", o), ("W", o), ("Z", oz)):
                setattr(h, name, s[name][at:].ctypes.data_as(C.POINTER(C.c_double)))
            h.Zsupp = s["Zsupp"][2 * o:].ctypes.data_as(C.POINTER(C.c_int))
            o += n
            oz += n * n
        s["recs"] = recs
        return s
    # serve: every request's D, E staged in device memory, results resident there
    rng = np.random.default_rng(seed)
    asked = rng.permutation(_serve_requests(case["count"])).tolist()
    N, NC = sum(n for n, _ in asked), sum(m for _, m in asked)
    D0 = torch.from_numpy(rng.uniform(-1.0, 1.0, N)).cuda()
    E0 = torch.from_numpy(rng.uniform(-1.0, 1.0, N)).cuda()
    s = dict(case=case, D0=D0, E0=E0, D=D0.clone(), E=E0.clone(),
             W=torch.zeros(N, dtype=torch.float64, device="cuda"),
             Z=torch.zeros(sum(n * m for n, m in asked), dtype=torch.float64, device="cuda"),
             Zsupp=torch.zeros(2 * NC, dtype=torch.int32, device="cuda"), server=M.Server(0))
    s["requests"] = []
    o = oz = oc = 0
    for n, m in asked:
        s["requests"].append(dict(
            jobz="V", range="A" if m == n else "I", il=1, iu=m, D=s["D"][o:o + n],
            E=s["E"][o:o + n], W=s["W"][o:o + n], Z=s["Z"][oz:oz + n * m],
            Zsupp=s["Zsupp"][2 * oc:2 * (oc + m)]))
        o += n
        oz += n * m
        oc += m
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "dense":
        return M.dsyeig(case["jobz"], case["range"], case["uplo"], state["A"], **state["kw"])
    if kind == "call":
        return M.mrrr(case["jobz"], case["range"], state["D"], state["E"], **state["kw"])
    if kind == "device":
        pb, st = state["pb"], state["stream"]
        with torch.cuda.stream(st):
            pb["D"].copy_(state["D0"])
            pb["E"].copy_(state["E0"])
        rc, res = M.mrrr_batched_device([pb], stream=st.cuda_stream)
        out = dict(info=rc, m=res[0].m, W=pb["W"][:res[0].m], D=pb["D"], E=pb["E"])
        if case["jobz"] == "V":
            out["Z"] = pb["Z"][:case["n"] * res[0].m]
            out["Zsupp"] = pb["Zsupp"][:2 * res[0].m]
        return out
    if kind == "batch":
        T, st = state["T"], state["stream"]
        with torch.cuda.stream(st):
            T["D"].copy_(T["D0"])
            T["E"].copy_(T["E0"])
        rc = state["solver"].solve(state["recs"], stream=st.cuda_stream)
        return dict(info=rc, m=np.array([q.m for q in state["recs"]]), W=T["W"], Z=T["Z"],
                    Zsupp=T["Zsupp"], D=T["D"], E=T["E"])
    if kind == "host_batch":
        state["D"][:] = state["D0"]
        state["E"][:] = state["E0"]
        rc = M.lib().mr3_batched(len(state["recs"]), state["recs"])
        return dict(info=rc, m=np.array([h.m for h in state["recs"]]),
                    **{k: state[k] for k in ("W", "Z", "Zsupp", "D", "E")})
    srv = state["server"]
    state["D"].copy_(state["D0"])
    state["E"].copy_(state["E0"])
    torch.cuda.current_stream().synchronize()   # the server's lanes have streams of their own
    tickets = [srv.submit_device(q) for q in state["requests"]]
    done = [srv.poll(t)[0] for t in tickets]
    return dict(info=max(r["info"] for r in done), m=np.array([r["m"] for r in done]),
                **{k: state[k] for k in ("W", "Z", "Zsupp", "D", "E")})


def work(case):
    """Bytes: D and E in, W, Z and the supports out.  Operations: a twisted
    factorisation and its back-substitution per eigenvector (13 a row), one
    Sturm count per eigenvalue (4 a row)."""
    kind = case["kind"]
    if kind in ("batch", "host_batch"):
        a, b, k = case["nmin"], case["nmax"], case["count"]
        ln = math.log(b / a)   # moments of the log-uniform sizes
        rows, pairs, entries, vec = k * (b - a) / ln, k * (b - a) / ln, k * (b * b - a * a) / 2 / ln, 1
    elif kind == "serve":
        asked, vec = _serve_requests(case["count"]), 1
        rows, pairs = sum(n for n, _ in asked), sum(m for _, m in asked)
        entries = sum(n * m for n, m in asked)
    else:
        n, vec = case["n"], int(case["jobz"] == "V")
        share = 1.0 if case["range"] == "A" else case["hi"] - case["lo"]
        rows, pairs, entries = n, share * n, share * n * n
        if kind == "dense":
            return {"bytes": 8 * n * n + 8 * pairs + 8 * entries * vec,
                    "flops": 4 / 3 * n ** 3 + vec * 2 * n * entries}
    return {"bytes": 16 * rows + 8 * pairs + vec * (8 * entries + 8 * pairs),
            "flops": entries * (17 if vec else 4)}


def _eigenvalues(A):
    A = torch.from_numpy(A)
    return torch.linalg.eigvalsh(A.cuda() if torch.cuda.is_available() else A).cpu().numpy()


def exact(case, seed):
    """The eigenvalues by a dense 64-bit solver.  An eigenvector is defined
    up to its sign, and one of a cluster only together with the cluster's
    others; D and E hold a representation that the solver chose: no value."""
    kind, n = case["kind"], case.get("n", 0)
    none = dict.fromkeys(("D", "E", "Z", "Zsupp", "info", "m", "il", "iu", "tryrac", "vl", "vu"))
    if kind in ("batch", "host_batch") and case["nmax"] <= 300:
        return none | {"W": np.concatenate([
            np.linalg.eigvalsh(np.diag(D) + np.diag(E[:-1], 1) + np.diag(E[:-1], -1))
            for D, E in _batch(case, seed)])}
    if kind not in ("call", "device", "dense") or n > 3500 or case.get("family") == "graded":
        return None   # (graded: a dense solver loses the small eigenvalues)
    if kind == "dense":
        A = _symmetric(n, seed)
        r = math.sqrt(n * 4 / 3)
        kw = _bounds(case, n, -r, r)
    else:
        D, E = _matrix(case["family"], n, seed)
        A = np.diag(D) + np.diag(E[:-1], 1) + np.diag(E[:-1], -1)
        kw = _bounds(case, n, *_span(D, E))
    w = _eigenvalues(A)
    if case["range"] == "I":
        w = w[kw["il"] - 1:kw["iu"]]
    elif case["range"] == "V":
        w = w[(w > kw["vl"]) & (w <= kw["vu"])]
    return none | {"W": w}
