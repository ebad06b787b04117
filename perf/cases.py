"""The calls that a user of this package makes, as cases to time and compare.

A program that uses the package enumerates the active sets of one problem
through the drop-in C call (``host.call_mpqp``, what main.py does for every
problem it loads), hands many problems to one launch sequence
(``solver.solve``), turns the optimal sets it found into laws and regions
(``mpqp_critical_regions``), and reduces a problem's rows before any of this
(``solver.reduce_constraints``).  All of these take host arrays and return
host arrays, so a pass is the whole call: upload, enumeration, download.

Problems are scaled as the driver scales them (``problems.scale_problem``).
A case's problems follow from its seed alone; sizes are this repository's own
workloads and test problems.
"""
from __future__ import annotations

import ctypes
import itertools
import math

import numpy as np

from mpqpcudasolver_gb300 import host
from mpqpcudasolver_gb300 import problems as P
from mpqpcudasolver_gb300 import solver

R_MIN, TOL = 1e-8, 1e-9          # region and optimality thresholds of the reference


def listed():
    return [
        # the smallest call of the driver's loop: one of its test problems, every |S| <= n
        dict(name="mpqp_n4", kind="mpqp", n=4, m=10, p=2, k=4),
        # an ordinary drop-in call: the mid-size problem to |S| = 4
        dict(name="mpqp_n10", kind="mpqp", n=10, m=43, p=4, k=4),
        # the driver's set of 43 small test problems in one call (n <= 5, m <= 16), every |S| <= n
        dict(name="small_set", kind="set", count=43, n_max=5, m_max=16, precision="mixed"),
        # the same kind of set, larger problems (n <= 7, m <= 22), in plain FP64, the default of solve()
        dict(name="small_set_fp64", kind="set", count=24, n_max=7, m_max=22, precision="fp64"),
        # the m = 62 problem to |S| = 4: a call of some milliseconds
        dict(name="m62_k4", kind="solve", n=12, m=62, p=6, k=4, count=1, budget=0, precision="mixed"),
        # the mid-size problem in plain FP64
        dict(name="n10_fp64", kind="solve", n=10, m=43, p=4, k=4, count=1, budget=0, precision="fp64"),
        # condensed MPC problems (sparse input and state bounds), many in one launch
        dict(name="mpc_64", kind="mpc", count=64, k=3, precision="mixed"),
        # ill-conditioned Q, near-duplicate rows, p = 8 (the screen's primal route)
        dict(name="illcond_k3", kind="illcond", count=1, k=3, precision="mixed"),
        # multiparametric LPs (Q = 0) of mixed sizes, every |S| <= n
        dict(name="mplp_32", kind="mplp", count=32, precision="mixed"),
        # laws, region rows and radii of the optimal sets a program holds
        dict(name="regions", kind="regions", n=12, m=62, p=6, sets=1024),
        # row reduction of a condensed MPC problem (72 rows)
        dict(name="reduce_mpc", kind="reduce", horizon=6),
        # the benchmark batch: the m = 62 problem to |S| = 6 and 32 problems of
        # mixed sizes under a budget each, the largest call
        dict(name="m62_batch", kind="batch", k=6, extra=32, budget=1 << 19, precision="mixed"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sets_up_to(m, k):
    return sum(math.comb(m, i) for i in range(min(k, m) + 1))


def _depth(m, n, most):
    """The largest k <= n whose sets of at most k rows number at most `most`."""
    k = 1
    while k < n and _sets_up_to(m, k + 1) <= most:
        k += 1
    return k


def draw(rng):
    kind = rng.choice(["mpqp", "mpqp", "set", "solve", "solve", "solve", "mpc", "illcond", "mplp", "regions", "reduce",
                       "batch"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind in ("mpqp", "solve", "regions"):
        n = rng.randint(3, 14)
        m = rng.randint(n + 4, 70)
        p = rng.randint(2, 7 if kind == "solve" else 6)
    if kind == "mpqp":
        return dict(kind=kind, n=n, m=m, p=p, k=_depth(m, n, _log_int(rng, 300, 2_000_000)))
    if kind == "set":
        return dict(kind=kind, count=_log_int(rng, 2, 64), n_max=rng.randint(3, 6), m_max=rng.randint(9, 18),
                    precision=precision)
    if kind == "solve":
        count = _log_int(rng, 1, 24)
        k = _depth(m, n, _log_int(rng, 1000, 200_000 if precision == "fp64" else 4_000_000) // count + 64)
        return dict(kind=kind, n=n, m=m, p=p, k=k, count=count, budget=rng.choice([0, 0, 1 << 15]),
                    precision=precision)
    if kind == "mpc":
        return dict(kind=kind, count=_log_int(rng, 1, 60 if precision == "mixed" else 8), k=rng.randint(2, 3),
                    precision=precision)
    if kind == "illcond":
        return dict(kind=kind, count=rng.randint(2, 4), k=rng.randint(2, 3), precision="mixed")
    if kind == "mplp":
        return dict(kind=kind, count=_log_int(rng, 1, 28 if precision == "mixed" else 8), precision=precision)
    if kind == "regions":
        return dict(kind=kind, n=n, m=m, p=p, sets=_log_int(rng, 1, 4096))
    if kind == "reduce":
        return dict(kind=kind, horizon=rng.randint(2, 8))
    return dict(kind=kind, k=rng.randint(4, 5), extra=rng.randint(1, 32), budget=1 << rng.randint(13, 18),
                precision="mixed")


def _seed(seed, i):
    return 100_003 * (seed % 20_000) + i


def _problems(case, seed):
    """The case's scaled problems, the largest |S| and the budget of each."""
    kind, count = case["kind"], case.get("count", 1)
    if kind in ("mpqp", "solve", "regions"):
        probs = [P.random_mpqp(case["n"], case["m"], case["p"], _seed(seed, i)) for i in range(count)]
        ks = [case.get("k", case["n"])] * count
    elif kind == "set":
        probs = P.pop_like_set(count, seed=seed % 20_000, n_max=case["n_max"], m_max=case["m_max"])
        ks = [p.n for p in probs]
    elif kind == "mpc":
        probs = [P.mpc_mpqp(_seed(seed, i)) for i in range(count)]
        ks = [case["k"]] * count
    elif kind == "illcond":
        probs = [P.illcond_n16_m62_p8(_seed(seed, i)) for i in range(count)]
        ks = [case["k"]] * count
    elif kind == "mplp":
        probs = [P.mplp_member(_seed(seed, i)) for i in range(count)]
        ks = [p.n for p in probs]
    elif kind == "reduce":
        probs, ks = [P.mpc_mpqp(_seed(seed, 0), horizon=case["horizon"])], [0]
    else:
        probs = [P.random_mpqp(12, 62, 6, _seed(seed, 0))] + [
            P.batch_member(_seed(seed, i)) for i in range(1, case["extra"] + 1)]
        ks = [case["k"]] + [p.n for p in probs[1:]]
    budgets = [case.get("budget", 0)] * len(probs)
    if kind == "batch":
        budgets[0] = 0
    return [P.scale_problem(p) for p in probs], ks, budgets


def _room(case):
    """Rows of the outputs that hold one entry per optimal set (the rest stay zero): the number of
    optimal sets is the answer of the call, and differs from problem to problem."""
    if case["kind"] in ("mpqp", "solve"):
        return min(1 << 19, case.get("count", 1) * _sets_up_to(case["m"], case["k"]))
    return 1 << 19


def _fill(room, a):
    if len(a) > room:
        raise ValueError("%d optimal sets, room for %d" % (len(a), room))
    out = np.zeros((room,) + a.shape[1:], dtype=a.dtype)
    out[:len(a)] = a
    return out


def prepare(case, seed):
    probs, ks, budgets = _problems(case, seed)
    kind = case["kind"]
    if kind == "mpqp":
        return dict(kind=kind, lib=host.load_mpqp_cuda(), lp=host.build_lp_data(host.MPQPProb.from_mpqp(probs[0])),
                    k=case["k"], room=_room(case))
    if kind == "regions":
        prob = probs[0]
        masks = _masks(_held_sets(prob, case["sets"], seed))
        n_sets, stride = len(masks), (2 * prob.m + prob.n + prob.ncp) * (prob.p + 1)
        return dict(kind=kind, lib=solver.load(), prob=prob, ps=solver._ProblemSet([prob]), masks=masks,
                    laws=np.zeros((n_sets, stride)), sizes=np.zeros((n_sets, 4), dtype=np.intc),
                    radius=np.zeros(n_sets), err=np.zeros(n_sets))
    if kind == "reduce":
        return dict(kind=kind, prob=probs[0])
    return dict(kind="solve", probs=probs, k=ks, budget=budgets, room=_room(case),
                precision=solver.MIXED if case["precision"] == "mixed" else solver.FP64)


def run(state):
    kind = state["kind"]
    if kind == "mpqp":
        return _run_mpqp(state)
    if kind == "regions":
        return _run_regions(state)
    if kind == "reduce":
        status, red = solver.reduce_constraints(state["prob"])
        full = state["prob"]
        return dict(status=status, rows=np.array([red.m, red.ncp]),
                    **{f: _fill(len(getattr(full, f)), getattr(red, f)) for f in ("A", "b", "F", "CRA", "CRb")})
    r = solver.solve(state["probs"], precision=state["precision"], k_max=state["k"], budget=state["budget"])
    # the answer: every optimal set with its margin, radius and stated error,
    # and per problem the numbers and digests of its sets (the counters of how
    # a verdict was reached, such as pivots, are no part of it)
    room = state["room"]
    sets = {f: _fill(room, r.opt[f]) for f in ("inst", "level", "region", "t", "r", "err")}
    counts = {f: r.inst[f] for f in ("candidates", "pruned", "feasible", "optimal", "regions", "last_level", "truncated")}
    bits = {f: _fill(room, r.opt[f]).view(np.int64) for f in ("mask_lo", "mask_hi")}
    bits |= {f: np.ascontiguousarray(r.inst[f]).view(np.int64)
             for f in ("feasible_digest", "optimal_digest", "region_digest")}
    return dict(sets=sets, counts=counts, bits=bits)


def _run_mpqp(state):
    lib, lp = state["lib"], state["lp"]
    res = host.call_mpqp(lib, lp, k_max=state["k"])
    g = res.contents
    if g.status != 0:
        raise solver.MpqpError(g.status, solver.last_error())
    nf, nx = g.n_final_lps, lp["num_x"]
    arr = lambda ptr, *shape: _fill(state["room"], np.ctypeslib.as_array(ptr, shape=shape))  # noqa: E731
    out = dict(active_sets=arr(g.active_sets, nf, nx), t=arr(g.t_star, nf), r=arr(g.radius, nf),
               region=arr(g.is_region, nf), err=arr(g.law_error, nf),
               counts=np.array([g.n_batches, g.n_feasible_lps, nf, g.n_regions, g.n_candidates, g.n_pruned]))
    lib.mpqp_free(res)
    return out


def _run_regions(state):
    dp = ctypes.POINTER(ctypes.c_double)
    laws, sizes, radius, err = (state[f] for f in ("laws", "sizes", "radius", "err"))
    rc = state["lib"].mpqp_critical_regions(
        state["ps"].arr, len(sizes), state["masks"].ctypes.data_as(ctypes.POINTER(ctypes.c_uint64)),
        laws.ctypes.data_as(dp), sizes.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), radius.ctypes.data_as(dp),
        err.ctypes.data_as(dp))
    if rc:
        raise solver.MpqpError(rc, solver.last_error())
    prob = state["prob"]
    m, n = prob.m, prob.n
    # a set has k <= n multiplier rows, n primal rows and n_cr region rows; what
    # is left of its slot is not part of the answer
    out = laws.reshape(len(sizes), -1, prob.p + 1)
    lagrange = np.where((np.arange(n)[None, :] < sizes[:, :1])[:, :, None], out[:, :n], 0.0)
    for i in np.flatnonzero(sizes[:, 3] < m + prob.ncp):
        out[i, m + n + sizes[i, 3]:] = 0.0
    return dict(lagrange=lagrange, primal_and_region=out[:, m:], sizes=sizes, radius=radius, err=err)


# ---------------------------------------------------------------------
# optimal sets in hand, and 64-bit values, in plain numpy
# ---------------------------------------------------------------------
def _kkt(prob):
    QiAT = np.linalg.solve(prob.Q, prob.A.T)
    QiH, Qic = np.linalg.solve(prob.Q, prob.H), np.linalg.solve(prob.Q, prob.c)
    return QiAT, QiH, Qic, prob.A @ QiAT, prob.A @ QiH + prob.F, prob.b + prob.A @ Qic


def _held_sets(prob, count, seed):
    """`count` active sets (repeats where fewer differ) that are optimal at parameters drawn from
    the box: a primal-dual active-set iteration on each, the converged ones kept."""
    rng = np.random.default_rng(seed)
    _, _, _, W, Wh, wc = _kkt(prob)
    found = {}
    lo, hi = -prob.CRb[prob.p:], prob.CRb[:prob.p]
    for _ in range(3 * count + 16):
        d = Wh @ (lo + (hi - lo) * rng.random(prob.p)) + wc      # slacks with no row active
        act = d < 0
        for _ in range(25):
            lam = np.zeros(prob.m)
            idx = np.flatnonzero(act)
            if len(idx) > prob.n:
                break
            if len(idx):
                lam[idx] = np.linalg.solve(W[np.ix_(idx, idx)], -d[idx])
            slack = d + W @ lam
            new = np.where(act, lam > 0, slack < 0)
            if (new == act).all():
                found.setdefault(tuple(idx.tolist()))
                break
            act = new
        if len(found) >= count:
            break
    sets = list(found) or [()]
    return [sets[i % len(sets)] for i in range(count)]


def _masks(sets):
    masks = np.zeros((len(sets), 2), dtype=np.uint64)
    for i, S in enumerate(sets):
        for j in S:
            masks[i, j // 64] |= np.uint64(1) << np.uint64(j % 64)
    return masks


def _set_rows(prob, kkt, S):
    """Laws and unscaled region rows [g | h] (g theta <= h) of the set S."""
    QiAT, QiH, Qic, W, Wh, wc = kkt
    S = list(S)
    one = np.hstack([Wh, wc[:, None]])
    Lam = np.linalg.solve(W[np.ix_(S, S)], one[S]) if S else np.zeros((0, prob.p + 1))
    lagrange = -Lam
    primal = QiAT[:, S] @ Lam - np.hstack([QiH, Qic[:, None]])
    slack = one - W[:, S] @ Lam                                   # b + F theta - A x, as [theta | 1]
    off = [i for i in range(prob.m) if i not in S]
    # lambda(theta) >= 0, the inactive rows, the parameter rows
    rows = np.vstack([np.hstack([Lam[:, :-1], -Lam[:, -1:]]),
                      np.hstack([-slack[off, :-1], slack[off, -1:]]),
                      np.hstack([prob.CRA, prob.CRb[:, None]])])
    return lagrange, primal, rows


def _lp_max(G, h, last):
    """max v s.t. G theta + last v <= h, by every basis of p + 1 rows (small problems)."""
    M = np.hstack([G, last[:, None]])
    idx = np.array(list(itertools.combinations(range(len(M)), M.shape[1])))
    B = M[idx]
    ok = np.abs(np.linalg.det(B)) > 1e-10
    x = np.linalg.solve(B[ok], h[idx[ok]][:, :, None])[:, :, 0]
    slack = h[None, :] - x @ M.T
    x = x[(slack > -1e-9).all(axis=1)]
    return x[:, -1].max() if len(x) else -np.inf


def _exact_sets(prob, k_max):
    """(set, t*, r*) of every optimal set in the order mpqp() lists them."""
    kkt, out = _kkt(prob), []
    p = prob.p
    for k in range(k_max + 1):
        for S in itertools.combinations(range(prob.m), k):
            rows = _set_rows(prob, kkt, S)[2]
            G, h = rows[:, :p], rows[:, p]
            t = _lp_max(G, h, np.concatenate([np.ones(prob.m), np.zeros(prob.ncp)]))
            if t > TOL:
                nrm = np.linalg.norm(G, axis=1)
                keep = nrm > 1e-12
                out.append((S, t, _lp_max(G[keep] / nrm[keep, None], h[keep] / nrm[keep], np.ones(int(keep.sum())))))
    return out


def exact(case, seed):
    """Laws, region rows and, for problems small enough to list every basis, the LP optima t* and
    r* of the optimal sets.  Larger enumerations would take plain numpy hours."""
    kind = case["kind"]
    if kind == "regions":
        prob = _problems(case, seed)[0][0]
        kkt, memo = _kkt(prob), {}
        n, top = prob.n, prob.n + prob.m + prob.ncp
        lag, rest = np.zeros((case["sets"], n, prob.p + 1)), np.zeros((case["sets"], top, prob.p + 1))
        for i, S in enumerate(_held_sets(prob, case["sets"], seed)):
            if S not in memo:
                lagrange, primal, cr = _set_rows(prob, kkt, S)
                zero = np.abs(cr[:, :-1]).max(axis=1) <= 1e-12 * np.maximum(1.0, np.abs(cr[:, -1]))
                zero[prob.m:] = False
                cr = cr[~zero]
                memo[S] = lagrange, np.vstack([primal, cr / np.linalg.norm(cr[:, :-1], axis=1, keepdims=True)])
            lagrange, low = memo[S]
            lag[i, :len(S)], rest[i, :len(low)] = lagrange, low
        return dict(lagrange=lag, primal_and_region=rest, sizes=None, radius=None, err=None)
    if kind == "mpqp":
        m, p, k = case["m"], case["p"], case["k"]
        if math.comb(m + 2 * p, p + 1) * _sets_up_to(m, k) > 1_000_000:
            return None
        found = _exact_sets(_problems(case, seed)[0][0], k)
        t, r = (_fill(_room(case), np.array([f[i] for f in found])) for i in (1, 2))
        return dict(active_sets=None, t=t, r=r, region=None, err=None, counts=None)
    return None


def work(case):
    """Every problem read once and every answer written once; for each candidate set the least an
    enumeration does: one pivot of its feasibility tableau and one elimination of its KKT rows."""
    probs, ks, budgets = _problems(case, 0)
    in_bytes = sum(8 * sum(a.size for a in (p.Q, p.c, p.H, p.A, p.b, p.F, p.CRA, p.CRb)) for p in probs)
    pr = probs[0]
    if case["kind"] == "regions":
        rows = 2 * pr.m + pr.n + pr.ncp
        k = pr.p
        flops = case["sets"] * (k ** 3 / 3 + 2 * (pr.p + 1) * (k * k + (pr.n + pr.m) * k) + 3 * rows * (pr.p + 1))
        return dict(bytes=in_bytes + case["sets"] * (16 + 8 * (rows - pr.m) * (pr.p + 1) + 32), flops=flops)
    if case["kind"] == "reduce":
        rows = pr.m + pr.ncp
        return dict(bytes=in_bytes + 4 * rows, flops=rows * 2.0 * rows * (pr.n + pr.p + 1))
    flops, cands = 0.0, 0.0
    for p, k, b in zip(probs, ks, budgets):
        c = _sets_up_to(p.m, k)
        c = min(c, b) if b else c
        cands += c
        flops += c * (2.0 * (p.m + p.ncp) * (p.n + p.p + 1) / 2 + 2.0 * k * (p.p + 1) * (k + 1))
    return dict(bytes=in_bytes + 16 * cands, flops=flops)
