"""Work that users of this framework have it do, as measurable cases.

Each case goes through the public binding (``comer2_b200.native.Handle``) the
way a program does: a handle with the default parameters holds an uploaded
database, and a pass takes the query (or the training batch) from host memory
and returns the results to host memory.

Kinds of case
  search   one query against the database: ranking DP, statistics, MAP
           alignments, hits and alignment strings back (what the ``comer2``
           program and the benchmark do per query);
  batch    a set of queries through the multi-query call, two workers;
  rank     phase 1 alone with its per-profile scores back (a ranking pass, as a
           host that keeps its own later stages makes it);
  logz     the differentiable alignment: log-partition of a set of pairs and
           its nine gradients per pair (a training step), for a batch of
           independent pairs or one query against several profiles.

Value distributions are those of ``comer2_b200.synth``: positions, transitions
and queries come from its generator (database positions drawn from a pool of
generated ones, so that large databases are quick to make), with planted
homologs as its benchmark configurations have them.
"""
import math
import random

import numpy as np
import torch

from comer2_b200 import params as P
from comer2_b200 import synth as S
from comer2_b200.native import HIT_DTYPE, SCORE_BF16_TC, SCORE_FP32, Handle

NAA, NCV = S.NUMAA, S.NCV
MODES = {"fp32": SCORE_FP32, "bf16": SCORE_BF16_TC}
# weights of the SS and context-vector terms in the training cases
WSS, WCV = 0.12, 0.15
POOL = 32768


def listed():
    return [
        # the smallest call: a short domain against a family-sized set, the
        # default score form (launches and host steps count most here)
        dict(name="search_small_fp32", kind="search", mode="fp32", lq=97, domains=1, nprof=300, lens="u",
             lo=30, hi=257, median=0, hom=0.02, nq=1),
        # benchmark configuration 0: one query of 150 vs 2,000 profiles of 50..500
        dict(name="search_c0_bf16", kind="search", mode="bf16", lq=150, domains=1, nprof=2000, lens="u",
             lo=50, hi=500, median=0, hom=0.0, nq=1),
        # benchmark configuration 1 (one query of 400, lognormal lengths, 2 %
        # homologs) at half its database: the largest single search here
        dict(name="search_c1_bf16", kind="search", mode="bf16", lq=400, domains=1, nprof=50000, lens="ln",
             lo=30, hi=2000, median=200, hom=0.02, nq=1),
        # the same configuration in the default FP32 score form
        dict(name="search_c1_fp32", kind="search", mode="fp32", lq=400, domains=1, nprof=20000, lens="ln",
             lo=30, hi=2000, median=200, hom=0.02, nq=1),
        # an ordinary long query of an odd length against an odd-sized set
        dict(name="search_odd_bf16", kind="search", mode="bf16", lq=1237, domains=1, nprof=4999, lens="ln",
             lo=30, hi=2000, median=250, hom=0.01, nq=1),
        # benchmark configuration 4: a six-domain query of 3,000 with 5 %
        # homologs (many alignments: the MAP stage leads)
        dict(name="search_c4_bf16", kind="search", mode="bf16", lq=3000, domains=6, nprof=4000, lens="ln",
             lo=30, hi=2000, median=300, hom=0.05, nq=1),
        # benchmark configuration 2: a set of queries, both score forms
        dict(name="batch_c2_bf16", kind="batch", mode="bf16", lq=250, domains=1, nprof=5000, lens="ln",
             lo=30, hi=2000, median=200, hom=0.02, nq=16),
        dict(name="batch_fp32", kind="batch", mode="fp32", lq=250, domains=1, nprof=1000, lens="ln",
             lo=30, hi=2000, median=200, hom=0.02, nq=7),
        # a ranking pass over an ordinary database
        dict(name="rank_fp32", kind="rank", mode="fp32", lq=250, domains=1, nprof=3000, lens="ln",
             lo=30, hi=2000, median=200, hom=0.02, nq=1),
        # benchmark configuration 3: 256 independent pairs of 100..600 positions
        dict(name="logz_c3", kind="logz", pairs=256, lo=100, hi=600, one_query=False),
        # one query's training step against a family (the torch wrapper's call)
        dict(name="logz_family", kind="logz", pairs=45, lo=60, hi=300, one_query=True),
        # short pairs, the smallest training step
        dict(name="logz_small", kind="logz", pairs=12, lo=20, hi=70, one_query=False),
    ]


def _loguni(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mean_len(c):
    return (c["lo"] + c["hi"]) / 2 if c["lens"] == "u" else min(c["hi"], c["median"] * math.exp(0.18))


def _cost(c):
    """Relative time of a case: ranking cells (the FP32 form about twice as
    dear), and the cells of the homologs' later stages."""
    if c["kind"] == "logz":
        return c["pairs"] * ((c["lo"] + c["hi"]) / 2) ** 2 * 30.0
    cells = c["nq"] * c["lq"] * c["nprof"] * _mean_len(c)
    w = 1.0 if c["mode"] == "bf16" else 2.0
    later = 0.0 if c["kind"] == "rank" else 40.0 * c["hom"] / c["nq"]
    return cells * (w + later)


def draw(rng: random.Random):
    limit = 0.8 * max(_cost(c) for c in listed())
    u = rng.random()
    if u < 0.25:
        lo = _loguni(rng, 20, 200)
        hi = min(600, max(lo + 1, int(lo * rng.uniform(1.5, 6.0))))
        return dict(kind="logz", pairs=_loguni(rng, 12, 256), lo=lo, hi=hi, one_query=rng.random() < 0.3)
    kind = "search" if u < 0.75 else "batch" if u < 0.9 else "rank"
    c = dict(kind=kind, mode=rng.choice(["fp32", "bf16"]), lq=_loguni(rng, 60, 3000 if kind == "search" else 500),
             domains=1, nprof=_loguni(rng, 300, 50000 if kind == "search" else 5000), lo=30, hi=2000, lens="ln",
             median=rng.choice([200, 250, 300]), hom=rng.choice([0.0, 0.01, 0.02, 0.05]), nq=1)
    if kind == "rank":
        c["mode"] = "fp32"
    if kind == "batch":
        c["nq"] = rng.randint(2, 16)
    if rng.random() < 0.3:
        c["lens"], c["lo"], c["hi"], c["median"] = "u", rng.randint(20, 60), rng.randint(200, 600), 0
    if c["lq"] >= 600:
        c["domains"] = rng.randint(1, 6)
    while _cost(c) > limit:
        c["nprof"] = max(50, int(c["nprof"] * 0.7))
        if c["nprof"] == 50:
            break
    return c


# ---------------------------------------------------------------------------
# inputs
def _gen(seed, salt):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, salt])


def _lengths(rng, c):
    if c["lens"] == "u":
        return rng.integers(c["lo"], c["hi"] + 1, c["nprof"]).astype(np.int64)
    return S.lognormal_lengths(rng, c["nprof"], c["median"], 0.6, c["lo"], c["hi"]).astype(np.int64)


def _query(rng, lq, domains):
    """One query; with several domains, independent parts joined end to end."""
    return S.random_profiles(rng, [lq]) if domains <= 1 else _joined(rng, lq, domains)


def _joined(rng, lq, domains):
    cuts = [lq * d // domains for d in range(domains + 1)]
    doms = [S.random_profiles(rng, [b - a]) for a, b in zip(cuts[:-1], cuts[1:])]
    q = S.concat(doms)
    trn = np.concatenate([doms[0].trn[:1]] + [d.trn[1:] for d in doms])
    return S.ProfileSet(np.array([lq], np.int32), np.zeros(1, np.int64), q.bkg[:1], q.eno[:1], trn, q.trg, q.cv,
                        q.cvprior, q.cvnorm2, q.ss, q.ssstate, q.aa, np.zeros((0, 7), np.int32),
                        np.zeros((0, NAA), np.int32))


def _take(a, idx):
    return torch.from_numpy(a).index_select(0, idx).numpy()


def _database(rng, lens, query, frac):
    """Profiles of these lengths: positions and transitions drawn from a pool
    of generated ones, a fraction of the profiles holding a perturbed segment
    of the query (as synth.planted_homolog does)."""
    pool = S.random_profiles(rng, [512] * (POOL // 512))
    nprof = lens.shape[0]
    hom = np.zeros(0, np.int64)
    segs = []
    if query is not None and frac > 0:
        lq = int(query.lengths[0])
        hom = np.sort(rng.choice(nprof, max(1, int(round(frac * nprof))), replace=False))
        for k in hom:
            ls = int(rng.integers(min(60, lq), min(300, lq) + 1))
            lens[k] = max(int(lens[k]), ls)
            segs.append((ls, int(rng.integers(0, lq - ls + 1)), int(rng.integers(0, int(lens[k]) - ls + 1))))
    n = int(lens.sum())
    offs = np.zeros(nprof, np.int64)
    offs[1:] = np.cumsum(lens[:-1])
    ip = torch.from_numpy(rng.integers(0, pool.npositions, n))
    it = torch.from_numpy(rng.integers(0, pool.trn.shape[0], n + nprof))
    db = S.ProfileSet(lens.astype(np.int32), offs, np.repeat(pool.bkg[:1], nprof, axis=0),
                      np.round(rng.uniform(1.0, 14.0, nprof), 1).astype(np.float32), _take(pool.trn, it),
                      _take(pool.trg, ip), _take(pool.cv, ip), _take(pool.cvprior, ip), _take(pool.cvnorm2, ip),
                      _take(pool.ss, ip), _take(pool.ssstate, ip), _take(pool.aa, ip), np.zeros((0, 7), np.int32),
                      np.zeros((0, NAA), np.int32))
    letters = np.frombuffer(S.AA, np.uint8)
    for k, (ls, qs, o) in zip(hom, segs):
        a = int(offs[k]) + o
        g = rng.standard_gamma(50.0 * query.trg[qs:qs + ls].astype(np.float64)) + 1e-12
        t = np.maximum(np.rint(g / g.sum(1, keepdims=True) * 10000.0), 1.0)
        t[np.arange(ls), t.argmax(1)] += 10000.0 - t.sum(1)
        db.trg[a:a + ls] = (t / 10000.0).astype(np.float32)
        db.aa[a:a + ls] = letters[t.argmax(1)]
        for f in ("cv", "cvprior", "cvnorm2", "ss", "ssstate"):
            getattr(db, f)[a:a + ls] = getattr(query, f)[qs:qs + ls]
        db.trn[a + k + 1:a + k + ls + 1] = query.trn[qs + 1:qs + ls + 1]
    return db


def _inputs(case, seed):
    """(queries, db, pair table) of a case: host arrays made from the seed."""
    c = case
    if c["kind"] == "logz":
        rng = _gen(seed, 3)
        nq = 1 if c["one_query"] else c["pairs"]
        qs = S.random_profiles(rng, rng.integers(c["lo"], c["hi"] + 1, nq))
        db = S.random_profiles(rng, rng.integers(c["lo"], c["hi"] + 1, c["pairs"]))
        qof = np.zeros(c["pairs"], np.int32) if c["one_query"] else np.arange(c["pairs"], dtype=np.int32)
        return qs, db, qof
    rng = _gen(seed, 1)
    if c["nq"] > 1:
        lqs = S.lognormal_lengths(rng, c["nq"], c["lq"], 0.6, 50, 1500)
        lqs = np.maximum(33, (lqs * min(1.0, c["lq"] * c["nq"] * 1.2 / lqs.sum())).astype(np.int64))
        queries = [_query(rng, int(x), 1) for x in lqs]
        qs = S.concat(queries)
        first = queries[0]
    else:
        qs = first = _query(rng, c["lq"], c["domains"])
    return qs, _database(rng, _lengths(rng, c), first, c["hom"]), None


class State:
    """What the caller's program holds: the handle, its queries, the pairs, and
    the result buffers of a fixed capacity that every search's hits go into."""

    def __init__(self, case, handle, queries, qof, theta):
        self.case, self.h, self.q, self.qof, self.theta = case, handle, queries, qof, theta
        if case["kind"] == "logz":
            self.pairs = np.arange(len(qof), dtype=np.int32)
        elif case["kind"] != "rank":
            cap = 256 * case["nq"] + int(2 * case["hom"] * case["nprof"])
            self.out = {k: np.zeros(cap, HIT_DTYPE[k]) for k in HIT_DTYPE.names}
            self.out["alignments"] = np.zeros(cap * 5 * 360, np.uint8)
            self.out["hits"] = np.zeros(case["nq"], np.int32)
            self.used = (0, 0)

    def store(self, results):
        """The hits of each query in turn into the result buffers."""
        n = nb = 0
        for i, (rec, aln) in enumerate(results):
            for k in HIT_DTYPE.names:
                self.out[k][n:n + len(rec)] = rec[k]
            size = int(5 * (rec["alnlen"].astype(np.int64) + 1).sum())
            self.out["alignments"][nb:nb + size] = aln[:size]
            self.out["hits"][i] = len(rec)
            n, nb = n + len(rec), nb + size
        for k in HIT_DTYPE.names:
            self.out[k][n:max(n, self.used[0])] = 0
        self.out["alignments"][nb:max(nb, self.used[1])] = 0
        self.used = (n, nb)
        return self.out


def _theta(seed):
    return _gen(seed, 7).normal(0.0, 0.05, 7).astype(np.float32)


def prepare(case, seed):
    qs, db, qof = _inputs(case, seed)
    h = Handle(P.load_default(), 0)
    if case["kind"] != "logz":
        h.set_score_mode(MODES[case["mode"]])
    h.upload_db(db)
    return State(case, h, qs, qof, _theta(seed))


def run(st):
    kind = st.case["kind"]
    if kind == "search":
        return st.store([st.h.search(st.q, arrays=True)])
    if kind == "batch":
        return st.store(st.h.search_batch(st.q, nworkers=2))
    if kind == "rank":
        st.h.set_query(st.q)
        st.h.run_phase1()
        best, coords = st.h.phase1()
        return {"best": best, "coords": coords}
    if st.case["one_query"]:
        st.h.set_query(st.q)
        z = st.h.logz_fwd(st.pairs, st.theta, WSS, WCV)
    else:
        st.h.set_query_batch(st.q)
        z = st.h.logz_fwd_batch(st.qof, st.pairs, st.theta, WSS, WCV)
    return {"logz": z, "grad": st.h.logz_bwd()}


def work(case):
    """Input fields read once, results written once; the arithmetic of the
    ranking cells (two contractions of 20 and 19 terms, three SS terms, the two
    logarithms and the DP's additions and maxima), or of the forward and
    backward log-sum-exp recursions."""
    c = case
    if c["kind"] == "logz":
        m = (c["lo"] + c["hi"]) / 2
        n = c["pairs"]
        pos = n * m + (m if c["one_query"] else n * m)
        return {"bytes": pos * 209.0 + n * 40.0, "flops": n * m * m * 400.0}
    pos = c["nprof"] * _mean_len(c)
    cells = c["nq"] * c["lq"] * pos
    return {"bytes": pos * 209.0 + c["nq"] * c["lq"] * 209.0 + c["nprof"] * 8.0, "flops": cells * 135.0}


# ---------------------------------------------------------------------------
# 64-bit values of the computed numbers, plain torch
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _t64(a, dev):
    return torch.from_numpy(np.ascontiguousarray(a)).to(dev).to(torch.float64)


def _trn(ps, k, dev):
    """MM MI MD IM II DM DD of every position of profile k, [L, 7]."""
    o = int(ps.offsets[k]) + k
    n = int(ps.lengths[k])
    r = _t64(ps.trn[o:o + n + 1], dev)
    a, b = r[:-1], r[1:]
    return torch.stack([a[:, 0], b[:, 1], a[:, 2], a[:, 3], b[:, 4], a[:, 5], a[:, 6]], 1)


def _parts(prm, qs, kq, db, kd, dev):
    """The three score terms of a pair, each [Lq, L]: amino acids, SS, CV."""
    qa, qn = int(qs.offsets[kq]), int(qs.lengths[kq])
    da, dn = int(db.offsets[kd]), int(db.lengths[kd])
    q, d = slice(qa, qa + qn), slice(da, da + dn)
    w = 0.5 * (_t64(qs.bkg[kq], dev) + _t64(db.bkg[kd], dev))
    shift = 0.002 if prm.mapaln else 0.0003
    s0 = torch.log((_t64(qs.trg[q], dev) / w) @ _t64(db.trg[d], dev).T) - shift
    # SS: table of the probabilities' bins, plus the helix term
    card = prm.ssss_card
    tab = _t64(prm.ssss, dev).reshape(card, card)

    def bins(ss):
        return [torch.from_numpy((10 * s + (ss[:, s] * np.float32(9.999)).astype(np.int32)).astype(np.int64)).to(dev)
                for s in range(3)]

    qss, dss = _t64(qs.ss[q], dev), _t64(db.ss[d], dev)
    qi, di = bins(qs.ss[q]), bins(db.ss[d])
    u = sum(qss[:, s:s + 1] * tab[qi[s]] for s in range(3))
    ss = sum(u[:, di[s]] * dss[:, s][None, :] for s in range(3))
    ss = ss + (qss[:, 2:3] + 0.1) * (dss[:, 2][None, :] + 0.1) * 0.1111111 - 0.05
    # CV: normal-inverse-Wishart log-odds, mapped through the score table
    kappa0, nu0 = 0.1, float(NCV)
    pw = -0.5 * (nu0 + 2.0)
    ct = (0.5 * NCV + pw) * (math.log(kappa0) - math.log(kappa0 + 2.0))
    ct += sum(math.log(nu0 + 1.0 - i) - math.log(2.0) for i in range(1, NCV + 1))
    dot = _t64(qs.cv[q], dev) @ _t64(db.cv[d], dev).T + 1.0 / kappa0
    cn = lambda ps, sl: _t64(ps.cvnorm2[sl], dev) + 1.0 + 1.0 / kappa0
    det = cn(qs, q)[:, None] * cn(db, d)[None, :] - dot * dot
    x = ct + pw * torch.log(det) - _t64(qs.cvprior[q], dev)[:, None] - _t64(db.cvprior[d], dev)[None, :]
    keys, vals = _t64(prm.cvs2s_keys, dev), _t64(prm.cvs2s_values, dev)
    ix = (prm.cvs2s_shift + torch.round(2.0 * x)).clamp(0, prm.cvs2s_card - 1).long()
    cv = torch.where(x <= keys[0], vals[0], torch.where(x >= keys[-1], vals[-1], vals[ix]))
    return s0, ss, cv


def _skew(a, steps):
    """[B, Lq, L] -> [steps, B, Lq]: element (i, j) at step i + j (0 elsewhere)."""
    b, lq, n = a.shape
    k = torch.arange(steps, device=a.device)[:, None]
    j = k - torch.arange(lq, device=a.device)[None, :]
    ok = (j >= 0) & (j < n)
    i = torch.arange(lq, device=a.device)[None, :].expand_as(j)
    g = a[:, i, j.clamp(0, n - 1)]
    return torch.where(ok, g, torch.zeros((), dtype=a.dtype, device=a.device)).permute(1, 0, 2)


def _skew_cols(t, lq, steps):
    """[B, L, 7] -> [steps, 7, B, Lq]: column values of the cell at step i + j."""
    n = t.shape[1]
    k = torch.arange(steps, device=t.device)[:, None]
    j = (k - torch.arange(lq, device=t.device)[None, :]).clamp(0, n - 1)
    return t[:, j, :].permute(1, 3, 0, 2)


def _shift(x, first):
    """Row i takes row i - 1's value; row 0 takes `first`."""
    return torch.cat([torch.full_like(x[:, :1], first), x[:, :-1]], 1)


def _recur(q7, t7s, s_s, left0, diag0, zero, soft):
    """The five-state recursion over anti-diagonals.  q7: 7 x [B, Lq]; t7s
    [steps, 7, B, Lq]; s_s [steps, B, Lq]; left0 / diag0: states of the column
    before the first one; zero: states of the row before the first one.  Yields
    MM per step.  soft: log-sum-exp with the local start, else maxima with 0."""
    steps, b, lq = s_s.shape
    if soft:
        two = torch.logaddexp

        def five(v, s):
            return torch.logsumexp(torch.stack([x + s for x in v] + [torch.zeros_like(s)]), 0)
    else:
        two = torch.maximum

        def five(v, s):
            m = v[0]
            for x in v[1:]:
                m = torch.maximum(m, x)
            return (m + s).clamp_min(0.0)
    qMM, qMI, qMD, qIM, qII, qDM, qDD = q7
    rows = torch.arange(lq, device=s_s.device)[None, :]
    cur = [torch.full((b, lq), z, dtype=torch.float64, device=s_s.device) for z in zero]
    up_prev = [_shift(x, z) for x, z in zip(cur, zero)]
    for k in range(steps):
        tMM, tMI, tMD, tIM, tII, tDM, tDD = t7s[k]
        up = [_shift(x, z) for x, z in zip(cur, zero)]
        left, diag = cur, up_prev
        if k < lq:
            at0 = rows == k
            left = [torch.where(at0, l0, x) for l0, x in zip(left0, left)]
            diag = [torch.where(at0, d0, x) for d0, x in zip(diag0, diag)]
        s = s_s[k]
        mm = five([diag[1] + qMM + tIM, diag[2] + qIM + tMM, diag[3] + qDM + tMM, diag[4] + qMM + tDM,
                   diag[0] + qMM + tMM], s)
        mi = two(up[0] + qMM + tMI, up[1] + qMM + tII)
        im = two(left[0] + qMI + tMM, left[2] + qII + tMM)
        dn = two(up[0] + qMD, up[3] + qDD)
        nd = two(left[0] + tMD, left[4] + tDD)
        up_prev = up
        cur = [mm, mi, im, dn, nd]
        yield mm


def _edge_states(tq, soft):
    """States of the column before the first (MM MI IM DN ND per row, and of
    the row before), with the 32-row block structure of the method."""
    z0 = -99.0 if soft else S.LOG0
    n = tq.shape[0]
    two = (lambda a, b: max(a, b) + math.log1p(math.exp(-abs(a - b)))) if soft else max
    t = tq.tolist()
    zero = [0.0, z0, z0, z0, z0] if soft else [0.0] * 5
    rows, pm, pd = [], 0.0, 0.0
    for r in range(n):
        mm, mi, md, im, ii, _, dd = t[r]
        um, ud = (zero[1], zero[3]) if r % 32 == 0 else (pm, pd)
        c1 = two(mm + z0, um + mm + z0)
        if r % 32 == 0:
            c2 = two(mi + z0, zero[2] + ii + z0)
        else:
            c2 = two(mi + z0, mi + z0 + ii + z0) if soft else mi + z0
        c3 = two(md, ud + dd)
        rows.append([0.0, c1, c2, c3, z0])
        pm, pd = c1, c3
    left = [zero if r % 32 == 31 else rows[r] for r in range(n)]
    diag = [zero if r % 32 in (0, 31) else rows[r - 1] for r in range(n)]
    return left, diag, zero


def _exact_rank(case, seed):
    dev = _dev()
    qs, db, _ = _inputs(case, seed)
    prm = P.load_default()
    lq = int(qs.lengths[0])
    tq = _trn(qs, 0, dev)
    left, diag, zero = _edge_states(tq, False)
    best = np.zeros(db.nprofiles, np.float64)
    order = np.argsort(-db.lengths, kind="stable")
    y = torch.arange(lq, device=dev)[:, None]
    for g in range(0, len(order), 250):
        ks = order[g:g + 250]
        n = int(db.lengths[ks].max())
        b = len(ks)
        sc = torch.full((b, lq, n), -1e4, dtype=torch.float64, device=dev)
        t7 = torch.full((b, n, 7), S.LOG0, dtype=torch.float64, device=dev)
        for i, k in enumerate(ks):
            ld = int(db.lengths[k])
            s0, ss, cv = _parts(prm, qs, 0, db, int(k), dev)
            x = torch.arange(ld, device=dev)[None, :]
            e = min(60, int(np.rint(np.float32(0.34) * np.float32(max(lq, ld)))))
            cut = ((lq <= y + e) & (x <= e + y - lq)) | ((ld - e + y <= x) & (y < e))
            sc[i, :, :ld] = torch.where(cut, -9.0, s0 + prm.ssswgt * ss + prm.cvswgt * cv)
            t7[i, :ld] = _trn(db, int(k), dev)
        steps = lq + n - 1
        sk, tk = _skew(sc, steps), _skew_cols(t7, lq, steps)
        q7 = [tq[:, i][None, :].expand(b, lq) for i in range(7)]
        l0 = [torch.tensor(v, dtype=torch.float64, device=dev)[None, :] for v in zip(*left)]
        d0 = [torch.tensor(v, dtype=torch.float64, device=dev)[None, :] for v in zip(*diag)]
        # (a padding column scores far below any path: its MM stays 0)
        acc = torch.zeros(b, dtype=torch.float64, device=dev)
        rows = torch.arange(lq, device=dev)
        for k, mm in enumerate(_recur(q7, tk, sk, l0, d0, zero, False)):
            ok = (rows <= k) & (k - rows < n)
            acc = torch.maximum(acc, torch.where(ok[None, :], mm, 0.0).amax(1))
        best[ks] = acc.cpu().numpy()
    return {"best": best, "coords": None}


def _exact_logz(case, seed):
    dev = _dev()
    qs, db, qof = _inputs(case, seed)
    prm = P.load_default()
    npair = len(qof)
    theta = torch.from_numpy(_theta(seed).astype(np.float64)).to(dev)
    z = np.zeros(npair, np.float64)
    grad = np.zeros((npair, 9), np.float64)
    lq_of = qs.lengths[qof].astype(np.int64)
    order = np.argsort(-(lq_of + db.lengths), kind="stable")
    for g in range(0, npair, 64):
        ks = order[g:g + 64]
        b, lq, n = len(ks), int(lq_of[ks].max()), int(db.lengths[ks].max())
        f64 = dict(dtype=torch.float64, device=dev)
        p0, p1, p2 = (torch.zeros(b, lq, n, **f64) for _ in range(3))
        t7, q7 = torch.zeros(b, n, 7, **f64), torch.zeros(b, lq, 7, **f64)
        l0, d0 = torch.zeros(5, b, lq, **f64), torch.zeros(5, b, lq, **f64)
        live = torch.zeros(b, lq, n, dtype=torch.bool, device=dev)
        for i, k in enumerate(ks):
            kq, a, m = int(qof[k]), int(lq_of[k]), int(db.lengths[k])
            p0[i, :a, :m], p1[i, :a, :m], p2[i, :a, :m] = _parts(prm, qs, kq, db, int(k), dev)
            t7[i, :m] = _trn(db, int(k), dev)
            q7[i, :a] = tq = _trn(qs, kq, dev)
            left, diag, zero = _edge_states(tq, True)
            l0[:, i, :a] = torch.tensor(left, **f64).T
            d0[:, i, :a] = torch.tensor(diag, **f64).T
            live[i, :a, :m] = True
        steps = lq + n - 1
        th = theta[None, :].repeat(b, 1).requires_grad_(True)
        w = torch.tensor([WSS, WCV], **f64)[None, :].repeat(b, 1).requires_grad_(True)
        s = p0 + w[:, 0, None, None] * p1 + w[:, 1, None, None] * p2
        sk, tk = _skew(s, steps), _skew_cols(t7, lq, steps)
        lk = _skew(live.double(), steps) > 0.5
        qth = [q7[:, :, i] + th[:, i, None] for i in range(7)]
        mms = torch.stack([torch.where(lk[k], mm, -1e30)
                           for k, mm in enumerate(_recur(qth, tk, sk, list(l0), list(d0), zero, True))])
        lz = torch.logsumexp(mms.permute(1, 0, 2).reshape(b, -1), 1)
        gt, gw = torch.autograd.grad(lz.sum(), [th, w])
        z[ks] = lz.detach().cpu().numpy()
        grad[ks] = torch.cat([gt, gw], 1).cpu().numpy()
    return {"logz": z, "grad": grad}


def exact(case, seed):
    """64-bit values of the ranking scores and of the log-partition and its
    gradients.  A search's statistics and alignments have none: they are
    defined on 32-bit integer bins of the scores and on an integer-coded
    exponential."""
    if case["kind"] == "rank" and case["lq"] * case["nprof"] <= 2_000_000:
        return _exact_rank(case, seed)
    if case["kind"] == "logz":
        return _exact_logz(case, seed)
    return None
