"""Performance cases of the search path.

Each case is one call that a program makes of this package: a search of one
query profile (or a batch of them) against a resident database chunk with
its results read back, the score matrices of a search read back whole, or
the phase-1 DP on device buffers the caller owns. The profiles are the
seeded synthetic ones of the benchmark configurations (cother_b200/synth.py):
lognormal database lengths (median 180 or 220, sigma 0.5), or uniform
500-1,500 for the long-query configuration, predicted distance lists on the
query's side and observed ones on the database's, 1 % planted homologs.

The sizes run from a query of 40 positions against 16 profiles, where the
launches and copies of a call count, to a query of 400 against 2,000
profiles (half a million positions, 200 million cells) and one of 1,500
against 60 profiles of up to 1,500.
"""
import ctypes
import math
import os

import numpy as np
import torch

import cother_b200 as cb
from cother_b200 import synth

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden")
LARGEST_CELLS = 200e6      # query positions x database positions of the largest case
FORMS = {"plain": cb.TC_PLAIN, "bf16": cb.TC_BF16X3, "tf32": cb.TC_TF32X3}

# a search with the options of the parity configuration
SEARCH = {"kind": "search", "qlen": 200, "ndb": 1000, "law": "lognormal", "mid": 220, "lo": 30, "hi": 1500,
          "window": 64, "form": "plain", "cvswgt": 0.0, "ddmswgt": 0.2, "dstsegm": 6, "mapaln": 1, "nq": 1}


def _search(name, **kw):
    return dict(SEARCH, name=name, **kw)


def listed():
    return [
        # the smallest call: a short query against a handful of profiles
        # (a hand-picked set, a test of a new profile): all latency
        _search("q40_db16", qlen=40, ndb=16),
        # benchmark configuration: 1 query of 200 against 1,000 profiles
        _search("q200_db1k", mid=180, hi=600),
        # the sweep's short query against a longer chunk
        _search("q64_db3k", qlen=64, ndb=3000),
        # the headline configuration's query and length law, on a chunk
        _search("q400_db2k", qlen=400, ndb=2000),
        # long-query stress: 1,500 positions, window 128, long profiles
        _search("q1500_db60", qlen=1500, ndb=60, law="uniform", lo=500, window=128),
        # the reference's default CVSWGT 0.15, at a ragged size
        _search("q333_db701_cvs", qlen=333, ndb=701, cvswgt=0.15),
        # the precision forms of the profile-profile term (the sweep's
        # middle and long query)
        _search("q256_db1k_bf16", qlen=256, ndb=1000, form="bf16"),
        _search("q1024_db250_tf32", qlen=1024, ndb=250, form="tf32"),
        # a search without the distance term (databases without structures):
        # the phase-1 DP and the HBM traffic of the matrices count
        _search("q400_db2k_noddms", qlen=400, ndb=2000, ddmswgt=0.0),
        # continuous batching: what a server slot searches in one pass
        _search("batch4_db500", kind="batch", nq=4, qlen=250, ndb=500),
        # the score matrices themselves, with phase-1 alignments instead of
        # the MAP realignment and short distance segments (analysis of one
        # family; an odd query length)
        _search("matrix_q97_db40", kind="matrix", qlen=97, ndb=40, mapaln=0, dstsegm=4),
        # the phase-1 DP alone, on a caller's device buffers of the largest
        # width that entry point takes
        {"name": "dp1_q256_64k", "kind": "dp1", "qlen": 256, "columns": 65536, "mid": 220},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search"] * 6 + ["batch", "matrix", "dp1"])
    if kind == "dp1":
        return {"kind": "dp1", "qlen": _logint(rng, 40, 512), "columns": _logint(rng, 1000, 65536),
                "mid": rng.choice([180, 220])}
    c = dict(SEARCH, kind=kind)
    c["qlen"] = _logint(rng, 40, 120 if kind == "matrix" else 600 if kind == "batch" else 1500)
    mean = 250
    if kind == "search" and rng.random() < 0.2:
        c.update(law="uniform", lo=500, hi=1500, window=128)
        mean = 1000
    elif rng.random() < 0.3:
        c.update(mid=180, hi=600)
        mean = 200
    if kind == "batch":
        c["nq"] = rng.randint(2, 4)
    most = LARGEST_CELLS / 1.5 / (c["qlen"] * c["nq"] * mean)
    c["ndb"] = max(4, _logint(rng, 8, min(3000, 48 if kind == "matrix" else max(9, most))))
    c["form"] = rng.choice(["plain", "plain", "plain", "bf16", "tf32"])
    c["cvswgt"] = rng.choice([0.0, 0.0, 0.0, 0.15])
    c["ddmswgt"] = rng.choice([0.2, 0.2, 0.2, 0.1, 0.0])
    c["dstsegm"] = rng.choice([6, 6, 6, 3, 5, 8])
    c["mapaln"] = rng.choice([1, 1, 1, 0])
    return c


def _lengths(case, n, seed):
    if case.get("law") == "uniform":
        return synth.uniform_lengths(n, case["lo"], case["hi"], seed)
    return synth.lognormal_lengths(n, case["mid"], case.get("lo", 30), case.get("hi", 1500), seed)


def _query_lengths(case, seed=0):
    if case["nq"] == 1:
        return [case["qlen"]]
    # requests of one batch: lengths about the case's, in the served range
    f = [1.0, 0.41, 1.73, 0.77][:case["nq"]]
    return [min(1200, max(40, int(case["qlen"] * x))) for x in f]


def _profiles(case, seed):
    # a case's database has the same lengths for every seed, so that its
    # outputs have the same shapes
    db = synth.make_profiles(_lengths(case, case["ndb"], 1), seed=seed * 1000 + 1, predicted=False,
                             window=case["window"])
    qs = [synth.make_profiles([L], seed=seed * 1000 + 2 + k, predicted=True, window=case["window"])
          for k, L in enumerate(_query_lengths(case))]
    if case["cvswgt"] > 0:
        synth.add_context_vectors(db, seed * 1000 + 1)
        for k, q in enumerate(qs):
            synth.add_context_vectors(q, seed * 1000 + 2 + k)
    for k, q in enumerate(qs):
        # 1 % homologs of each query, two at least so that every search has
        # pairs to realign
        synth.plant_homologs(q, db, max(0.01, 2.0 / case["ndb"]), seed=seed * 1000 + 50 + k)
    return qs, db


def _dp1_lengths(case):
    """Whole profiles that fill the columns; the last one is cut to fit."""
    lens, left = [], case["columns"]
    for x in synth.lognormal_lengths(4096, case["mid"], 30, 1500, 1):
        lens.append(min(int(x), left))
        left -= lens[-1]
        if left == 0:
            break
    return np.asarray(lens, np.int32)


def _dp1_scores(case, seed, device):
    """Cell scores as searches give them: about -0.9 on average with a
    spread of 0.7, and some diagonal runs of similarity."""
    Lq, n = case["qlen"], case["columns"]
    g = torch.Generator(device=device).manual_seed(seed)
    s = torch.randn((Lq, n), generator=g, device=device) * 0.7 - 0.9
    rows = torch.arange(Lq, device=device)
    cols = torch.randint(0, n, (max(1, n // 2000),), generator=g, device=device)
    c = cols[:, None] + rows[None, :]
    ok = c < n
    s[rows[None, :].expand_as(c)[ok], c[ok]] += 1.5
    return s


def prepare(case, seed):
    if case["kind"] == "dp1":
        dev = torch.device("cuda:0")
        lens = _dp1_lengths(case)
        q = synth.make_profiles([case["qlen"]], seed=seed * 1000 + 2, predicted=True)
        db = synth.make_profiles(lens, seed=seed * 1000 + 1, predicted=False)
        Lq, n, P = case["qlen"], case["columns"], db.nprofiles
        put = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev)  # noqa: E731
        return {"kind": "dp1", "lib": cb.load_library(), "qlen": Lq, "n": n, "P": P,
                "scores": _dp1_scores(case, seed, dev), "qtrn": put(q.trn), "dtrn": put(db.trn),
                "lens": put(db.lens), "starts": put(db.starts),
                "btck": torch.zeros((Lq, n), dtype=torch.uint8, device=dev),
                "max": torch.zeros(P, dtype=torch.float32, device=dev),
                "xy": torch.zeros(P, dtype=torch.int32, device=dev)}
    o = cb.Options.defaults()
    o.tc_form = FORMS[case["form"]]
    o.cvswgt, o.ddmswgt, o.dstsegm, o.mapaln = case["cvswgt"], case["ddmswgt"], case["dstsegm"], case["mapaln"]
    qs, db = _profiles(case, seed)
    bp = cb.BatchProcessing(np.load(os.path.join(GOLDEN, "ssss.npy")), o)
    if case["cvswgt"] > 0:
        cvs = np.load(os.path.join(GOLDEN, "cvs2s.npz"))
        bp.set_cvs2s_map(cvs["keys"], cvs["scores"])
    bp.transfer_cpm_data(db)
    if case["ndb"] >= 250:
        # a chunk of a database of 50,000 profiles, for its E-values; a
        # smaller set of profiles is searched for itself
        bp.set_db_details(db.npositions * 50000 // db.nprofiles, 50000)
    return {"kind": case["kind"], "bp": bp, "queries": qs, "db": db}


MOST_ALIGNMENTS = 64


def _results(bp, q, db):
    """The results of a search as a program keeps them: the fields of each
    profile's hit record (0 for the profiles without one), each profile's
    place among the reported hits, from 1 (0: not reported), and the
    alignments of the hits in reported order, 64 at most."""
    t = cb.records_table(bp.hit_records())
    who = t["org_pro_no"].astype(np.int64)
    out = {}
    for k, v in t.items():
        if k in ("org_pro_no", "pro_new_dst"):
            continue
        if k == "log_evalue_pair":
            v = v.view(np.int32)     # after realignment, the alignment's length
        out[k] = np.zeros(db.nprofiles, np.int64 if v.dtype.kind in "ui" else np.float32)
        out[k][who] = v
    order, alns = bp.hit_list(), bp.alignments(q.npositions)
    out["place"] = np.zeros(db.nprofiles, np.int64)
    out["place"][who[order]] = np.arange(1, len(order) + 1)
    out["alignments"] = np.zeros((min(db.nprofiles, MOST_ALIGNMENTS), 5, q.npositions + int(db.lens.max())), np.uint8)
    for i, k in enumerate(order[:MOST_ALIGNMENTS]):
        for r in range(5):
            a = np.frombuffer(alns[k][r].encode(), np.uint8)
            out["alignments"][i, r, :len(a)] = a
    return out


def run(state):
    if state["kind"] == "dp1":
        s = state
        rc = s["lib"].cbp_dp1_noalloc(
            s["scores"].data_ptr(), s["n"], s["qlen"], s["qtrn"].data_ptr(), s["n"], s["P"], s["dtrn"].data_ptr(),
            s["lens"].data_ptr(), s["starts"].data_ptr(), 0, s["P"], 0, s["btck"].data_ptr(), s["max"].data_ptr(),
            s["xy"].data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError(s["lib"].cbp_last_error().decode())
        return {"btck": s["btck"], "max": s["max"], "xy": s["xy"]}
    bp, qs = state["bp"], state["queries"]
    if state["kind"] == "batch":
        bp.process_batch(qs)
        out = []
        for k in range(len(qs)):
            bp.select_query(k)
            r = _results(bp, qs[k], state["db"])
            out.append({x: r[x] for x in ("score", "log_evalue", "beg_coords", "end_coords", "identities", "gaps",
                                          "log_evalue_pair", "place", "alignments")})
        return out
    bp.process_score_matrix(qs[0])
    if state["kind"] == "matrix":
        s, m, _ = bp.read_score_matrix(qs[0].npositions, state["db"].npositions)
        return {"scores": s, "modscores": m, "hits": _results(bp, qs[0], state["db"])}
    return _results(bp, qs[0], state["db"])


def _ddms_steps(L1, L2, dstsegm):
    """Steps of four list elements that the distance term of one cell runs
    for lists of L1 and L2 distances."""
    if L1 < dstsegm or L2 < dstsegm:
        return 0
    n = sum((max(0, min(L1, L2 - j)) + 3) // 4 for j in range(L2 >> 2, -1, -2))
    return n + sum((max(0, min(L2, L1 - i)) + 3) // 4 for i in range(L1 >> 2, 0, -2))


def work(case):
    """Bytes: the profiles' fields and, where a call returns them, the
    matrices. Operations of a cell: 20 quotients summed (60), the secondary
    structure term (30), 37 of the DP, and of the distance term, for each
    step of four elements, two interpolated scores (4), four running sums
    clamped at zero (8), four segment lengths (4) and the best of the step
    (4)."""
    if case["kind"] == "dp1":
        cells = case["qlen"] * case["columns"]
        return {"bytes": 5.0 * cells + 28 * case["columns"], "flops": 37.0 * cells}
    lens = _lengths(case, case["ndb"], 1).astype(np.float64)
    n = float(lens.sum())
    ql = _query_lengths(case)
    cells = n * sum(ql)
    ops = 97.0 + (60.0 if case["cvswgt"] > 0 else 0.0)
    if case["ddmswgt"] > 0:
        # a position's list holds its nearest residues, 99 at most
        size = lambda L: int(min(99, L - 2))  # noqa: E731
        top = {L: max(1, n_) for L, n_ in zip(*np.unique(np.minimum(lens, 101), return_counts=True))}
        steps = {L: _ddms_steps(size(min(ql[0], 101)), size(L), case["dstsegm"]) for L in top}
        share = {L: lens[np.minimum(lens, 101) == L].sum() / n for L in top}
        ops += 20.0 * sum(share[L] * steps[L] for L in top)
    out = 8.0 * cells if case["kind"] == "matrix" else 0.0
    return {"bytes": 255.0 * (n + sum(ql)) + out, "flops": ops * cells}


def _device():
    return torch.device("cuda:0" if torch.cuda.is_available() else "cpu")


def _dist64(q, db, dstsegm, dev):
    """The distance-distribution match sums of all cells, in 64 bits, as
    multiples of 0.00125 (every pair score and every mean of two is one):
    for each diagonal of the two lists, segments of positive running sums,
    the best of each step of four offered to a register of the three best
    that do not intersect. None for cells whose lists are too short."""
    def lists(p):
        v = torch.from_numpy(p.dd[1:].T.astype(np.int64)).to(dev)
        n = torch.from_numpy(p.dd[0].astype(np.int64)).to(dev)
        v = torch.where(v == 255, 21, v.clamp(max=20))
        v = torch.where(torch.arange(99, device=dev)[None] < n[:, None], v, 21)
        return torch.cat([v, torch.full((len(v), 40), 21, device=dev)], 1), n
    ql, qn = lists(q)
    dl, dn = lists(db)
    a = torch.arange(22, device=dev, dtype=torch.float64)
    hi, lo = torch.maximum(a[:, None], a[None]), torch.minimum(a[:, None], a[None])
    T = 280 - 30 * hi + 16 * lo
    T[21] = -800
    T[:, 21] = -800
    sums = torch.zeros((len(ql), len(dl)), dtype=torch.float64, device=dev)
    D = len(dl)
    for r in range(len(ql)):
        L1 = int(qn[r])
        ms = torch.zeros((3, D), dtype=torch.float64, device=dev)
        mb = torch.zeros((3, 2, D), dtype=torch.int64, device=dev)
        me = torch.zeros((3, 2, D), dtype=torch.int64, device=dev)

        def cross(b, e, k):
            return ((torch.minimum(e, me[k]) >= torch.maximum(b, mb[k])).any(0)) & (ms[k] > 0)

        def offer(s, b, e):
            x0, x1 = cross(b, e, 0), cross(b, e, 1)
            pos = s > 0
            first = pos & (ms[0] <= s)
            second = pos & ~first & (ms[1] <= s) & ~x0
            third = pos & ~first & (ms[1] > s) & (ms[2] <= s) & ~x0 & ~x1
            a1 = torch.where(x0, 0.0, ms[0])
            a2 = torch.where(x1, 0.0, ms[1])
            up = a1 == 0
            n1, n2 = torch.where(up, a2, a1), torch.where(up, 0.0, a2)
            o0, o1 = ms[0].clone(), ms[1].clone()
            ob, oe = mb.clone(), me.clone()
            ms[0] = torch.where(first, s, o0)
            ms[1] = torch.where(first, n1, torch.where(second, s, o1))
            ms[2] = torch.where(first, n2, torch.where(second, a2, torch.where(third, s, ms[2])))
            for new, old, m in ((b, ob, mb), (e, oe, me)):
                m[0] = torch.where(first, new, old[0])
                m[1] = torch.where(first & ~up, old[0], torch.where(second, new, old[1]))
                m[2] = torch.where(first | second, old[1], torch.where(third, new, old[2]))

        def diagonal(oq, od, lim, on):
            # offsets into the two lists (od per column), steps while x < lim
            at = lambda e: T[ql[r, oq + e], dl.gather(1, (od + e)[:, None])[:, 0]]  # noqa: E731
            s0 = at(0)
            t = s0.clamp(min=0.0)
            beg = torch.zeros(D, dtype=torch.int64, device=dev)
            for x in range(0, int(lim.max()) if D else 0, 4):
                go = on & (x < lim)
                s2, s4 = at(x + 2), at(x + 4)
                best = torch.zeros_like(t)
                bb = torch.zeros_like(beg)
                bk = torch.zeros_like(beg)
                for k, v in enumerate(((s0 + s2) / 2, s2, (s2 + s4) / 2, s4), 1):
                    beg = torch.where(t == 0, x + k, beg)
                    t = (t + v).clamp(min=0.0)
                    better = (best < t) & (x + k - beg + 1 >= dstsegm)
                    best, bb, bk = (torch.where(better, n, o) for n, o in
                                    ((t, best), (beg, bb), (torch.full_like(bk, x + k), bk)))
                offer(torch.where(go, best, 0.0), torch.stack([oq + bb, od + bb]), torch.stack([oq + bk, od + bk]))
                s0 = s4

        on = (dn >= dstsegm) & (L1 >= dstsegm)
        for step in range(0, 14):
            j = (dn >> 2) - 2 * step
            live = on & (j >= 0)
            if bool(live.any()):
                j = j.clamp(min=0)
                diagonal(0, j, torch.where(live, torch.minimum(torch.full_like(dn, L1), dn - j), 0), live)
        for i in range(L1 >> 2, 0, -2):
            diagonal(i, torch.zeros_like(dn), torch.where(on, torch.minimum(dn, torch.full_like(dn, L1 - i)), 0), on)
        sums[r] = torch.where(on, ms.sum(0), math.nan)
    return sums * 0.00125


def _matrix64(case, seed):
    """Scores and modular scores of all cells in 64 bits (no context
    vectors)."""
    dev = _device()
    (q,), db = _profiles(case, seed)
    f64 = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev).double()  # noqa: E731
    pro = torch.from_numpy(np.repeat(np.arange(db.nprofiles), db.lens)).to(dev)
    den = 0.5 * (f64(q.bkg) + f64(db.bkg)[:, pro])
    s = torch.log(f64(q.tf).T @ (f64(db.tf) / den)) - (0.002 if case["mapaln"] else 0.0003)
    T = f64(np.load(os.path.join(GOLDEN, "ssss.npy")))
    qs, ds = f64(q.ss), f64(db.ss)
    # the table's row and column of a probability, in its own precision
    bins = lambda x: torch.from_numpy((x.astype(np.float32) * np.float32(9.999)).astype(np.int64)).to(dev)  # noqa: E731
    qi, di = bins(q.ss), bins(db.ss)
    ss = torch.zeros_like(s)
    for i in range(3):
        for j in range(3):
            ss += qs[i][:, None] * ds[j][None] * T[(10 * i + qi[i])[:, None], (10 * j + di[j])[None]]
    ss = torch.where(ss > -99, (ss + (qs[2] + 0.1)[:, None] * (ds[2] + 0.1)[None] * 0.1111111 - 0.05) * 0.12, ss)
    s, m = s + ss, ss.clone()
    w = case["ddmswgt"]
    if w > 0:
        d = (0.053 * 16 * _dist64(q, db, case["dstsegm"], dev) - 1.235) * w
        on = ~torch.isnan(d)
        s = torch.where(on, s + d, s)
        m = torch.where(on, m + d - 0.2 * w, m)
    return {"scores": s, "modscores": m, "hits": None}


def _dp64(case, seed):
    """The maxima of the phase-1 DP in 64 bits: a max-plus recurrence over
    the states MM, MI, IM, DN, ND, swept along anti-diagonals with all
    profiles at once. State 0 outside the matrix; the two corners score -9;
    column -1 as bands of 32 query rows leave it."""
    dev = _device()
    lens = _dp1_lengths(case)
    q = synth.make_profiles([case["qlen"]], seed=seed * 1000 + 2, predicted=True)
    db = synth.make_profiles(lens, seed=seed * 1000 + 1, predicted=False)
    S = _dp1_scores(case, seed, dev).double()
    f64 = lambda x: torch.from_numpy(np.ascontiguousarray(x)).to(dev).double()  # noqa: E731
    Lq, P = case["qlen"], db.nprofiles
    qt, dt = f64(q.trn), f64(db.trn)
    L = torch.from_numpy(db.lens.astype(np.int64)).to(dev)[:, None]
    start = torch.from_numpy(db.starts).to(dev)[:, None]
    t0 = start + torch.arange(P, device=dev)[:, None]
    r = torch.arange(Lq, device=dev)[None]
    MM, MI, MD, IM, II, DM, DD = range(7)
    qMM, qIM, qDM, qMD, qDD = (qt[k, :Lq][None] for k in (MM, IM, DM, MD, DD))
    qMIc, qIIc = qt[MI, 1:Lq + 1][None], qt[II, 1:Lq + 1][None]
    left0 = torch.zeros((5, Lq), dtype=torch.float64, device=dev)
    dn = 0.0
    for k in range(Lq):
        if k % 32 != 31:
            dn = max(float(qt[MD, k]), (0.0 if k % 32 == 0 else dn) + float(qt[DD, k]))
            left0[1, k] = left0[2, k] = left0[4, k] = -32768.0
            left0[3, k] = dn
    diag0 = torch.roll(left0, 1, 1)
    diag0[:, 0] = 0.0
    diag0[:, 31::32] = 0.0
    edge = torch.round(0.34 * torch.maximum(L, torch.full_like(L, Lq)).float()).long().clamp(max=60)
    p1 = torch.zeros((5, P, Lq), dtype=torch.float64, device=dev)
    p2 = torch.zeros_like(p1)

    def above(p):
        o = torch.zeros_like(p)
        o[:, :, 1:] = p[:, :, :-1]
        return o

    most = torch.zeros(P, dtype=torch.float64, device=dev)
    for s in range(Lq + int(L.max()) - 1):
        c = s - r
        on = (c >= 0) & (c < L)
        cc = torch.where(on, c, torch.zeros_like(c))
        dMM, dIM, dDM, dMD, dDD = (dt[k][t0 + cc] for k in (MM, IM, DM, MD, DD))
        dMIc, dIIc = dt[MI][t0 + cc + 1], dt[II][t0 + cc + 1]
        first = (c == 0).expand(P, Lq)
        le = torch.where(first, left0[:, None], p1)
        up = above(p1)
        dg = torch.where(first, diag0[:, None], above(p2))
        corner = ((Lq <= r + edge) & (c <= edge + r - Lq)) | ((L - edge + r <= c) & (r < edge))
        sc = torch.where(corner, -9.0, S[r.expand(P, Lq), start + cc])
        m = torch.stack([dg[1] + qMM + dIM, dg[2] + qIM + dMM, dg[3] + qDM + dMM, dg[4] + qMM + dDM,
                         dg[0] + qMM + dMM]).amax(0)
        cur = torch.stack([(m + sc).clamp(min=0.0), torch.maximum(up[0] + qMM + dMIc, up[1] + qMM + dIIc),
                           torch.maximum(le[0] + qMIc + dMM, le[2] + qIIc + dMM),
                           torch.maximum(up[0] + qMD, up[3] + qDD), torch.maximum(le[0] + dMD, le[4] + dDD)])
        cur = torch.where(on, cur, 0.0)
        most = torch.maximum(most, torch.where(on, cur[0], 0.0).amax(1))
        p2, p1 = p1, cur
    return {"btck": None, "max": most, "xy": None}


def exact(case, seed):
    if case["kind"] == "matrix" and case["cvswgt"] == 0 and case["form"] == "plain":
        return _matrix64(case, seed)
    if case["kind"] == "dp1":
        return _dp64(case, seed)
    # the other calls return the selected hits' records and alignments, whose
    # scores, statistics and posteriors come from restated 32-bit functions
    # (the path's own exponential and logarithm): no 64-bit values
    return None
