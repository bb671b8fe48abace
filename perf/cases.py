"""The workloads the covariation engine is timed on, each through its public
entry points (covgpu.Engine, covgpu.Batch): the E-valued analysis of one
alignment from the smallest family to rRNA scale, many families in one call,
score matrices and pair probabilities, null simulation, alignment preparation,
power analysis and the learned null.

Alignments are host arrays, as a program that has parsed its Stockholm file
holds them; a context (its device buffers) and the tree are made once per
alignment size, and score matrices and pair probabilities are read into arrays
that are made once too (R-scape's mi->COV and mi->pp), as programs keep them.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "r-scape_gb300")


def _load(name, filename):
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, os.path.join(PKG, filename))
        sys.modules[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(sys.modules[name])
    return sys.modules[name]


cg = _load("covgpu", "covgpu.py")
ln = _load("learned_null", "learned_null.py")

RESULT_INTS = ("status", "nshuffle", "Nt", "nhit", "h_nb", "h_imin", "h_imax", "h_cmin", "h_n", "h_Nc", "h_No")
RESULT_FLOATS = ("w", "minCOV", "maxCOV", "null_minCOV", "null_maxCOV", "pmass", "newmass", "mu", "lambda_", "tau",
                 "sc_thresh", "h_bmin", "h_xmin", "h_xmax", "h_phi")


def listed():
    return [
        # a small family (a riboswitch or a snoRNA seed alignment), every
        # option left at its default: the shortest call a user makes
        dict(name="rscape_30x61", kind="rscape", N=30, L=61, nulls=-1, types="GTp", counter="default", scores=False),
        # one ordinary small alignment with planted helices, default options
        dict(name="rscape_100x120", kind="rscape", N=100, L=120, nulls=-1, types="GTp", counter="default",
             scores=True),
        # a long non-coding RNA of odd sizes scored with three statistics and
        # both corrections, the score matrices read back for further analysis
        dict(name="rscape_301x773", kind="rscape", N=301, L=773, nulls=20, types="GTp,MIa,RAFSp", counter="tensor",
             scores=True),
        # many nulls for one alignment (a finer null tail): N=500, L=400, 200 nulls
        dict(name="rscape_500x400_200nulls", kind="rscape", N=500, L=400, nulls=200, types="GTp", counter="tensor",
             scores=True),
        # rRNA scale: N=2,000, L=3,000, 20 nulls, four statistics
        dict(name="rscape_2000x3000", kind="rscape", N=2000, L=3000, nulls=20, types="GTp,MIp,CHIp,RAFp",
             counter="tensor", scores=False),
        # a deep alignment scored with four statistics, score matrices out
        dict(name="score_20000x1500", kind="score", N=20000, L=1500, types="GTp,CHIp,OMESp,CCFp", counter="tensor",
             probs=False),
        # scores and the pair probabilities that structure prediction reads,
        # with the default counter
        dict(name="score_400x351", kind="score", N=400, L=351, types="GTp", counter="default", probs=True),
        # a database slice: ragged families (N 20-2,000, L 50-1,500) in one call
        dict(name="families_64", kind="families", families=64, maxN=2000, maxL=1500),
        # simulated alignments on a given tree and structure, read back
        dict(name="simulate_1000x1201_8", kind="simulate", N=1000, L=1201, reps=8),
        # alignment preparation: tree weights and the gap-column filter
        dict(name="weights_900x700", kind="weights", N=900, L=700),
        # substitutions on the tree and the power of every pair
        dict(name="power_701x650", kind="power", N=701, L=650),
        # E-values with the learned null: 20 quick nulls and the shipped network
        dict(name="learned_400x300", kind="learned", N=400, L=300),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rscape", "rscape", "rscape", "score", "families", "simulate", "weights", "power", "learned"])
    if kind == "rscape":
        N, L = _log(rng, 20, 2000), _log(rng, 45, 3000)
        counter = rng.choice(["default", "tensor", "tensor"])
        if counter == "default":   # the plain counting path: kept to alignments it is used for
            N, L = min(N, 600), min(L, 500)
        nulls = rng.choice([-1, 20, 20, 100]) if L <= 600 else 20
        types = rng.choice(["GTp", "GTp", "GTp,MIa,RAFSp", "GTp,MIp,CHIp,RAFp", "MIrp,OMESp", "CHIp,MIgp"])
        return dict(kind=kind, N=N, L=L, nulls=nulls, types=types, counter=counter, scores=L <= 800)
    if kind == "score":
        if rng.random() < 0.5:
            return dict(kind=kind, N=_log(rng, 50, 800), L=_log(rng, 60, 500),
                        types=rng.choice(["GTp", "CHIp,GTa", "GTp,RAFp"]), counter="default", probs=True)
        return dict(kind=kind, N=_log(rng, 1000, 20000), L=_log(rng, 200, 1500),
                    types=rng.choice(["GTp,CHIp,OMESp,CCFp", "GTp", "MIp,RAFp"]), counter="tensor", probs=False)
    if kind == "families":
        return dict(kind=kind, families=_log(rng, 8, 64), maxN=_log(rng, 200, 2000), maxL=_log(rng, 200, 1500))
    if kind == "simulate":
        return dict(kind=kind, N=_log(rng, 50, 2000), L=_log(rng, 60, 2000), reps=rng.randint(1, 8))
    if kind == "weights":
        return dict(kind=kind, N=_log(rng, 50, 2000), L=_log(rng, 60, 1500))
    if kind == "power":
        return dict(kind=kind, N=_log(rng, 30, 1500), L=_log(rng, 60, 1200))
    return dict(kind=kind, N=_log(rng, 60, 1500), L=_log(rng, 80, 1000))


def _synth(N, L, seed, tree_len=1.5, gap_rate=0.08):
    """An alignment on a coalescent tree with a third of its columns paired."""
    nbp = max(1, L // 6)
    nhelix = max(1, nbp // 10)
    return cg.Synth(N, L, tree_len, nbp, nhelix, min(4, nbp // nhelix), max(14, -(-nbp // nhelix)), gap_rate,
                    seed=seed)


def _families(case, seed):
    fams = []
    for k in range(case["families"]):
        f = ln.draw_family(1000003 * (seed % 1000) + 131 * k + 1)
        while f["N"] > case["maxN"] or f["L"] > case["maxL"]:
            f = ln.draw_family(f["seed"] + 7919)
        fams.append(ln.make_family(f)[0])
    return fams


def _counter(case):
    return {"counter": cg.TENSOR} if case["counter"] == "tensor" else {}


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case)
    if kind == "families":
        st["families"] = [dict(ax=s.ax, parent=s.parent, left=s.left, right=s.right) for s in _families(case, seed)]
        st["batch"] = cg.Batch()
        return st
    N, L = case["N"], case["L"]
    s = _synth(N, L, seed, gap_rate=0.0 if kind == "simulate" else 0.08)
    st["s"], st["ax"] = s, s.ax
    if kind == "rscape":
        ns = case["nulls"]
        if ns < 0:   # R-scape's own number of nulls: at most 300
            ns = 300 if L < 40 or N < 4 else (200 if L < 50 or N * L < 1000 else 20)
        st["w"] = cg.weights_pb(s.ax)
        st["e"] = cg.Engine(N, L, maxslots=ns + 1, maxnull=ns)
    elif kind == "score":
        st["w"] = cg.weights_pb(s.ax)
        st["e"] = cg.Engine(N, L)
    elif kind == "simulate":
        st["model"] = cg.synth_model()
        st["e"] = cg.Engine(N, L, maxslots=case["reps"], maxnull=0)
    elif kind == "weights":
        st["e"] = cg.Engine(N, L)
    elif kind == "power":
        x = np.arange(0.0, 200.0)
        st["curve"] = (x, 1.0 - np.exp(-x / 40.0))
        st["e"] = cg.Engine(N, L, maxslots=2, maxnull=1)
    elif kind == "learned":
        st["w"] = cg.weights_pb(s.ax)
        st["net"] = ln.load(os.path.join(PKG, "learned_null_gtp.npz"))
        st["tree_len"] = ln.tree_depth(s.parent, s.left, s.right, s.ld, s.rd)
        st["e"] = cg.Engine(N, L, maxslots=201, maxnull=200)
    ntypes = len(case.get("types", "").split(","))
    if kind == "score" or case.get("scores"):
        st["COV"] = [np.zeros((L, L)) for _ in range(ntypes)]
    if case.get("probs"):
        st["probs"] = [np.zeros((L, L, 16)), np.zeros((L, L)), np.zeros((L, L)), np.zeros((L, 4)), np.zeros((L, 5))]
    if kind not in ("score", "weights"):
        st["e"].set_tree(s.parent, s.left, s.right)
    return st


def _scores(st):
    """The score matrices of the last call into the program's own arrays."""
    e = st["e"]
    for q, out in enumerate(st["COV"]):
        e._ck(cg.lib().covgpu_get_cov(e.h, 0, q, out.reshape(-1)))
    return st["COV"]


def _results(rows):
    """Result dicts as one array per field, and the hit lists one after the
    other in arrays with room for 256 hits per list (the rest zero)."""
    out = {f: np.array([r[f] for r in rows], dtype=np.float64) for f in RESULT_FLOATS}
    out.update({f: np.array([r[f] for r in rows], dtype=np.int64) for f in RESULT_INTS})
    hits = [h for r in rows for h in r["hits"]]
    table = np.zeros((5, 256 * len(rows)))
    hits = hits[:table.shape[1]]
    if hits:
        table[:, :len(hits)] = np.array(hits, dtype=np.float64).T
    out["hit_i"], out["hit_j"] = table[0].astype(np.int64), table[1].astype(np.int64)
    out["hit_score"], out["hit_E"], out["hit_pval"] = table[2], table[3], table[4]
    return out


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    if kind == "families":
        res = st["batch"].rscape(st["families"], ["GTp"], counter=cg.TENSOR)
        return _results([r for rows in res for r in rows])
    e = st["e"]
    if kind == "rscape":
        types = case["types"].split(",")
        res = e.rscape(st["ax"], st["w"], types, nshuffle=case["nulls"], **_counter(case))
        out = _results(res)
        if case["scores"]:
            out["COV"] = _scores(st)
        return out
    if kind == "score":
        types = case["types"].split(",")
        e.set_weights(st["w"])
        e.set_alignment(0, st["ax"])
        mm = e.score(types, **_counter(case))
        out = {"minmax": mm, "COV": _scores(st)}
        if case["probs"]:
            e._ck(cg.lib().covgpu_get_probs(e.h, 0, st["w"].ctypes.data, *[a.ctypes.data for a in st["probs"]]))
            out["pp"], out["nseff"], out["ngap"], out["pm"], out["ps"] = st["probs"]
        return out
    if kind == "simulate":
        s, (Q4, pi4, Q16, pi16) = st["s"], st["model"]
        e.simulate(s.ld, s.rd, Q4, pi4, Q16, pi16, s.ct, gap_rate=0.08, gap_mean=3.0, seed=7, nrep=case["reps"])
        return [e.get_alignment(k) for k in range(case["reps"])]
    if kind == "weights":
        e.set_alignment(0, st["ax"])
        w = e.weights_gsc(0) if case["N"] <= 1000 else e.weights_pb(0)   # R-scape's rule
        return {"w": w, "keep": e.gapfilter(0, w)}
    if kind == "power":
        e.set_alignment(0, st["ax"])
        nsubs, ndouble, njoin = e.substitutions(0)
        return {"nsubs": nsubs, "ndouble": ndouble, "njoin": njoin,
                "power": e.power(single=st["curve"], join=st["curve"], double=st["curve"])}
    res, used = e.rscape_learned(st["ax"], st["w"], st["net"], st["tree_len"], nquick=20, nshuffle=200,
                                 counter=cg.TENSOR)
    out = _results([res])
    out["used_net"] = used
    return out


def _alignments(case):
    """Alignments that are counted in one pass."""
    if case["kind"] == "score":
        return 1
    if case["kind"] == "learned":
        return 21
    N, L, ns = case["N"], case["L"], case["nulls"]
    if ns < 0:
        ns = 300 if L < 40 or N < 4 else (200 if L < 50 or N * L < 1000 else 20)
    return ns + 1


def work(case):
    """Bytes: the alignment(s) in and the outputs out.  Flops: the pair counts,
    16 cells x one multiply-add per sequence and column pair of every
    alignment counted, however the weights are represented."""
    kind = case["kind"]
    if kind == "families":
        # the sizes drawn are uniform in N and log-uniform in L, cut at maxN and maxL
        N = 0.5 * (20 + case["maxN"])
        L2 = (case["maxL"] ** 2 - 50.0 ** 2) / (2.0 * math.log(case["maxL"] / 50.0))
        L = (case["maxL"] - 50.0) / math.log(case["maxL"] / 50.0)
        return {"bytes": case["families"] * N * (L + 12.0), "flops": case["families"] * 21 * 16.0 * N * L2}
    N, L = case["N"], case["L"]
    P = 0.5 * L * (L - 1)
    if kind in ("rscape", "score", "learned"):
        nt = len(case.get("types", "GTp").split(","))
        out = 400.0 * nt
        if kind == "score" or case.get("scores"):
            out += 8.0 * L * L * nt
        if case.get("probs"):
            out += 8.0 * L * L * 18 + 72.0 * L
        return {"bytes": N * L + 8.0 * N + out, "flops": 32.0 * N * P * _alignments(case)}
    if kind == "simulate":
        # every node's states once (the internal nodes' are written and read by the children)
        return {"bytes": 1.0 * case["reps"] * N * L + 16.0 * N + 4.0 * L, "flops": 0.0}
    if kind == "weights":
        # identities of all sequence pairs: one comparison and one sum per column
        gsc = N <= 1000
        return {"bytes": 1.0 * N * L + 8.0 * N + L, "flops": N * (N - 1.0) * L if gsc else 2.0 * N * L}
    # power: three integer counts per pair over the 2(N-1) branches, one bit each
    return {"bytes": 1.0 * N * L + 8.0 * L * L + 24.0 * P, "flops": 6.0 * P * (2 * (N - 1) / 32.0)}


# ---------------------------------------------------------------------------
# score matrices and pair probabilities in 64 bits, from the definitions
# ---------------------------------------------------------------------------
ALLOWED = torch.zeros(4, 4, dtype=torch.float64)
for _x, _y in ((0, 3), (3, 0), (1, 2), (2, 1), (2, 3), (3, 2)):
    ALLOWED[_x, _y] = 1.0


def _counts(ax, w):
    """C[i][x][j][y]: weighted joint counts of every column pair."""
    N, L = ax.shape
    X = torch.stack([(ax == k).to(torch.float64) for k in range(4)], dim=2).reshape(N, 4 * L)
    return (X.t() @ (X * w[:, None])).reshape(L, 4, L, 4).permute(0, 2, 1, 3)   # [i][j][x][y]


def _raf(ax):
    N, L = ax.shape
    one = torch.ones(N, dtype=torch.float64, device=ax.device)
    n = _counts(ax, one) * ALLOWED.to(ax.device)
    nA = n.sum((2, 3))
    c = nA * nA - 0.5 * ((n.sum(3) ** 2).sum(2) + (n.sum(2) ** 2).sum(2))
    return 2.0 * c / (N * (N - 1.0)) - (N - nA) / N


def _score64(ax, w, types):
    N, L = ax.shape
    C = _counts(ax, w)
    nseff = C.sum((2, 3))
    cp = C + 1e-10
    pp = cp / cp.sum((2, 3), keepdim=True)
    del cp
    off = ~torch.eye(L, dtype=torch.bool, device=ax.device)
    use = (off & (nseff > 0)).to(torch.float64)
    pm = (pp.sum(3) * use[:, :, None]).sum(1)
    tot = pm.sum(1, keepdim=True)
    pm = torch.where(tot > 0, pm / tot, torch.full_like(pm, 0.25))
    out, e = {}, None
    need = {t.rstrip("pa") for t in types}
    if need & {"GT", "MI", "MIr", "MIg"}:
        lp = pp.log()
        mi = (pp * (lp - pm.log()[:, None, :, None] - pm.log()[None, :, None, :])).sum((2, 3))
        H = -(pp * lp).sum((2, 3))
        out["MI"], out["GT"] = mi, 2.0 * nseff * mi
        out["MIr"] = torch.where(H > 1e-2, mi / H, torch.zeros_like(mi))
        out["MIg"] = torch.where(nseff > 0, mi - (w.sum() - nseff) / nseff, mi)
    if need & {"CHI", "OMES"}:
        e = pm[:, None, :, None] * pm[None, :, None, :]
        d2 = (pp - e) ** 2
        out["CHI"] = nseff * torch.where(e > 0, d2 / e, torch.zeros_like(e)).sum((2, 3))
        out["OMES"] = nseff * d2.sum((2, 3))
    if "CCF" in need:
        up = torch.triu(nseff, 1).sum(1)
        mp = (up[:, None] * pm).sum(0)
        mp = mp / mp.sum() if float(mp.sum()) != 0.0 else torch.full_like(mp, 0.25)
        a = ((nseff[:, :, None] * pm[:, None, :] - mp) ** 2).sum(2)
        out["CCF"] = torch.sqrt(a * a.t())
    if need & {"RAF", "RAFS"}:
        raf = _raf(ax)
        out["RAF"] = raf
        s = 2.0 * raf
        s[1:, :-1] = s[1:, :-1] + raf[:-1, 1:]                       # (i - 1, j + 1)
        i = torch.arange(L, device=ax.device)
        inner = torch.zeros_like(raf)
        inner[:-1, 1:] = raf[1:, :-1]                                # (i + 1, j - 1)
        s = s + torch.where(i[:, None] < i[None, :] - 2, inner, torch.zeros_like(inner))
        u = torch.triu(0.25 * s, 1)
        out["RAFS"] = u + u.t()
    covs, mms = [], []
    for t in types:
        base, corr = (t[:-1], t[-1]) if t[-1] in "pa" else (t, "")
        v = torch.where(off, out[base], torch.zeros_like(out[base]))
        cx = v.sum(1) / (L - 1.0)
        avg = cx.sum() / L
        if corr == "p":
            v = v - cx[:, None] * cx[None, :] / avg
        elif corr == "a":
            v = v - (cx[:, None] + cx[None, :] - avg)
        x = v[off]
        mms.append([float(x.min()), float(x.max())])
        v = torch.where(off, v, torch.full_like(v, -math.inf))
        covs.append(v.cpu().numpy())
    return covs, np.array(mms), (pp, nseff, pm, off)


def exact(case, seed):
    if case["kind"] not in ("rscape", "score") or case["N"] <= 8 or case["L"] <= 50 or case["N"] * case["L"] ** 2 > 5e10:
        return None   # no closed form (simulated nulls), the two-cell class, or too large for 64 bits
    if case["kind"] == "rscape" and case["L"] > 1500:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    s = _synth(case["N"], case["L"], seed)
    wh = cg.weights_pb(s.ax)
    ax, w = torch.from_numpy(s.ax).to(dev), torch.from_numpy(wh).to(dev)
    types = case["types"].split(",")
    covs, mm, (pp, nseff, pm, off) = _score64(ax, w, types)
    if case["kind"] == "rscape":
        out = {f: None for f in RESULT_FLOATS + RESULT_INTS + ("hit_i", "hit_j", "hit_score", "hit_E", "hit_pval")}
        out["minCOV"], out["maxCOV"] = mm[:, 0].copy(), mm[:, 1].copy()
        if case["scores"]:
            out["COV"] = covs
        return out
    out = {"minmax": mm.reshape(1, -1, 2), "COV": covs}
    if case["probs"]:
        L = case["L"]
        o = off.to(torch.float64)
        ps = torch.stack([((ax == k).to(torch.float64) * w[:, None]).sum(0) for k in range(5)], dim=1) + 1e-5
        out["pp"] = (pp * o[:, :, None, None]).reshape(L, L, 16).cpu().numpy()
        out["nseff"] = (nseff * o).cpu().numpy()
        out["ngap"] = torch.triu(w.sum() - nseff, 1).cpu().numpy()
        out["pm"] = pm.cpu().numpy()
        out["ps"] = (ps / ps.sum(1, keepdim=True)).cpu().numpy()
    return out
