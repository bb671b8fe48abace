"""Kernel variants at the sizes where they can go wrong: tile edges, the
smallest and largest of a variant's range, remainders (needs a GB300)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from parity_tol import stat_close

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,L", [(40, 51), (9, 64), (64, 65), (33, 97)])
@pytest.mark.parametrize("cells", [6, 9, 16])
def test_statistics_at_tile_edges(covgpu, oracle, N, L, cells):
    """The pair-by-pair statistics (two columns to a thread, counts staged a
    row of cells ahead, RAF's counts staged for up to six allowed cells) at
    column counts around the 32-column tile and with more allowed cells than
    are staged."""
    s = covgpu.Synth(N, L, 1.5, 8, 1, 4, 8, 0.15, seed=N + L, tree_kind=1)
    w = covgpu.weights_pb(s.ax) * np.random.default_rng(L).uniform(0.6, 1.4, N)
    allow = covgpu.default_allow()
    extra = [k for k in range(16) if allow[k] == 0.0]
    allow[extra[:cells - 6]] = 1.0
    e = covgpu.Engine(N, L)
    e.set_weights(w)
    e.set_alignment(0, s.ax)
    iu = np.triu_indices(L, 1)
    for types in (["GT", "RAF"], ["CHIp", "RAFa", "MIrp", "OMES"], ["MIg", "CCF", "MIp"], ["RAFp"]):
        mm = e.score(types, allow=allow)
        for q, t in enumerate(types):
            ref, (rmin, rmax) = oracle.cov_calculate(t, s.ax, w, allow=allow)
            got = e.get_cov(0, q)
            ok, rel, small = stat_close(got[iu], ref[iu])
            assert ok, "%s rel %g small %g" % (t, rel, small)
            assert mm[0, q, 0] == got[iu].min() and mm[0, q, 1] == got[iu].max()
    e.close()


@pytest.mark.parametrize("N,L,ns", [(2, 33, 2), (3, 17, 1), (300, 64, 40), (40, 1100, 2), (5600, 33, 1)])
def test_nulls_on_every_route(covgpu, oracle, N, L, ns):
    """Null alignments byte for byte on each route: one launch per null
    cluster (1 CTA, 4 CTAs), a launch per depth (more than 1,024 columns), and
    the reconstruction of a tree too deep for shared memory; with ambiguity
    codes and a root of two leaves."""
    s = covgpu.Synth(N, L, 1.5, 4, 1, 4, 4, 0.15, seed=N + L)
    rng = np.random.default_rng(N)
    for code in (5, 15, 17):
        s.ax[rng.integers(0, N, 4 + N // 50), rng.integers(0, L, 4 + N // 50)] = code
    e = covgpu.Engine(N, L, maxslots=ns + 1, maxnull=ns)
    e.set_alignment(0, s.ax)
    e.set_tree(s.parent, s.left, s.right)
    e.make_nulls(7, 5, ns, 1)
    T = oracle.TreeArrays(s.parent, s.left, s.right, s.ld, s.rd)
    for q in sorted({0, ns // 2, ns - 1}):
        assert np.array_equal(e.get_alignment(1 + q), oracle.null_msa(s.ax, T, 7, 5 + q)), q
    e.close()


@pytest.mark.parametrize("N,L", [(2, 20), (129, 31), (5600, 33)])
def test_reconstruction_with_ambiguity_codes(covgpu, oracle, N, L):
    """Substitutions per column and pair on the Fitch reconstruction, in shared
    memory and (the deepest tree) in global rows."""
    s = covgpu.Synth(N, L, 1.5, 4, 1, 4, 4, 0.15, seed=N)
    s.ax[0, : L // 2] = 15
    e = covgpu.Engine(N, L)
    e.set_alignment(0, s.ax)
    e.set_tree(s.parent, s.left, s.right)
    T = oracle.TreeArrays(s.parent, s.left, s.right, s.ld, s.rd)
    for got, ref in zip(e.substitutions(0, seed=9), oracle.substitutions(s.ax, T, 9, 0xFFFFFFFF)):
        assert np.array_equal(got, ref)
    e.close()


@pytest.mark.parametrize("N,L", [(7, 20), (256, 40), (257, 40), (513, 60), (1025, 24)])
def test_gsc_weights_at_cluster_edges(covgpu, oracle, N, L):
    """GSC weights around the sizes where the merges' cluster (8 or 16 CTAs) and
    the rows per lane change, with many equal distances (short, duplicated
    rows), against the oracle."""
    s = covgpu.Synth(N, L, 0.6, 2, 1, 1, 2, 0.1, seed=N, tree_kind=1)
    rng = np.random.default_rng(N)
    for k in range(N // 4):
        i, j = rng.integers(0, N, size=2)
        s.ax[j] = s.ax[i]
    e = covgpu.Engine(N, L)
    e.set_alignment(0, s.ax)
    g = e.weights_gsc(0, set=False)
    e.close()
    assert np.allclose(g, oracle.weights_gsc(s.ax), rtol=1e-10, atol=1e-13)


@pytest.mark.parametrize("N,L", [(3, 31), (31, 33), (9000, 40)])
def test_position_weights_and_gap_filter_by_slices(covgpu, oracle, N, L):
    """Column counts in packed bytes (emptied every 255 rows of a slice) and
    the gap filter's sums by slices of the sequences."""
    s = covgpu.Synth(N, L, 1.0, 2, 1, 1, 2, 0.3, seed=N)
    e = covgpu.Engine(N, L)
    e.set_alignment(0, s.ax)
    w = e.weights_pb(0, set=False)
    assert np.allclose(w, oracle.weights_pb(s.ax), rtol=1e-12, atol=1e-15)
    for thr in (0.5, 0.7, 0.75):
        for wgt in (None, w):
            assert np.array_equal(e.gapfilter(0, wgt, thr), oracle.gapfilter(s.ax, wgt, thr) == 1)
    e.close()


@pytest.mark.parametrize("N,L,ns,pmass,w0,want", [
    # ~300 bins: one warp per block, 17 bins near mu at each of six points
    (8, 40, 1, 0.05, 0.05, [(0.830686218287233, 0.5717117980558083), (10.803158200648957, 0.2815148742465867)]),
    # coarse bins, half of the histogram in the tail
    (8, 40, 1, 0.5, 0.5, [(1.822823517103002, 0.7979367241135228), (16.611265927604805, 0.8372782766560288)]),
    # ~10^4 bins: more than one item per thread, every SM in the grid
    (60, 100, 8, 0.3, 0.001, [(0.1162342608351604, 0.9960794172969336), (7.804012852676134, 1.2917766699223328)]),
    # a tail of a few dozen bins, a third or more of them near mu
    (60, 100, 8, 0.0005, 0.05, [(0.3792700169111325, 0.8599124467420373), (36.04358169921398, 1.492509473769629)]),
])
def test_tail_fit_at_list_edges(covgpu, oracle, N, L, ns, pmass, w0, want):
    """The tail fit on the grid and on one block (in a batch): the histogram of
    the oracle; lambda and tau of the serial evaluation of the same search (a
    thread per bin, its incomplete gammas one after the other), which only the
    order of operations could change (1e-9); both forms within 1e-6 of one
    another (the search's convergence)."""
    s = covgpu.Synth(N, L, 1.5, 8, 1, 8, 14, 0.08, seed=5)
    w = np.ones(N)
    kw = dict(pmass=pmass, w0=w0, nshuffle=ns, thresh=10.0)
    T = oracle.TreeArrays(s.parent, s.left, s.right, s.ld, s.rd)
    e = covgpu.Engine(N, L, maxslots=ns + 1, maxnull=ns)
    e.set_tree(s.parent, s.left, s.right)
    types = ["GTp", "MI"]
    one = e.rscape(s.ax, w, types, counter=covgpu.TENSOR, **kw)
    e.close()
    b = covgpu.Batch()
    fam = dict(ax=s.ax, parent=s.parent, left=s.left, right=s.right, wgt=w)
    grp = b.rscape([fam, fam], types, counter=covgpu.TENSOR, **kw)
    b.close()
    for q, t in enumerate(types):
        ref = oracle.rscape(s.ax, w, T, covtype=t, **kw)
        lam, tau = want[q]
        assert abs(one[q]["lambda_"] - lam) <= 1e-9 * lam, (t, one[q]["lambda_"], lam)
        assert abs(one[q]["tau"] - tau) <= 1e-9 * tau, (t, one[q]["tau"], tau)
        for g in (one[q], grp[0][q], grp[1][q]):
            for k in ("h_nb", "h_imin", "h_imax", "h_cmin", "h_n", "h_Nc", "h_No"):
                assert g[k] == ref[k], (t, k)
            assert abs(g["lambda_"] - lam) <= 1e-6 * lam


@pytest.mark.parametrize("N,L", [(9, 40), (8, 64), (2, 65), (33, 97)])
@pytest.mark.parametrize("rate,mean", [(0.3, 3.0), (1.0, 1.0), (0.02, 400.0), (1e-12, 2.0)])
def test_simulated_gap_runs_by_words(covgpu, oracle, N, L, rate, mean):
    """Rows that end inside, at and after a word of 32 columns; every column
    open, runs across many words, hardly any: the oracle's alignment."""
    s = covgpu.Synth(N, L, 1.5, max(1, L // 6), 1, 1, L // 6, 0.0, seed=3)
    e = covgpu.Engine(N, L, maxslots=3, maxnull=0)
    e.set_tree(s.parent, s.left, s.right)
    Q4, pi4, Q16, pi16 = covgpu.synth_model()
    e.simulate(s.ld, s.rd, Q4, pi4, Q16, pi16, s.ct, gap_rate=rate, gap_mean=mean, seed=9, rep0=1, nrep=3)
    P4, P16 = e.sim_tables()
    T = oracle.TreeArrays(s.parent, s.left, s.right, s.ld, s.rd)
    for r in range(3):
        ref = oracle.simulate(T, L, s.ct, P4, P16, pi4, pi16, None, rate, mean, 9, 1 + r)
        assert np.array_equal(e.get_alignment(r), ref)
    e.close()


@pytest.mark.parametrize("L", [1, 15, 16, 17, 31, 32, 33, 47, 63, 95, 97, 130])
def test_alignment_rows_round_trip(covgpu, L):
    """Rows of every offset in a word, lengths around 16 and 32, two slots of
    different content: what was set is what is read."""
    rng = np.random.default_rng(L)
    e = covgpu.Engine(37, L, maxslots=2, maxnull=0)
    ax = [rng.integers(0, 18, (37, L)).astype(np.uint8) for _ in range(2)]
    for k in (0, 1):
        e.set_alignment(k, ax[k])
    for k in (1, 0):
        assert np.array_equal(e.get_alignment(k), ax[k])
    e.close()


@pytest.mark.parametrize("N", [2, 15, 16, 17, 33, 129])
@pytest.mark.parametrize("L", [17, 32, 65, 97])
@pytest.mark.parametrize("weights", ["limbs", "equal"])
def test_plain_counts_at_chunk_edges(covgpu, oracle, N, L, weights):
    """The plain counting path at the edges of its chunks of 16 sequences, its
    half tiles and the single-column frequencies' chunks of 128: the counts
    are exact, so the probabilities equal the tensor path's in every bit; the
    frequencies (of the weights as given) within 1e-12 of the oracle's."""
    rng = np.random.default_rng(N * 100 + L)
    ax = rng.integers(0, 6, (N, L)).astype(np.uint8)
    ax[ax == 5] = 15   # N: neither residue nor gap
    w = rng.uniform(0.2, 3.0, N) if weights == "limbs" else np.full(N, 0.7)
    got = []
    for counter in (covgpu.SIMT, covgpu.TENSOR):
        e = covgpu.Engine(N, L)
        e.set_weights(w)
        e.set_alignment(0, ax)
        e.score(["GTp", "RAF"], counter=counter)
        got.append(e.get_probs(0, w) + (e.get_cov(0, 1),))
        e.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)
    assert np.allclose(got[0][4], oracle.probs(ax, w)[4], rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("w0", [0.05, 0.002, 0.0004])
@pytest.mark.parametrize("doexp", [0, 1])
def test_survival_tables(covgpu, oracle, w0, doexp):
    """E-values read from survival tables of hundreds to ~10^5 bins, two lanes
    or one to a bin, on the grid and in a batch: the oracle's within 1e-4, as
    in the pipeline's parity tests."""
    s = covgpu.Synth(60, 100, 1.5, 16, 2, 4, 14, 0.08, seed=7)
    w = covgpu.weights_pb(s.ax)
    kw = dict(nshuffle=8, thresh=10.0, w0=w0, doexpfit=doexp)
    e = covgpu.Engine(60, 100, maxslots=9, maxnull=8)
    e.set_tree(s.parent, s.left, s.right)
    one = e.rscape(s.ax, w, ["GTp"], counter=covgpu.TENSOR, **kw)[0]
    e.close()
    b = covgpu.Batch()
    grp = b.rscape([dict(ax=s.ax, parent=s.parent, left=s.left, right=s.right, wgt=w)], ["GTp"],
                   counter=covgpu.TENSOR, **kw)[0][0]
    b.close()
    ref = oracle.rscape(s.ax, w, oracle.TreeArrays(s.parent, s.left, s.right, s.ld, s.rd), covtype="GTp", **kw)
    rh = {(i, j): E for (i, j, sc, E, p) in ref["hits"]}
    assert len(rh) >= 5
    for r in (one, grp):
        gh = {(i, j): E for (i, j, sc, E, p) in r["hits"]}
        assert set(gh) == set(rh)
        for k in rh:
            assert abs(gh[k] - rh[k]) <= 1e-4 * rh[k] + 1e-300, (k, gh[k], rh[k])


@pytest.mark.parametrize("members", [0, 1, 3])
def test_network_rows_equal_products(covgpu, members):
    """The forward pass by rows (up to 1024 rows) gives the bits of the layers'
    products (more rows)."""
    rng = np.random.default_rng(members)
    net = covgpu.MLP(batch_cap=2048)
    p = net.params()
    if members:
        net.set_members(np.stack([p + 0.02 * rng.normal(size=p.shape).astype(np.float32) for _ in range(members)]))
    X = rng.normal(size=(1025, 64)).astype(np.float32)
    Y = net.forward(X)
    for n in (1, 2, 1024):
        assert np.array_equal(net.forward(X[:n]), Y[:n]), n
    net.close()


@pytest.mark.parametrize("copies", [1, 3, 25, 70, 160])
def test_batch_fit_does_not_depend_on_its_cluster(covgpu, copies):
    """One family many times in a batch: clusters of eight, eight, six and two
    blocks per fit and one block; lambda and tau keep their bits."""
    s = covgpu.Synth(40, 60, 1.5, 9, 1, 4, 14, 0.08, seed=3)
    fam = dict(ax=s.ax, parent=s.parent, left=s.left, right=s.right)
    b = covgpu.Batch()
    want = b.rscape([fam, fam], ["GTp"], counter=covgpu.TENSOR, nshuffle=20)[0][0]
    for rows in b.rscape([fam] * copies, ["GTp"], counter=covgpu.TENSOR, nshuffle=20):
        for k in ("lambda_", "tau", "sc_thresh", "nhit"):
            assert rows[0][k] == want[k], k
    b.close()


@pytest.mark.parametrize("N,L", [(200, 12), (5, 40), (60, 70)])
@pytest.mark.parametrize("curve", ["rising", "unsorted", "one"])
def test_power_tabled_and_scanned(covgpu, oracle, N, L, curve):
    """Few pairs (each scans its curve) and many (the curves are tabled): the
    oracle's step at every pair's counts, also for a curve whose points do not
    rise and for a single point."""
    s = covgpu.Synth(N, L, 1.5, max(1, L // 6), 1, 1, L // 6, 0.1, seed=4)
    e = covgpu.Engine(N, L, maxslots=1, maxnull=0)
    e.set_tree(s.parent, s.left, s.right)
    e.set_alignment(0, s.ax)
    ns, nd, nj = e.substitutions(0)
    x = {"rising": np.arange(-1.0, 30.0, 1.5), "unsorted": np.array([0.0, 3.0, 2.0, 9.0, 1.0, 4.0]),
         "one": np.array([1.0])}[curve]
    y = np.linspace(0.05, 0.95, len(x))
    got = e.power(single=(x, y), join=(x, y[::-1].copy()), double=(x, y))
    e.close()
    i, j = np.triu_indices(L, 1)
    for g, n, p in zip(got, (ns[i] + ns[j], nj[i, j], nd[i, j]), (y, y[::-1], y)):
        assert np.array_equal(g, [oracle.power_step(float(v), x, np.ascontiguousarray(p)) for v in n])


@pytest.mark.parametrize("N,L", [(64, 40), (96, 16), (97, 33), (200, 65), (1001, 48)])
@pytest.mark.parametrize("thr", [0.5, 0.75, 0.25])
def test_gap_filter_on_the_threshold(covgpu, oracle, N, L, thr):
    """Columns whose weighted fraction lies exactly on the threshold: every
    weight is held by four sequences, 1 - thr of them with a residue, so that
    the rounding of the sums decides.  The sums run over the sequences in their
    order, as the oracle's: the same columns."""
    rng = np.random.default_rng(N + L)
    n4 = N // 4
    w = np.concatenate([np.repeat(rng.uniform(0.1, 3.0, n4), 4), rng.uniform(0.1, 3.0, N - 4 * n4)])
    ax = np.full((N, L), 17, dtype=np.uint8)   # the sequences beyond 4 n4: missing, not counted
    for c in range(L):
        for k in range(n4):
            res = rng.permutation(4) < 4 * (1 - thr)
            ax[4 * k:4 * k + 4, c] = np.where(res, rng.choice([0, 1, 2, 3, 7, 15], 4), rng.choice([4, 16], 4))
    p = rng.permutation(N)
    ax, w = np.ascontiguousarray(ax[p]), np.ascontiguousarray(w[p])
    ref = oracle.gapfilter(ax, w, thr) == 1
    e = covgpu.Engine(N, L)
    e.set_alignment(0, ax)
    assert np.array_equal(e.gapfilter(0, w, thr), ref)
    assert np.array_equal(e.gapfilter(0, None, thr), oracle.gapfilter(ax, None, thr) == 1)
    e.close()


@pytest.mark.parametrize("shift", [0, 39, 41])
@pytest.mark.parametrize("weights", ["limbs", "equal"])
def test_statistics_at_the_weights_scale(covgpu, oracle, shift, weights):
    """Weights of the size of one and 2^39 or 2^41 times smaller, where the pair
    counts lie far below the prior of 1e-10, against the oracle to 1e-7 of the
    largest score.  The prior is the FP32 number next to 1e-10, 1.34e-8 above
    it, and MI goes as its inverse square there: 2.7e-8; the double-float terms
    (2^-44 of p |ln p|, |ln p| up to 28) add less than 2e-8 of a largest MI of
    9e-5.  Counts that lose their low word in the addition of the prior (a
    two-sum for operands in the other order) put the scores off by 3e-7 and
    1e-6."""
    N, L = 40, 60
    s = covgpu.Synth(N, L, 1.5, 8, 1, 4, 8, 0.15, seed=11, tree_kind=1)
    w = np.random.default_rng(3).integers(1 << 29, 1 << 33, N) * 2.0 ** -32
    w = (w if weights == "limbs" else np.full(N, 1.0 + 2.0 ** -20 + 2.0 ** -22)) * 2.0 ** -shift
    e = covgpu.Engine(N, L)
    e.set_weights(w)
    e.set_alignment(0, s.ax)
    iu = np.triu_indices(L, 1)
    types = ["MI", "MIr", "CHI", "GT"]
    for counter in (covgpu.SIMT, covgpu.TENSOR):
        e.score(types, covclass=covgpu.C16, counter=counter)
        for q, t in enumerate(types):
            ref = oracle.cov_calculate(t, s.ax, w, covclass=covgpu.C16)[0][iu]
            err = np.abs(e.get_cov(0, q)[iu] - ref).max()
            assert err <= 1e-7 * np.abs(ref).max(), (t, err, np.abs(ref).max())
    e.close()


@pytest.mark.parametrize("N,L,ns", [(3100, 33, 3), (5400, 17, 2), (5400, 290, 15), (16400, 17, 2), (29000, 20, 1)])
def test_nulls_of_deep_trees(covgpu, oracle, N, L, ns):
    """Null alignments byte for byte in every form of the reconstruction beyond
    the deepest tree that lies in shared memory with 16 columns: eight columns,
    four columns, rows in global memory (many columns), four columns with the
    tree in global memory, and everything in global memory; the reconstruction
    itself in the same forms."""
    s = covgpu.Synth(N, L, 1.5, 2, 1, 2, 2, 0.15, seed=N + L)
    rng = np.random.default_rng(N)
    for code in (5, 15, 17):
        s.ax[rng.integers(0, N, N // 50), rng.integers(0, L, N // 50)] = code
    e = covgpu.Engine(N, L, maxslots=ns + 1, maxnull=ns)
    e.set_alignment(0, s.ax)
    e.set_tree(s.parent, s.left, s.right)
    e.make_nulls(7, 5, ns, 1)
    T = oracle.TreeArrays(s.parent, s.left, s.right, s.ld, s.rd)
    for q in sorted({0, ns - 1}):
        assert np.array_equal(e.get_alignment(1 + q), oracle.null_msa(s.ax, T, 7, 5 + q)), q
    for got, ref in zip(e.substitutions(0, seed=9), oracle.substitutions(s.ax, T, 9, 0xFFFFFFFF)):
        assert np.array_equal(got, ref)
    e.close()


@pytest.mark.parametrize("deep", [(5400, 33), (3100, 60), (5400, 250)])
def test_batch_with_a_deep_family(covgpu, deep):
    """A deep family beside small ones: the batch's null scores (the forms of
    the reconstruction by the deepest family of the chunk) are the single
    calls'."""
    fams = []
    for k, (N, L) in enumerate([(30, 61), deep, (90, 64)]):
        s = covgpu.Synth(N, L, 1.5, 4, 1, 4, 4, 0.1, seed=k + 2)
        fams.append(dict(ax=s.ax, parent=s.parent, left=s.left, right=s.right, wgt=covgpu.weights_pb(s.ax)))
    b = covgpu.Batch()
    got = b.rscape(fams, ["GTp"], counter=covgpu.TENSOR, nshuffle=20)
    b.close()
    for f, rows in zip(fams, got):
        e = covgpu.Engine(*f["ax"].shape, maxslots=21, maxnull=20)
        e.set_tree(f["parent"], f["left"], f["right"])
        one = e.rscape(f["ax"], f["wgt"], ["GTp"], counter=covgpu.TENSOR, nshuffle=20)[0]
        e.close()
        for k in ("null_minCOV", "null_maxCOV", "h_nb", "h_imin", "h_imax", "h_n", "nhit"):
            assert rows[0][k] == one[k], k


def _gsc_merge_by_merge(ax):
    """GSC weights on UPGMA in numpy, a merge at a time in FP64: the closest
    pair, ties to the first in row-major order; the operations of the oracle,
    whose search over all pairs takes too long beyond a thousand sequences."""
    N, L = ax.shape
    X = np.stack([(ax == k) for k in range(4)], 2).reshape(N, -1).astype(np.float32)
    n = (ax < 4).sum(1).astype(np.float64)
    mn = np.minimum(n[:, None], n[None, :])
    D = np.where(mn > 0, 1.0 - (X @ X.T).astype(np.float64) / np.maximum(mn, 1.0), 1.0)
    np.fill_diagonal(D, np.inf)
    up = np.array([(D[a, a + 1:].min(), a + 1 + D[a, a + 1:].argmin()) if a + 1 < N else (np.inf, 0)
                   for a in range(N)])
    rmin, rarg = up[:, 0].copy(), up[:, 1].astype(int)
    w, cl = np.zeros(N), np.arange(N)
    size, height, cw, alive = np.ones(N), np.zeros(N), np.zeros(N), np.ones(N, dtype=bool)

    def rescan(r):
        k = D[r, r + 1:].argmin() if r + 1 < N else 0
        rmin[r], rarg[r] = (D[r, r + 1 + k], r + 1 + k) if r + 1 < N else (np.inf, 0)

    for _ in range(N - 1):
        a = int(rmin.argmin())
        b = int(rarg[a])
        h = D[a, b] / 2.0
        bl = [max(h - height[k], 0.0) for k in (a, b)]
        for k, x in ((a, bl[0]), (b, bl[1])):
            m = cl == k
            w[m] += x * w[m] / cw[k] if cw[k] > 0 else x / size[k]
        cl[cl == b] = a
        x = (D[a] * size[a] + D[b] * size[b]) / (size[a] + size[b])
        alive[b] = False
        x[~alive] = np.inf
        x[a] = np.inf
        D[a], D[:, a] = x, x
        D[b], D[:, b] = np.inf, np.inf
        cw[a] = (cw[a] + bl[0]) + (cw[b] + bl[1])
        size[a], height[a], rmin[b] = size[a] + size[b], h, np.inf
        lost = alive & ((rarg == a) | (rarg == b))
        lost[a] = True
        below = np.flatnonzero(alive[:a] & ~lost[:a])
        better = below[(x[below] < rmin[below]) | ((x[below] == rmin[below]) & (a < rarg[below]))]
        rmin[better], rarg[better] = x[better], a
        for r in np.flatnonzero(lost):
            rescan(r)
    return w * N / w.sum()


@pytest.mark.parametrize("N,L", [(300, 40), (2100, 60), (4097, 30), (8200, 48)])
def test_gsc_weights_of_deep_alignments(covgpu, oracle, N, L):
    """16 and 32 rows per lane, and the weights' state in global memory (8,200
    sequences), against a merge at a time on the host; the smallest size also
    against the oracle."""
    s = covgpu.Synth(N, L, 1.0, 2, 1, 1, 2, 0.1, seed=N, tree_kind=1)
    rng = np.random.default_rng(N)
    dup = rng.integers(0, N, size=(N // 20, 2))
    s.ax[dup[:, 1]] = s.ax[dup[:, 0]]
    ref = _gsc_merge_by_merge(s.ax)
    if N <= 1000:
        assert np.allclose(ref, oracle.weights_gsc(s.ax), rtol=1e-10, atol=1e-13)
    e = covgpu.Engine(N, L)
    e.set_alignment(0, s.ax)
    g = e.weights_gsc(0, set=False)
    e.close()
    assert np.allclose(g, ref, rtol=1e-10, atol=1e-13)


def _hard_quotients(rng, n, near):
    """x, b whose quotient lies within 2^-105 of the middle of two numbers: b an
    odd 53-bit integer, m the odd 54-bit middle with m b = -+1 mod 2^54, x = (m b
    +- 1) / 2^54.  near: b near a power of two."""
    xs, bs = [], []
    while len(xs) < n:
        b = int(rng.integers(1 << 52, 1 << 53)) | 1
        if near:
            k = int(rng.integers(0, 1 << 12)) | 1
            b = (1 << 52) + k if len(xs) & 1 else (1 << 53) - k
        for sgn in (1, -1):
            m = (-sgn * pow(b, -1, 1 << 54)) % (1 << 54)
            if m < 1 << 53:
                continue
            x = (m * b + sgn) >> 54
            xs.append(float(x))
            bs.append(float(b))
    return np.array(xs[:n]), np.array(bs[:n])


@pytest.mark.parametrize("kind", ["div_fast", "div_by"])
def test_quotients_against_cuda_division(tmp_path, kind):
    """The corrected quotients beside CUDA's division: random operands over
    div_range and at its ends, operands next to powers of two, equal quotients
    and small integers, and the hardest cases for rounding.  div_by is the
    rounded quotient everywhere; div_fast too, but for the hardest cases, where
    it may be the neighbour (its reciprocal may be an ulp off); outside
    div_range nothing is claimed of div_fast."""
    here = os.path.dirname(os.path.abspath(__file__))
    so = str(tmp_path / "quotients.so")
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-Xcompiler", "-fPIC", "-shared", "-I", os.path.join(here, "..", "r-scape_gb300", "csrc"),
                    os.path.join(here, "quotients.cu"), "-o", so], check=True)
    lib = ctypes.CDLL(so)
    rng = np.random.default_rng(17)
    n = 1 << 22

    def run(x, b):
        x, b = (np.ascontiguousarray(v, dtype=np.float64) for v in np.broadcast_arrays(x, b))
        q, r, ok = np.zeros(len(x)), np.zeros(len(x)), np.zeros(len(x), dtype=np.int32)
        assert lib.quotients(int(kind == "div_by"), *[ctypes.c_void_p(v.ctypes.data) for v in (x, b)], len(x),
                             *[ctypes.c_void_p(v.ctypes.data) for v in (q, r, ok)]) == 0
        return q, r, ok

    def mantissa(size):
        return rng.uniform(1.0, 2.0, size) * rng.choice([-1.0, 1.0], size)

    sets = [(mantissa(n) * 2.0 ** rng.integers(-98, 99, n), mantissa(n) * 2.0 ** rng.integers(-98, 99, n)),
            (mantissa(n) * 2.0 ** rng.choice([-98, 98], n), mantissa(n) * 2.0 ** rng.choice([-98, 98], n)),
            (1.0 + 2.0 ** -52 * rng.integers(0, 64, n), 2.0 - 2.0 ** -52 * rng.integers(1, 64, n)),
            (2.0 - 2.0 ** -52 * rng.integers(1, 64, n), 1.0 + 2.0 ** -52 * rng.integers(0, 64, n)),
            (rng.integers(0, 5000, n).astype(float), rng.integers(1, 5000, n).astype(float))]
    for x, b in sets:
        q, r, ok = run(x, b)
        assert np.array_equal(q, r)
    for near in (False, True):
        x, b = _hard_quotients(rng, 20000, near)
        q, r, ok = run(x, b)
        off = q != r
        print("%s: %d of %d hard quotients the other neighbour" % (kind, off.sum(), len(x)))
        assert np.all(np.abs(q - r) <= np.spacing(np.abs(r)))
        if kind == "div_by":
            assert not off.any()
    # the ends of div_range
    e = np.array([0.0, 0.99e-30, 1.01e-30, 0.99e30, 1.01e30, np.inf, np.nan])
    ok = run(e, np.full(len(e), 1.0))[2]
    assert ok.tolist() == [0, 0, 1, 1, 0, 0, 0]


def test_null_buffers_hold_what_the_generator_uses(covgpu):
    """A context's device memory per null: the null's internal rows and its
    branch counters (200 bytes per sequence); of the reconstruction only the
    root's row is kept."""
    import torch
    N, L, Lp, ns = 4000, 500, 512, 200

    def used(maxnull):
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        e = covgpu.Engine(N, L, maxslots=1, maxnull=maxnull)
        after = torch.cuda.mem_get_info()[0]
        e.close()
        return before - after

    used(1)
    per = (used(ns) - used(1)) / (ns - 1)
    assert per <= 1.05 * N * (Lp + 200), per / N


@pytest.mark.parametrize("N,L,ns", [(5, 40, 30), (60, 100, 3)])
def test_reconstruction_and_nulls_share_a_buffer(covgpu, oracle, N, L, ns):
    """More nulls than internal nodes and fewer: nulls, the reconstruction of
    the same context, the nulls again."""
    s = covgpu.Synth(N, L, 1.5, 4, 1, 4, 4, 0.1, seed=N)
    e = covgpu.Engine(N, L, maxslots=ns + 1, maxnull=ns)
    e.set_alignment(0, s.ax)
    e.set_tree(s.parent, s.left, s.right)
    T = oracle.TreeArrays(s.parent, s.left, s.right, s.ld, s.rd)
    for _ in range(2):
        e.make_nulls(7, 0, ns, 1)
        for q in (0, ns - 1):
            assert np.array_equal(e.get_alignment(1 + q), oracle.null_msa(s.ax, T, 7, q)), q
        for got, ref in zip(e.substitutions(0, seed=9), oracle.substitutions(s.ax, T, 9, 0xFFFFFFFF)):
            assert np.array_equal(got, ref)
    e.close()


def test_a_large_workspace_is_given_back(covgpu):
    """covgpu_power takes 24 bytes per pair of columns (108 MB here); the context
    keeps no more than 64 MB of workspace after the call, and its results do not
    depend on what it kept."""
    import torch
    N, L = 6, 3000
    s = covgpu.Synth(N, L, 1.5, 8, 1, 4, 8, 0.1, seed=2)
    e = covgpu.Engine(N, L)
    e.set_tree(s.parent, s.left, s.right)
    e.set_alignment(0, s.ax)
    subs = e.substitutions(0)
    x = np.arange(8.0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    first = e.power(single=(x, x / 8), join=(x, x / 8), double=(x, x / 8))
    assert before - torch.cuda.mem_get_info()[0] <= 66 << 20
    e.set_alignment(0, s.ax)
    for a, b in zip(subs, e.substitutions(0)):
        assert np.array_equal(a, b)
    for a, b in zip(first, e.power(single=(x, x / 8), join=(x, x / 8), double=(x, x / 8))):
        assert np.array_equal(a, b)
    e.close()


@pytest.mark.parametrize("scale", [1.0, 2.0 ** -140, 2.0 ** -300, 2.0 ** 120, 2.0 ** 1000])
@pytest.mark.parametrize("thr", [0.5, 0.25, 1.0, 1.0 - 1e-7, 1.5, 0.0, -0.5])
def test_gap_filter_at_the_edges_of_its_sums(covgpu, oracle, scale, thr):
    """Weights out of FP32's range and with zeros among them, columns without a
    counted sequence or with weights of 0 alone, thresholds of 0 and below and
    above 1, fractions from far to one part in 1e7 of the threshold: the
    oracle's columns; so for a negative weight and one that is not finite."""
    N, L = 333, 70
    rng = np.random.default_rng(5)
    w = rng.uniform(0.5, 2.0, N) * scale
    w[rng.integers(0, N, 20)] = 0.0
    ax = np.where(rng.random((N, L)) < rng.uniform(0, 1, L), 4, rng.choice([0, 1, 2, 3, 9, 16, 17], (N, L)))
    ax[:, 0], ax[:, 1], ax[:, 2] = 17, np.where(w == 0.0, 2, 17), 4
    half = rng.permutation(N)[:N // 2]
    for k in range(8):   # residues and gaps of equal weight, then one residue's weight more by a little
        ax[:, 10 + k] = 17
        ax[half, 10 + k] = 1
    w2 = w.copy()
    other = np.setdiff1d(np.arange(N), half)[:len(half)]
    w2[other] = w2[half]
    for k in range(8):
        ax[other, 10 + k] = 4
    w2[half[np.flatnonzero(w2[half] > 0)[0]]] *= 1.0 + 1e-5
    e = covgpu.Engine(N, L)
    ax = np.ascontiguousarray(ax.astype(np.uint8))
    e.set_alignment(0, ax)
    cases = [w, w2]
    for v in (-0.25 * scale, np.inf, np.nan):
        w3 = w.copy()
        w3[7] = v
        cases.append(w3)
    for x in cases:
        with np.errstate(all="ignore"):
            assert np.array_equal(e.gapfilter(0, x, thr), oracle.gapfilter(ax, x, thr) == 1)
    assert np.array_equal(e.gapfilter(0, None, thr), oracle.gapfilter(ax, None, thr) == 1)
    e.close()
