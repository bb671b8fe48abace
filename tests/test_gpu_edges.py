"""Kernel variants at the sizes where they can go wrong: tile edges, the
smallest and largest of a variant's range, remainders (needs a GB300)."""
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
