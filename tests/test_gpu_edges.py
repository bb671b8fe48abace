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
