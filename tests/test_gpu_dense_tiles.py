"""Far lines of crowded mixed tiles (summed at the tile's nodes): where they may be taken, what they round,
and what a gradient makes of the opacity they leave."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(L, lo, hi, n, teff=4500.0, wl=None):
    from korg_gb300 import synthetic
    w = synthetic.Workload("dense", teff, 4.4, 0.0, L, wl or (lo, hi), synthetic.synthetic_linelist(n, lo, hi, seed=n))
    return synthetic.prepare(w)


def _lines_only(gpu_lib, inp, ll, cutoff=3e-4):
    """The opacity of the lines alone in mixed precision, and how many lines reach the grid."""
    from korg_gb300 import line_absorption_
    from korg_gb300.api import ContinuumInterpolant
    from korg_gb300.data import default_partition_funcs
    ctx = gpu_lib.Context(0)
    a = np.zeros((len(inp.wls), len(inp.T)))
    line_absorption_(a, ll, inp.wls, inp.T, inp.ne, inp.number_densities, default_partition_funcs(), inp.xi,
                     ContinuumInterpolant(inp.cntm_knots, inp.cntm_vals), cutoff_threshold=cutoff, precision="mixed",
                     ctx=ctx)
    n = ctx.stats().lines_in_window
    ctx.close()
    return a, n


def test_series_of_far_lines_in_fp64(gpu_lib):
    """9,000 lines, all far from the only tile (three tile widths and more) and weakly damped, so that every one
    is given by its wing cubic there: the tile's opacity is the polynomial of degree 15 through the nodes.  In
    FP32 are its terms from the fourth on, 2 (1 + n) 14^-n of the mean, off by n^2 2^-24 of themselves at most
    (n^2 from the rounded argument): 4e-10 in all, so 1e-9."""
    from korg_gb300 import synthetic
    inp = _inputs(14, 5000, 5006, 300, wl=(5000.0, 5001.27))
    assert len(inp.wls) == 128
    ll = synthetic.synthetic_linelist(9000, 5005.1, 5006, seed=1, molecular=True)
    ll.gamma_rad[:] = 1e7
    a, n = _lines_only(gpu_lib, inp, ll, cutoff=1e-20)
    assert n == 9000
    w = inp.wls.all_wls
    V = np.polynomial.chebyshev.chebvander((w - w[0]) / (0.5 * (w[-1] - w[0])) - 1, 15)
    fit = V @ np.linalg.lstsq(V, a, rcond=None)[0]
    assert np.max(np.abs(a / fit - 1)) <= 1e-9


def test_sparse_tiles_of_an_unsorted_list(gpu_lib):
    """Forty lines below 5100 A and 14,000 weak ones above 5150 A, which come in reverse: for an unsorted
    list the candidate runs are whole tiers, more than the limit for far lines, but the tiles below 5100 A are as
    sparse as before.  Their lines stand first in the list, in one chunk of candidates and one batch either way:
    the same terms in the same order, so the same bits."""
    from korg_gb300 import synthetic
    inp = _inputs(14, 5000, 5200, 300)
    few = synthetic.synthetic_linelist(40, 5005, 5090, seed=2, loggf=(-3.0, -1.0))
    many = synthetic.synthetic_linelist(14000, 5150, 5199, seed=3, loggf=(-6.0, -5.0), molecular=True)
    ll = few.concat(many)
    order = np.arange(len(ll))
    order[40:] = order[:39:-1]
    (a, n), (b, _) = _lines_only(gpu_lib, inp, ll), _lines_only(gpu_lib, inp, ll.subset(order))
    assert n >= 8192 + 40 and np.all(a[:10001].max(axis=0) > 0)
    assert np.array_equal(a[:10001], b[:10001])
    np.testing.assert_allclose(b, a, rtol=1e-5, atol=0)
