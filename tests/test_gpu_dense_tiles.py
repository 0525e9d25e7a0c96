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


@pytest.mark.parametrize("n,hi", [(20000, 5020.0), (9000, 5120.0)])
@pytest.mark.parametrize("L", [56, 72])
def test_batch_gradient_of_dense_tiles(gpu_lib, L, n, hi):
    """Above the limit (20,000 lines on 20 A) and a long list whose tiles are below it: a batch's gradient that
    reuses its forward equals the recomputed one and the single spectrum's, as for short lists (1e-9), and the
    mixed gradient lies as near to FP64's as the mixed reverse mode's own comparison asks (2e-3)."""
    from korg_gb300.api import GRAD_FIELDS, synthesize_vjp
    from korg_gb300.batch import BatchSynthesis
    inps = [_inputs(L, 5000, hi, k) for k in (n, 300)]
    b = BatchSynthesis(inps, precision="mixed", use_graph=False)
    rng = np.random.default_rng(3)
    dF, dC = (b.torch.as_tensor(rng.normal(size=(len(inps), b.nwl)), device=b.dev) for _ in range(2))
    b.run()
    got = {"reuse": b.vjp(dF, dC, reuse_forward=True)}
    b.torch.cuda.synchronize()
    got = {k: [{f: v.cpu().numpy() for f, v in g.items()} for g in gs] for k, gs in got.items()}
    got["again"] = [{f: v.cpu().numpy() for f, v in g.items()} for g in b.vjp(dF, dC, reuse_forward=True)]
    got["recompute"] = [{f: v.cpu().numpy() for f, v in g.items()} for g in b.vjp(dF, dC, reuse_forward=False)]
    for k, inp in enumerate(inps):
        args = (inp, dF[k].cpu().numpy(), dC[k].cpu().numpy())
        ref, ref64 = (synthesize_vjp(*args, precision=p, ctx=b.ctx) for p in ("mixed", "fp64"))
        for f in GRAD_FIELDS:
            scale = max(float(np.max(np.abs(ref[f]))), 1e-300)
            for name, g in got.items():
                assert np.max(np.abs(g[k][f].reshape(ref[f].shape) - ref[f])) <= 1e-9 * scale, (k, f, name)
            assert np.max(np.abs(ref[f] - ref64[f])) <= 2e-3 * np.max(np.abs(ref64[f])), (k, f)


@pytest.mark.parametrize("hydrogen", [True, False])
@pytest.mark.parametrize("tw", [None, 64, 256])
def test_gradient_reusing_a_dense_forward(gpu_lib, hydrogen, tw):
    """The single spectrum's reuse against its recomputation, element by element as for short lists, at the
    default and other tile widths, and when the width changes between the forward and its reuse."""
    from korg_gb300.api import rectified_loss, synthesize_prepared, synthesize_vjp
    ctx = gpu_lib.Context(0)
    inp = _inputs(56, 5000, 5020, 20000)
    inp.hydrogen_lines = hydrogen
    shape = lambda w: ctx.check(ctx.lib.korg_set_tile_config(ctx.h, 56, gpu_lib.KORG_MIXED, w, 0, 1))
    if tw:
        shape(tw)
    r = synthesize_prepared(inp, precision="mixed", ctx=ctx)
    obs = r.flux / r.cntm * (1 + 0.01 * np.random.default_rng(5).standard_normal(len(r.flux)))
    _, dF, dC = rectified_loss(r.flux, r.cntm, obs)
    kw = dict(precision="mixed", ctx=ctx)
    want = synthesize_vjp(inp, dF, dC, **kw)
    synthesize_prepared(inp, precision="mixed", ctx=ctx)
    got = synthesize_vjp(inp, dF, dC, reuse_forward=True, **kw)
    for k in want:
        np.testing.assert_allclose(got[k], want[k], rtol=1e-9, atol=1e-14 * np.max(np.abs(want[k])) + 1e-300)
    if tw:  # another width moves the roundings of single terms, but leaves no far lines behind
        synthesize_prepared(inp, precision="mixed", ctx=ctx)
        shape(128)
        got = synthesize_vjp(inp, dF, dC, reuse_forward=True, **kw)
        for k in want:
            np.testing.assert_allclose(got[k], want[k], rtol=1e-9, atol=1e-14 * np.max(np.abs(want[k])) + 1e-300)
    ctx.close()


def test_reuse_after_a_batch_size_that_only_the_new_width_takes(gpu_lib):
    """Forward at 256 wavelengths a tile, then a shape of 64 whose batches of 510 lines would not fit 256: the
    reuse goes by the forward's width and the default batches, as the forward did."""
    from korg_gb300.api import synthesize_prepared, synthesize_vjp
    ctx = gpu_lib.Context(0)
    inp = _inputs(56, 5000, 5010, 12000)
    inp.hydrogen_lines = False
    shape = lambda *s: ctx.check(ctx.lib.korg_set_tile_config(ctx.h, 56, gpu_lib.KORG_MIXED, *s))
    shape(256, 0, 1)
    dF = np.random.default_rng(1).standard_normal(len(inp.wls))
    want = synthesize_vjp(inp, dF, precision="mixed", ctx=ctx)
    synthesize_prepared(inp, precision="mixed", ctx=ctx)
    assert ctx.lib.korg_set_tile_config(ctx.h, 56, gpu_lib.KORG_MIXED, 256, 510, 1) == 1
    shape(64, 510, 1)
    got = synthesize_vjp(inp, dF, precision="mixed", reuse_forward=True, ctx=ctx)
    ctx.close()
    for k in want:
        np.testing.assert_allclose(got[k], want[k], rtol=1e-9, atol=1e-14 * np.max(np.abs(want[k])) + 1e-300)
