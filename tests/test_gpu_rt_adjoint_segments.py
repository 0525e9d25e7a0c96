"""The reverse transfer's continuum pass at the nodes of the knot intervals against the same cotangents
taken in pieces of the grid too short for that (each column by itself)."""
import copy

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
FIELDS = ("T", "cntm_vals", "alpha_ref_cntm", "log_gf")


@pytest.mark.parametrize("special", [None, np.inf, np.nan])
@pytest.mark.parametrize("wls,L", [((5000, 5020), 56), ((5000, 5020), 128), ((3640, 3655), 56), ((8195, 8215), 33)])
def test_node_pass_matches_column_passes(gpu_lib, wls, L, special):
    """FP64 sums of the same terms in another order, and series of 8 nodes good to 1e-16: 1e-11 of the
    largest.  (3640-3655 A holds the Balmer edge: intervals that are no series.)"""
    from korg_gb300 import Wavelengths, synthetic
    from korg_gb300.api import synthesize_vjp
    w = synthetic.Workload("rta", 5000.0, 4.0, 0.0, L, (*wls, 0.002), synthetic.synthetic_linelist(3, wls[0], wls[0] + 3, seed=1))
    w.hydrogen_lines = False
    inp = synthetic.prepare(w)
    n, limit = len(inp.wls.all_wls), 16 * (len(inp.cntm_knots) - 1)
    piece = 250
    assert n >= limit > piece and n > 152 * 8 * 4
    rng = np.random.default_rng(2)
    dF, dC = rng.normal(size=n), rng.normal(size=n)
    if special is not None:
        dC[n // 2 + 7] = special
    ctx = gpu_lib.Context(0)
    got = synthesize_vjp(inp, dF, dC, hydrogen=False, ctx=ctx)
    ref = None
    for i in range(0, n, piece):
        part = copy.copy(inp)
        part.wls = Wavelengths.from_array(inp.wls.all_wls[i:i + piece])
        g = synthesize_vjp(part, dF[i:i + piece], dC[i:i + piece], hydrogen=False, ctx=ctx)
        ref = {k: g[k] + (ref[k] if ref else 0.0) for k in FIELDS}
    ctx.close()
    for k in FIELDS:
        scale = np.max(np.abs(ref[k][np.isfinite(ref[k])]), initial=0.0)
        np.testing.assert_allclose(got[k], ref[k], rtol=0, atol=1e-11 * scale, err_msg=k)
