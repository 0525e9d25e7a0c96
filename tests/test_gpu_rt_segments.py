"""The planar transfer's continuum series per knot interval and Planck series per block against the
FP64 oracle: grids with and without enough points per interval, blocks that straddle knots, an
ionisation edge (Balmer, Paschen), a gap, coarse grids whose blocks span too much for the series, and
both block sizes."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 1

GRIDS = [((5000, 5020), 1.0), ((5000, 5003), 1.0), ((3640, 3655), 1.0), ((8195, 8215), 1.0), ((5000, 5020), 7.0),
         ([(5000, 5010), (5060, 5070)], 1.0), ((4000, 9000, 5.0), 1.0), ((4000, 9000, 5.0), 200.0),
         ((15000, 15250, 0.005), 1.0)]


@pytest.mark.parametrize("teff", [4200.0, 6500.0])
@pytest.mark.parametrize("wls,step", GRIDS)
def test_continuum_and_flux_match_oracle(gpu_lib, oracle_lib, wls, step, teff):
    """Both transfers to 1e-12 of the oracle, as the transfer's own parity test asks (no lines but three
    weak ones, so that the flux is a transfer of its own)."""
    from korg_gb300 import synthetic
    from korg_gb300.api import synthesize_prepared
    from korg_gb300.data import stark_profiles
    lo = wls[0][0] if isinstance(wls, list) else wls[0]
    w = synthetic.Workload("rt", teff, 4.0, 0.0, 56, wls, synthetic.synthetic_linelist(3, lo, lo + 3, seed=1))
    w.hydrogen_lines = False
    inp = synthetic.prepare(w, cntm_step=step)
    flux, cntm, _, _, _ = oracle_lib.synthesize(inp, inp.linelist, inp.linelist5, stark_profiles(), inp.wls.all_wls,
                                                nthreads=NT)
    ctx = gpu_lib.Context(0)
    r = synthesize_prepared(inp, precision="fp64", ctx=ctx)
    ctx.close()
    np.testing.assert_allclose(r.cntm, cntm, rtol=1e-12, atol=0)
    np.testing.assert_allclose(r.flux, flux, rtol=1e-12, atol=0)
