"""The planar transfer of long grids (a thread per column) against the FP64 oracle: blocks that span too much
for the Planck series, a gap between ranges inside a block, a fine grid across the Balmer edge, and one
column more than a block boundary."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 1


@pytest.mark.parametrize("teff", [4200.0, 6500.0])
@pytest.mark.parametrize("wls", [(3000, 10000, 0.1), [(5000, 5120.37), (5180, 5300)], (3635, 3660, 0.001),
                                 (5000, 5204.8)])
def test_continuum_and_flux_of_long_grids(gpu_lib, oracle_lib, wls, teff):
    """Both transfers to 1e-12 of the oracle, as the transfer's own parity test asks (three weak lines only)."""
    from korg_gb300 import synthetic
    from korg_gb300.api import synthesize_prepared
    from korg_gb300.data import stark_profiles
    lo = wls[0][0] if isinstance(wls, list) else wls[0]
    w = synthetic.Workload("rt", teff, 4.0, 0.0, 56, wls, synthetic.synthetic_linelist(3, lo, lo + 3, seed=1))
    w.hydrogen_lines = False
    inp = synthetic.prepare(w)
    assert len(inp.wls) > 20000
    flux, cntm, _, _, _ = oracle_lib.synthesize(inp, inp.linelist, inp.linelist5, stark_profiles(), inp.wls.all_wls,
                                                nthreads=NT)
    ctx = gpu_lib.Context(0)
    r = synthesize_prepared(inp, precision="fp64", ctx=ctx)
    ctx.close()
    np.testing.assert_allclose(r.cntm, cntm, rtol=1e-12, atol=0)
    np.testing.assert_allclose(r.flux, flux, rtol=1e-12, atol=0)
