"""Transfers of many layers, on both sides of the layer counts where the Planck rows (597), the continuum
intervals (1,329) and the warp-per-column form (1,775) no longer fit the shared memory, up to the 1,790
that every form of the call takes, against the FP64 oracle."""
import ctypes as C
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 1


@pytest.mark.parametrize("hi", [5010.0, 5300.0])
@pytest.mark.parametrize("L", [597, 598, 1329, 1330, 1775, 1776, 1790])
def test_transfers_of_many_layers(gpu_lib, oracle_lib, L, hi):
    """A synthesis without any lines, whose layer count only the transfer bounds (flux and continuum are the same
    transfer then), and the transfer of its opacity with the Planck function as a given source: 1,001 columns go
    by warps, 30,001 by threads.  The transfer's own parity tolerance, 1e-12, of ten times the layers."""
    import dataclasses
    from korg_gb300 import synthetic
    from korg_gb300.api import synthesize_prepared
    from korg_gb300.data import stark_profiles
    w = synthetic.Workload("deep", 5200.0, 4.0, 0.0, 56, (5000.0, hi), synthetic.synthetic_linelist(3, 5000, 5003, seed=1))
    w.hydrogen_lines = False
    inp = synthetic.prepare(w)
    none = inp.linelist.subset(np.arange(0))
    x, x0 = np.linspace(0, 55, L), np.arange(56.0)
    f = lambda a: np.exp(np.interp(x, x0, np.log(a)))
    r = lambda a: np.stack([np.interp(x, x0, row) for row in np.atleast_2d(a)])
    deep = dataclasses.replace(
        inp, linelist=none, linelist5=none, T=f(inp.T), ne=f(inp.ne), tau_ref=f(inp.tau_ref), xi=f(inp.xi),
        n_eff_vdW=f(inp.n_eff_vdW), n_div_U=r(inp.n_div_U), nH_I=f(inp.nH_I), nHe_I=f(inp.nHe_I), UH_I=f(inp.UH_I),
        alpha_ref_cntm=f(inp.alpha_ref_cntm), cntm_vals=np.exp(r(np.log(inp.cntm_vals.T)).T))
    wl = deep.wls.all_wls
    flux, cntm, alpha, _, _ = oracle_lib.synthesize(deep, none, none, stark_profiles(), wl, nthreads=NT)
    ctx = gpu_lib.Context(0)
    out = synthesize_prepared(deep, precision="fp64", ctx=ctx)
    np.testing.assert_allclose(out.flux, flux, rtol=1e-11, atol=0)
    np.testing.assert_allclose(out.cntm, cntm, rtol=1e-11, atol=0)
    S = 2 * 6.62607015e-27 * 2.99792458e10 ** 2 / wl[:, None] ** 5 / np.expm1(1.43877687750393 / (wl[:, None] * deep.T))
    F = np.full(len(wl), np.nan)
    keep = [np.ascontiguousarray(a, np.float64) for a in (alpha, S, deep.tau_ref, deep.alpha_ref_cntm)]
    p = lambda a: a.ctypes.data_as(C.POINTER(C.c_double))
    ctx.check(ctx.lib.korg_radiative_transfer(ctx.h, p(keep[0]), p(keep[1]), L, len(wl), p(keep[2]), p(keep[3]), p(F)))
    ctx.close()
    np.testing.assert_allclose(F, oracle_lib.rt_flux_expint(*keep, NT), rtol=1e-11, atol=0)
