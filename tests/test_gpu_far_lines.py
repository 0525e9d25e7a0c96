"""Far lines of the line tiles (evaluated at 16 Chebyshev nodes per tile and interpolated) against the
FP64 oracle, at the sizes where the split can go wrong: tiles cut short by the grid's end, every
layers-per-group template, other tile widths, a non-uniform grid with a gap, and mixed tiles above the
candidate limit."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NT = os.cpu_count() or 1


def _inputs(L, lo, hi, n, teff=5000.0):
    from korg_gb300 import synthetic
    w = synthetic.Workload("far", teff, 4.4, 0.0, L, (lo, hi), synthetic.synthetic_linelist(n, lo, hi, seed=n))
    return synthetic.prepare(w)


def _opacity(gpu_lib, oracle_lib, inp, wls, precision, tile=None):
    from korg_gb300 import Wavelengths, line_absorption_
    from korg_gb300.api import ContinuumInterpolant, _prec
    from korg_gb300.data import default_partition_funcs
    ctx = gpu_lib.Context(0)
    if tile:
        ctx.check(ctx.lib.korg_set_tile_config(ctx.h, len(inp.T), _prec(precision), *tile))
    a0 = np.stack([np.interp(wls, inp.cntm_knots, v) for v in inp.cntm_vals], axis=1)
    got, ref = a0.copy(), a0.copy()
    n = line_absorption_(got, inp.linelist, Wavelengths.from_array(wls), inp.T, inp.ne, inp.number_densities,
                         default_partition_funcs(), inp.xi, ContinuumInterpolant(inp.cntm_knots, inp.cntm_vals),
                         precision=precision, ctx=ctx)
    ctx.close()
    n_ref = oracle_lib.line_absorption(ref, inp.linelist, wls, inp.T, inp.ne, inp.n_eff_vdW, inp.xi, inp.n_div_U,
                                       inp.cntm_knots, inp.cntm_vals, cutoff=3e-4, nthreads=NT)
    assert n == n_ref
    return got, ref


@pytest.mark.parametrize("L,tile", [(56, None), (56, (64, 0, 1)), (56, (96, 0, 0)), (56, (128, 169, 1)), (80, None), (130, None)])
@pytest.mark.parametrize("extra", [0, 1, 63, 64, 65, 127])
def test_fp64_far_lines_match_oracle(gpu_lib, oracle_lib, L, tile, extra):
    """The sum of a few hundred positive terms and the 16-node series both round at 1e-15 each: 1e-12."""
    if (L != 56 or tile) and extra not in (1, 64):
        pytest.skip("the remainders are covered at 56 layers")
    inp = _inputs(L, 5000, 5010, 400)
    wls = inp.wls.all_wls[:512 + extra] if extra else inp.wls.all_wls[:512]
    got, ref = _opacity(gpu_lib, oracle_lib, inp, wls, "fp64", tile)
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=0)


@pytest.mark.parametrize("lo,hi", [(7.0, 9.0), (9.5, 11.5), (8.0, 12.5)])
def test_fp64_profile_branches_match_oracle(gpu_lib, oracle_lib, lo, hi):
    """Damping from a = 1e-4 to some 30, so that every branch of the Hjerting function and both far
    series occur; each term is a few roundings of positive factors: 1e-12."""
    inp = _inputs(56, 5000, 5010, 120)
    inp.linelist.gamma_rad[:] = 10.0 ** np.random.default_rng(3).uniform(lo, hi, 120)
    got, ref = _opacity(gpu_lib, oracle_lib, inp, inp.wls.all_wls[:700], "fp64")
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=0)


@pytest.mark.parametrize("L", [33, 51, 56, 64, 80])
@pytest.mark.parametrize("n", [641, 5057])
def test_fp64_parts_of_groups_match_whole_groups(gpu_lib, oracle_lib, L, n):
    """The first n points of a grid long enough for whole layer groups per CTA, and by themselves in parts
    of groups (2 layers or half; of 33 and 51 layers the last ones are padding): the same terms, in the
    order of their tiers, which the grid's end may change: 1e-13."""
    inp = _inputs(L, 5000, 5270, 2000)
    wls = inp.wls.all_wls
    assert (len(wls) + 127) // 128 * ((L + 15) // 16) >= 4 * 152
    whole, _ = _opacity(gpu_lib, oracle_lib, inp, wls, "fp64")
    part, ref = _opacity(gpu_lib, oracle_lib, inp, wls[:n], "fp64")
    np.testing.assert_allclose(part, ref, rtol=1e-12, atol=0)
    np.testing.assert_allclose(part[:n // 128 * 128], whole[:n // 128 * 128], rtol=1e-13, atol=0)


def test_fp64_far_lines_on_an_uneven_grid(gpu_lib, oracle_lib):
    """Steps that grow along the grid, repeated wavelengths and a 20 A gap inside a tile."""
    inp = _inputs(56, 5000, 5040, 800)
    d = np.concatenate([np.full(300, 0.004), np.linspace(0.002, 0.03, 300), [0.0, 0.0, 20.0], np.full(300, 0.01)])
    wls = (5002.0 + np.cumsum(d)) * 1e-8
    got, ref = _opacity(gpu_lib, oracle_lib, inp, wls, "fp64")
    np.testing.assert_allclose(got, ref, rtol=1e-12, atol=0)


@pytest.mark.parametrize("L", [56, 80, 130])
def test_mixed_far_lines_match_oracle(gpu_lib, oracle_lib, L):
    """FP32 evaluations (a few 1e-7 each) of lines whose sum is dominated by no single one; the seams
    of the Hjerting branches are the exceptions."""
    inp = _inputs(L, 5000, 5020, 20000, teff=4500.0)
    wls = inp.wls.all_wls[:1000 + 65]
    got, ref = _opacity(gpu_lib, oracle_lib, inp, wls, "mixed")
    rel = np.abs(got / ref - 1)
    assert np.percentile(rel, 99.9) <= 2e-6 and rel.max() <= 1e-3


@pytest.mark.parametrize("L", [56, 80, 130])
def test_mixed_far_lines_of_a_batch(gpu_lib, L):
    """A batch's far lines (a launch over spectra, one of them sparse) against single spectra's: FP32
    roundings of 6e-8 of the far opacity move the flux by less than 1e-7 of it."""
    from korg_gb300.batch import BatchSynthesis
    from korg_gb300.api import synthesize_prepared
    inps = [_inputs(L, 5000, 5020, n, teff=4500.0) for n in (20000, 300)]
    b = BatchSynthesis(inps, precision="mixed", use_graph=False)
    b.run()
    f, c = b.results()
    for i, inp in enumerate(inps):
        r = synthesize_prepared(inp, precision="mixed")
        np.testing.assert_allclose(f[i], r.flux, rtol=1e-7, atol=0)
        np.testing.assert_allclose(c[i], r.cntm, rtol=1e-12, atol=0)
