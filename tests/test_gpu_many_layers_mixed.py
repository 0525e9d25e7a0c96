"""Mixed line opacity of 225 to 256 layers, for lists whose prologue blocks hold one warp and all eight: its
boundaries of 256 padded layers a warp, beside the kernel's own tables, go above 48 KB there."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", [224, 225, 256])
@pytest.mark.parametrize("n", [20, 80000])
def test_mixed_lines_of_many_layers(gpu_lib, L, n):
    """Against FP64, at the mixed opacity's own tolerance (99.9 % within 1e-5, seams of the branches 1e-2)."""
    from korg_gb300 import line_absorption_, synthetic
    from korg_gb300.api import ContinuumInterpolant
    from korg_gb300.data import default_partition_funcs
    w = synthetic.Workload("deep", 4500.0, 4.4, 0.0, L, (5000.0, 5000.63), synthetic.synthetic_linelist(n, 4998, 5003, seed=n))
    inp = synthetic.prepare(w, continuum="gpu", chemistry="gpu")
    out = {}
    for precision in ("mixed", "fp64"):
        out[precision] = np.zeros((len(inp.wls), L))
        ctx = gpu_lib.Context(0)
        line_absorption_(out[precision], inp.linelist, inp.wls, inp.T, inp.ne, inp.number_densities,
                         default_partition_funcs(), inp.xi, ContinuumInterpolant(inp.cntm_knots, inp.cntm_vals),
                         precision=precision, ctx=ctx)
        ctx.close()
    ok = out["fp64"] > 0
    rel = np.abs(out["mixed"][ok] / out["fp64"][ok] - 1)
    assert np.percentile(rel, 99.9) <= 1e-5 and rel.max() <= 1e-2
