"""Rotation on both sides of the lines between its forms (3 and 10 points in half a window, a step of 5e-6 of the
wavelength), one to seventeen spectra, against the FP64 restatement: both forms are the same map."""
import functools

import numpy as np
import pytest

import postprocess_oracle as po
from korg_gb300.wavelengths import Wavelengths

pytestmark = pytest.mark.gpu

C = 299792.458
# grid, points in half the window at the grid's end
CASES = [((5000, 5003, 0.01), m) for m in (0.4, 1.5, 2.99, 3.01, 9.99, 10.01)] + \
        [((5000, 5008, 0.02499), 12.0), ((5000, 5008, 0.02501), 12.0), ([(5000, 5001, 0.01), (5002, 5012, 0.1)], 20.0),
         ((15000, 15001, 0.005), 10.01), ((5000, 5300, 1.0), 2.0), ((5000, 5300, 1.0), 4.0)]


@functools.lru_cache(maxsize=None)
def _case(k):
    g = Wavelengths(CASES[k][0])
    vsini = max(CASES[k][1] * C / (start / step + n - 1) for start, step, n in g.ranges[:1])
    return g, vsini, np.stack([po.apply_rotation(e, g.all_wls, g.ranges, vsini, 0.6) for e in np.eye(len(g))], axis=1)


@pytest.mark.parametrize("k", range(len(CASES)))
@pytest.mark.parametrize("nspec", [1, 5, 17])
def test_rotation_and_its_transpose(gpu_lib, k, nspec):
    """At most 40 weights a point, differences of integrals rounded at 1e-16: 1e-11 relative, as the
    restatement's own comparison asks, and 1e-12 absolute for values of order 1."""
    torch = pytest.importorskip("torch")
    from korg_gb300.postprocess import Rotation
    g, vsini, M = _case(k)
    rng = np.random.default_rng(k + nspec)
    f, y = rng.random((nspec, len(g))), rng.standard_normal((nspec, len(g)))
    dev = torch.device("cuda", 0)
    tf = torch.as_tensor(f, device=dev).requires_grad_(True)
    z = Rotation.apply(tf, torch.as_tensor(g.all_wls, device=dev), g, vsini, 0.6)
    z.backward(torch.as_tensor(y, device=dev))
    np.testing.assert_allclose(z.detach().cpu().numpy(), f @ M.T, rtol=1e-11, atol=1e-12)
    np.testing.assert_allclose(tf.grad.cpu().numpy(), y @ M, rtol=1e-11, atol=1e-12)
