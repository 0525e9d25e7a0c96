"""Rotation in blocks: the kernel integrals' quartics and their direct evaluation, on both sides of the
sizes where the kernels change course (block and chunk edges, one to seventeen spectra, windows wider
than a chunk and wider than the grid, ranges of 1 to 65 points), against the FP64 restatement."""
import functools

import numpy as np
import pytest

import postprocess_oracle as po
from korg_gb300.wavelengths import Wavelengths

pytestmark = pytest.mark.gpu

GRIDS = [[(5000, 5000.63, 0.01)], [(5000, 5000.64, 0.01)], [(5000, 5003.2, 0.01), (5003.5, 5003.5, 0.01)],
         [(15000, 15001, 0.005), (15001.5, 15001.8, 0.01)], [(5000, 5120, 1.0)]]


@functools.lru_cache(maxsize=None)
def _matrix(k, vsini):
    g = Wavelengths(GRIDS[k] if len(GRIDS[k]) > 1 else GRIDS[k][0])
    return g, np.stack([po.apply_rotation(e, g.all_wls, g.ranges, vsini, 0.6) for e in np.eye(len(g))], axis=1)


@pytest.mark.parametrize("k", range(len(GRIDS)))
@pytest.mark.parametrize("vsini", [3.0, 40.0, 300.0])
@pytest.mark.parametrize("nspec", [1, 3, 17])
def test_rotation_and_its_transpose(gpu_lib, k, vsini, nspec):
    """Sums of at most a few thousand weights that are differences of integrals rounded at 1e-16:
    1e-11 relative, as the restatement's own comparison asks, and 1e-12 absolute for values of order 1."""
    torch = pytest.importorskip("torch")
    from korg_gb300.postprocess import Rotation
    g, M = _matrix(k, vsini)
    n = len(g)
    rng = np.random.default_rng(n + nspec)
    f, y = rng.random((nspec, n)), rng.standard_normal((nspec, n))
    dev = torch.device("cuda", 0)
    tf = torch.as_tensor(f, device=dev).requires_grad_(True)
    z = Rotation.apply(tf, torch.as_tensor(g.all_wls, device=dev), g, vsini, 0.6)
    z.backward(torch.as_tensor(y, device=dev))
    np.testing.assert_allclose(z.detach().cpu().numpy(), f @ M.T, rtol=1e-11, atol=1e-12)
    np.testing.assert_allclose(tf.grad.cpu().numpy(), y @ M, rtol=1e-11, atol=1e-12)
