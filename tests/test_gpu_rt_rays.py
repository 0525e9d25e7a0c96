"""The one-pass ray kernel (anchored optical depth, linear and flux-only solutions) against the FP64
oracle: columns around its 32-column blocks, rays that reach the bottom, stop at some layer or touch one
layer only, inward rays on all rays, and opacities that end a ray early."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nwl", [1, 31, 32, 33, 100])
@pytest.mark.parametrize("R", [None, 7e10, 3e8])
@pytest.mark.parametrize("I_scheme", [0, 1])
@pytest.mark.parametrize("inward", [0, 1])
def test_rays_match_oracle(gpu_lib, oracle_lib, nwl, R, I_scheme, inward):
    L, n_mu = 56, 9
    rng = np.random.default_rng(nwl)
    tau_ref = 10.0 ** np.linspace(-5, 2, L)
    z = np.linspace(2e7, -8e7, L)
    ref = np.exp(np.linspace(-20, -12, L))
    alpha = np.ascontiguousarray(ref * 10.0 ** rng.uniform(-1, 3, (nwl, 1)))
    S = np.ascontiguousarray(np.linspace(1.0, 30.0, L) * rng.uniform(0.9, 1.1, (nwl, L)))
    spatial = z if R is None else R + z
    mu, w = np.polynomial.legendre.leggauss(n_mu)
    mu, w = mu / 2 + 0.5, w / 2
    want = oracle_lib.rt_general(alpha, S, spatial, R is not None, tau_ref, ref, mu, w, bool(inward), 0, I_scheme)
    ctx = gpu_lib.default_context()
    F, I = np.empty(nwl), np.empty((n_mu, nwl))
    keep = [np.ascontiguousarray(a, np.float64) for a in (alpha, S, spatial, tau_ref, ref, mu, w, F, I)]
    p = [a.ctypes.data_as(C.POINTER(C.c_double)) for a in keep]
    ctx.check(ctx.lib.korg_radiative_transfer_general(ctx.h, p[0], p[1], L, nwl, p[2], int(R is not None), p[3], p[4],
                                                      p[5], p[6], n_mu, inward, 0, I_scheme, p[7], p[8]))
    np.testing.assert_allclose(keep[7], want, rtol=1e-9, atol=0)  # the other schemes' tolerance
