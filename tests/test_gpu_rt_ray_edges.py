"""The one-pass ray kernel at its limits: layer counts whose columns need more than 48 KB, the most rays, the
surface intensity of every ray, segments without optical depth, layers that are not finite, and columns
that do not depend on their neighbours."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MU = {m: tuple(a / 2 + b for a, b in zip(np.polynomial.legendre.leggauss(m), (0.5, 0.0))) for m in (1, 9, 32, 64)}


def _atmosphere(L, nwl, seed=0):
    rng = np.random.default_rng(seed)
    ref = np.exp(np.linspace(-20, -12, L))
    alpha = np.ascontiguousarray(ref * 10.0 ** rng.uniform(-1, 3, (nwl, 1)))
    S = np.ascontiguousarray(np.linspace(1.0, 30.0, L) * rng.uniform(0.9, 1.1, (nwl, L)))
    return alpha, S, np.linspace(2e7, -8e7, L), 10.0 ** np.linspace(-5, 2, L), ref


def _rays(gpu_lib, alpha, S, spatial, spherical, tau, ref, mu_w, inward, scheme):
    nwl, L = alpha.shape
    mu, w = mu_w
    n_mu = len(mu)
    F, I = np.full(nwl, np.nan), np.full((n_mu, nwl), np.nan)
    ctx = gpu_lib.default_context()
    keep = [np.ascontiguousarray(a, np.float64) for a in (alpha, S, spatial, tau, ref, mu, w, F, I)]
    p = [a.ctypes.data_as(C.POINTER(C.c_double)) for a in keep]
    ctx.check(ctx.lib.korg_radiative_transfer_general(ctx.h, p[0], p[1], L, nwl, p[2], int(spherical), p[3], p[4], p[5],
                                                      p[6], n_mu, int(inward), 0, scheme, p[7], p[8]))
    return keep[7], keep[8]


@pytest.mark.parametrize("L,n_mu,inward", [(2, 1, False), (89, 9, True), (90, 9, True), (128, 32, True), (128, 64, False)])
@pytest.mark.parametrize("nwl", [1, 31, 33])
@pytest.mark.parametrize("scheme", [0, 1])
def test_intensity_of_every_ray(gpu_lib, L, n_mu, inward, nwl, scheme):
    """Each ray's intensity is that of a call with this ray alone, whose flux is 2 pi mu of it, and the flux is
    their sum (a few roundings).  64 rays leave no room for inward ones: planar."""
    alpha, S, z, tau, ref = _atmosphere(L, nwl, L + nwl)
    shell = n_mu < 64
    z = z + 7e10 * shell
    F, I = _rays(gpu_lib, alpha, S, z, shell, tau, ref, MU[n_mu], inward, scheme)
    mu, w = MU[n_mu]
    for u in range(n_mu):
        one, _ = _rays(gpu_lib, alpha, S, z, shell, tau, ref, (mu[u:u + 1], np.ones(1)), inward, scheme)
        np.testing.assert_allclose(I[u], one / (2 * np.pi * mu[u]), rtol=1e-14, atol=0)
    np.testing.assert_allclose(F, 2 * np.pi * (I.T @ (w * mu)), rtol=1e-12)


def test_segments_without_optical_depth(gpu_lib, oracle_lib):
    """Layers without opacity: the flux-only form takes the slope over 1, the linear one is not a number."""
    alpha, S, z, tau, ref = _atmosphere(56, 40)
    alpha[:, 10:14] = 0.0
    F, _ = _rays(gpu_lib, alpha, S, z, False, tau, ref, MU[9], False, 1)
    want = oracle_lib.rt_general(alpha, S, z, False, tau, ref, *MU[9], False, 0, 1)
    np.testing.assert_allclose(F, want, rtol=1e-9)
    F, _ = _rays(gpu_lib, alpha, S, z, False, tau, ref, MU[9], False, 0)
    assert np.all(np.isnan(F))


@pytest.mark.parametrize("inward", [False, True])
@pytest.mark.parametrize("scheme", [0, 1])
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("layer", [3, 55])
def test_layers_that_are_not_finite(gpu_lib, oracle_lib, inward, scheme, bad, layer):
    """An opacity or source value that is not finite, above or far below the depth where rays end (all do by then
    at 700): the flux is a number where the oracle's is (the flux-only form with an infinitely opaque last
    layer), else it is not, and the other columns keep their bits."""
    alpha, S, z, tau, ref = _atmosphere(56, 40)
    alpha *= 700.0
    clean = _rays(gpu_lib, alpha, S, 7e10 + z, True, tau, ref, MU[9], inward, scheme)
    alpha[5, layer], S[17, layer] = bad, bad
    F, I = _rays(gpu_lib, alpha, S, 7e10 + z, True, tau, ref, MU[9], inward, scheme)
    with np.errstate(all="ignore"):
        want = oracle_lib.rt_general(alpha, S, 7e10 + z, True, tau, ref, *MU[9], inward, 0, scheme)
    np.testing.assert_allclose(F, want, rtol=1e-9, atol=0, equal_nan=True)
    ok = ~np.isin(np.arange(40), (5, 17))
    assert np.array_equal(F[ok], clean[0][ok]) and np.array_equal(I[:, ok], clean[1][:, ok])


@pytest.mark.parametrize("inward", [False, True])
def test_columns_do_not_depend_on_each_other(gpu_lib, inward):
    """An opaque column among transparent ones, whose rays go on below its end, with a source function that
    would show what lies there: the same bits as by itself."""
    L = 56
    alpha, _, z, tau, ref = _atmosphere(L, 40)
    alpha = np.tile(ref * 1e-3, (40, 1))
    alpha[7] = ref * 1e3
    S = np.tile(10.0 ** np.linspace(0, 25, L), (40, 1))
    F, I = _rays(gpu_lib, alpha, S, 7e10 + z, True, tau, ref, MU[9], inward, 0)
    F1, I1 = _rays(gpu_lib, alpha[7:8], S[7:8], 7e10 + z, True, tau, ref, MU[9], inward, 0)
    assert F[7] == F1[0] and np.array_equal(I[:, 7], I1[:, 0])


def _long_double(alpha, S, z, shell, tau, ref, mu, inward, scheme):
    """Surface intensities by the same formulas in extended precision (RadiativeTransfer.jl:92-139, 244-324)."""
    LD, out = np.longdouble, []
    for u in mu:
        n, ds = len(z), np.full(len(z), 1 / u)
        if shell:
            b = z[0] * np.sqrt(1 - u * u)
            if b >= z[-1]:
                n = int(np.argmin(np.abs(z - b)))
                n = n if z[n] < b else n + 1
            ds = z[:n] / np.sqrt(z[:n] ** 2 - b * b)
        ib = alpha[:, :n].astype(LD) * (tau[:n] / ref[:n] * ds).astype(LD)
        d = LD(0.5) * (ib[:, 1:] + ib[:, :-1]) * np.diff(np.log(tau[:n])).astype(LD)
        e, Sx = np.exp(-d), S[:, :n].astype(LD)
        m = np.diff(Sx, axis=1) / d
        T, up, down = np.ones(len(S), LD), np.zeros(len(S), LD), np.zeros(len(S), LD)
        for k in range(n - 1):
            up += T * (Sx[:, k] + m[:, k] - e[:, k] * (Sx[:, k + 1] + m[:, k]))
            down = e[:, k] * down + Sx[:, k + 1] - m[:, k] - e[:, k] * (Sx[:, k] - m[:, k])
            T = T * e[:, k]
        out.append(up + T * down if inward or n < len(z) else up)
    return np.array(out, np.float64)


@pytest.mark.parametrize("seed", range(8))
@pytest.mark.parametrize("shell", [False, True])
@pytest.mark.parametrize("scheme", [0, 1])
def test_intensities_where_slopes_cancel(gpu_lib, seed, shell, scheme):
    """Thin segments with source slopes of 1e6 and more, and rays through a shell that leave on the other side:
    each ray's intensity to 1e-9 of an evaluation in extended precision, as the schemes' own comparison asks."""
    L = (20, 56, 100)[seed % 3]
    alpha, S, z, tau, ref = _atmosphere(L, 32, seed)
    mu, w = np.polynomial.legendre.leggauss(8)
    mu, w = mu / 2 + 0.5, w / 2
    z = z + 7e10 * shell
    inward = bool(seed % 2)
    _, I = _rays(gpu_lib, alpha, S, z, shell, tau, ref, (mu, w), inward, scheme)
    np.testing.assert_allclose(I, _long_double(alpha, S, z, shell, tau, ref, mu, inward, scheme), rtol=1e-9, atol=0)
