"""Calls of two threads, a context each, whose launches of one kernel need different amounts of shared memory:
neither may be refused because of the other's size."""
import ctypes as C
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
REPS = 400


def _together(calls):
    """Runs each of `calls` REPS times in a thread of its own; the errors they raised."""
    errors, start = [], threading.Barrier(len(calls))

    def work(call):
        start.wait()
        try:
            for _ in range(REPS):
                call()
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    return errors


def test_rays_of_different_layer_counts(gpu_lib):
    def rays(L, n_mu):
        ctx = gpu_lib.Context(0)
        tau, z, ref = 10.0 ** np.linspace(-5, 2, L), np.linspace(0, -1e8, L), np.exp(np.linspace(-20, -12, L))
        alpha, S = np.tile(ref, (40, 1)), np.tile(np.linspace(1, 30, L), (40, 1))
        mu, w = np.polynomial.legendre.leggauss(n_mu)
        keep = [np.ascontiguousarray(a) for a in (alpha, S, z, tau, ref, mu / 2 + 0.5, w / 2, np.empty(40))]
        p = [a.ctypes.data_as(C.POINTER(C.c_double)) for a in keep]
        return lambda: ctx.check(ctx.lib.korg_radiative_transfer_general(
            ctx.h, p[0], p[1], L, 40, p[2], 0, p[3], p[4], p[5], p[6], n_mu, 0, 0, 0, p[7], None)) or keep

    assert _together([rays(128, 40), rays(8, 2)]) == []


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_line_tiles_of_different_batches(gpu_lib, precision):
    from korg_gb300 import synthetic
    from korg_gb300.api import synthesize_prepared
    inp = synthetic.prepare(synthetic.Workload("two", 5000.0, 4.4, 0.0, 56, (5000, 5003),
                                               synthetic.synthetic_linelist(30, 5000, 5003, seed=1)))
    inp.hydrogen_lines = False
    prec = gpu_lib.KORG_MIXED if precision == "mixed" else gpu_lib.KORG_FP64
    ctxs = [gpu_lib.Context(0) for _ in range(2)]
    for ctx, stage in zip(ctxs, (128, 4)):  # lines per batch: shared memory of the launch
        ctx.check(ctx.lib.korg_set_tile_config(ctx.h, 56, prec, 128, stage, 1))
    assert _together([lambda c=c: synthesize_prepared(inp, precision=precision, ctx=c) for c in ctxs]) == []


def test_reverse_modes_of_different_layer_counts(gpu_lib):
    from korg_gb300 import synthetic
    from korg_gb300.api import synthesize_vjp
    calls = []
    for L in (128, 14):
        inp = synthetic.prepare(synthetic.Workload("two", 5000.0, 4.4, 0.0, L, (5000, 5001),
                                                   synthetic.synthetic_linelist(5, 5000, 5001, seed=1)))
        inp.hydrogen_lines = False
        ctx, d = gpu_lib.Context(0), np.ones(len(inp.wls))
        calls.append(lambda inp=inp, ctx=ctx, d=d: synthesize_vjp(inp, d, precision="fp64", ctx=ctx))
    assert _together(calls) == []
