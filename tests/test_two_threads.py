"""Two threads with a context each: geometries in turn, with memory to set buffers aside and without."""

import threading

import numpy as np
import pytest

from cphf_gb300 import Context, synth

pytestmark = pytest.mark.gpu

SIZES = [dict(nao=96, naux=150, nocc=(12,), natm=3, decay=12.0), dict(nao=120, naux=200, nocc=(15,), natm=4, decay=12.0)]


def _geometry(ctx, s):
    ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
    ctx.make_response_preparation(s.mo_coeff[0], s.mo_occ[0], s.mo_energy[0])
    return ctx.solve_dimless_cphf(s.rhs[0])


def _both(work):
    errors = []

    def guard(i):
        try:
            work(i)
        except BaseException as e:  # reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=guard, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def test_geometries_in_two_threads():
    """Solves reach a residual of 1e-8; answers of two contexts agree to 1e-7."""
    systems = [[synth.make_system(d, seed=k) for k in (1, 2)] for d in SIZES]
    ref = [[_geometry(Context(precision="mixed"), s) for s in both] for both in systems]

    def work(i):
        ctx = Context(precision="mixed")
        for _ in range(4):
            for s, x in zip(systems[i], ref[i]):
                assert np.abs(_geometry(ctx, s) - x).max() < 1e-7
        ctx.close()

    _both(work)


def test_geometries_with_little_memory_left():
    """Nothing is set aside then: every preparation frees and allocates beside the other thread's."""
    import torch
    systems = [synth.make_system(d, seed=3) for d in SIZES]
    ctxs = [Context(precision="mixed") for _ in SIZES]
    ref = [_geometry(c, s) for c, s in zip(ctxs, systems)]
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - (3 << 30), dtype=torch.uint8, device="cuda")

    def work(i):
        for _ in range(5):
            assert np.abs(_geometry(ctxs[i], systems[i]) - ref[i]).max() < 1e-7

    try:
        _both(work)
    finally:
        del held
        torch.cuda.empty_cache()
