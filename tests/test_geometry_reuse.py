"""Successive preparations of one context reuse the split-precision buffers and give fresh results."""

import numpy as np
import pytest

from cphf_gb300 import Context, synth

pytestmark = pytest.mark.gpu

BASE = dict(nao=96, naux=150, nocc=(12,), natm=3, decay=12.0)
GRID = dict(nao=96, naux=150, nocc=(12,), natm=3, decay=12.0, grid=True, points=(500, 800), window=20)


def _prepare(ctx, s):
    ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
    assert not ctx.tensor_cores_active
    if s.grid is not None:
        ctx.set_grid(s.grid.ao, s.grid.weights, s.grid.fxc, s.nspin, s.grid.atom_offsets)
    one = lambda v: v if s.nspin == 2 else v[0]
    ctx.make_response_preparation(one(s.mo_coeff), one(s.mo_occ), one(s.mo_energy))
    assert ctx.tensor_cores_active


@pytest.mark.parametrize("graphs", [0, 1])
@pytest.mark.parametrize("steps", [
    [(BASE, 1), (BASE, 2), (BASE, 1)],                                            # same sizes
    [(BASE, 1), (dict(BASE, nocc=(17,)), 2), (dict(BASE, naux=140), 3), (BASE, 4)],  # other sizes between
    [(GRID, 1), (GRID, 2)],
])
def test_each_preparation_matches_a_fresh_context(steps, graphs):
    """Solves reach a residual of 1e-8; answers of two contexts agree to 1e-7."""
    ctx = Context(precision="mixed", cuda_graphs=graphs)
    for dims, seed in steps:
        s = synth.make_system(dims, seed=seed)
        fresh = Context(precision="mixed", cuda_graphs=graphs)
        out = []
        for c in (ctx, fresh):
            _prepare(c, s)
            out.append([c.solve_dimless_cphf(s.rhs[0]) for _ in range(2)])
            assert c.last_stats["residual_max"] < 1e-8
        for a, b in zip(*out):
            assert np.abs(a - b).max() < 1e-7


def test_repeated_geometry_allocates_nothing_more():
    s = synth.make_system(BASE, seed=1)
    ctx = Context(precision="mixed")
    sizes = []
    for _ in range(3):
        _prepare(ctx, s)
        ctx.solve_dimless_cphf(s.rhs[0])
        sizes.append(ctx.device_bytes)
    assert sizes[1] == sizes[2]
