"""Preparations that take over the split-precision buffers on a kept grid, or after a change of settings."""

import numpy as np
import pytest

from cphf_gb300 import Context, synth

pytestmark = pytest.mark.gpu

DIMS = dict(nao=96, naux=150, nocc=(12,), natm=3, decay=12.0, grid=True, points=(500, 800), window=20)


def _orbitals(ctx, s):
    ctx.make_response_preparation(s.mo_coeff[0], s.mo_occ[0], s.mo_energy[0])


def _fresh(s, grid, **cfg):
    ctx = Context(precision="mixed", **cfg)
    ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
    ctx.set_grid(grid.ao, grid.weights, grid.fxc, 1, grid.atom_offsets)
    _orbitals(ctx, s)
    return ctx


def _solve(ctx, s):
    x = ctx.solve_dimless_cphf(s.rhs[0])
    assert ctx.last_stats["residual_max"] < 1e-8
    return x


@pytest.mark.parametrize("graphs", [0, 1])
def test_new_orbitals_and_cderi_on_a_kept_grid(graphs):
    """Solves reach a residual of 1e-8; answers of two contexts agree to 1e-7."""
    a, b = synth.make_system(DIMS, seed=1), synth.make_system(DIMS, seed=2)
    ctx = _fresh(a, a.grid, cuda_graphs=graphs)
    _solve(ctx, a)
    for s, cderi in ((b, False), (b, True), (a, True)):  # orbitals alone, then with their cderi
        if cderi:
            ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
        _orbitals(ctx, s)
        other = _fresh(s, a.grid, cuda_graphs=graphs) if cderi else None
        if other is None:
            other = Context(precision="mixed", cuda_graphs=graphs)
            other.set_cderi(a.cderi, a.scale_j, a.scale_k)
            other.set_grid(a.grid.ao, a.grid.weights, a.grid.fxc, 1, a.grid.atom_offsets)
            _orbitals(other, s)
        for _ in range(2):
            assert np.abs(_solve(ctx, s) - _solve(other, s)).max() < 1e-7


@pytest.mark.parametrize("change", [dict(tensor_cores=0), dict(aux_chunk=40), dict(xc_chunk_points=700),
                                    dict(residual_dfloat=1), dict(verify_residual=1)])
def test_settings_changed_between_preparations(change):
    s = synth.make_system(DIMS, seed=3)
    ctx = _fresh(s, s.grid)
    _solve(ctx, s)
    for cfg in (change, {}, change):
        ctx.set_config(**{"tensor_cores": 1, "aux_chunk": 0, "xc_chunk_points": 0, "residual_dfloat": 2,
                          "verify_residual": 2, **cfg})
        ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
        _orbitals(ctx, s)
        assert np.abs(_solve(ctx, s) - _solve(_fresh(s, s.grid, **cfg), s)).max() < 1e-7
