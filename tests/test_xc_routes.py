"""FP64 XC contractions: dense fixed-point products, per-batch GEMMs and grouped kernels agree.

Bar: 1e-12 of the largest element, the FP64 plugins' (the dense route's digits keep 62 bits of each
operand row's and column's maximum).
"""

import numpy as np
import pytest

from conftest import rel_err
from cphf_gb300 import Context, synth
from oracle import xc

pytestmark = pytest.mark.gpu

# nao, nocc, natm, points per atom, window, vectors: few / many points, narrow / full windows, odd sizes
LDA = [(33, (5,), 3, (300, 420), 8, 7), (64, (9,), 4, (700, 1300), 20, 12), (83, (11, 10), 6, (900, 1201), 27, 18),
       (131, (4,), 2, (1500, 1801), 131, 9), (97, (13, 1), 9, (65, 130), 5, 24)]


def _system(nao, nocc, natm, points, window):
    return synth.make_system(dict(nao=nao, naux=40, nocc=nocc, natm=natm, decay=12.0, grid=True, points=points,
                                  window=window), seed=nao)


def _context(s, **cfg):
    ctx = Context(**cfg)
    ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
    ctx.set_grid(s.grid.ao, s.grid.weights, s.grid.fxc, s.nspin, s.grid.atom_offsets)
    one = lambda v: v if s.nspin == 2 else v[0]
    ctx.make_response_preparation(one(s.mo_coeff), one(s.mo_occ), one(s.mo_energy))
    return ctx


def _bra(s, nb, seed):
    rng = np.random.default_rng(seed)
    return [rng.standard_normal((s.nao, n, nb)) for n in s.nocc]


def _run(ctx, s, bra):
    got = ctx.get_response_bra(bra if s.nspin == 2 else bra[0], plugin="xc")
    return got if s.nspin == 2 else [got]


@pytest.mark.parametrize("nao,nocc,natm,points,window,nb", LDA)
@pytest.mark.parametrize("chunk", [0, 1000])
def test_lda_routes_match_oracle(nao, nocc, natm, points, window, nb, chunk):
    s = _system(nao, nocc, natm, points, window)
    g, bra = s.grid, _bra(s, nb, 1)
    mocc = [s.mo_coeff[t][:, :s.nocc[t]] for t in range(s.nspin)]
    if s.nspin == 1:
        ref = [xc.rks_response_bra(g.ao, g.weights, g.fxc, bra[0], mocc[0])]
    else:
        ref = xc.uks_response_bra(g.ao, g.weights, g.fxc, bra, mocc)
    for tc in (1, 0):
        ctx = _context(s, tensor_cores=tc, xc_chunk_points=chunk)
        for a, b in zip(_run(ctx, s, bra), ref):
            assert rel_err(a, b) < 1e-12


def test_dense_route_runs_on_the_tensor_cores():
    s = _system(*LDA[2][:5])
    ctx = _context(s)
    bra = _bra(s, LDA[2][5], 1)
    _run(ctx, s, bra)
    ctx.profile(True)
    _run(ctx, s, bra)
    assert ctx.profile_report()["gemm_fp64_tcgen05"]["launches"] == 4  # two contractions of two spins


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_non_finite_elements_stay_in_their_windows(bad):
    """A non-finite AO row reaches the points and AOs of the batches that hold it, on every route."""
    s = _system(*LDA[2][:5])
    bra = _bra(s, LDA[2][5], 2)
    bra[0][0, 3, 2] = bad
    with np.errstate(all="ignore"):
        got = [_run(_context(s, tensor_cores=tc), s, [b.copy() for b in bra]) for tc in (1, 0)]
    for a, b in zip(*got):
        assert np.array_equal(np.isfinite(a), np.isfinite(b))
        ok = np.isfinite(b)
        assert not ok.all() and ok.any()
        assert rel_err(a[ok], b[ok]) < 1e-12


@pytest.mark.parametrize("den", ["sigma", "tau"])
@pytest.mark.parametrize("nao,nocc,natm,points,window,nb", [LDA[1], LDA[2], LDA[4]])
def test_gradient_components_in_one_product(nao, nocc, natm, points, window, nb, den):
    s = _system(nao, nocc, natm, points, window)
    ao, fx = synth.make_mgga_grid(s.grid, den, seed=3, nspin=s.nspin)
    one = lambda v: v if s.nspin == 2 else v[0]
    bra, got = _bra(s, nb, 3), []
    for tc in (1, 0):
        ctx = Context(tensor_cores=tc)
        ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
        ctx.set_grid_ex(den, ao, s.grid.weights, fx, s.nspin, s.grid.atom_offsets)
        ctx.make_response_preparation(one(s.mo_coeff), one(s.mo_occ), one(s.mo_energy))
        got.append(_run(ctx, s, bra))
    for a, b in zip(*got):
        assert rel_err(a, b) < 1e-12


@pytest.mark.parametrize("nao,nocc,natm,points,window,nb", LDA + [(300, (6,), 2, (1500, 1801), 290, 4)])
def test_tensor_core_xc_at_tile_edges(nao, nocc, natm, points, window, nb):
    """Mixed-precision XC on CTA pairs: split FP16 to 1e-5 of the operator, the exact-slice residual to
    1e-9 max(1, max |x|) (the operators' bars)."""
    s = _system(nao, nocc, natm, points, window)
    one = lambda v: v if s.nspin == 2 else v[0]
    c64, lp = _context(s), _context(s, precision="mixed")
    rng = np.random.default_rng(5)
    mo1 = [rng.standard_normal((nao, n, nb)) for n in nocc]
    a, b = lp.response_dimless_cphf_lowp(one(mo1)), c64.response_dimless_cphf(one(mo1))
    for u, v in zip(a if s.nspin == 2 else [a], b if s.nspin == 2 else [b]):
        assert rel_err(u, v) < 1e-5
    mx = _context(s, precision="mixed", residual_dfloat=2, max_refine=1, residual_tol=1.0, verify_residual=0)
    x = mx.solve_dimless_cphf(one(s.rhs))
    xs = x if s.nspin == 2 else [x]
    y = c64.response_dimless_cphf(x)
    r = np.concatenate([(p - q - w).reshape(-1, 3 * natm, order="F")
                        for p, q, w in zip(s.rhs, xs, y if s.nspin == 2 else [y])])
    ref = float(np.linalg.norm(r, axis=0).max())
    assert abs(mx.last_stats["residual_max"] - ref) < 1e-9 * max(1.0, max(np.abs(q).max() for q in xs))
