"""Split-K contractions of the RI-K term on CTA pairs (csrc/tc_pair.cu) at the edges of their tiles.

The pairs' tile is 256 (i, a) columns by a multiple of 32 AO rows (at most 256 split FP16, 128
exact slices), in K blocks of 64 / 32: nao around multiples of these, and columns around 256.

Tolerances, relative to the largest response element: split FP16 keeps 22 bits of each operand
row's maximum and accumulates in FP32, ~2^-21 per product times the spread of the row maxima: 1e-5
with room for 2^4 of spread; six exact slices keep 36 bits and drop terms below 2^-34, so a
residual of vectors of order max|x| agrees with FP64 to 1e-9 max(1, max|x|).
"""

import numpy as np
import pytest

from conftest import rel_err
from cphf_gb300 import Context, synth
from oracle import cphf, rijk

pytestmark = pytest.mark.gpu

# nao, naux, nocc, natm
EDGES = [(33, 40, 5, 2), (63, 30, 9, 3), (65, 30, 16, 5), (97, 37, 17, 5), (128, 20, 29, 3), (129, 20, 13, 7),
         (223, 11, 12, 7), (257, 9, 11, 8)]


def _system(nao, naux, nocc, natm):
    return synth.make_system(dict(nao=nao, naux=naux, nocc=(nocc,), natm=natm, decay=12.0), seed=nao + nocc)


def _context(s, **cfg):
    ctx = Context(precision="mixed", **cfg)
    ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
    ctx.make_response_preparation(s.mo_coeff[0], s.mo_occ[0], s.mo_energy[0])
    return ctx


def _oracle(s):
    plug = lambda b: rijk.rhf_response_bra(s.cderi, s.mo_coeff[0], s.mo_occ[0], b, s.scale_j, s.scale_k)
    return cphf.RHF(s.mo_coeff[0], s.mo_occ[0], s.mo_energy[0], [plug], s.natm)


@pytest.mark.parametrize("nao,naux,nocc,natm", EDGES)
def test_split_fp16_operator_at_tile_edges(nao, naux, nocc, natm):
    s = _system(nao, naux, nocc, natm)
    ctx = _context(s, aux_chunk=8)
    mo1 = np.random.default_rng(nao).standard_normal((nao, nocc, 3 * natm))
    got = ctx.response_dimless_cphf_lowp(mo1)
    assert ctx.tensor_cores_active
    assert rel_err(got, _oracle(s).response_dimless_cphf(mo1)) < 1e-5


@pytest.mark.parametrize("nao,naux,nocc,natm", EDGES)
def test_exact_slice_residual_at_tile_edges(nao, naux, nocc, natm):
    s = _system(nao, naux, nocc, natm)
    ctx = _context(s, residual_dfloat=2, max_refine=1, residual_tol=1.0, verify_residual=0, aux_chunk=8)
    x = ctx.solve_dimless_cphf(s.rhs[0])
    assert ctx.last_stats["residual_mode"] == 2
    y = _oracle(s).response_dimless_cphf(x)
    r = (s.rhs[0] - x - y).reshape(-1, 3 * natm, order="F")
    ref = float(np.linalg.norm(r, axis=0).max())
    assert abs(ctx.last_stats["residual_max"] - ref) < 1e-9 * max(1.0, np.abs(x).max()), ref


@pytest.mark.parametrize("nocc", [1, 31, 32, 33, 63, 64, 65, 127, 128, 129])
def test_t_generation_at_column_tile_edges(nocc):
    """T generation keeps the bra tile for nocc <= 128, in column tiles of 32, 64 or 128."""
    s = _system(161, 21, nocc, 1)
    ctx = _context(s, aux_chunk=8)
    mo1 = np.random.default_rng(nocc).standard_normal((161, nocc, 3))
    got = ctx.response_dimless_cphf_lowp(mo1)
    assert ctx.tensor_cores_active
    assert rel_err(got, _oracle(s).response_dimless_cphf(mo1)) < 1e-5


@pytest.mark.parametrize("naux,chunk", [(21, 8), (20, 7), (1, 0)])
@pytest.mark.parametrize("nocc", [1, 31, 32, 33, 64, 65])
def test_exact_generation_at_column_tile_edges(nocc, naux, chunk):
    """T and W of the exact slices come two aux functions to a column tile for nocc <= 32."""
    s = _system(131, naux, nocc, 2)
    ctx = _context(s, residual_dfloat=2, max_refine=1, residual_tol=1.0, verify_residual=0, aux_chunk=chunk)
    x = ctx.solve_dimless_cphf(s.rhs[0])
    assert ctx.last_stats["residual_mode"] == 2
    r = (s.rhs[0] - x - _oracle(s).response_dimless_cphf(x)).reshape(-1, 6, order="F")
    ref = float(np.linalg.norm(r, axis=0).max())
    assert abs(ctx.last_stats["residual_max"] - ref) < 1e-9 * max(1.0, np.abs(x).max())
