"""Fixed-point FP64 GEMM: operands of wide range, its accuracy bound, its less common forms, each with
the route asserted.

The slices are fixed point relative to each row's and column's maximum, so the error of an element is
bounded by the maxima, not by sum |a||b|:  with |a| < 2^e_a, |b| < 2^e_b for a row and a column, a
product loses 2^-62 to the rounding of both operands and 7 2^14 2^48 2^-124 = 7 2^-62 to the digit
pairs left out, so  K 8 2^-62 2^(e_a + e_b) <= K 2^-57 max|a| max|b|  over K products, plus a rounding
of each K range (2^-53 of its sum) and of each of their additions.
"""

import numpy as np
import pytest

from conftest import rel_err
from cphf_gb300 import Context, synth
from oracle import krylov, rijk

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _orbitals(nao, nocc, rng):
    occ = np.zeros(nao)
    occ[:nocc] = 2.0
    e = np.concatenate([np.linspace(-9, -1, nocc), np.linspace(0.5, 5, nao - nocc)])
    return np.asfortranarray(rng.standard_normal((nao, nao))), occ, e


def _s1mo(C, occ, e, s1, routed=True, **cfg):
    ctx = Context(**cfg)
    ctx.set_nao(C.shape[0])
    ctx.make_response_preparation(C, occ, e)
    ctx.profile(True)
    out = ctx.compute_dimless_cphf_rhs(None, None, s1)[2]
    assert ("gemm_fp64_tcgen05" in ctx.profile_report()) == routed
    return out


@pytest.mark.parametrize("octaves", [6, 20, 40, 70])
def test_error_against_the_maxima(octaves):
    """s1mo = C^T (s1ao Cocc) with entries over many octaves along every row and column."""
    nao, nocc, natm = 137, 33, 40
    rng = np.random.default_rng(octaves)
    C, occ, e = _orbitals(nao, nocc, rng)
    C *= np.exp2(-rng.uniform(0, octaves, C.shape))
    s1 = np.asfortranarray(rng.standard_normal((nao, nao, 3, natm)) * np.exp2(-rng.uniform(0, octaves, (nao, nao, 3, natm))))
    got = _s1mo(C, occ, e, s1).reshape(nao, nocc, -1, order="F")[:, :, ::40]
    sel = s1.reshape(nao, nao, -1, order="F")[:, :, ::40]
    Cl, Co = C.astype(np.longdouble), C[:, :nocc]
    for k in range(sel.shape[2]):
        S = sel[:, :, k]
        mid = S.astype(np.longdouble) @ Cl[:, :nocc]
        ref = Cl.T @ mid
        top = lambda v, axis: np.abs(v).max(axis=axis).astype(float)
        e1 = nao * 2.0 ** -57 * np.outer(top(S, 1), top(Co, 0)) + 2 * U * np.abs(mid).astype(float)
        e2 = nao * 2.0 ** -57 * np.outer(top(C, 0), top(mid, 0)) + 2 * U * np.abs(ref).astype(float)
        bound = e2 + np.abs(C).T @ e1
        assert (np.abs(got[:, :, k] - ref).astype(float) <= bound).all()


@pytest.mark.parametrize("shift", [-900, -430, 430, 700])
def test_exponents_near_the_ends_of_the_range(shift):
    """A power of two on an operand comes out of the product exactly (nothing subnormal here)."""
    rng = np.random.default_rng(1)
    nao, nocc, natm = 150, 40, 30
    C, occ, e = _orbitals(nao, nocc, rng)
    s1 = np.asfortranarray(rng.standard_normal((nao, nao, 3, natm)))
    np.testing.assert_array_equal(_s1mo(C, occ, e, np.ldexp(s1, shift)), np.ldexp(_s1mo(C, occ, e, s1), shift))


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
def test_non_finite_operands_leave_the_digit_route(value):
    rng = np.random.default_rng(2)
    nao, nocc, natm = 150, 40, 30
    C, occ, e = _orbitals(nao, nocc, rng)
    s1 = np.asfortranarray(rng.standard_normal((nao, nao, 3, natm)))
    s1[3, 7, 1, 11] = value
    with np.errstate(all="ignore"):
        ref = np.einsum("up,uvxa,vi->pixa", C, s1, C[:, :nocc], optimize=True)
    got = _s1mo(C, occ, e, s1)
    ok = np.isfinite(ref)
    np.testing.assert_array_equal(np.isfinite(got), ok)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    np.testing.assert_array_equal(_s1mo(C, occ, e, s1, routed=False, tensor_cores=0)[~ok], got[~ok])
    assert rel_err(got[ok], ref[ok]) < 1e-13


@pytest.mark.parametrize("nao,naux,nocc,nb,chunk", [(101, 301, 11, 6, 0), (129, 333, 17, 3, 0), (101, 301, 11, 6, 97)])
def test_split_sums_with_beta_and_any_alpha(nao, naux, nocc, nb, chunk):
    """The exchange products: few columns, a long odd K in ranges, alpha = -0.3 scale_k, added to J's result."""
    s = synth.make_system(dict(nao=nao, naux=naux, nocc=(nocc,), natm=2, decay=12.0), seed=nao)
    ctx = Context(aux_chunk=chunk)
    ctx.set_cderi(s.cderi, 0.7, 0.3)
    ctx.make_response_preparation(s.mo_coeff[0], s.mo_occ[0], s.mo_energy[0])
    bra = np.random.default_rng(3).standard_normal((nao, nocc, nb))
    ctx.profile(True)
    got = ctx.get_response_bra(bra)
    assert ctx.profile_report()["gemm_fp64_tcgen05"]["launches"] > 0
    assert rel_err(got, rijk.rhf_response_bra(s.cderi, s.mo_coeff[0], s.mo_occ[0], bra, 0.7, 0.3)) < 1e-12


def test_several_passes_over_the_rows():
    """Z_P of 2300 aux functions has 3.3 GB of digits, beyond the 3 GiB of one pass."""
    import torch
    nao, naux, nocc = 300, 2300, 16
    gen = torch.Generator(device="cuda").manual_seed(5)
    cderi = torch.randn((naux, nao * (nao + 1) // 2), generator=gen, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    rng = np.random.default_rng(5)
    C, occ, e = _orbitals(nao, nocc, rng)
    bra = rng.standard_normal((nao, nocc, 2))
    out = []
    for tc in (1, 0):
        ctx = Context(tensor_cores=tc)
        ctx.set_cderi(cderi.t(), 1.0, 0.0)  # (J: Z alone)
        ctx.profile(True)
        ctx.make_response_preparation(C, occ, e)
        assert ("gemm_fp64_tcgen05" in ctx.profile_report()) == bool(tc)
        out.append(ctx.get_response_bra(bra))
        del ctx
    assert rel_err(*out) < 1e-12


@pytest.mark.parametrize("spread", [0, 6])
def test_balanced_basis_updates(spread):
    """Krylov updates with basis vectors of opposing scales (balanced along k before the slicing)."""
    rng = np.random.default_rng(7)
    n, nset = 3001, 48
    d = rng.uniform(-0.3, 0.3, n)
    b = rng.standard_normal((n, nset)) * 10.0 ** np.linspace(-spread / 2, spread / 2, nset)
    op = lambda v: d[:, None] * v
    ctx = Context()
    ctx.profile(True)
    x = ctx.krylov_block(op, b, tol=1e-8, lindep=1e-24)
    assert ctx.profile_report()["gemm_fp64_tcgen05"]["launches"] > 0
    ref = krylov.krylov_block(op, b, tol=1e-8, lindep=1e-24)
    assert (np.abs(x - ref).max(axis=0) <= 1e-9 * np.abs(ref).max(axis=0) + 1e-10 * np.abs(ref).max() * 10.0 ** -spread).all()


@pytest.mark.parametrize("octaves", [0, 12])
def test_balanced_triangular_solve(octaves):
    """cderi = j3c L^-T with a graded metric: every column as accurate as the native route's."""
    nao, naux = 60, 700
    rng = np.random.default_rng(8)
    q = np.linalg.qr(rng.standard_normal((naux, naux)))[0]
    g = np.exp2(rng.permutation(np.linspace(-octaves, octaves, naux)))
    j2c = g[:, None] * ((q * rng.uniform(0.5, 2.0, naux)) @ q.T) * g[None, :]
    j2c = np.asfortranarray(0.5 * (j2c + j2c.T))
    j3c = np.asfortranarray(rng.standard_normal((nao * (nao + 1) // 2, naux)) * g)
    out = []
    for tc in (1, 0):
        ctx = Context(tensor_cores=tc)
        ctx.profile(True)
        ctx.set_j3c(j3c, j2c)
        assert ("gemm_fp64_tcgen05" in ctx.profile_report()) == bool(tc)
        out.append(ctx.get_cderi())
    diff = np.abs(out[0] - out[1]).max(axis=0) / np.abs(out[1]).max(axis=0)
    assert diff.max() < 1e-12
