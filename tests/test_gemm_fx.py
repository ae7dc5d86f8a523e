"""Fixed-point FP64 GEMM on the tensor cores (csrc/gemm_fx.cu)."""

import math
from fractions import Fraction

import numpy as np
import pytest

from cphf_gb300 import Context

S, BITS = 8, 62


def _digits(v):
    """The kernel's balanced base-256 digits of round(v 2^62), |v| < 1, restated on Python integers."""
    f = math.floor(Fraction(abs(float(v))) * 2 ** BITS + Fraction(1, 2)) * (-1 if v < 0 else 1)
    u = f + int("80" * (S - 1), 16)
    q = [u >> (8 * (S - 1))]
    q += [((u >> (8 * (S - 1 - t))) & 0xFF) - 128 for t in range(1, S)]
    return f, q


def test_digits_reconstruct_and_stay_in_range():
    rng = np.random.default_rng(1)
    vals = np.concatenate([rng.uniform(-1, 1, 200), [0.0, 0.5, -0.5, 1 - 2.0 ** -53, -1 + 2.0 ** -53, 1 / 3, 2.0 ** -40]])
    for v in vals:
        f, q = _digits(v)
        assert sum(d * 256 ** (S - 1 - t) for t, d in enumerate(q)) == f
        assert abs(q[0]) <= 64 and all(-128 <= d <= 127 for d in q[1:])
        if abs(v) >= 2.0 ** -9:  # 53-bit values within 2^-9 of the row maximum are exact
            assert Fraction(f, 2 ** BITS) == Fraction(float(v))


def test_group_sums_stay_exact():
    """Sums of |q_t q_u| over the K blocks between two drains stay within 2^23 (group_kb)."""
    for g in range(S):
        bound = sum((64 if t == 0 else 128) * (64 if g == t else 128) for t in range(g + 1))
        p = 32
        while p > 2 and bound * 32 * p > 2 ** 23:
            p //= 2
        assert bound * 32 * p <= 2 ** 23


def _rhs_inputs(nao, nocc, natm, seed):
    rng = np.random.default_rng(seed)
    C = np.asfortranarray(rng.standard_normal((nao, nao)))
    occ = np.zeros(nao)
    occ[:nocc] = 2.0
    e = np.concatenate([np.linspace(-9, -1, nocc), np.linspace(0.5, 5, nao - nocc)])
    s1 = np.asfortranarray(rng.standard_normal((nao, nao, 3, natm)) * np.exp2(rng.uniform(-6, 0, (nao, nao, 3, natm))))
    return C, occ, e, s1


def _context(C, occ, e, **cfg):
    ctx = Context(**cfg)
    ctx.set_nao(C.shape[0])
    ctx.make_response_preparation(C, occ, e)
    return ctx


@pytest.mark.gpu
@pytest.mark.parametrize("nao,nocc,natm", [(128, 64, 3), (129, 33, 4), (191, 65, 2), (257, 31, 2), (320, 130, 1),
                                           (128, 64, 40), (129, 33, 60), (191, 65, 24), (257, 31, 24), (320, 130, 8)])
def test_against_extended_precision(nao, nocc, natm):
    """s1mo = C^T (s1ao Cocc), two GEMMs at the edges of the 128 x 64 tiles and of the 32-wide K
    blocks: the slices add 2^-62 |a||b| and each product one rounding, so the error stays within
    3 2^-53 |C|^T |s1ao| |Cocc| (two results rounded, the first one's error carried on)."""
    C, occ, e, s1 = _rhs_inputs(nao, nocc, natm, nao)
    ctx = _context(C, occ, e)
    ctx.profile(True)
    _, _, got = ctx.compute_dimless_cphf_rhs(None, None, s1)
    if natm >= 8:  # (small products are left to the native kernel)
        assert ctx.profile_report()["gemm_fp64_tcgen05"]["launches"] > 0
    sel = (s1.reshape(nao, nao, -1, order="F")[:, :, ::max(1, natm)]).astype(np.longdouble)
    got = got.reshape(nao, nocc, -1, order="F")[:, :, ::max(1, natm)]
    Cl = C.astype(np.longdouble)
    for k in range(sel.shape[2]):
        ref = Cl.T @ (sel[:, :, k] @ Cl[:, :nocc])
        bound = np.abs(C).T @ (np.abs(sel[:, :, k]).astype(float) @ np.abs(C[:, :nocc]))
        assert (np.abs(got[:, :, k] - ref).astype(float) <= 3 * 2.0 ** -53 * bound).all()


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_non_finite_operands_take_the_native_kernel(value):
    C, occ, e, s1 = _rhs_inputs(150, 40, 2, 5)
    s1[3, 7, 1, 1] = value
    out = [_context(C, occ, e, tensor_cores=tc).compute_dimless_cphf_rhs(None, None, s1)[2] for tc in (0, 1)]
    np.testing.assert_array_equal(out[0], out[1])
    assert not np.isfinite(out[1]).all()
