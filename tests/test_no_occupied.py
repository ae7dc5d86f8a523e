"""Solves without an occupied orbital: empty vectors, as before any sweep over rows."""

import numpy as np
import pytest

from cphf_gb300 import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nspin", [1, 2])
def test_no_occupied_orbital(precision, nspin):
    rng = np.random.default_rng(1)
    nao, naux = 12, 20
    ctx = Context(precision=precision)
    ctx.set_cderi(np.asfortranarray(0.1 * rng.standard_normal((nao * (nao + 1) // 2, naux))), 1.0, 0.5)
    C, e = np.asfortranarray(rng.standard_normal((nao, nao))), np.linspace(-2, 2, nao)
    two = lambda v: [v, v.copy()] if nspin == 2 else v
    ctx.make_response_preparation(two(C), two(np.zeros(nao)), two(e))
    x = ctx.solve_dimless_cphf(two(np.zeros((nao, 0, 3, 2), order="F")))
    assert all(v.shape == (nao, 0, 3, 2) for v in (x if nspin == 2 else [x]))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_one_spin_without_an_occupied_orbital(precision):
    rng = np.random.default_rng(2)
    nao, naux, no = 14, 25, 4
    ctx = Context(precision=precision)
    ctx.set_cderi(np.asfortranarray(0.05 * rng.standard_normal((nao * (nao + 1) // 2, naux))), 1.0, 0.5)
    C = np.asfortranarray(np.linalg.qr(rng.standard_normal((nao, nao)))[0])
    e = np.concatenate([np.linspace(-9, -6, no), np.linspace(2, 5, nao - no)])
    ctx.make_response_preparation([C, C.copy()], [np.r_[np.ones(no), np.zeros(nao - no)], np.zeros(nao)], [e, e.copy()])
    b = np.asfortranarray(rng.standard_normal((nao, no, 3, 2)))
    x, empty = ctx.solve_dimless_cphf([b, np.zeros((nao, 0, 3, 2), order="F")])
    assert empty.shape == (nao, 0, 3, 2)
    y, _ = ctx.response_dimless_cphf([x, empty])
    assert np.abs(b - x - y).max() < 1e-7
