"""The Krylov solver's orthogonalisation sweep and projected solve at their edges, against the oracle."""

import numpy as np
import pytest

from cphf_gb300 import Context
from oracle import krylov

pytestmark = pytest.mark.gpu


def _compare(apply, gpu_op, b, **kw):
    ctx = Context()
    x = ctx.krylov_block(gpu_op, b, **kw)
    calls = []

    def counted(v):
        calls.append(v.shape[1])
        return apply(v)

    ref = krylov.krylov_block(counted, b, **kw)
    assert ctx.last_stats["aop_calls"] == len(calls)
    assert ctx.last_stats["aop_columns"] == sum(calls)
    # both stop on the same trial norm; the answers differ by the rounding of the sweeps
    assert np.abs(x - ref).max() <= 1e-10 * np.abs(ref).max()


@pytest.mark.parametrize("n,nset", [(37, 1), (37, 3), (53, 4), (53, 5), (641, 17), (900, 36), (1300, 23)])
def test_block_widths(n, nset):
    """Panels of four with every remainder, one and several blocks, LU panels of 16 with remainders."""
    rng = np.random.default_rng(n + nset)
    A = rng.standard_normal((n, n))
    A *= 0.4 / np.linalg.norm(A, 2)
    b = rng.standard_normal((n, nset))
    _compare(lambda v: A @ v, np.asfortranarray(A), b, tol=1e-9, lindep=1e-20)


@pytest.mark.parametrize("kind", ["near", "exact", "zero", "scaled"])
def test_dependent_columns_take_single_projections(kind):
    """Panels whose columns nearly or exactly depend on one another, are zero or differ in scale."""
    rng = np.random.default_rng(11)
    n, nset = 700, 10
    A = rng.standard_normal((n, n))
    A *= 0.3 / np.linalg.norm(A, 2)
    b = rng.standard_normal((n, nset))
    if kind == "near":
        b[:, 2] = b[:, 0] + 1e-2 * rng.standard_normal(n)
        b[:, 5] = b[:, 4] - b[:, 3] + 1e-3 * rng.standard_normal(n)
    elif kind == "exact":
        b[:, 3] = 2.0 * b[:, 1]
        b[:, 7] = b[:, 6]
    elif kind == "zero":
        b[:, [0, 5]] = 0.0
    else:
        b *= 10.0 ** np.linspace(-4, 2, nset)
    _compare(lambda v: A @ v, np.asfortranarray(A), b, tol=1e-8, lindep=1e-14)


def test_rows_beyond_the_shared_memory_stage():
    rng = np.random.default_rng(3)
    n, nset = 400_000, 6
    d = rng.uniform(-0.3, 0.3, n)
    b = rng.standard_normal((n, nset))
    _compare(lambda v: d[:, None] * v, lambda v: d[:, None] * v, b, tol=1e-6, lindep=1e-14)
