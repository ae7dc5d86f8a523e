"""Accuracy of the orthogonalisation sweep on correlated columns, against serial Gram-Schmidt.

The operator callback of krylov_block receives the orthogonalised block.  The sweep projects up to
four columns at once where they are nearly independent of one another, which keeps its errors within
twice those of column-by-column projections of the same vectors with exact dot products (restated
here; both against extended precision), a factor left for the dot products' own sums.
"""

import numpy as np
import pytest

from cphf_gb300 import Context

pytestmark = pytest.mark.gpu


def _serial(v):
    """Right-looking Gram-Schmidt in v's precision, dot products in extended precision."""
    v = v.copy()
    for i in range(v.shape[1] - 1):
        dots = v[:, i].astype(np.longdouble) @ v[:, i:].astype(np.longdouble)
        v[:, i + 1:] -= np.outer(v[:, i], (dots[1:] / dots[0]).astype(v.dtype))
    return v


def _sweep(b):
    seen = []

    def op(v):
        seen.append(v.copy())
        return np.zeros_like(v)

    Context().krylov_block(op, b, tol=1e-6, lindep=1e-20)
    assert seen[0].shape == b.shape
    return seen[0]


@pytest.mark.parametrize("n,m", [(741, 36), (4000, 36), (641, 7)])
@pytest.mark.parametrize("noise", [100.0, 3.0, 1.0, 0.5, 0.2])
def test_errors_within_twice_the_serial_sweep(n, m, noise):
    err = [[], []]
    for seed in range(4):
        rng = np.random.default_rng(seed)
        base = rng.standard_normal(n)
        b = np.stack([base] + [base + noise * rng.standard_normal(n) for _ in range(m - 1)], axis=1)
        ref = _serial(b.astype(np.longdouble)).astype(float)
        norm = np.linalg.norm(ref, axis=0)
        for e, v in zip(err, (_serial(b), _sweep(b))):
            e.append(np.linalg.norm(v - ref, axis=0) / norm)
    serial, got = (np.sqrt(np.mean(np.square(e))) for e in err)
    assert got <= 2.0 * serial
