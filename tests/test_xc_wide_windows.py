"""Mixed-precision LDA with a batch window wider than the exact slices' K range (3072 AOs)."""

import numpy as np
import pytest

from cphf_gb300 import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nao", [3071, 3073, 3200])
def test_window_beyond_one_exact_range(nao):
    """The mixed residual agrees with the FP64 operator's to 1e-9 max(1, max |x|), its bar elsewhere."""
    rng = np.random.default_rng(nao)
    nmo, nocc, ng = 7, 2, 300
    off = np.array([0, 170, 170, ng])
    ao = np.asfortranarray(0.05 * rng.standard_normal((ng, nao)))
    ao[170:, 1500:] = 0.0  # a second, narrow window
    cderi = np.asfortranarray(1e-3 * rng.standard_normal((nao * (nao + 1) // 2, 3)))
    C = np.asfortranarray(np.linalg.qr(rng.standard_normal((nao, nmo)))[0])
    occ, e = np.array([2.0] * nocc + [0.0] * (nmo - nocc)), np.concatenate([np.linspace(-3, -2, nocc), np.linspace(1, 3, nmo - nocc)])
    rhs = np.asfortranarray(rng.standard_normal((nmo, nocc, 3, 2)))

    def context(**cfg):
        ctx = Context(**cfg)
        ctx.set_cderi(cderi, 1.0, 0.5)
        ctx.set_grid(ao, np.full(ng, 1e-2), -rng.random(ng), 1, off)
        ctx.make_response_preparation(C, occ, e)
        return ctx

    state = rng.bit_generator.state
    mx = context(precision="mixed", residual_dfloat=2, max_refine=1, residual_tol=1.0, verify_residual=0)
    x = mx.solve_dimless_cphf(rhs)
    assert mx.last_stats["residual_mode"] == 2
    rng.bit_generator.state = state  # the same kernel values
    r = (rhs - x - context(tensor_cores=0).response_dimless_cphf(x)).reshape(-1, 6, order="F")
    assert abs(mx.last_stats["residual_max"] - np.linalg.norm(r, axis=0).max()) < 1e-9 * max(1.0, np.abs(x).max())
