"""FP64 products whose output has millions of columns (csrc/gemm_simt.cu).

O_P = Cocc^T Z_P of a preparation has nocc naux columns: here one tile row of 32 columns more than
65535 tiles of 32, and more than 65535 tiles of 64.  Both arithmetics of the FP64 GEMMs agree to the
plugins' 1e-12 of the largest element.
"""

import numpy as np
import pytest

from conftest import rel_err
from cphf_gb300 import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nao,naux,nocc", [(34, 65665, 32), (66, 65666, 64)])
def test_more_column_tiles_than_a_grid_dimension(nao, naux, nocc):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(nao)
    cderi = torch.randn((naux, nao * (nao + 1) // 2), generator=gen, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()  # the context reads it on a stream of its own
    rng = np.random.default_rng(nao)
    C = np.linalg.qr(rng.standard_normal((nao, nao)))[0]
    occ = np.zeros(nao)
    occ[:nocc] = 2.0
    bra = rng.standard_normal((nao, nocc, 2))
    out = []
    for tc in (0, 1):
        ctx = Context(tensor_cores=tc)
        ctx.set_cderi(cderi.t(), 0.0, 1.0)
        ctx.make_response_preparation(np.asfortranarray(C), occ, np.linspace(-2, 2, nao))
        out.append(ctx.get_response_bra(bra))
        del ctx
    assert np.isfinite(out[0]).all() and rel_err(out[0], out[1]) < 1e-12
