"""FP32 GEMMs of the inner operator on the CUDA cores (csrc/gemm_simt.cu) at tile edges and K splits.

Bar: FP32 products and sums of up to 3e4 terms, ~2^-24 sqrt(3e4) = 1e-5 of the largest element.
"""

import numpy as np
import pytest

from conftest import rel_err
from cphf_gb300 import Context, synth
from oracle import cphf, rijk

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nao,naux,nocc,natm", [(24, 30, 1, 1), (64, 63, 4, 7), (65, 257, 17, 5), (128, 64, 16, 2),
                                                (129, 300, 31, 21), (200, 128, 32, 22), (256, 513, 8, 43)])
def test_inner_operator_on_the_cuda_cores(nao, naux, nocc, natm):
    s = synth.make_system(dict(nao=nao, naux=naux, nocc=(nocc,), natm=natm, decay=12.0), seed=nao)
    ctx = Context(precision="mixed", tensor_cores=0)
    ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
    ctx.make_response_preparation(s.mo_coeff[0], s.mo_occ[0], s.mo_energy[0])
    mo1 = np.random.default_rng(nao).standard_normal((nao, nocc, 3 * natm))
    plug = lambda b: rijk.rhf_response_bra(s.cderi, s.mo_coeff[0], s.mo_occ[0], b, s.scale_j, s.scale_k)
    ref = cphf.RHF(s.mo_coeff[0], s.mo_occ[0], s.mo_energy[0], [plug], natm).response_dimless_cphf(mo1)
    assert rel_err(ctx.response_dimless_cphf_lowp(mo1), ref) < 1e-5
