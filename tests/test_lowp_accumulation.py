"""FP32 accumulation of the inner operator's exchange term (csrc/tc_pair.cu).

The tensor cores drop the low bits of a partial sum at every MMA: half an ulp on average, 2^-25 of the
final sum over a sum that grows evenly.  An accumulator of the large products takes one MMA per 16
products, of at most 32 nao products (32 aux functions of term 1), so the exchange term stays within
2 nao 2^-25 of FP64, rounded up to whole K blocks of 64, plus the planes' 2^-21.
"""

import numpy as np
import pytest

from cphf_gb300 import Context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nao,naux,nocc,natm", [(400, 1333, 40, 12), (330, 1000, 50, 10), (97, 2100, 9, 1), (64, 33, 64, 2)])
def test_exchange_sums_stay_short(nao, naux, nocc, natm):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(nao)
    draw = lambda *shape: torch.randn(shape, generator=gen, dtype=torch.float64, device="cuda")
    nu, mu = torch.tril_indices(nao, nao, device="cuda")
    cderi = draw(naux, mu.numel()) * 0.3 * torch.exp((mu - nu).double() / 20.0)
    torch.cuda.synchronize()  # the context reads it on a stream of its own
    occ = np.zeros(nao)
    occ[:nocc] = 2.0
    ctx = Context(precision="mixed")
    ctx.set_cderi(cderi.t(), 0.0, 1.0)
    ctx.make_response_preparation(np.asfortranarray(torch.linalg.qr(draw(nao, nao))[0].cpu().numpy()), occ,
                                  np.concatenate([np.linspace(-9, -1, nocc), np.linspace(0.5, 5, nao - nocc)]))
    mo1 = np.asfortranarray(draw(nao, nocc, 3, natm).cpu().numpy())
    got, ref = ctx.response_dimless_cphf_lowp(mo1), ctx.response_dimless_cphf(mo1)
    assert ctx.tensor_cores_active
    assert np.linalg.norm(got - ref) <= (32 * -(-nao // 64) * 4 * 2.0 ** -25 + 2.0 ** -21) * np.linalg.norm(ref)
