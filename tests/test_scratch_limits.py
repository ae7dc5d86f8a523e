"""FP64 calls with little device memory left: the fixed-point products' scratch is not needed to answer."""

import numpy as np
import pytest

from conftest import rel_err
from cphf_gb300 import Context, synth

pytestmark = pytest.mark.gpu

RIJK = dict(nao=200, naux=600, nocc=(20,), natm=18, decay=12.0)
LDA = dict(nao=83, naux=40, nocc=(11, 10), natm=6, decay=12.0, grid=True, points=(900, 1201), window=27)


class _Filled:
    """All device memory but about ``left`` bytes (24 MiB) held by torch."""

    def __init__(self, left=24 << 20):
        self.left = left

    def __enter__(self):
        import torch
        torch.cuda.empty_cache()
        self.held = []
        for keep in (1 << 30, 256 << 20, 0):
            n = torch.cuda.mem_get_info()[0] - self.left - keep
            if n > 0:
                self.held.append(torch.empty(n, dtype=torch.uint8, device="cuda"))
        assert torch.cuda.mem_get_info()[0] < self.left + (40 << 20)

    def __exit__(self, *exc):
        import torch
        self.held = None
        torch.cuda.empty_cache()


def _context(s, kind):
    ctx = Context(tensor_cores=0)
    ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
    if kind == "lda":
        ctx.set_grid(s.grid.ao, s.grid.weights, s.grid.fxc, s.nspin, s.grid.atom_offsets)
    elif kind == "sigma":
        ao, fx = synth.make_mgga_grid(s.grid, "sigma", seed=3, nspin=s.nspin)
        ctx.set_grid_ex("sigma", ao, s.grid.weights, fx, s.nspin, s.grid.atom_offsets)
    one = lambda v: v if s.nspin == 2 else v[0]
    ctx.make_response_preparation(one(s.mo_coeff), one(s.mo_occ), one(s.mo_energy))
    return ctx


@pytest.mark.parametrize("dims,kind", [(RIJK, "rijk"), (LDA, "lda"), (LDA, "sigma")])
def test_no_memory_for_digit_planes(dims, kind):
    s = synth.make_system(dims, seed=4)
    ctx = _context(s, kind)
    rng = np.random.default_rng(1)
    bra = [rng.standard_normal((s.nao, n, 54)) for n in s.nocc]
    bra = bra if s.nspin == 2 else bra[0]
    plugin = "rijk" if kind == "rijk" else "xc"
    ref = ctx.get_response_bra(bra, plugin=plugin)  # (the native route's scratch is in place now)
    ctx.set_config(tensor_cores=1)
    with _Filled():
        got = ctx.get_response_bra(bra, plugin=plugin)
    ctx.profile(True)
    ctx.get_response_bra(bra, plugin=plugin)
    assert ctx.profile_report()["gemm_fp64_tcgen05"]["launches"] > 0  # (with memory the digits are used)
    for a, b in zip(got if s.nspin == 2 else [got], ref if s.nspin == 2 else [ref]):
        assert rel_err(a, b) < 1e-12


SMALL = dict(nao=96, naux=150, nocc=(12,), natm=3, decay=12.0)
MIXED = dict(nao=200, naux=600, nocc=(20,), natm=6, decay=12.0)


def _mixed(s, ctx=None):
    ctx = ctx or Context(precision="mixed")
    ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
    ctx.make_response_preparation(s.mo_coeff[0], s.mo_occ[0], s.mo_energy[0])
    return ctx


def test_parked_buffers_serve_another_context():
    """The buffers that one context keeps for its next preparation are freed for another's allocation."""
    s, t = synth.make_system(MIXED, seed=1), synth.make_system(SMALL, seed=2)
    ctx, other = _mixed(s), Context()
    ref = ctx.solve_dimless_cphf(s.rhs[0])
    ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
    kept = ctx.device_bytes
    with _Filled():
        _mixed(t, other)
        # (the buffers that other now needs in earnest come to more than the memory left)
        other.krylov_block(np.asfortranarray(0.1 * np.eye(40)), np.ones((40, 2)))
        big = np.zeros((3000, 3000), order="F")
        other.krylov_block(big, np.ones((3000, 1)))  # 72 MB
        assert ctx.device_bytes < kept
    ctx.make_response_preparation(s.mo_coeff[0], s.mo_occ[0], s.mo_energy[0])
    assert np.abs(ctx.solve_dimless_cphf(s.rhs[0]) - ref).max() < 1e-7  # (residual 1e-8)


def test_buffers_are_parked_only_while_memory_is_plenty():
    s = synth.make_system(MIXED, seed=1)
    ctx = _mixed(s)
    ctx.solve_dimless_cphf(s.rhs[0])
    held = ctx.device_bytes
    ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
    assert ctx.device_bytes == held
    ctx = _mixed(s)
    ctx.solve_dimless_cphf(s.rhs[0])
    with _Filled():
        ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
        assert ctx.device_bytes < held // 2


def test_chunks_follow_the_memory_of_each_preparation():
    """Prepared while memory was short, a context works in small chunks; prepared again, as a fresh one."""
    s = synth.make_system(dict(MIXED, natm=18), seed=1)
    mo1 = np.random.default_rng(2).standard_normal((s.nao, 20, 54))

    def launches(ctx):
        ctx.response_dimless_cphf_lowp(mo1)  # (the first call of a shape also tunes its launches)
        before = ctx.kernel_launches
        ctx.response_dimless_cphf_lowp(mo1)
        return ctx.kernel_launches - before

    ctx = Context(precision="mixed")
    ctx.set_cderi(s.cderi, s.scale_j, s.scale_k)
    with _Filled(left=3 << 29):  # planes and chunks: T alone is 0.6 GB in one chunk
        _mixed(s, ctx)
        short = launches(ctx)
    again, fresh = launches(_mixed(s, ctx)), launches(_mixed(s))
    assert again == fresh < short
