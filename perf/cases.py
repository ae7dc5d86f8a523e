"""Performance cases: what a user of the CPHF/CPKS response library has it do.

Every case goes through ``cphf_gb300.Context``.  The kinds:

* ``response``  ``get_response_bra`` on a prepared context (the plugin call of a host program
  that keeps its own solver), all 3 natm nuclear displacements at once;
* ``solve``     ``solve_dimless_cphf`` on a prepared context, the call that dominates a Hessian;
* ``hessian``   right-hand side, solve, ``finalize_cphf`` and ``get_cphf_hess`` in a row;
* ``setup``     ``set_j3c`` (metric decomposition and triangular solve) and the cderi read back;
* ``geometry``  a new geometry on a kept context: ``set_cderi``, the response preparation, solve.

Systems are synthetic with the distributions of the repository's generator
(``cphf_gb300/synth.py``), drawn on the GPU: cderi Gaussian with an exponential decay in the AO
distance, orthogonal orbitals, occupied energies on [-20, -0.3], virtual ones on [0.05, 5], the
scale of B (and of the XC kernel) set so that the response operator's norm on the vir-occ block
is about half the smallest gap; XC grids in per-atom batches with block-sparse AO values.
"""

import math
import sys
from pathlib import Path
from types import SimpleNamespace

import numpy as np
import torch

_PKG = Path.cwd() / "rstsr-showcase-hessian_gb300"
if str(_PKG) not in sys.path:
    sys.path.insert(0, str(_PKG))

import cphf_gb300  # noqa: E402

DEV = "cuda"
F64 = torch.float64


def _case(kind, nao, naux, nocc, natm, precision="fp64", xc="none", npts=0, learned=False, name=None):
    """``nocc``: one count (restricted) or (alpha, beta); ``npts``: mean grid points per atom."""
    two = isinstance(nocc, tuple)
    c = dict(kind=kind, precision=precision, xc=xc, nao=nao, naux=naux, nocc_a=nocc[0] if two else nocc,
             nocc_b=nocc[1] if two else 0, unrestricted=two, natm=natm, npts=npts, learned=learned)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one plugin call for a molecule of a few atoms: launches and host work
        _case("response", 24, 84, 5, 4, name="response_rhf_nao24"),
        # default (FP64) solves: a small molecule with odd sizes, and an ordinary one
        _case("solve", 57, 211, 13, 6, name="solve_rhf_nao57"),
        _case("solve", 180, 600, 18, 18, name="solve_rhf_nao180"),
        # open-shell LDA on a small uneven grid, FP64
        _case("solve", 83, 245, (11, 10), 6, xc="lda", npts=1100, name="solve_uks_lda_nao83"),
        # gradient-corrected functional, FP64
        _case("solve", 96, 320, 15, 8, xc="gga", npts=700, name="solve_rks_gga_nao96"),
        # mixed-precision solves: ordinary and odd, then the 60-atom configuration with the learned
        # preconditioner (the benchmark's default options)
        _case("solve", 243, 811, 27, 24, precision="mixed", name="mixed_rhf_nao243"),
        _case("solve", 600, 2000, 60, 60, precision="mixed", learned=True, name="mixed_rhf_nao600"),
        # mixed precision with an LDA functional, and an open-shell one with two ragged spins
        _case("solve", 300, 1000, 30, 30, precision="mixed", xc="lda", npts=2500, name="mixed_rks_lda_nao300"),
        _case("solve", 210, 700, (33, 29), 14, precision="mixed", name="mixed_uhf_nao210"),
        # the metric decomposition and the cderi build
        _case("setup", 200, 667, 1, 1, name="setup_j3c_nao200"),
        # a new geometry on a kept context, mixed precision
        _case("geometry", 400, 1333, 40, 12, precision="mixed", name="geometry_mixed_nao400"),
        # a whole Hessian's response part, FP64
        _case("hessian", 120, 400, 20, 10, name="hessian_rhf_nao120"),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["response", "solve", "solve", "solve", "hessian", "setup", "geometry"])
    while True:
        mixed = kind in ("solve", "geometry") and rng.random() < 0.5
        xc = rng.choice(["none", "none", "lda", "gga"]) if kind in ("response", "solve") else "none"
        two = kind != "setup" and rng.random() < 0.25
        if mixed:
            nao = _logint(rng, 90, 560 if xc == "none" else 320 if xc == "lda" else 150)
        else:
            nao = _logint(rng, 20, 190 if xc == "none" else 110)
        naux = int(nao * rng.uniform(2.7, 3.6))
        na = max(2, int(nao * rng.uniform(0.08, 0.16)))
        nocc = (na, max(1, na - rng.randrange(0, 4))) if two else na
        natm = max(2, int(nao / rng.uniform(8.0, 14.0)))
        npts = _logint(rng, 400, 2500) if xc != "none" else 0
        c = _case(kind, nao, naux, nocc, natm, "mixed" if mixed else "fp64", xc, npts, mixed and rng.random() < 0.3)
        # no dearer than the largest listed case
        if _response_flops(c) <= (1.5e13 if mixed else 8e10):
            return c


# ---- the systems ----------------------------------------------------------------------------
def _nocc(case):
    return [case["nocc_a"], case["nocc_b"]] if case["unrestricted"] else [case["nocc_a"]]


def _forder(*shape):
    """An uninitialised F-ordered (col-major) float64 tensor."""
    t = torch.empty(tuple(reversed(shape)), dtype=F64, device=DEV)
    return t.permute(*reversed(range(len(shape))))


def _to_f(t):
    out = _forder(*t.shape)
    out.copy_(t)
    return out


def _packed_index(nao):
    nu, mu = torch.tril_indices(nao, nao, device=DEV)  # element mu <= nu at nu (nu + 1) / 2 + mu
    return mu, nu


def _dense(packed, nao, dtype):
    """[naux, nao, nao] from packed rows [naux, nao_tp]."""
    mu, nu = _packed_index(nao)
    full = torch.empty((nao, nao), dtype=torch.int64, device=DEV)
    k = torch.arange(mu.numel(), device=DEV)
    full[mu, nu] = k
    full[nu, mu] = k
    return packed.to(dtype)[:, full.reshape(-1)].reshape(-1, nao, nao)


def _grid(case, gen):
    nao, natm = case["nao"], case["natm"]
    lo_p, hi_p = max(8, int(0.7 * case["npts"])), int(1.3 * case["npts"]) + 9
    counts = torch.randint(lo_p, hi_p, (natm,), generator=gen, device=DEV).cpu().numpy()
    off = np.zeros(natm + 1, dtype=np.int64)
    off[1:] = np.cumsum(counts)
    ng = int(off[-1])
    ncomp = 4 if case["xc"] == "gga" else 1
    per, window = max(1, nao // natm), 80 if nao >= 240 else max(8, nao // 3)
    ao = torch.zeros((ncomp, nao, ng), dtype=F64, device=DEV)
    mu = torch.arange(nao, device=DEV)
    for a in range(natm):
        lo, hi = min(a * per, nao - 1), (a + 1) * per if a < natm - 1 else nao
        d = torch.clamp(torch.maximum(lo - mu, mu - (hi - 1)), min=0).to(F64)
        env = torch.where(d <= window, torch.exp(-(2.0 * d / window) ** 2), 0.0)
        g0, g1 = int(off[a]), int(off[a + 1])
        cols = torch.nonzero(env).reshape(-1)
        v = torch.randn((ncomp, cols.numel(), g1 - g0), generator=gen, dtype=F64, device=DEV)
        ao[:, cols, g0:g1] = v * env[cols][None, :, None]
    w = 1e-2 * (1.0 - torch.rand(ng, generator=gen, dtype=F64, device=DEV))
    rho = torch.exp(torch.rand((2, ng), generator=gen, dtype=F64, device=DEV) * math.log(1e7) + math.log(1e-6))
    nvar, ns = (4 if ncomp == 4 else 1), len(_nocc(case))
    f = torch.zeros((nvar * ns, nvar * ns, ng), dtype=F64, device=DEV)  # index x + nvar * spin
    base = rho[0] ** (-2.0 / 3.0)
    if nvar > 1:
        x = torch.randn((nvar * ns, nvar * ns, ng), generator=gen, dtype=F64, device=DEV) * 0.1 * base
        f = 0.5 * (x + x.transpose(0, 1))
    for s in range(ns):
        for t in range(ns):
            f[nvar * s, nvar * t] = -rho[s] ** (-2.0 / 3.0) if s == t else -0.1 * (rho[0] * rho[1]) ** (-1.0 / 3.0)
    return SimpleNamespace(ao=ao, w=w, f=f, off=off, nvar=nvar, ng=ng)


def _system(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 7919 + 17)
    randn = lambda *s: torch.randn(s, generator=gen, dtype=F64, device=DEV)  # noqa: E731
    rand = lambda *s: torch.rand(s, generator=gen, dtype=F64, device=DEV)  # noqa: E731
    nao, naux, natm, nocc = case["nao"], case["naux"], case["natm"], _nocc(case)
    ns = len(nocc)
    s = SimpleNamespace(nao=nao, naux=naux, natm=natm, nocc=nocc, ns=ns, sj=1.0, sk=0.5 if ns == 1 else 1.0)
    mu, nu = _packed_index(nao)
    sigma = 0.3 * torch.exp(-(nu - mu).to(F64) / (20.0 if nao >= 100 else 6.0))
    s.packed = randn(naux, mu.numel()).mul_(sigma)
    s.C, s.e = [], []
    for no in nocc:
        s.C.append(torch.linalg.qr(randn(nao, nao))[0])
        eo = torch.sort(-20.0 + 19.7 * rand(no))[0]
        ev = torch.sort(0.05 + 4.95 * rand(nao - no))[0]
        s.e.append(torch.cat([eo, ev]))
    s.grid = _grid(case, gen) if case["xc"] != "none" else None
    s.s1, s.f1, s.rhs = [], [], []
    for t, no in enumerate(nocc):
        eo, dif = s.e[t][:no], s.e[t][no:, None] - s.e[t][None, :no]
        s1 = 0.1 * randn(nao, no, 3, natm)
        r = 0.1 * randn(nao, no, 3, natm)
        r[:no] = -0.5 * s1[:no]
        f1 = 0.1 * randn(nao, no, 3, natm)
        f1[no:] = -r[no:] * dif[:, :, None, None] + s1[no:] * eo[None, :, None, None]
        s.s1.append(s1), s.f1.append(f1), s.rhs.append(r)
    # scale of the response: half the smallest gap
    gap = min(float(s.e[t][no] - s.e[t][no - 1]) for t, no in enumerate(nocc))
    dense = _dense(s.packed, nao, torch.float32)
    x0 = [randn(nao - no, no) for no in nocc]
    n_jk = _norm(s, x0, lambda c1: _jk(s, dense, c1))
    del dense
    total = n_jk
    if s.grid is not None:
        s.grid.f *= n_jk / _norm(s, x0, lambda c1: _xc(s, c1))
        total = 2.0 * n_jk
    k = min(1.0, 0.5 * gap / total)
    s.packed *= math.sqrt(k)
    if s.grid is not None:
        s.grid.f *= k
    return s


def _norm(s, x, op, iterations=8):
    lam = 1.0
    for _ in range(iterations):
        nrm = math.sqrt(sum(float((v * v).sum()) for v in x))
        c1 = [(s.C[t][:, no:] @ (x[t] / nrm))[:, :, None].float() for t, no in enumerate(s.nocc)]
        x = [s.C[t][:, no:].T @ r[:, :, 0].to(F64) for t, (no, r) in enumerate(zip(s.nocc, op(c1)))]
        lam = math.sqrt(sum(float((v * v).sum()) for v in x))
    return lam


def _jk(s, dense, bra):
    """The RI-JK response of bra [nao, nocc, nb] per spin, in the dtype of ``dense`` and ``bra``."""
    dt = dense.dtype
    occ = [s.C[t][:, :no].to(dt) for t, no in enumerate(s.nocc)]
    z = [(dense.reshape(-1, s.nao) @ m).reshape(s.naux, s.nao, -1) for m in occ]
    d = sum(2.0 * z[t].reshape(s.naux, -1) @ bra[t].reshape(-1, bra[t].shape[2]) for t in range(s.ns))
    jfac = 2.0 * s.sj * (1.0 if s.ns == 1 else 0.5)
    out = []
    for t, no in enumerate(s.nocc):
        nb = bra[t].shape[2]
        r = jfac * (z[t].reshape(s.naux, -1).T @ d).reshape(s.nao, no, nb)
        o = torch.matmul(occ[t].T, z[t])                                       # [P, j, i]
        step = max(1, (1 << 28) // max(1, s.nao * no * nb))
        for p in range(0, s.naux, step):
            b, zz, oo = dense[p:p + step], z[t][p:p + step], o[p:p + step]
            tm = torch.einsum("vja,Pji->Pvia", bra[t], oo)
            r -= s.sk * (b.permute(1, 0, 2).reshape(s.nao, -1) @ tm.reshape(-1, no * nb)).reshape(s.nao, no, nb)
            w = torch.einsum("Pvi,vja->Pjia", zz, bra[t])
            r -= s.sk * (zz.permute(1, 0, 2).reshape(s.nao, -1) @ w.reshape(-1, no * nb)).reshape(s.nao, no, nb)
        out.append(r)
    return out


def _xc(s, bra):
    """The XC response of bra per spin, point chunks, in the dtype of ``bra``."""
    g, dt = s.grid, bra[0].dtype
    nc, fac = g.ao.shape[0], 4.0 if s.ns == 1 else 2.0
    out = [torch.zeros_like(b) for b in bra]
    nb = bra[0].shape[2]
    step = max(64, (1 << 26) // (nc * max(s.nocc) * nb))
    for g0 in range(0, g.ng, step):
        g1 = min(g.ng, g0 + step)
        phi = g.ao[:, :, g0:g1].to(dt).transpose(1, 2)                          # [c, g, mu]
        aob = [torch.matmul(phi, s.C[t][:, :no].to(dt)) for t, no in enumerate(s.nocc)]
        rho = []
        for t, no in enumerate(s.nocc):
            ket = torch.matmul(phi, bra[t].reshape(s.nao, -1)).reshape(nc, g1 - g0, no, nb)
            for x in range(g.nvar):
                v = torch.einsum("gi,gia->ga", aob[t][0], ket[x])
                if x > 0:
                    v = v + torch.einsum("gi,gia->ga", aob[t][x], ket[0])
                rho.append(v)
        rho = torch.stack(rho)                                                  # [(x, s), g, a]
        wv = torch.einsum("xyg,xga->yga", g.f[:, :, g0:g1].to(dt), rho) * g.w[g0:g1].to(dt)[None, :, None]
        for t, no in enumerate(s.nocc):
            v = wv[g.nvar * t:g.nvar * (t + 1)]
            q0 = sum(v[x][:, None, :] * aob[t][x][:, :, None] for x in range(g.nvar))
            acc = phi[0].T @ q0.reshape(g1 - g0, -1)
            for x in range(1, g.nvar):
                acc += phi[x].T @ (v[x][:, None, :] * aob[t][0][:, :, None]).reshape(g1 - g0, -1)
            out[t] += fac * acc.reshape(out[t].shape)
    return out


# ---- prepare and run ------------------------------------------------------------------------
def _set_grid(ctx, case, s):
    g = s.grid
    ao = g.ao.permute(2, 1, 0)                                                  # [g, mu, c], F-order
    if case["xc"] == "lda":
        f = _to_f(g.f.permute(2, 0, 1)) if s.ns == 2 else g.f[0, 0].contiguous()
        ctx.set_grid(ao[:, :, 0], g.w, f, s.ns, g.off)
    else:
        f = g.f.permute(2, 0, 1)
        if s.ns == 2:
            f = f.reshape(g.ng, 2, 4, 2, 4).permute(0, 2, 1, 4, 3)
        ctx.set_grid_ex("sigma", ao, g.w, _to_f(f), s.ns, g.off)


def _one(v):
    return v if len(v) > 1 else v[0]


def _orbitals(s):
    occ = [torch.cat([torch.full((no,), 2.0 if s.ns == 1 else 1.0, dtype=F64), torch.zeros(s.nao - no, dtype=F64)])
           .to(DEV) for no in s.nocc]
    return _one([_to_f(c) for c in s.C]), _one(occ), _one(list(s.e))


def _metric(case, seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 104729 + 5)
    nao, naux = case["nao"], case["naux"]
    mu, nu = _packed_index(nao)
    sigma = 0.3 * torch.exp(-(nu - mu).to(F64) / 20.0)
    j3c = torch.randn((naux, mu.numel()), generator=gen, dtype=F64, device=DEV).mul_(sigma)
    q = torch.linalg.qr(torch.randn((naux, naux), generator=gen, dtype=F64, device=DEV))[0]
    ev = torch.exp(torch.rand(naux, generator=gen, dtype=F64, device=DEV) * math.log(1e4) + math.log(1e-3))
    j2c = (q * ev) @ q.T
    return j3c, 0.5 * (j2c + j2c.T)


def _ao_derivatives(s, seed):
    """Skeleton derivatives whose transforms are the system's f1mo and s1mo (orthogonal C)."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 15485863 + 3)
    c, no = s.C[0], s.nocc[0]
    np3 = 3 * s.natm
    core = 0.05 * torch.randn((s.nao, s.nao, np3), generator=gen, dtype=F64, device=DEV)
    sm = 0.1 * torch.randn((s.nao, s.nao, np3), generator=gen, dtype=F64, device=DEV)
    core, sm = 0.5 * (core + core.transpose(0, 1)), 0.5 * (sm + sm.transpose(0, 1))
    el = 0.05 * torch.randn((s.nao, no, np3), generator=gen, dtype=F64, device=DEV)
    shape = (3, s.natm)
    return (core.reshape(s.nao, s.nao, *shape), el.reshape(s.nao, no, *shape), sm.reshape(s.nao, s.nao, *shape))


def prepare(case, seed):
    kind = case["kind"]
    ctx = cphf_gb300.Context(precision=case["precision"])
    st = SimpleNamespace(case=case, ctx=ctx)
    if kind == "setup":
        j3c, j2c = _metric(case, seed)
        st.j3c, st.j2c, st.out = j3c.t(), j2c.t(), _forder(j3c.shape[1], case["naux"])
        torch.cuda.synchronize()
        return st
    s = _system(case, seed)
    st.scale_j, st.scale_k = s.sj, s.sk
    if case["learned"]:
        ctx.set_mlp_weights(np.load(Path(cphf_gb300.__file__).with_name("mlp_weights.npy")))
        ctx.set_config(use_learned_guess=1)
    st.orbitals = _orbitals(s)
    torch.cuda.synchronize()
    if kind == "geometry":
        st.cderi = s.packed.t()
    else:
        ctx.set_cderi(s.packed.t(), s.sj, s.sk)
        if s.grid is not None:
            _set_grid(ctx, case, s)
        ctx.make_response_preparation(*st.orbitals)
    if kind == "response":
        st.bra = _one([_to_f(torch.einsum("up,pixa->uixa", s.C[t], s.rhs[t])) for t in range(s.ns)])
    elif kind == "hessian":
        st.derivs = tuple(_to_f(v) for v in _ao_derivatives(s, seed))
    else:
        st.rhs = _one([_to_f(r) for r in s.rhs])
        st.out = _one([_forder(*r.shape) for r in s.rhs])
    torch.cuda.synchronize()
    return st


def run(st):
    ctx, kind = st.ctx, st.case["kind"]
    if kind == "response":
        return ctx.get_response_bra(st.bra)
    if kind == "setup":
        ctx.set_j3c(st.j3c, st.j2c)
        return ctx.get_cderi(out=st.out)
    if kind == "hessian":
        rhs, f1mo, s1mo = ctx.compute_dimless_cphf_rhs(*st.derivs)
        mo1 = ctx.solve_dimless_cphf(rhs)
        mo1, mo_e1 = ctx.finalize_cphf(f1mo, s1mo, mo1)
        return {"mo1": mo1, "mo_e1": mo_e1, "de": ctx.get_cphf_hess(f1mo, s1mo, mo1, mo_e1)}
    if kind == "geometry":
        ctx.set_cderi(st.cderi, st.scale_j, st.scale_k)
        ctx.make_response_preparation(*st.orbitals)
    return ctx.solve_dimless_cphf(st.rhs, out=st.out)


# ---- work -----------------------------------------------------------------------------------
def _response_flops(case):
    """One application of the response to all 3 natm columns."""
    nao, naux, nb = case["nao"], case["naux"], 3 * case["natm"]
    f = 0.0
    for no in _nocc(case):
        f += nb * (2.0 * nao * nao * naux * no + 6.0 * nao * naux * no * no + 4.0 * nao * naux * no)
        if case["xc"] != "none":
            ng = case["natm"] * case["npts"]
            win = nao if case["xc"] == "gga" else min(nao, 2 * (80 if nao >= 240 else max(8, nao // 3)) + nao // case["natm"])
            f += 4.0 * ng * win * no * nb * (4 if case["xc"] == "gga" else 1)
    return f


def work(case):
    nao, naux, nb, kind = case["nao"], case["naux"], 3 * case["natm"], case["kind"]
    tp = nao * (nao + 1) // 2
    if kind == "setup":
        return {"bytes": 8.0 * (2 * tp * naux + naux * naux), "flops": naux ** 3 / 3.0 + float(tp) * naux * naux}
    vec = 8.0 * nao * sum(_nocc(case)) * nb
    grid = 8.0 * case["natm"] * case["npts"] * nao * (4 if case["xc"] == "gga" else 1)
    mo = sum(4.0 * nao * nao * no * nb for no in _nocc(case))  # C x and C^T r
    one = _response_flops(case) + mo
    # a solve needs about five applications at this operator norm, a Hessian one more, its
    # transforms and pair sums
    flops = {"response": _response_flops(case), "solve": 5 * one, "geometry": 5 * one, "hessian": 6 * one}[kind]
    if kind == "hessian":
        flops += sum(8.0 * nao * nao * no * nb + 6.0 * nb * nb * nao * no for no in _nocc(case))
    if kind == "geometry":
        flops += sum(2.0 * nao * nao * no * naux for no in _nocc(case))
    extra = 8.0 * 2 * nao * nao * nb if kind == "hessian" else 0.0
    return {"bytes": 8.0 * tp * naux + grid + 2 * vec + extra, "flops": flops}


# ---- 64-bit values --------------------------------------------------------------------------
def _respond(s, dense, bra):
    out = _jk(s, dense, bra)
    if s.grid is not None:
        out = [a + b for a, b in zip(out, _xc(s, bra))]
    return out


def _pair_fields(s, t, g0, g1):
    """Density fields of the (vir, occ) pairs of spin t: [nvar, points, nvir * nocc]."""
    no = s.nocc[t]
    phi = s.grid.ao[:, :, g0:g1].transpose(1, 2)
    m = torch.matmul(phi, s.C[t])
    v, o = m[:, :, no:], m[:, :, :no]
    x = [v[0][:, :, None] * o[0][:, None, :]]
    for c in range(1, s.grid.nvar):
        x.append(v[c][:, :, None] * o[0][:, None, :] + v[0][:, :, None] * o[c][:, None, :])
    return torch.stack([f.reshape(g1 - g0, -1) for f in x])


def _vir_operator(s, dense):
    """The dimensionless operator on the vir-occ block, dense [n, n] over both spins."""
    sizes = [(s.nao - no) * no for no in s.nocc]
    off = np.concatenate([[0], np.cumsum(sizes)])
    a = torch.zeros((int(off[-1]), int(off[-1])), dtype=F64, device=DEV)
    mo = []
    for t, no in enumerate(s.nocc):
        half = torch.matmul(dense, s.C[t])
        mo.append(torch.matmul(s.C[t].T, half))
    jfac = 4.0 * s.sj if s.ns == 1 else 2.0 * s.sj
    for t, no in enumerate(s.nocc):
        bt = mo[t][:, no:, :no].reshape(s.naux, -1)
        for u, nu in enumerate(s.nocc):
            bu = mo[u][:, nu:, :nu].reshape(s.naux, -1)
            a[off[t]:off[t + 1], off[u]:off[u + 1]] = jfac * (bt.T @ bu)
        nv = s.nao - no
        blk = a[off[t]:off[t + 1], off[t]:off[t + 1]].view(nv, no, nv, no)
        vv, oo = mo[t][:, no:, no:].reshape(s.naux, -1), mo[t][:, :no, :no].reshape(s.naux, -1)
        blk -= s.sk * (vv.T @ oo).view(nv, nv, no, no).permute(0, 2, 1, 3)
        blk -= s.sk * (bt.T @ bt).view(nv, no, nv, no).permute(0, 3, 2, 1)
    if s.grid is not None:
        fac, nv, g = 4.0 if s.ns == 1 else 2.0, s.grid.nvar, s.grid
        step = max(64, (1 << 28) // (nv * int(off[-1])))
        for g0 in range(0, g.ng, step):
            g1 = min(g.ng, g0 + step)
            x = [_pair_fields(s, t, g0, g1) for t in range(s.ns)]
            fw = g.f[:, :, g0:g1] * (fac * g.w[g0:g1])
            for t in range(s.ns):
                for u in range(s.ns):
                    for i in range(nv):
                        y = sum(fw[nv * u + j, nv * t + i][:, None] * x[u][j] for j in range(nv))
                        a[off[t]:off[t + 1], off[u]:off[u + 1]] += x[t][i].T @ y
    dif = torch.cat([(s.e[t][no:, None] - s.e[t][None, :no]).reshape(-1) for t, no in enumerate(s.nocc)])
    return a / dif[:, None], dif, off


def _solved(s, rhs):
    """(I + A) x = rhs, per-spin [nao, nocc, 3, natm]."""
    dense, nb = _dense(s.packed, s.nao, F64), 3 * s.natm
    b = [r.reshape(s.nao, no, nb) for r, no in zip(rhs, s.nocc)]
    occ_bra = [torch.einsum("up,pia->uia", s.C[t][:, :no], b[t][:no]) for t, no in enumerate(s.nocc)]
    r = _respond(s, dense, occ_bra)
    a, dif, off = _vir_operator(s, dense)
    r = torch.cat([torch.einsum("up,uia->pia", s.C[t][:, no:], r[t]).reshape(-1, nb) for t, no in enumerate(s.nocc)])
    v = torch.cat([b[t][no:].reshape(-1, nb) for t, no in enumerate(s.nocc)]) - r / dif[:, None]
    a.diagonal().add_(1.0)
    x = torch.linalg.solve(a, v)
    out = []
    for t, no in enumerate(s.nocc):
        full = b[t].clone()
        full[no:] = x[off[t]:off[t + 1]].reshape(s.nao - no, no, nb)
        out.append(full)
    return out, dense


def exact(case, seed):
    kind, nb = case["kind"], 3 * case["natm"]
    if kind == "setup":
        j3c, j2c = _metric(case, seed)
        low = torch.linalg.cholesky(j2c)
        return torch.linalg.solve_triangular(low, j3c, upper=False).t()
    n = sum((case["nao"] - no) * no for no in _nocc(case))
    ng = case["natm"] * case["npts"] * (16 if case["xc"] == "gga" else 1)
    if kind != "response" and (n > 18000 or 2.0 * n * n * ng > 1.2e13):
        return None  # the dense 64-bit system takes too long
    s = _system(case, seed)
    shape = lambda t, rows: (rows, s.nocc[t], 3, s.natm)  # noqa: E731
    if kind == "response":
        bra = [torch.einsum("up,pia->uia", s.C[t], s.rhs[t].reshape(s.nao, no, nb)) for t, no in enumerate(s.nocc)]
        out = _respond(s, _dense(s.packed, s.nao, F64), bra)
        return _one([o.reshape(shape(t, s.nao)) for t, o in enumerate(out)])
    if kind != "hessian":
        out, _ = _solved(s, s.rhs)
        return _one([o.reshape(shape(t, s.nao)) for t, o in enumerate(out)])
    if s.ns == 2:
        return None
    core, el, sm = _ao_derivatives(s, seed)
    c, no, e = s.C[0], s.nocc[0], s.e[0]
    f1 = torch.einsum("up,uixa->pixa", c, torch.einsum("uvxa,vi->uixa", core, c[:, :no]) + el)
    s1 = torch.einsum("up,uixa->pixa", c, torch.einsum("uvxa,vi->uixa", sm, c[:, :no]))
    dif = e[:, None] - e[None, :no]
    b1 = f1 - s1 * e[None, :no, None, None]
    rhs = torch.cat([-0.5 * s1[:no], -b1[no:] / dif[no:, :, None, None]])
    (x,), dense = _solved(s, [rhs])
    resp = _respond(s, dense, [torch.einsum("up,pia->uia", c, x)])[0]
    b1 = b1 + torch.einsum("up,uia->pia", c, resp).reshape(b1.shape)
    x = x.reshape(b1.shape)
    mo_e1 = b1[:no] + x[:no] * dif[:no, :, None, None]
    mo1 = torch.cat([x[:no], -b1[no:] / dif[no:, :, None, None]])
    m, ff, ss = mo1.reshape(-1, nb), f1.reshape(-1, nb), s1.reshape(-1, nb)
    se = (s1 * e[None, :no, None, None]).reshape(-1, nb)
    gq = 4.0 * m.T @ ff - 4.0 * m.T @ se - 2.0 * mo_e1.reshape(-1, nb).T @ s1[:no].reshape(-1, nb)
    # column r = x natm + a in these C-ordered reshapes; de[x, y, b, a] takes the b <= a pair
    gq = gq.reshape(3, s.natm, 3, s.natm).permute(0, 2, 1, 3)                   # [x, y, b, a] = G[(x, b), (y, a)]
    low = torch.tril(torch.ones((s.natm, s.natm), dtype=torch.bool, device=DEV), -1)  # b > a
    de = torch.where(low[None, None], gq.permute(1, 0, 3, 2), gq)
    return {"mo1": mo1, "mo_e1": mo_e1, "de": de}
