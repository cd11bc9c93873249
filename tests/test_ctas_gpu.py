"""The kernels with one CTA per work slot and with clusters of 2, 4 and 8, on the same problems.

A launch picks the CTAs by its number of items, and a test has few: ``ctas`` runs them through the kernels
that large launches take as well.  Tolerance 1e-10 relative (max norm of a block), as for every FP64 result;
gradients 1e-9: sums of |G|^4-sized terms over energies and blocks, on well-conditioned devices."""
import numpy as np
import pytest
import torch

from oracle import rgf_oracle
from tests.test_block_inverse import E0
from tests.test_block_inverse import _device as _singular_leading_device
from tests.test_block_sizes_gpu import ETA, _device
from tests.test_products_gpu import _lead_blocks, _rand, _torch_lead_adjoint

pytestmark = pytest.mark.gpu
RTOL, GRAD_RTOL = 1e-10, 1e-9
CTAS = [1, 2, 4, 8]
TAGS = ("g_trans", "grd", "grl", "gru", "gr_lc", "gr_left")


def _t(x):
    return torch.as_tensor(np.ascontiguousarray(x), dtype=torch.complex128, device="cuda")


def _problem(dims, B, seed):
    from dpnegf_b200 import rgf_plan
    hd, hu, hl, sd, su, sl, se = _device(dims, seed)
    E = np.linspace(-0.7, 0.9, B)
    seL, seR = ([(1 + 0.1j * k) * s for k in range(B)] for s in se)
    geom = rgf_plan.Geometry([rgf_plan.DeviceBlocks(*[[_t(x) for x in xs] for xs in (hd, hu, hl, sd, su, sl)])])
    gpu = (geom, [_t(E)], [_t(np.stack(seL))], [_t(np.stack(seR))])
    return gpu, (E, hl, hd, hu, sd, su, sl, np.stack(seL), np.stack(seR))


def _close(got, want, what, rtol=RTOL):
    if isinstance(want, list):
        assert len(got) == len(want), what
        for q, (g, w) in enumerate(zip(got, want)):
            _close(g, w, (what, q), rtol)
        return
    got = got.cpu().numpy()
    err = np.abs(got - want).max() / np.abs(want).max()
    assert got.shape == want.shape and err <= rtol, (what, err)


@pytest.mark.parametrize("ctas", CTAS)
@pytest.mark.parametrize("dims", [[24, 32, 20], [33, 32, 34], [65, 64, 66, 40], [130, 129, 131], [256, 255, 192], [300, 70]])
def test_retarded_sweep(dims, ctas):
    from dpnegf_b200 import rgf_plan
    args, host = _problem(dims, 3, sum(dims))
    ref = rgf_oracle.rgf(*host, eta=ETA, need_gr_lc=True)
    T = rgf_oracle.transmission(ref["g_trans"], rgf_oracle.gamma_from_se(host[7]), rgf_oracle.gamma_from_se(host[8]))
    D = rgf_oracle.dos(ref["grd"], ref["grl"], ref["gru"], *host[4:7])
    res = rgf_plan.run(*args, eta=ETA, outputs=TAGS, trans=True, dos=True, ctas=ctas)
    for tag in TAGS:
        _close(res.blocks[0][tag], ref[tag], tag)
    for kw in (dict(trans=True, dos=True), dict(trans=True), dict(dos=True), dict(trans=True, refine=True)):
        some = rgf_plan.run(*args, eta=ETA, outputs=(), ctas=ctas, **kw)
        if "trans" in kw:
            _close(some.trans, T, kw)
        if "dos" in kw:
            _close(some.dos, D, kw)


@pytest.mark.parametrize("ctas", CTAS)
@pytest.mark.parametrize("dims", [[24, 32, 20], [40, 72, 40], [130, 129, 131]])
@pytest.mark.parametrize("which", ["lesser", "greater", "both"])
def test_lesser_and_greater_sweeps(dims, which, ctas):
    from dpnegf_b200 import rgf_plan
    B = 3
    args, host = _problem(dims, B, sum(dims) + 1)
    f = np.linspace(0.1, 0.9, B)
    kw, ref_kw = {}, {}
    if which != "greater":
        ref_kw.update(need_lesser=True, s_in=rgf_oracle.s_in_from_se(host[7], host[8], f, 1 - f, dims))
        kw.update(s_in=[[_t(s) for s in ref_kw["s_in"]]])
    if which != "lesser":
        ref_kw.update(need_greater=True, s_out=rgf_oracle.s_in_from_se(host[7], host[8], 1 - f, f, dims))
        kw.update(s_out=[[_t(s) for s in ref_kw["s_out"]]])
    ref = rgf_oracle.rgf(*host, eta=ETA, **ref_kw)
    res = rgf_plan.run(*args, eta=ETA, outputs=("grd",), ctas=ctas, **kw)
    tags = ["grd"] + (["gnd", "gnl", "gnu", "gin_left"] if "s_in" in kw else [])
    tags += ["gpd", "gpl", "gpu", "gip_left"] if "s_out" in kw else []
    for tag in tags:
        _close(res.blocks[0][tag], ref[tag], tag)


@pytest.mark.parametrize("ctas", CTAS)
@pytest.mark.parametrize("inverse,inv_ob", [("block", 32), ("block", 64), ("block", 512), ("gj", 64), ("gj", 512)])
def test_singular_leading_block_falls_back(inverse, inv_ob, ctas):
    """The pivoted inverse that a failed probe falls back to, for every outer block width of a one-CTA launch."""
    from dpnegf_b200 import rgf_plan
    hd, hu, hl, sd, su, sl, seL, seR = _singular_leading_device()
    geom = rgf_plan.Geometry([rgf_plan.DeviceBlocks(*[[_t(x) for x in xs] for xs in (hd, hu, hl, sd, su, sl)])])
    E = np.array([E0, E0 + 0.2], dtype=complex)
    sL, sR = (np.stack([s, s]) for s in (seL, seR))
    res = rgf_plan.run(geom, [_t(E)], [_t(sL)], [_t(sR)], eta=0.0, outputs=("g_trans", "grd"), trans=True,
                       inverse=inverse, inv_ob=inv_ob, ctas=ctas)
    ref = rgf_oracle.rgf(E, hl, hd, hu, sd, su, sl, sL, sR, eta=0.0)
    _close(res.blocks[0]["grd"], ref["grd"], "grd")
    _close(res.blocks[0]["g_trans"], ref["g_trans"], "g_trans")


@pytest.mark.parametrize("ctas", CTAS)
@pytest.mark.parametrize("n", [20, 48, 130])
def test_singular_block_is_reported(n, ctas):
    from dpnegf_b200 import rgf_plan
    z = lambda: torch.zeros(n, n, dtype=torch.complex128, device="cuda")
    eye = torch.eye(n, dtype=torch.complex128, device="cuda")
    geom = rgf_plan.Geometry([rgf_plan.DeviceBlocks([z(), eye], [0.1 * eye], [0.1 * eye], [eye, eye], [z()], [z()])])
    E = torch.zeros(2, dtype=torch.complex128, device="cuda")  # z S - H = 0 in the first block
    with pytest.raises(torch.linalg.LinAlgError, match="singular"):
        rgf_plan.run(geom, [E], [None], [None], eta=0.0, outputs=("grd",), ctas=ctas)


def _dense_gradients(host, w, wd):
    """Gradients of sum w T + wd DOS by torch autograd through dense inverses, in 64 bits on the host."""
    E, hl, hd, hu, sd, su, sl, seL, seR = host
    K = len(hd)
    off = np.concatenate([[0], np.cumsum([h.shape[0] for h in hd])])
    leaf = {k: [torch.as_tensor(x.copy()).requires_grad_(True) for x in v]
            for k, v in dict(hd=hd, hu=hu, hl=hl, sd=sd, su=su, sl=sl).items()}
    leaf["se_l"], leaf["se_r"] = (torch.as_tensor(s.copy()).requires_grad_(True) for s in (seL, seR))
    place = lambda q, p, x: torch.nn.functional.pad(x, (int(off[p]), int(off[-1] - off[p + 1]),
                                                        int(off[q]), int(off[-1] - off[q + 1])))
    full = lambda d, u, l: (sum(place(q, q, leaf[d][q]) for q in range(K))
                            + sum(place(q, q + 1, leaf[u][q]) + place(q + 1, q, leaf[l][q]) for q in range(K - 1)))
    H, S = full("hd", "hu", "hl"), full("sd", "su", "sl")
    loss, n0, nN = 0.0, int(off[1]), int(off[-1] - off[-2])
    for b in range(len(E)):
        sL, sR = leaf["se_l"][b], leaf["se_r"][b]
        G = torch.linalg.inv((E[b] + 1j * ETA) * S - H - place(0, 0, sL) - place(K - 1, K - 1, sR))
        gL, gR = 1j * (sL - sL.mH), 1j * (sR - sR.mH)
        g = G[:n0, -nN:]
        loss = loss + float(w[b]) * torch.trace(gL @ g @ gR @ g.mH).real
        if wd is not None:  # S is block-tridiagonal, so the trace over its blocks is the whole trace
            loss = loss - float(wd[b]) * (2.0 / np.pi) * torch.trace(G @ S).imag
    loss.backward()
    return {k: [x.grad.numpy() for x in v] if isinstance(v, list) else v.grad.numpy() for k, v in leaf.items()}


@pytest.mark.parametrize("ctas", CTAS)
@pytest.mark.parametrize("dims", [[20, 24, 18, 22, 20], [40, 33, 48, 36, 40], [70, 66, 90]])
@pytest.mark.parametrize("density,checkpoint", [(False, 0), (True, 0), (False, 2), (True, 2)])
def test_gradients(dims, density, checkpoint, ctas):
    from dpnegf_b200 import rgf_plan
    B = 3
    args, host = _problem(dims, B, sum(dims) + 2)
    w = np.linspace(0.5, 1.5, B)
    wd = np.linspace(-0.3, 0.8, B) if density else None
    want = _dense_gradients(host, w, wd)
    got = rgf_plan.run(*args, eta=ETA, outputs=(), adjoint_w=torch.as_tensor(w),
                       adjoint_w_dos=None if wd is None else torch.as_tensor(wd), checkpoint=checkpoint, ctas=ctas).grads
    for k, v in want.items():
        if k in ("sd", "su", "sl") or isinstance(v, list):
            scale = max(np.abs(x).max() for x in v)
            err = max(np.abs(g.cpu().numpy() - x).max() for g, x in zip(got[k], v))
            assert err <= GRAD_RTOL * scale, (k, err / scale)
        else:
            _close(got[k], v, k, GRAD_RTOL)


@pytest.mark.parametrize("form", [0, 1, 2])
@pytest.mark.parametrize("n", [17, 48, 96, 130, 260])
def test_lead_kernels_are_bitwise_the_same(n, form):
    """Decimation, Sigma and the lead adjoint in clusters do one CTA's operations in its order."""
    from dpnegf_b200 import surface_green as sg
    from dpnegf_b200.products import lead_adjoint
    gen = torch.Generator().manual_seed(60 + n + form)
    nc, b, B, eta = n // 2 + 1, n - 3, 4, 1e-2
    lead = _lead_blocks(n, gen)
    lead = [lead[0], lead[1] / np.sqrt(n / 8), lead[2], lead[3] / np.sqrt(n / 8)]
    hDL, sDL = (_rand((nc, b), gen, 0.4).cuda(), _rand((nc, b), gen, 0.02).cuda()) if form == 0 else (None, None)
    E = np.linspace(-0.8, 1.1, B)
    arena = sg.LeadArena([sg.LeadBlocks(*lead, hDL, sDL)], device="cuda")
    m = nc if form == 0 else n
    gsig = _rand((B, m, m), gen).cuda()
    runs = []
    for ctas in CTAS:
        res = sg.self_energies(arena, [0] * B, E, eta, want_gs=True, ctas=ctas)
        gs, sig = torch.stack(res.gs), torch.stack(res.sigma)
        grads = lead_adjoint(*lead, hDL, sDL, E, eta, gs, gsig, form, ctas=ctas)
        runs.append(([gs, sig] + [g for g in grads if g is not None], list(res.iters)))
    for out, iters in runs[1:]:
        assert iters == runs[0][1]
        assert all(torch.equal(x, y) for x, y in zip(out, runs[0][0]))
    want = [x for x in _torch_lead_adjoint(*lead, hDL, sDL, E, eta, runs[0][0][0], gsig, form) if x is not None]
    for x, y in zip(runs[0][0][2:], want):
        assert float((x - y).abs().max()) <= GRAD_RTOL * float(y.abs().max())


def test_ctas_that_cannot_run_are_refused():
    from dpnegf_b200 import _lib, rgf_plan, surface_green as sg
    args, _ = _problem([40, 40], 2, 5)
    for kw in (dict(ctas=3), dict(ctas=16), dict(ctas=-1), dict(ctas=2, precision="mixed")):
        with pytest.raises(_lib.NegfError, match="invalid argument"):
            rgf_plan.run(*args, eta=ETA, outputs=(), trans=True, **kw)
    arena = sg.LeadArena([sg.LeadBlocks(*_lead_blocks(20, torch.Generator().manual_seed(1)))], device="cuda")
    with pytest.raises(_lib.NegfError, match="invalid argument"):
        sg.self_energies(arena, [0], [0.1], 1e-3, ctas=5)


@pytest.mark.parametrize("ctas", CTAS)
def test_deferred_plan_keeps_its_ctas_and_is_captured(ctas):
    from dpnegf_b200 import rgf_plan
    args, _ = _problem([70, 66, 90], 3, 8)
    kw = dict(eta=ETA, outputs=(), trans=True, dos=True, ctas=ctas)
    want = rgf_plan.run(*args, **kw)
    plan = rgf_plan.run(*args, defer=True, **kw)
    plan.launch()
    torch.cuda.synchronize()
    plan.check()
    assert torch.equal(plan.result.trans, want.trans)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.launch()
    plan.result.trans.zero_()
    graph.replay()
    torch.cuda.synchronize()
    plan.check()
    assert torch.equal(plan.result.trans, want.trans) and torch.equal(plan.result.dos, want.dos)
