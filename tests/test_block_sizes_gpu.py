"""The sweep at block sizes where its kernels change form: the in-register inverse (row and column
edges of its 16, 32 and 64-wide layouts), the block inverse just above it, and ragged GEMM tiles."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

ETA = 1e-3
# The blocks are well conditioned (eta and the retarded self-energies bound |G| by O(10)), each entry
# of a Green's-function block is a sum of at most K n products, so a backward-stable sweep leaves
# K n eps cond ~ 4 * 130 * 2.2e-16 * 1e2 ~ 1e-11 relative to the block's norm.
TOL = 1e-10


def _device(dims, seed):
    rng = np.random.default_rng(seed)
    c = lambda m, n, s: (rng.normal(size=(m, n)) + 1j * rng.normal(size=(m, n))) * s
    herm = lambda x: (x + x.conj().T) / 2
    hd = [herm(c(n, n, 0.5 / np.sqrt(n))) + np.diag(rng.uniform(-2, 2, n)) for n in dims]
    sd = [np.eye(n) + herm(c(n, n, 0.02 / np.sqrt(n))) for n in dims]
    hu = [c(a, b, 0.5 / np.sqrt(max(a, b))) for a, b in zip(dims, dims[1:])]
    su = [c(a, b, 0.01 / np.sqrt(max(a, b))) for a, b in zip(dims, dims[1:])]
    se = []
    for n in (dims[0], dims[-1]):
        x = c(n, n, 0.5 / np.sqrt(n))
        se.append(herm(c(n, n, 0.3 / np.sqrt(n))) - 1j * (x @ x.conj().T + 0.2 * np.eye(n)))
    return hd, hu, [u.conj().T for u in hu], sd, su, [s.conj().T for s in su], se


@pytest.mark.parametrize("n", [1, 2, 5, 8, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65, 95, 97, 130])
def test_blocks_match_oracle(n):
    from dpnegf_b200.recursive_green_cal import recursive_gf
    dims = [n, max(1, n - 1), n + 1]
    hd, hu, hl, sd, su, sl, (seL, seR) = _device(dims, 100 + n)
    B = 3
    E = np.linspace(-0.7, 0.9, B)
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.complex128, device="cuda")
    ts = lambda xs: [t(x) for x in xs]
    rep = lambda s: t(s).expand(B, -1, -1)
    got = recursive_gf(torch.as_tensor(E).cuda(), ts(hl), ts(hd), ts(hu), ts(sd), ts(su), ts(sl), rep(seL), rep(seR),
                       eta=ETA, need_gr_lc=True)
    A = np.zeros((sum(dims), sum(dims)), complex)
    off = np.concatenate([[0], np.cumsum(dims)])
    for e in range(B):
        z = E[e] + 1j * ETA
        A[:] = 0
        for q in range(3):
            A[off[q]:off[q + 1], off[q]:off[q + 1]] = z * sd[q] - hd[q]
        for q in range(2):
            A[off[q]:off[q + 1], off[q + 1]:off[q + 2]] = z * su[q] - hu[q]
            A[off[q + 1]:off[q + 2], off[q]:off[q + 1]] = z * sl[q] - hl[q]
        A[:dims[0], :dims[0]] -= seL
        A[-dims[2]:, -dims[2]:] -= seR
        G = np.linalg.inv(A)
        blk = lambda i, j: G[off[i]:off[i + 1], off[j]:off[j + 1]]
        pairs = [(got[0][e], blk(0, 2))] + [(got[1][q][e], blk(q, 2)) for q in range(3)]
        pairs += [(got[2][q][e], blk(q, q)) for q in range(3)]
        pairs += [(got[3][q][e], blk(q + 1, q)) for q in range(2)] + [(got[4][q][e], blk(q, q + 1)) for q in range(2)]
        for x, y in pairs:
            x = x.cpu().numpy()
            assert np.linalg.norm(x - y) <= TOL * max(np.linalg.norm(y), 1e-3 * np.linalg.norm(G)), (n, e)


@pytest.mark.parametrize("overlap", [True, False])
@pytest.mark.parametrize("dims", [[20, 24, 16, 24], [70, 66, 90]])
def test_every_output_selection_agrees(dims, overlap):
    """The sweep forms only the products its outputs need: each output alone equals the same output
    of a sweep that returns everything (the same products in another association at most: TOL)."""
    from dpnegf_b200 import rgf_plan
    hd, hu, hl, sd, su, sl, (seL, seR) = _device(dims, 7)
    if not overlap:
        su, sl, sd = [0 * x for x in su], [0 * x for x in sl], [np.eye(n) for n in dims]
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.complex128, device="cuda")
    ts = lambda xs: [t(x) for x in xs]
    geom = rgf_plan.Geometry([rgf_plan.DeviceBlocks(ts(hd), ts(hu), ts(hl), ts(sd), ts(su), ts(sl))])
    B = 4
    E = [torch.linspace(-0.7, 0.9, B, dtype=torch.float64).cuda()]
    L, R = [t(seL).expand(B, -1, -1)], [t(seR).expand(B, -1, -1)]
    run = lambda **kw: rgf_plan.run(geom, E, L, R, eta=ETA, **kw)
    tags = ("g_trans", "grd", "grl", "gru", "gr_lc")
    full = run(outputs=tags, trans=True, dos=True, orb_dos=True, orb_g=True, orb_ar=True,
               s_in=[[torch.zeros(B, n, n, dtype=torch.complex128, device="cuda") for n in dims]])
    same = lambda x, y: float((x - y).abs().max()) <= TOL * float(y.abs().max())
    for key in ("trans", "dos", "orb_dos", "orb_g", "orb_ar"):
        assert same(getattr(run(outputs=(), **{key: True}), key), getattr(full, key)), key
    both = run(outputs=(), trans=True, dos=True)
    assert same(both.trans, full.trans) and same(both.dos, full.dos)
    for tag in tags:
        got, want = run(outputs=(tag,)).blocks[0][tag], full.blocks[0][tag]
        for x, y in [(got, want)] if tag == "g_trans" else zip(got, want):
            assert same(x, y), tag


def test_packed_arena_equals_the_blocks():
    """One launch packs blocks of any stride, conjugated views and transposes exactly; zero couplings
    (and only those) are marked; other types and host blocks take the copy path with the same arena."""
    from dpnegf_b200 import rgf_plan
    gen = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.complex(*(torch.randn(*s, generator=gen, dtype=torch.float64, device="cuda") for _ in range(2)))
    dims = [3, 40, 33]
    wide = r(80, 80)
    hd = [r(3, 3).mT, wide[::2, 1::2], r(33, 33).mH]
    hu = [r(40, 3).mH, r(1, 33).expand(40, 33)]
    hl = [u.mH for u in hu]
    sd = [torch.eye(n, dtype=torch.complex128, device="cuda") for n in dims]
    su = [torch.zeros(3, 40, dtype=torch.complex128, device="cuda"), r(40, 33)]
    sl = [-torch.zeros(40, 3, dtype=torch.complex128, device="cuda"), su[1].mH]
    su[1] = su[1].clone()
    g = rgf_plan.Geometry([rgf_plan.DeviceBlocks(hd, hu, hl, sd, su, sl)])
    host = rgf_plan.Geometry([rgf_plan.DeviceBlocks(*[[t.cpu().resolve_conj() for t in x] for x in (hd, hu, hl, sd, su, sl)])])
    assert torch.equal(g.hs, host.hs) and (g.blocks == host.blocks).all()
    b = g.blocks
    assert b[0]["su"] == b[0]["sl"] == b[0]["suT"] == b[0]["slT"] == -1
    assert all(b[1][k] >= 0 for k in ("hu", "hl", "su", "sl", "suT", "slT")) and b[0]["hu"] >= 0


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32])
def test_small_ctas_agree_with_large(n):
    """More items than SMs with blocks of up to 32 run on two-warp CTAs; the same sweep with fewer
    slots runs on eight-warp ones.  Only the order of reductions and of the inverse's panels differs
    (TOL); n at the edges of the inverse's 8, 16 and 32-wide layouts."""
    from dpnegf_b200 import rgf_plan
    dims = [n, max(1, n - 1), n, n]
    hd, hu, hl, sd, su, sl, (seL, seR) = _device(dims, 300 + n)
    t = lambda x: torch.as_tensor(np.ascontiguousarray(x), dtype=torch.complex128, device="cuda")
    ts = lambda xs: [t(x) for x in xs]
    geom = rgf_plan.Geometry([rgf_plan.DeviceBlocks(ts(hd), ts(hu), ts(hl), ts(sd), ts(su), ts(sl))])
    B = 460
    E = [torch.linspace(-0.7, 0.9, B, dtype=torch.float64).cuda()]
    L, R = [t(seL).expand(B, -1, -1)], [t(seR).expand(B, -1, -1)]
    s_in = [[torch.ones(B, 1, 1, dtype=torch.complex128, device="cuda") * t(np.eye(m)) for m in dims]]
    for kw in (dict(outputs=(), trans=True, dos=True, orb_g=True, orb_ar=True),
               dict(outputs=("grd", "gru"), trans=True, s_in=s_in)):
        a = rgf_plan.run(geom, E, L, R, eta=ETA, **kw)
        b = rgf_plan.run(geom, E, L, R, eta=ETA, n_slots=100, **kw)
        same = lambda x, y: float((x - y).abs().max()) <= TOL * float(y.abs().max())
        for key in ("trans", "dos", "orb_g", "orb_ar"):
            if getattr(a, key) is not None:
                assert same(getattr(a, key), getattr(b, key)), key
        for tag in a.blocks[0]:
            for x, y in zip(a.blocks[0][tag], b.blocks[0][tag]):
                assert same(x, y), tag
    w = torch.linspace(0.2, 1.0, B, dtype=torch.float64)
    g = [rgf_plan.run(geom, E, L, R, eta=ETA, outputs=(), adjoint_w=w, adjoint_w_dos=w, n_slots=m).grads for m in (B, 100)]
    for key in ("hd", "hu", "sd", "sl"):
        for x, y in zip(g[0][key], g[1][key]):
            assert same(x, y), key
