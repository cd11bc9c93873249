"""The work a transport calculation has the package do, as cases that can be timed and checked.

Every case goes through a public entry point on the GPU.  ``listed()`` spans the
range from a single-orbital chain to 256-wide blocks; ``draw(rng)`` gives more
cases of the same kinds and ranges.  Kinds:

  tdos    ``transport.transmission_dos`` with a packed geometry: T(E) and DOS(E)
  green   ``recursive_gf``: every Green's-function block, with the lesser blocks
          when ``lesser``; ``energies == 1`` is the scalar call
  scf     the density sweep of one self-consistent iteration: a deferred plan
          (``rgf_plan.run(..., defer=True)``) that is launched again and again
  batch   ``Ozaki.uneven_batch``: decimation, sweep and density of several devices
  fit     T and DOS through ``adjoint.transmission_dos`` and the gradient of a
          current + density loss w.r.t. the device blocks and self-energies
  lead    ``adjoint.lead_self_energy``, forward or forward + backward

Devices are random Hermitian tight-binding matrices (onsite U[-2, 2] plus a
Hermitian Gaussian, couplings of norm about one, S = I plus a small Hermitian
part), self-energies are random retarded matrices, all made from the seed.
"""
import math

import numpy as np
import torch

from dpnegf_b200 import adjoint, density, recursive_green_cal, rgf_plan, surface_green, transport

C128 = torch.complex128
F64 = torch.float64
ETA = 1e-5
ETA_LEAD_FIT = 1e-3  # lead broadening where lead parameters are fitted (their gradient amplifies by 1 / eta)
KT = 0.025          # eV
BIAS = 0.3          # V


def listed():
    return [
        # the textbook check of a transport code: a 1-D chain with a two-site layer, a defect in the
        # middle and a fine energy grid (the smallest blocks; S = I)
        dict(name="chain", kind="tdos", b=2, blocks=10, energies=1000, ragged=False, overlap=False, precision="fp64"),
        # one energy of a small junction with all its blocks: what a loop over energies calls
        dict(name="one_energy", kind="green", b=64, blocks=8, energies=1, ragged=False, lesser=False),
        # a 2072-orbital carbon nanotube in 18 uneven blocks, one batch of 50 energies
        dict(name="nanotube_batch50", kind="tdos", b=115, blocks=18, energies=50, ragged=True, overlap=True,
             precision="fp64"),
        # a spectrum of a long junction
        dict(name="spectrum_b128", kind="tdos", b=128, blocks=48, energies=512, ragged=False, overlap=True,
             precision="fp64"),
        # G^< of a short junction under bias, all blocks returned
        dict(name="lesser_b128", kind="green", b=128, blocks=6, energies=64, ragged=False, lesser=True),
        # the headline shape (256-wide blocks), in both precisions; the largest work
        dict(name="spectrum_b256", kind="tdos", b=256, blocks=32, energies=256, ragged=False, overlap=True,
             precision="fp64"),
        dict(name="mixed_b256", kind="tdos", b=256, blocks=32, energies=256, ragged=False, overlap=True,
             precision="mixed"),
        # many devices of different block size and length at once: decimation, sweep and density
        dict(name="uneven_density", kind="batch", b_min=16, b_max=240, devices=6, blocks=24, poles=32, gauss=47),
        # one density sweep of a self-consistent loop: 64 poles, the far pole and 64 bias-window points
        dict(name="scf_sweep", kind="scf", b=64, blocks=16, energies=129, poles=65),
        # a fitting step: current + density loss and its gradient
        dict(name="fit_b96", kind="fit", b=96, blocks=32, energies=256),
        # lead self-energies of the headline device, and a lead-parameter gradient
        dict(name="lead_b256", kind="lead", n=256, energies=128, backward=False),
        dict(name="lead_fit_n96", kind="lead", n=96, energies=64, backward=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _fit_energies(rng, per_energy, lo, hi, most=9.0e12):
    """A number of energies in [lo, hi], log-uniform, within the work of the largest listed case."""
    return _log_int(rng, lo, max(lo, min(hi, int(most / per_energy))))


def draw(rng):
    kind = rng.choice(["tdos", "tdos", "tdos", "green", "scf", "batch", "fit", "lead", "lead"])
    if kind == "tdos":
        b = _log_int(rng, 2, 300)
        L = rng.randint(6, 64) if b <= 160 else rng.randint(4, 24)
        mixed = b >= 96 and rng.random() < 0.25
        return dict(kind="tdos", b=b, blocks=L, energies=_fit_energies(rng, 72.0 * b ** 3 * L, 16, 1500),
                    ragged=rng.random() < 0.4, overlap=rng.random() < 0.7, precision="mixed" if mixed else "fp64")
    if kind == "green":
        lesser = rng.random() < 0.5
        b = _log_int(rng, 16, 160)
        return dict(kind="green", b=b, blocks=rng.randint(3, 6 if lesser else 12), lesser=lesser,
                    energies=rng.choice([1, _log_int(rng, 2, 96)]), ragged=rng.random() < 0.5)
    if kind == "scf":
        poles = rng.randint(20, 80)
        return dict(kind="scf", b=_log_int(rng, 16, 160), blocks=rng.randint(6, 32), poles=poles,
                    energies=poles + rng.randint(0, 100))
    if kind == "batch":
        return dict(kind="batch", b_min=16, b_max=rng.randint(96, 240), devices=rng.randint(2, 6),
                    blocks=rng.randint(8, 24), poles=rng.randint(16, 40), gauss=rng.randint(16, 48))
    if kind == "fit":
        return dict(kind="fit", b=_log_int(rng, 24, 128), blocks=rng.randint(6, 32), energies=_log_int(rng, 32, 160))
    n = _log_int(rng, 12, 256)
    return dict(kind="lead", n=n, energies=_log_int(rng, 16, 128 if n > 96 else 512), backward=rng.random() < 0.4)


# ----------------------------------------------------------------------------- inputs
def _dims(case):
    b, L = case["b"], case["blocks"]
    if not case.get("ragged"):
        return [b] * L
    return [max(1, b + ((5 * q) % 7 - 3) * max(1, b // 20)) for q in range(L)]


def _batch_shapes(case):
    """(block size, blocks) of every device of a batch: sizes spread over [b_min, b_max], lengths with them."""
    nd = case["devices"]
    return [(int(case["b_min"] + (case["b_max"] - case["b_min"]) * i / max(1, nd - 1)) // 8 * 8 or 8,
             max(3, case["blocks"] - 3 * ((2 * i) % 5))) for i in range(nd)]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _cgauss(gen, shape, sigma):
    re = torch.randn(*shape, generator=gen, dtype=F64, device="cuda")
    im = torch.randn(*shape, generator=gen, dtype=F64, device="cuda")
    return (sigma / math.sqrt(2.0)) * torch.complex(re, im)


def _herm(x):
    return 0.5 * (x + x.mH)


def _device(gen, dims, overlap=True):
    """hd, hu, hl, sd, su, sl of a random Hermitian tight-binding device."""
    hd, sd, hu, su = [], [], [], []
    for n in dims:
        h = _herm(_cgauss(gen, (n, n), 0.3 / math.sqrt(n)))
        e = torch.rand(n, generator=gen, dtype=F64, device="cuda") * 4.0 - 2.0
        hd.append((h - torch.diag(torch.diagonal(h)) + torch.diag(e.to(C128))).contiguous())
        s = torch.eye(n, dtype=C128, device="cuda")
        sd.append((s + _herm(_cgauss(gen, (n, n), 0.01 / math.sqrt(n)))).contiguous() if overlap else s)
    for n0, n1 in zip(dims, dims[1:]):
        hu.append(_cgauss(gen, (n0, n1), 1.0 / math.sqrt(max(n0, n1))))
        su.append(_cgauss(gen, (n0, n1), 0.01 / math.sqrt(max(n0, n1))) if overlap
                  else torch.zeros(n0, n1, dtype=C128, device="cuda"))
    return hd, hu, [u.mH.contiguous() for u in hu], sd, su, [u.mH.contiguous() for u in su]


def _chain(gen, blocks):
    """The 2-site-layer chain (onsite 0, hopping -1) with a random defect in the middle."""
    h = torch.tensor([[0, -1], [-1, 0]], dtype=C128, device="cuda")
    u = torch.tensor([[0, 0], [-1, 0]], dtype=C128, device="cuda")
    hd = [h.clone() for _ in range(blocks)]
    hd[blocks // 2][0, 0] += torch.rand((), generator=gen, dtype=F64, device="cuda")
    zero = torch.zeros(2, 2, dtype=C128, device="cuda")
    K = blocks - 1
    return (hd, [u.clone() for _ in range(K)], [u.mT.contiguous() for _ in range(K)],
            [torch.eye(2, dtype=C128, device="cuda") for _ in range(blocks)], [zero.clone() for _ in range(K)],
            [zero.clone() for _ in range(K)])


def _chain_se(E, eta):
    """Both lead self-energies of the chain: the surface Green's function of a half chain, t = -1."""
    z = E.to(C128) + 1j * eta
    r = torch.sqrt(z * z - 4.0)
    g = torch.where(((z - r) / 2.0).imag <= 0, (z - r) / 2.0, (z + r) / 2.0)
    seL = torch.zeros(len(E), 2, 2, dtype=C128, device="cuda")
    seR = seL.clone()
    seL[:, 0, 0] = g
    seR[:, 1, 1] = g
    return seL, seR


def _self_energy(gen, B, n):
    a = _cgauss(gen, (B, n, n), 0.5 / math.sqrt(n))
    c = _cgauss(gen, (B, n, n), 0.5 / math.sqrt(n))
    return (_herm(a) - 1j * (c @ c.mH + 0.05 * torch.eye(n, dtype=C128, device="cuda"))).contiguous()


def _eta_lead(case):
    return ETA_LEAD_FIT if case["backward"] else ETA


def _fermi(E, mu):
    return 1.0 / (1.0 + torch.exp((E - mu) / KT))


def _lead(gen, n):
    """A principal layer and its couplings: [H, H01, S, S01, H_DL, S_DL]."""
    (h, _), (h01, ), _, (s, _), (s01, ), _ = _device(gen, [n, n])
    return [h, h01, s, s01, h01.clone(), s01.clone()]


def _inputs(case, seed):
    """The case's input tensors (what ``exact`` starts from too)."""
    gen, kind = _gen(seed), case["kind"]
    if kind == "lead":
        d = dict(lead=_lead(gen, case["n"]), E=torch.linspace(-3, 3, case["energies"], dtype=F64) + 0.01 * (seed % 7))
        w = torch.randn(case["energies"], case["n"], case["n"], generator=gen, dtype=F64, device="cuda")
        return dict(d, weight=w)
    if kind == "batch":
        devs = [_device(gen, [b] * L) for b, L in _batch_shapes(case)]
        pairs = []
        for hd, hu, hl, sd, su, sl in devs:
            pairs.append(((hd[0], hl[0], sd[0], sl[0], hl[0], sl[0]), (hd[-1], hu[-1], sd[-1], su[-1], hu[-1], su[-1])))
        return dict(devices=devs, leads=pairs)
    dims, B = _dims(case), case["energies"]
    chain = kind == "tdos" and case["b"] == 2 and not case["overlap"] and not case["ragged"]
    blocks = _chain(gen, case["blocks"]) if chain else _device(gen, dims, case.get("overlap", True))
    if kind == "fit":
        E = torch.linspace(-0.3, 0.3, B, dtype=F64, device="cuda")
    elif kind == "scf":
        x = torch.linspace(-BIAS, BIAS, max(1, B - case["poles"]), dtype=F64, device="cuda")[:B - case["poles"]]
        poles = 1j * math.pi * KT * (2 * torch.arange(case["poles"], dtype=F64, device="cuda") + 1)
        E = torch.cat([poles, x.to(C128)])
    else:
        E = torch.linspace(-3, 3, B, dtype=F64, device="cuda") if B > 1 else torch.tensor([0.37], dtype=F64, device="cuda")
    seL, seR = _chain_se(E, ETA) if chain else (_self_energy(gen, B, dims[0]), _self_energy(gen, B, dims[-1]))
    d = dict(blocks=blocks, E=E, seL=seL, seR=seR)
    if kind == "green" and case["lesser"]:
        s = [torch.zeros(B, n, n, dtype=C128, device="cuda") for n in dims]
        s[0] = s[0] + 1j * (seL - seL.mH) * (1j * _fermi(E, BIAS / 2)).view(B, 1, 1)
        s[-1] = s[-1] + 1j * (seR - seR.mH) * (1j * _fermi(E, -BIAS / 2)).view(B, 1, 1)
        d["s_in"] = s
    if kind == "fit":
        dE = 0.6 / (B - 1)
        d["w_t"] = (_fermi(E, BIAS / 2) - _fermi(E, -BIAS / 2)) * dE
        d["w_d"] = _fermi(E, 0.0) * dE
        hd, hu, _, sd, su, _ = blocks
        d["leaves"] = [torch.stack(x) for x in (hd, hu, sd, su)] + [seL, seR]
    return d


# ----------------------------------------------------------------------------- the calls
def prepare(case, seed):
    d, kind = _inputs(case, seed), case["kind"]
    st = dict(case=case, d=d)
    if kind == "tdos":
        st["geometry"] = rgf_plan.Geometry([rgf_plan.DeviceBlocks(*d["blocks"])])
    elif kind == "scf":
        geom = rgf_plan.Geometry([rgf_plan.DeviceBlocks(*d["blocks"])])
        bias = case["energies"] > case["poles"]
        st["plan"] = rgf_plan.run(geom, [d["E"].to(C128)], [d["seL"]], [d["seR"]], eta=ETA, outputs=(), orb_g=True,
                                  orb_ar=bias, defer=True)
    elif kind == "batch":
        st["ozaki"] = density.Ozaki(R=1e3, M_cut=case["poles"], n_gauss=case["gauss"])
        st["devices"] = [rgf_plan.DeviceBlocks(*x) for x in d["devices"]]
        st["leads"] = [tuple(surface_green.LeadBlocks(*x) for x in p) for p in d["leads"]]
    elif kind == "fit":
        st["leaves"] = [x.clone().requires_grad_(True) for x in d["leaves"]]
    elif kind == "lead":
        st["lead"] = [x.clone().requires_grad_(case["backward"]) for x in d["lead"]]
    return st


def run(st):
    case, d = st["case"], st["d"]
    kind = case["kind"]
    if kind == "tdos":
        T, D, _ = transport.transmission_dos(*d["blocks"], d["E"], d["seL"], d["seR"], eta=ETA,
                                             geometry=st["geometry"], precision=case["precision"])
        return {"T": T, "dos": D}
    if kind == "green":
        hd, hu, hl, sd, su, sl = d["blocks"]
        one = case["energies"] == 1
        pick = (lambda x: x[0]) if one else (lambda x: x)
        kw = {}
        if case["lesser"]:
            kw = dict(s_in=[pick(s) for s in d["s_in"]], need_lesser=True)
        r = recursive_green_cal.recursive_gf(pick(d["E"]), hl, hd, hu, sd, su, sl, pick(d["seL"]), pick(d["seR"]),
                                             eta=ETA, **kw)
        return dict(zip(recursive_green_cal.TAGS, r))
    if kind == "scf":
        st["plan"].launch()
        r = st["plan"].result
        return {"g": r.orb_g, "a": r.orb_ar}
    if kind == "batch":
        f = [(lambda e, mu=mu: _fermi(e, mu)) for mu in (BIAS / 2, -BIAS / 2)]
        return st["ozaki"].uneven_batch(st["devices"], st["leads"], KT, 0.0, vL=BIAS / 2, vR=-BIAS / 2, fermi_L=f[0],
                                        fermi_R=f[1], eta_lead=ETA, eta_device=ETA)
    if kind == "fit":
        return _fit_step(st["leaves"], d, lambda hd, hu, hl, sd, su, sl, seL, seR: adjoint.transmission_dos(
            hd, hu, hl, sd, su, sl, d["E"], seL, seR, eta=ETA))
    sig = adjoint.lead_self_energy(*st["lead"][:4], d["E"], _eta_lead(case), hDL=st["lead"][4], sDL=st["lead"][5])
    if not case["backward"]:
        return {"sigma": sig}
    return {"sigma": sig.detach(), "grad": torch.autograd.grad((d["weight"] * sig.real).sum(), st["lead"])}


def _fit_step(leaves, d, tdos):
    Hd, Hu, Sd, Su, seL, seR = leaves
    hd, hu, sd, su = (list(x.unbind(0)) for x in (Hd, Hu, Sd, Su))
    T, D = tdos(hd, hu, [u.mH for u in hu], sd, su, [u.mH for u in su], seL, seR)
    loss = (d["w_t"] * T).sum() + (d["w_d"] * D).sum()
    return {"T": T.detach(), "dos": D.detach(), "grad": torch.autograd.grad(loss, leaves)}


# ----------------------------------------------------------------------------- the work
def work(case):
    """Bytes in and out once, and the flops (8 per complex multiply-add) of the algorithm the results need:
    per block one inverse and seven products for T and DOS, and so on."""
    kind = case["kind"]
    if kind == "lead":
        n, B = case["n"], case["energies"]
        steps = 14 if case["backward"] else 20  # doubling steps at these broadenings
        fl = 8.0 * n ** 3 * B * (19.0 / 3.0 * steps + (4.0 * steps if case["backward"] else 0))
        return {"bytes": 16.0 * n * n * (6 + B + (0.5 * B + 6 if case["backward"] else 0)), "flops": fl}
    if kind == "batch":
        nE = 1 + case["poles"] + case["gauss"]
        fl = by = 0.0
        for b, L in _batch_shapes(case):
            fl += 8.0 * b ** 3 * nE * (7 * L + 2 * 19.0 / 3.0 * 20)
            by += 16.0 * b * b * 6 * L + 8.0 * nE + 16.0 * b * L
        return {"bytes": by, "flops": fl}
    dims, B = _dims(case), case["energies"]
    n3 = float(sum(n ** 3 for n in dims))
    n2 = float(sum(n * n for n in dims))
    K = len(dims)
    by = 16.0 * (6 * n2 + B * (dims[0] ** 2 + dims[-1] ** 2))
    if kind == "tdos":
        return {"bytes": by + 16.0 * B, "flops": 8.0 * B * n3 * (8 if case["overlap"] else 7)}
    if kind == "scf":
        return {"bytes": by + 24.0 * B * sum(dims), "flops": 8.0 * B * n3 * 7}
    if kind == "fit":
        return {"bytes": 2 * by, "flops": 8.0 * B * n3 * 25}
    fam = 7 if case["lesser"] else 4
    return {"bytes": by + 16.0 * B * n2 * fam, "flops": 8.0 * B * n3 * (22 if case["lesser"] else 8)}


# ----------------------------------------------------------------------------- 64-bit values
def _sweep(blocks, z, seL, seR, s_in=None):
    """The block-tridiagonal recursion in plain complex128 torch; every tag of ``recursive_gf``."""
    hd, hu, hl, sd, su, sl = blocks
    K, zz = len(hd), z.view(-1, 1, 1)
    A = [zz * s - h for h, s in zip(hd, sd)]
    A[0] = A[0] - seL
    A[-1] = A[-1] - seR
    U = [h - zz * s for h, s in zip(hu, su)]
    L = [h - zz * s for h, s in zip(hl, sl)]
    g, gin = [], []
    for q in range(K):
        D = A[q] if q == 0 else A[q] - L[q - 1] @ g[q - 1] @ U[q - 1]
        g.append(torch.linalg.solve(D, torch.eye(D.shape[-1], dtype=C128, device=D.device).expand(D.shape)))
        if s_in is not None:
            s = s_in[q] if q == 0 else s_in[q] + L[q - 1] @ gin[q - 1] @ U[q - 1]
            gin.append(g[q] @ s @ g[q].mH)
    grd, grl, gru, gc = [None] * K, [None] * (K - 1), [None] * (K - 1), [None] * K
    gnd, gnl = [None] * K, [None] * (K - 1)
    grd[-1] = gc[-1] = g[-1]
    if s_in is not None:
        gnd[-1] = gin[-1]
    for q in range(K - 2, -1, -1):
        gU = g[q] @ U[q]
        grl[q] = grd[q + 1] @ L[q] @ g[q]
        gru[q] = gU @ grd[q + 1]
        grd[q] = g[q] + gU @ grl[q]
        gc[q] = gU @ gc[q + 1]
        if s_in is not None:
            t = gnd[q + 1] @ L[q] @ g[q].mH
            gnl[q] = grd[q + 1] @ L[q] @ gin[q] + t
            gnd[q] = gin[q] + gU @ t + gin[q] @ U[q] @ gru[q].mH + gru[q] @ L[q] @ gin[q]
    r = dict(g_trans=gc[0], gc=gc, grd=grd, grl=grl, gru=gru, gr_left=g)
    if s_in is not None:
        r.update(gnd=gnd, gnl=gnl, gnu=[x.mH for x in gnl], gin_left=gin)
    return r


def _t_dos(blocks, z, seL, seR):
    r = _sweep(blocks, z, seL, seR)
    _, _, _, sd, su, sl = blocks
    gam = [1j * (s - s.mH) for s in (seL, seR)]
    gt = r["g_trans"]
    T = torch.einsum("bij,bij->b", gam[0] @ gt @ gam[1], gt.conj()).real
    tr = lambda a, b: (a * b.mT).sum((-2, -1))
    D = sum(tr(a, s) for a, s in zip(r["grd"], sd)) + sum(tr(a, s) for a, s in zip(r["grl"], su)) + \
        sum(tr(a, s) for a, s in zip(r["gru"], sl))
    return T, -2.0 / math.pi * D.imag


def _spectra(blocks, z, seL, seR):
    r = _sweep(blocks, z, seL, seR)
    gam = 1j * (seR - seR.mH)
    g = torch.cat([x.diagonal(dim1=-2, dim2=-1) for x in r["grd"]], -1)
    a = torch.cat([((x @ gam) * x.conj()).sum(-1).real for x in r["gc"]], -1)
    gL = 1j * (seL - seL.mH)
    T = ((gL @ r["g_trans"] @ gam) * r["g_trans"].conj()).sum((-2, -1)).real
    return g, a, T


def _decimate(lead, E, eta):
    """Sigma(E) of one lead by the doubling iteration, batched over E."""
    h, h01, s, s01, hdl, sdl = lead
    E = E.to(C128).view(-1, 1, 1)
    z = E + 1j * eta
    al, be = h01.mH - z * s01.mH, h01 - z * s01
    eps = epss = h.expand(len(E), -1, -1)
    n = h.shape[-1]
    for _ in range(60):
        x = torch.linalg.solve(z * s - eps, torch.cat([al, be], -1))
        xa, xb = x[..., :n], x[..., n:]
        bxa = be @ xa
        eps, epss = eps + al @ xb + bxa, epss + bxa
        al, be = al @ xa, be @ xb
        if float((al.abs() + be.abs()).max().detach()) < 1e-40:
            break
    g = torch.linalg.inv(z * s - epss)
    return (E * sdl - hdl) @ g @ (E * sdl.mH - hdl.mH)


def _chunks(B, n):
    step = max(1, min(B, int(6e7 / max(1, n))))
    return [(a, min(B, a + step)) for a in range(0, B, step)]


def exact(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    if kind == "lead":
        lead = [x.clone().requires_grad_(case["backward"]) for x in d["lead"]]
        sigs, grads = [], None
        for a, b in _chunks(case["energies"], (200 if case["backward"] else 10) * case["n"] ** 2):
            sig = _decimate(lead, d["E"][a:b].cuda(), _eta_lead(case))
            sigs.append(sig.detach())
            if case["backward"]:
                g = torch.autograd.grad((d["weight"][a:b] * sig.real).sum(), lead)
                grads = g if grads is None else tuple(x + y for x, y in zip(grads, g))
        sig = torch.cat(sigs)
        return {"sigma": sig, "grad": grads} if case["backward"] else {"sigma": sig}
    if kind == "batch":
        oz = density.Ozaki(R=1e3, M_cut=case["poles"], n_gauss=case["gauss"])  # its nodes and weights only
        xl, xu = -BIAS / 2 - 8 * KT, BIAS / 2 + 8 * KT
        x, w = (torch.tensor(v) for v in np.polynomial.legendre.leggauss(case["gauss"]))
        x, w = x * (0.5 * (xu - xl)) + 0.5 * (xu + xl), w * (0.5 * (xu - xl))
        p, res = oz.poles.to(F64), oz.residues.to(F64).cuda()
        zs = torch.cat([torch.tensor([1j * 1e3], dtype=C128), 1j * p * KT, x.to(C128)]).cuda()
        df = (_fermi(x, -BIAS / 2) - _fermi(x, BIAS / 2)).cuda()
        out = []
        for blocks, (lL, lR) in zip(d["devices"], d["leads"]):
            seL, seR = _decimate(lL, zs, ETA), _decimate(lR, zs, ETA)
            g, a, T = _spectra(blocks, zs + 1j * ETA, seL, seR)
            P = len(p)
            n_eq = (1j * 1e3 * g[0]).real - ((-4j * KT) * g[1:1 + P] * res.view(-1, 1)).imag.sum(0)
            n_neq = ((w.cuda() * df).view(-1, 1) * a[1 + P:]).sum(0)
            out.append({"n_eq": n_eq, "n_neq": n_neq, "energy": x, "trans": T[1 + P:]})
        return out
    z = d["E"].to(C128) + 1j * ETA
    n_el = sum(n * n for n in _dims(case))
    if kind == "fit":
        leaves = [x.clone().requires_grad_(True) for x in d["leaves"]]
        acc = None
        for a, b in _chunks(case["energies"], 6 * n_el):
            part = {k: d[k][a:b] for k in ("w_t", "w_d")}
            mine = leaves[:4] + [x[a:b].detach().requires_grad_(True) for x in leaves[4:]]
            r = _fit_step(mine, part, lambda hd, hu, hl, sd, su, sl, L, R: _t_dos((hd, hu, hl, sd, su, sl), z[a:b], L, R))
            if acc is None:
                acc = {"T": [r["T"]], "dos": [r["dos"]], "grad": [list(r["grad"][:4]), [r["grad"][4]], [r["grad"][5]]]}
            else:
                acc["T"].append(r["T"])
                acc["dos"].append(r["dos"])
                acc["grad"][0] = [x + y for x, y in zip(acc["grad"][0], r["grad"][:4])]
                acc["grad"][1].append(r["grad"][4])
                acc["grad"][2].append(r["grad"][5])
        return {"T": torch.cat(acc["T"]), "dos": torch.cat(acc["dos"]),
                "grad": tuple(acc["grad"][0]) + (torch.cat(acc["grad"][1]), torch.cat(acc["grad"][2]))}
    if kind == "green":
        r = _sweep(d["blocks"], z, d["seL"], d["seR"], d.get("s_in"))
        r = {t: r.get(t) for t in recursive_green_cal.TAGS}
        if case["energies"] == 1:
            r = {t: None if v is None else (v[0] if torch.is_tensor(v) else [x[0] for x in v]) for t, v in r.items()}
        return r
    parts = []
    for a, b in _chunks(case["energies"], 12 * n_el):
        args = (d["blocks"], z[a:b], d["seL"][a:b], d["seR"][a:b])
        parts.append(_t_dos(*args) if kind == "tdos" else _spectra(*args))
    if kind == "tdos":
        return {"T": torch.cat([p[0] for p in parts]), "dos": torch.cat([p[1] for p in parts])}
    bias = case["energies"] > case["poles"]
    return {"g": torch.cat([p[0].reshape(-1) for p in parts]),
            "a": torch.cat([p[1].reshape(-1) for p in parts]) if bias else None}
