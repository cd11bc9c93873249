"""How calls reach the kernels: packing, empty problems, little memory, the inverse's
widths, threads."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_geometry_is_built_under_capture():
    """With detect_zero_offdiag=False a Geometry of device tensors reads nothing back, so it can be captured; a
    replay packs the blocks' new values."""
    from dpnegf_b200 import rgf_plan
    gen = torch.Generator(device="cuda").manual_seed(11)
    r = lambda *s: torch.complex(*(torch.randn(*s, generator=gen, dtype=torch.float64, device="cuda") for _ in range(2)))
    parts = [[r(3, 3), r(5, 5)], [r(3, 5)], [r(5, 3)], [r(3, 3), r(5, 5)], [r(3, 5)], [r(5, 3)]]
    build = lambda: rgf_plan.Geometry([rgf_plan.DeviceBlocks(*parts)], detect_zero_offdiag=False)
    build()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        geom = build()
    for t in (t for p in parts for t in p):
        t.copy_(r(*t.shape))
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(geom.hs, build().hs)


def test_no_devices():
    """A plan over no devices launches nothing and has empty results; a direct call is refused."""
    from dpnegf_b200 import _lib, rgf_plan
    kw = dict(eta=1e-5, outputs=(), trans=True, dos=True)
    plan = rgf_plan.run(rgf_plan.Geometry([]), [], [], [], defer=True, **kw)
    plan.launch()
    plan.check()
    assert plan.result.trans.numel() == plan.result.dos.numel() == 0 and plan.result.blocks == []
    with pytest.raises(_lib.NegfError, match="invalid argument"):
        rgf_plan.run(rgf_plan.Geometry([]), [], [], [], **kw)


def _device(K, n, B, seed):
    from dpnegf_b200 import rgf_plan, workload
    d = workload.random_device(n, K, seed=seed)
    geom = rgf_plan.Geometry([rgf_plan.DeviceBlocks(d.hd, d.hu, d.hl, d.sd, d.su, d.sl)])
    E = workload.energy_grid(B).to(torch.complex128).cuda()
    seL, seR = (workload.random_self_energy(B, n, seed=seed + k).cuda() for k in (1, 2))
    return geom, [E], [seL], [seR]


def test_gradient_fits_where_only_the_kept_products_do_not():
    """Memory for everything but half of the kept L g: the gradient call does without it.  L g alone is one
    product regrouped, so the results agree to rounding."""
    from dpnegf_b200 import rgf_plan
    K, n, B = 64, 64, 80
    args = _device(K, n, B, 40)
    w = torch.linspace(0.2, 1.0, B, dtype=torch.float64)
    run = lambda: rgf_plan.run(*args, eta=1e-3, outputs=(), adjoint_w=w)
    run()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.reset_peak_memory_stats()
    want = run()
    peak = torch.cuda.max_memory_allocated()
    want = want.trans.clone(), [x.clone() for x in want.grads["hd"]]
    torch.cuda.empty_cache()
    kept = B * K * n * n * 16
    total = torch.cuda.get_device_properties(0).total_memory
    torch.cuda.set_per_process_memory_fraction((peak - kept // 2) / total)
    try:
        got = run()
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert float((got.trans - want[0]).abs().max()) <= 1e-10 * float(want[0].abs().max())
    for x, y in zip(got.grads["hd"], want[1]):
        assert float((x - y).abs().max()) <= 1e-10 * float(y.abs().max())


@pytest.mark.parametrize("K,n,keeps", [(4, 64, True), (320, 64, False)])
def test_deferred_plan_keeps_little(K, n, keeps):
    """A deferred plan holds its scratch for its life: L g is kept where it is small, and only there."""
    from dpnegf_b200 import _lib, rgf_plan
    sms = _lib.load().negf_sm_count()
    plan = rgf_plan.run(*_device(K, n, sms, 41), eta=1e-3, outputs=(), trans=True, dos=True, defer=True)
    kept = sms * K * n * n * 16
    assert (kept <= torch.cuda.get_device_properties(0).total_memory // 64) == keeps
    assert bool(plan.prob.flags & _lib.KEEP_LG) == keeps


@pytest.mark.parametrize("K,n,many", [(4, 8, True), (256, 32, False)])
def test_deferred_plan_takes_extra_slots_where_they_are_small(K, n, many):
    from dpnegf_b200 import _lib, rgf_plan
    sms = _lib.load().negf_sm_count()
    plan = rgf_plan.run(*_device(K, n, 3 * sms, 42), eta=1e-3, outputs=(), trans=True, dos=True, defer=True)
    assert plan.prob.n_slots == (3 * sms if many else sms)


def test_deferred_plan_takes_nothing_large_of_a_half_full_gpu():
    from dpnegf_b200 import _lib, rgf_plan
    sms = _lib.load().negf_sm_count()
    args = _device(96, 32, 3 * sms, 43)
    build = lambda: rgf_plan.run(*args, eta=1e-3, outputs=(), trans=True, dos=True, defer=True)
    full = torch.empty(int(0.52 * torch.cuda.get_device_properties(0).total_memory), dtype=torch.uint8, device="cuda")
    plan = build()
    del full
    assert plan.prob.n_slots == sms and not plan.prob.flags & _lib.KEEP_LG
    plan = build()
    assert plan.prob.n_slots == 3 * sms and plan.prob.flags & _lib.KEEP_LG


def test_outer_block_width_is_honoured_with_few_items():
    """inverse="gj" runs with the outer block width it is given, however few the items: two widths sum in two
    orders, so they agree to rounding (TOL of test_rgf_gpu's blocks) and not bitwise."""
    from dpnegf_b200 import rgf_plan
    args = _device(3, 160, 2, 43)
    grd = [rgf_plan.run(*args, eta=1e-3, outputs=("grd",), inverse="gj", inv_ob=ob).blocks[0]["grd"][0]
           for ob in (32, 64, 128)]
    for x in grd[1:]:
        assert not torch.equal(x, grd[0])
        assert float((x - grd[0]).abs().max()) <= 1e-10 * float(grd[0].abs().max())


@pytest.mark.parametrize("K,packs", [(1, 0), (2, 1), (5, 1)])
def test_one_block_is_copied(K, packs, monkeypatch):
    """A device of one block has three pieces, fewer than a pack launch pays for."""
    from dpnegf_b200 import _lib, rgf_plan
    lib, calls = _lib.load(), []
    run = lib.negf_pack_run
    monkeypatch.setattr(lib, "negf_pack_run", lambda *a: calls.append(a) or run(*a))
    eye = torch.eye(7, dtype=torch.complex128, device="cuda")
    geom = rgf_plan.Geometry([rgf_plan.DeviceBlocks([eye] * K, *([[2 * eye] * (K - 1)] * 2), [3 * eye] * K,
                                                    *([[4 * eye] * (K - 1)] * 2))])
    assert len(calls) == packs
    for off, v in ((geom.blocks[0]["hd"], 1), (geom.blocks[K - 1]["sd"], 3)):
        assert torch.equal(geom.hs[int(off):int(off) + 49].view(7, 7), v * eye)


@pytest.mark.parametrize("ctas", [0, 1])
def test_threads_launch_problems_of_different_sizes(ctas):
    """Two threads on two streams launch sweeps that need different amounts of shared memory: neither may take
    the other's limit away between setting it and launching."""
    import threading
    from dpnegf_b200 import rgf_plan
    plans = [rgf_plan.run(*_device(1, n, 1, 44 + n), eta=1e-3, outputs=(), trans=True, defer=True, ctas=ctas)
             for n in (40, 256)]
    for p in plans:
        p.launch()
    torch.cuda.synchronize()
    want, errors = [p.result.trans.clone() for p in plans], []

    def work(p):
        s = torch.cuda.Stream()
        try:
            for k in range(3000):
                p.launch(s)
                if k % 64 == 0:
                    s.synchronize()
            s.synchronize()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(p,)) for p in plans]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors
    for p, w in zip(plans, want):
        p.check()
        assert torch.equal(p.result.trans, w)
