"""How calls reach the kernels: packing under stream capture, empty problems."""
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
