"""A server whose budget holds a handful of samples at a time serves renders and
queries tile by tile, with the results of unlimited ones."""
import numpy as np
import pytest

from cgspline_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("budget,width", [(12 << 10, 1), (40 << 10, 3), (100 << 10, 11)])
def test_server_of_a_few_kilobytes(budget, width):
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import rt
    g = rt.GpuScene(S.scene_c2(nu=16, nv=16))
    cam = S.camera_c2()
    rays = rt.camera_rays(cam, 8, 6)
    want = g.intersect(rays)
    whole = rt.Request.alloc(0, cam, width, 4, linear=True)
    rt.RayTracer(rt.Options(recursion_depth=1)).render_batch([whole], g)
    torch.cuda.synchronize()
    sv = rt.Server(g, slots=1, memory_budget=budget, max_batch_requests=1, options=rt.Options(recursion_depth=1))
    req = rt.Request.alloc(0, cam, width, 4, linear=True)
    try:
        a = sv.submit_render(req)
        b, hits = sv.submit_query(0, rays)
        for t in (a, b):
            sv.wait(t, 60.0)
    finally:
        sv.close()
    assert torch.equal(req.linear, whole.linear)
    for k in want:
        assert torch.equal(hits[k], want[k]), k
    g.close()
