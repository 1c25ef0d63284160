"""A render's queries (closest hits and shadow rays of each level) have the long
candidate lists to themselves, one after another: a level whose rays take all of
them leaves the next level as many.  Counted by node visits: the bounce level of a
frame over stacked patches costs what a query of the same rays alone costs."""
import numpy as np
import pytest

from cgspline_gb300 import scenes as S

pytestmark = pytest.mark.gpu

SIDE, COPIES = 8, 100


def scene():
    """A floor and, in the direction of its mirror rays, a ceiling: each 100 copies of a field, 1/64 apart, so that a ray
    has some 100 candidates.  One of the floor's 64 cells is a mirror."""
    s = S.heightfield(5, sigma=0.01, n=SIDE)
    pts, idx = [], []
    for c in range(COPIES):
        p = s.points.copy()
        p[:, 2] -= np.float32(c) / np.float32(64.0)
        pts.append(p)
        idx.append(s.indices + np.uint32(c * p.shape[0]))
    surf = S.Surface(np.concatenate(pts), np.concatenate(idx).astype(np.uint32))
    mirror = (np.arange(surf.patch_count) % (SIDE * SIDE) == SIDE * SIDE // 2 + SIDE // 2).astype(np.uint32)
    mats = [S.Material(roughness=1.0), S.Material(roughness=0.0)]  # a rough one reflects nothing
    l2w, w2l = S.IDENTITY16.copy(), S.IDENTITY16.copy()
    up, down = S.IDENTITY16.copy(), S.IDENTITY16.copy()
    up[13], up[14] = 9.0, 5.5
    down[13], down[14] = -9.0, -5.5
    none = np.zeros_like(mirror)
    return S.Scene([surf], [S.Object(0, l2w, w2l, mats[0], mirror, mats), S.Object(0, up, down, mats[0], none, mats)], [],
                   name="floor"), mirror


# a one-launch query and one of separate kernels
@pytest.mark.parametrize("width,height", [(160, 100), (480, 300)])
def test_bounce_level_has_the_lists_again(width, height):
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import rt
    sc, mirror = scene()
    eye = (SIDE / 2, -9.0, 9.0)
    cam = S.Camera(rotation=S.look_at(eye, (SIDE / 2, SIDE / 2, 0.0)), position=eye, fovy=0.65)
    g = rt.GpuScene(sc)
    nodes = []
    for depth in (0, 1):
        f = rt.Frame(width, height)
        rt.RayTracer(rt.Options(recursion_depth=depth)).render(f, cam, g)
        torch.cuda.synchronize()
        c = g.counters()
        nodes.append(c["nodes"])
        rays_traced = c["rays"]
        assert c["device_errors"] == 0
    prim = rt.camera_rays(cam, width, height)
    h = g.intersect(prim)
    at = torch.nonzero((h["object"] == 0) & (torch.from_numpy(mirror.astype(np.int64)).cuda()[h["patch"].long().clamp(min=0)] > 0)
                       ).reshape(-1)
    n = width * height
    needy = int((h["object"] == 0).sum())
    lists = n // 48 + 32
    assert needy > 4 * lists and 30 < at.numel() <= lists and rays_traced == n + at.numel()
    d, t = prim[3:6, at], h["t"][at]
    nrm = rt.normal(g, 0, h["patch"][at], h["u"][at], h["v"][at])
    r = d - 2.0 * (d * nrm).sum(0) * nrm
    bounce = torch.cat([prim[0:3, at] + t * d + 1e-4 * r, r, torch.full((1, at.numel()), float("inf"), device="cuda")])
    b = g.intersect(bounce)
    assert ((b["object"] == 1).float().mean() > 0.5)
    alone = g.counters()["nodes"]
    level = nodes[1] - nodes[0]
    assert level <= 1.05 * alone, (level, alone)
    g.close()
