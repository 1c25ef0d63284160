"""The query engine's walk trees against the reference traversal.

A store of the reference split collects a ray's candidates on a second tree
over the same leaves and restores the reference traversal's order from the
reference tree's boxes.  Where that could go wrong is where the order decides:
roots at exactly equal distances (here: copies of the same patches and
objects), and where a ray's candidates do not fit in its list (here: stacks of
up to 150 patches over every ray, lists of 4 to 64 entries).  The parity build
is held bit for bit to the oracle, which walks the reference tree alone."""
import struct

import numpy as np
import pytest

from cgspline_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def stacked(copies: int, n: int = 2, objects: int = 1) -> S.Scene:
    """`copies` copies of an n x n field: pairs at the same height (ties), the pairs 1/64 apart."""
    s = S.heightfield(5, n=n)
    pts, idx = [], []
    for c in range(copies):
        p = s.points.copy()
        p[:, 2] -= np.float32(c // 2) / np.float32(64.0)
        pts.append(p)
        idx.append(s.indices + np.uint32(c * p.shape[0]))
    surf = S.Surface(np.concatenate(pts), np.concatenate(idx).astype(np.uint32))
    obs = []
    for k in range(objects):
        l2w, w2l = S.IDENTITY16.copy(), S.IDENTITY16.copy()
        l2w[12], w2l[12] = np.float32(k // 2), -np.float32(k // 2)  # objects 2i and 2i + 1 coincide
        obs.append(S.Object(0, l2w, w2l))
    return S.Scene([surf], obs, S.scene_c1().lights, name=f"stacked{copies}")


def field_rays(n: int, side: int = 40) -> np.ndarray:
    """Oblique rays over an n x n field: from above, from below and along it, with the field's lines among them."""
    g = np.linspace(0.0, n, side)
    x, y = (v.reshape(-1) for v in np.meshgrid(g, g, indexing="ij"))
    rays = []
    for d in ((0.3, 0.2, -0.9), (-0.2, 0.4, 0.9), (0.99, 0.05, -0.12), (0.0, 0.6, -0.8)):
        d = np.array(d) / np.sqrt(np.dot(d, d))
        o = np.stack([x, y, np.zeros_like(x)]) - 6.0 * d[:, None]
        rays.append(np.concatenate([o, np.repeat(d[:, None], x.size, 1), np.full((1, x.size), np.inf)]))
    return np.ascontiguousarray(np.concatenate(rays, axis=1), dtype=np.float32)


@pytest.mark.parametrize("copies,objects,engine", [
    (1, 1, {}), (2, 1, {}), (3, 3, {}), (15, 1, {}), (15, 5, {}), (31, 1, {}), (64, 1, {}), (150, 1, {}), (150, 2, {}),
    (15, 3, {"queue_chunk": 4, "passes": 8}), (64, 1, {"queue_chunk": 8, "passes": 3}),
    (15, 5, {"queue_chunk": 16, "passes": 4, "backtrack_cache": 0}), (64, 2, {"passes": 1, "packet_width": 1}),
])
def test_ties_and_full_lists_match_the_reference_order(copies, objects, engine, oracle_mod):
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import _capi, rt
    sc = stacked(copies, objects=objects)
    rays = field_rays(2)
    scene = oracle_mod.OracleScene(sc)
    ref = scene.intersect(rays, method=oracle_mod.CLIP_DEVICE)
    occluded = scene.intersect(rays, method=oracle_mod.CLIP_DEVICE, any_hit=True)["patch"] >= 0
    assert (ref["patch"] >= 0).mean() > 0.4
    lib = _capi.load(_capi.LIB_NOFMA_PATH)
    import ctypes as C
    base = _capi.EngineConfig()
    _capi.check(lib.cgs_engine_config_get(C.byref(base)), "get")
    cfg = _capi.EngineConfig(**{**{k: getattr(base, k) for k, _ in base._fields_}, **engine})
    g = rt.GpuScene(sc, lib_path=_capi.LIB_NOFMA_PATH)
    try:
        _capi.check(lib.cgs_engine_config_set(C.byref(cfg)), "set")
        dev = torch.from_numpy(rays).cuda()
        got = {k: v.cpu().numpy() for k, v in g.intersect(dev).items()}
        free = g.intersect(dev, any_hit=True)["patch"].cpu().numpy() < 0
        assert g.counters()["device_errors"] == 0
    finally:
        lib.cgs_engine_config_set(C.byref(base))
        g.close()
    for k in ("t", "u", "v", "patch", "object"):
        assert np.array_equal(got[k], ref[k]), (k, int((got[k] != ref[k]).sum()))
    assert np.array_equal(free, ~occluded)


@pytest.mark.parametrize("copies,objects", [(31, 1), (32, 1), (90, 1), (120, 1), (130, 1), (150, 2), (15, 7)])
@pytest.mark.parametrize("n", [37, 70001])
def test_long_lists_match_the_reference(copies, objects, n, oracle_mod):
    """A few rays whose candidates outgrow their chunk, alone and among 70,000 rays that miss: they go on in long lists
    (one of 256 entries each), which are sorted by a warp; past that, on the reference tree."""
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import _capi, rt
    sc = stacked(copies, objects=objects)
    rays = np.ascontiguousarray(field_rays(2)[:, :: 173])  # 37 rays
    ref = oracle_mod.OracleScene(sc).intersect(rays, method=oracle_mod.CLIP_DEVICE)
    assert rays.shape[1] <= 37 and (ref["patch"] >= 0).mean() > 0.4
    at = np.linspace(0, n - 1, rays.shape[1]).astype(np.int64)
    many = np.zeros((7, n), np.float32)
    many[2], many[5], many[6] = 50.0, 1.0, np.inf
    many[:, at] = rays
    g = rt.GpuScene(sc, lib_path=_capi.LIB_NOFMA_PATH)
    dev = torch.from_numpy(many).cuda()
    got = {k: v.cpu().numpy() for k, v in g.intersect(dev).items()}
    free = g.intersect(dev, any_hit=True)["patch"].cpu().numpy() < 0
    assert g.counters()["device_errors"] == 0
    g.close()
    for k in ("t", "u", "v", "patch", "object"):
        assert np.array_equal(got[k][at], ref[k]), (k, int((got[k][at] != ref[k]).sum()))
    assert (np.delete(got["patch"], at) < 0).all()
    assert np.array_equal(free[at], ref["patch"] < 0)


def test_loaded_store_walks_its_own_trees(tmp_path):
    """A store read back gives the built one's hits; one whose file hides the root's left half behind an empty box is
    walked as the file says."""
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import rt
    sc = stacked(15)
    rays = torch.from_numpy(field_rays(2)).cuda()
    g = rt.GpuScene(sc)
    want = {k: v.cpu().numpy() for k, v in g.intersect(rays).items()}
    nodes = g.counters()["nodes"]
    path = tmp_path / "store.cgs"
    g.save(str(path))
    left = g.bvh(0)
    g.close()
    h = rt.GpuScene.load(str(path))
    got = {k: v.cpu().numpy() for k, v in h.intersect(rays).items()}
    assert h.counters()["nodes"] == nodes
    h.close()
    for k in want:
        assert np.array_equal(got[k], want[k]), k
    data = bytearray(path.read_bytes())
    at = 6 * 4
    for width in (4, 4):  # the surface's points and indices
        at += 4 + struct.unpack_from("<I", data, at)[0] * width
    struct.pack_into("<6f", data, at + 4, *([1e30] * 3 + [2e30] * 3))  # the root's left box
    path.write_bytes(bytes(data))
    h = rt.GpuScene.load(str(path))
    got = h.intersect(rays)["patch"].cpu().numpy()
    h.close()
    # pre-order: the right half's leaves are those from the root's right child on
    first = int(left["nodes"][0, 13])
    leaves = [int(left["indices"][n[13]]) for n in left["nodes"][first:] if n[12] == 0xFFFFFFFF]
    assert (got >= 0).any() and np.isin(got[got >= 0], leaves).all()
