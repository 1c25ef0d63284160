"""The query engine's separate kernels (queries of more than 65,536 rays, 32,768 for
subdivision, or on compressed nodes) where the order and the lists decide: the
stacked copies of test_gpu_walk.py and the union scene, over settings that park
rays, resume them and change the blocks, bit for bit against the oracle; and
the lending tests' rays among many.  That the kernels in question ran is told by
the launch count: a smaller query is one launch."""
import ctypes as C

import numpy as np
import pytest

from cgspline_gb300 import scenes as S

from test_gpu_lending import scene_and_rays
from test_gpu_walk import field_rays, stacked

pytestmark = pytest.mark.gpu

KEYS = ("t", "u", "v", "patch", "object")


class Engine:
    """The parity build's engine settings, set for a while."""

    def __init__(self, **settings):
        from cgspline_gb300 import _capi
        self.capi, self.lib = _capi, _capi.load(_capi.LIB_NOFMA_PATH)
        self.base = _capi.EngineConfig()
        _capi.check(self.lib.cgs_engine_config_get(C.byref(self.base)), "get")
        self.now = _capi.EngineConfig(**{**{k: getattr(self.base, k) for k, _ in self.base._fields_}, **settings})

    def __enter__(self):
        self.capi.check(self.lib.cgs_engine_config_set(C.byref(self.now)), "set")

    def __exit__(self, *exc):
        self.capi.check(self.lib.cgs_engine_config_set(C.byref(self.base)), "set")


def hits(g, rays, **kw):
    """Host copies of the hits, and the query's launches."""
    h = {k: v.cpu().numpy() for k, v in g.intersect(rays, **kw).items()}
    c = g.counters()
    assert c["device_errors"] == 0
    return h, c["kernel_launches"]


SETTINGS = [
    {}, {"queue_chunk": 4, "passes": 8}, {"queue_chunk": 4, "passes": 1, "collect_threads": 128, "resolve_threads": 64},
    {"queue_chunk": 8, "passes": 3, "collect_threads": 128, "backtrack_cache": 0},
    {"queue_chunk": 16, "passes": 4, "resolve_threads": 64, "packet_width": 32},
    {"compressed_nodes": 1}, {"compressed_nodes": 1, "queue_chunk": 8, "passes": 2, "packet_width": 1},
]


@pytest.mark.parametrize("copies,objects", [(3, 3), (15, 5), (64, 1), (150, 2)])
def test_ties_and_full_lists(copies, objects, oracle_mod):
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import _capi, rt
    sc = stacked(copies, objects=objects)
    rays = field_rays(2, side=20)
    n = rays.shape[1]
    scene = oracle_mod.OracleScene(sc)
    ref = scene.intersect(rays, method=oracle_mod.CLIP_DEVICE)
    occluded = scene.intersect(rays, method=oracle_mod.CLIP_DEVICE, any_hit=True)["patch"] >= 0
    assert (ref["patch"] >= 0).mean() > 0.4
    many = 66000 // n + 1
    order = np.random.RandomState(copies).permutation(many * n) % n
    g = rt.GpuScene(sc, lib_path=_capi.LIB_NOFMA_PATH)
    dev = torch.from_numpy(np.ascontiguousarray(rays[:, order])).cuda()
    for s in SETTINGS:
        if s.get("compressed_nodes"):  # its wider boxes let rays that run in a box's face meet more
            continue
        with Engine(**s):
            got, launches = hits(g, dev)
            assert launches > 4
            for k in KEYS:
                assert np.array_equal(got[k], ref[k][order]), (s, k, int((got[k] != ref[k][order]).sum()))
            free, launches = hits(g, dev, any_hit=True)
            assert launches > 4
            assert np.array_equal(free["patch"] >= 0, occluded[order]), s
    g.close()


@pytest.mark.parametrize("settings", SETTINGS)
def test_union_scene_across_list_chunks(settings, oracle_mod):
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import _capi, rt
    sc, cam = S.scene_c4(5), S.camera_c4(5)[0]
    rays = oracle_mod.camera_rays(cam, 280, 240)
    ref = oracle_mod.OracleScene(sc).intersect(rays, method=oracle_mod.CLIP_DEVICE)
    g = rt.GpuScene(sc, lib_path=_capi.LIB_NOFMA_PATH)
    with Engine(**settings):
        got, launches = hits(g, torch.from_numpy(rays).cuda())
    g.close()
    assert launches > 4
    for k in KEYS:
        assert np.array_equal(got[k], ref[k]), (k, int((got[k] != ref[k]).sum()))


@pytest.mark.parametrize("name", ["stacked", "torus"])
@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("any_hit", [False, True])
@pytest.mark.parametrize("resolve_threads", [64, 128])
def test_lending_among_many_rays(name, method, any_hit, resolve_threads):
    """The rays of the lending tests, a few hundred of them spread over a query that the separate kernels run."""
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import _capi, rt
    sc, rays = scene_and_rays(name)
    g = rt.GpuScene(sc, lib_path=_capi.LIB_NOFMA_PATH)
    whole, launches = hits(g, torch.from_numpy(rays).cuda(), method=method, any_hit=any_hit)
    assert launches == 1
    keys = ["patch"] if any_hit else KEYS
    n = rays.shape[1]
    for total in (66000, 150001):
        order = np.random.RandomState(total).randint(0, n, total)
        with Engine(resolve_threads=resolve_threads):
            got, launches = hits(g, torch.from_numpy(np.ascontiguousarray(rays[:, order])).cuda(), method=method,
                                 any_hit=any_hit)
        assert launches > 4
        for k in keys:
            assert np.array_equal(got[k], whole[k][order]), (k, int((got[k] != whole[k][order]).sum()))
    g.close()


def test_autotune_keeps_settings_without_effect():
    """On a batch whose queries are one launch each the block sizes and occupancies do nothing: the autotuner leaves them
    as they were set."""
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import rt
    g = rt.GpuScene(S.scene_c2(nu=16, nv=16))
    base = rt.engine_config()
    req = [rt.Request.alloc(0, S.camera_c2(), 64, 36)]
    try:
        for ct, rtn, occ in ((128, 64, 6), (256, 128, 0), (128, 128, 0), (256, 64, 3)):
            rt.set_engine_config(**{**base, "collect_threads": ct, "resolve_threads": rtn, "collect_occupancy": occ,
                                    "compressed_nodes": 0})
            cfg, ms = rt.autotune(g, req, rt.Options(recursion_depth=1), repeats=1)
            assert ms > 0 and cfg == rt.engine_config()
            if not cfg["compressed_nodes"]:
                assert (cfg["collect_threads"], cfg["resolve_threads"], bool(cfg["collect_occupancy"])) == (ct, rtn, bool(occ))
    finally:
        rt.set_engine_config(**base)
        g.close()
