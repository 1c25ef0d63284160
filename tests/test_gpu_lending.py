"""Lanes without rays borrow intervals of their warp's longest searches, so how a
search is split depends on what else runs.  Its result must not: the same rays
alone, in small sets and in one large set, in both orders, give the same hits bit
for bit, for both intersectors, closest and any hit, and the closest hits of the
parity build are the oracle's.  The field of stacked copies has roots at equal
distances; the rays along it have the longest searches."""
import numpy as np
import pytest

from cgspline_gb300 import scenes as S

from test_gpu_walk import field_rays, stacked

pytestmark = pytest.mark.gpu


def scene_and_rays(name):
    if name == "stacked":
        return stacked(9, n=2), field_rays(2, side=20)
    sc = S.scene_c2(nu=32, nv=32)
    return sc, S.grazing_rays(sc.surfaces[0], 1500, seed=8, max_deg=4.0)


@pytest.mark.parametrize("name", ["stacked", "torus"])
@pytest.mark.parametrize("method", [0, 1])
@pytest.mark.parametrize("any_hit", [False, True])
def test_results_do_not_depend_on_the_batch(name, method, any_hit, oracle_mod):
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import _capi, rt
    sc, rays = scene_and_rays(name)
    g = rt.GpuScene(sc, lib_path=_capi.LIB_NOFMA_PATH)
    keys = ["patch"] if any_hit else ["t", "u", "v", "patch", "object"]

    def run(r):
        h = g.intersect(torch.from_numpy(np.ascontiguousarray(r)).cuda(), method=method, any_hit=any_hit)
        return {k: h[k].cpu().numpy() for k in keys}

    whole = run(rays)
    n = rays.shape[1]
    back = run(rays[:, ::-1])
    many = run(np.tile(rays, (1, 40)))
    for k in keys:
        assert np.array_equal(whole[k], back[k][::-1]), k
        assert np.array_equal(np.tile(whole[k], 40), many[k]), k
    for size in (1, 3, 33):
        for at in range(0, min(n, 40 * size), size):
            part = run(rays[:, at:at + size])
            for k in keys:
                assert np.array_equal(part[k], whole[k][at:at + size]), (k, size, at)
    assert g.counters()["device_errors"] == 0
    g.close()
    ref = oracle_mod.OracleScene(sc).intersect(rays, method=oracle_mod.SUBDIV if method else oracle_mod.CLIP_DEVICE,
                                               any_hit=any_hit)
    if any_hit:
        assert np.array_equal(whole["patch"] >= 0, ref["patch"] >= 0)
        return
    for k in keys:
        assert np.array_equal(whole[k], ref[k]), (k, int((whole[k] != ref[k]).sum()))
