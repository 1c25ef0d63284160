"""Loading a store builds its walk trees on all of the host's cores, as building one
does: many surfaces side by side, one large surface's tree in subtrees; the same
trees as a build's."""
import os
import time

import numpy as np
import pytest

from cgspline_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def store(name):
    if name == "large":
        return S.scene_c2(nu=600, nv=300)
    fields = [S.heightfield(k, n=68) for k in range(1, 41)]  # 4,624 patches each
    obs = []
    for k in range(len(fields)):  # side by side
        l2w, w2l = S.IDENTITY16.copy(), S.IDENTITY16.copy()
        l2w[12], l2w[13] = 70.0 * (k % 8), 70.0 * (k // 8)
        w2l[12:14] = -l2w[12:14]
        obs.append(S.Object(k, l2w, w2l))
    return S.Scene(fields, obs, S.scene_c1().lights, name="fields")


@pytest.mark.parametrize("name", ["large", "many"])
def test_walk_trees_of_a_loaded_store_are_built_by_all_cores(name, tmp_path):
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import rt
    if (os.cpu_count() or 1) < 8:
        pytest.skip("needs eight cores")
    sc = store(name)
    g = rt.GpuScene(sc)
    cam = S.camera_c2() if name == "large" else S.Camera(rotation=S.look_at((34.0, -30.0, 40.0), (34.0, 34.0, 0.0)),
                                                         position=(34.0, -30.0, 40.0), fovy=0.9)
    rays = rt.camera_rays(cam, 160, 120)
    want = {k: v.cpu().numpy() for k, v in g.intersect(rays).items()}
    nodes = g.counters()["nodes"]
    assert (want["patch"] >= 0).mean() > 0.1
    path = str(tmp_path / "store.cgs")
    g.save(path)
    g.close()
    rt.GpuScene.load(path).close()
    # processor time over elapsed time: 1.0 and 1.2 where one thread does it, 2.8 and 3.9 on 16 cores
    wall, cpu = time.perf_counter(), time.process_time()
    h = rt.GpuScene.load(path)
    wall, cpu = time.perf_counter() - wall, time.process_time() - cpu
    got = {k: v.cpu().numpy() for k, v in h.intersect(rays).items()}
    assert h.counters()["nodes"] == nodes
    h.close()
    for k in want:
        assert np.array_equal(got[k], want[k]), k
    assert cpu >= 1.7 * wall, (cpu, wall)
