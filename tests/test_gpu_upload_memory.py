"""Making a store resident takes the device memory that it holds afterwards and no
staging copy of its patches and nodes beside it."""
import threading

import numpy as np
import pytest

from cgspline_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def test_upload_needs_no_second_copy_on_the_device():
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import _capi, rt
    fields = [S.heightfield(k, n=68) for k in range(1, 9)]
    pts = np.concatenate([f.points for f in fields])
    base = np.cumsum([0] + [f.points.shape[0] for f in fields[:-1]])
    idx = np.concatenate([f.indices + np.uint32(b) for f, b in zip(fields, base)])
    surf = S.Surface(pts, np.tile(idx, 14))  # 517,888 patches: 133 MB of them, 133 MB of nodes and their mirror
    sc = S.Scene([surf], [S.Object(0, S.IDENTITY16, S.IDENTITY16)], S.scene_c1().lights, name="tiled")
    g = rt.GpuScene(sc, split=rt.SPLIT_LONGEST, build=False)
    torch.cuda.synchronize()
    _capi.check(g.lib.cgs_bvh_build(g.h), "build")
    before = torch.cuda.mem_get_info()[0]
    low, stop = [before], threading.Event()

    def watch():
        while not stop.is_set():
            low.append(torch.cuda.mem_get_info()[0])

    t = threading.Thread(target=watch)
    t.start()
    status = g.lib.cgs_hash_build(g.h, None)
    stop.set()
    t.join()
    torch.cuda.synchronize()
    held = before - torch.cuda.mem_get_info()[0]
    assert held > 200 << 20, (held, status)
    # (the hash build of a large table keeps its own scratch, which held counts)
    assert before - min(low) <= held + (32 << 20), (before - min(low), held, len(low))
    g.close()
