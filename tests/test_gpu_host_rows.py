"""Host queries copy rows that follow one another in one allocation together.
Rows that are neighbours in memory but page-locked one by one, or only some of
them, have their own copies (a copy may not span such ranges), and every layout
gives the same hits."""
import ctypes as C
import mmap

import numpy as np
import pytest

from cgspline_gb300 import scenes as S

pytestmark = pytest.mark.gpu

N = 16384  # a row of 64 KiB: whole pages


class Rows:
    """`count` neighbouring rows of whole pages, each of them page-locked by itself where `locked` says so."""

    def __init__(self, torch, count, locked):
        self.mem = mmap.mmap(-1, count * N * 4)
        self.array = np.frombuffer(self.mem, np.float32).reshape(count, N)
        self.rt = torch.cuda.cudart()
        self.at = [self.array[k].ctypes.data for k in range(count) if locked(k)]
        for p in self.at:
            assert int(self.rt.cudaHostRegister(p, N * 4, 0)) == 0

    def close(self):
        for p in self.at:
            assert int(self.rt.cudaHostUnregister(p)) == 0


@pytest.mark.parametrize("n", [N, N - 1, 513, 512, 33])
@pytest.mark.parametrize("any_hit", [False, True])
def test_rows_of_several_allocations(n, any_hit):
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import _capi, rt
    sc = S.scene_c2(nu=16, nv=16)
    g = rt.GpuScene(sc)
    cam = rt.camera_rays(S.camera_c2(), 128, 128).cpu().numpy()
    cam = cam[:, np.random.RandomState(7).permutation(N)]
    want = g.intersect(np.ascontiguousarray(cam[:, :n]), any_hit=any_hit)
    assert (want["patch"] >= 0).any()
    for locked in (lambda k: True, lambda k: k % 2 == 0, lambda k: k % 3 == 1, lambda k: False):
        rays, out = Rows(torch, 7, locked), Rows(torch, 5, locked)
        try:
            # rows of n: the first of whole pages as they lie; shorter ones at the pages' starts are not neighbours,
            # so those are laid out end to end
            if n < 1000:
                base, res = rays.array.reshape(-1)[: 7 * n].reshape(7, n), out.array.reshape(-1)[: 5 * n].reshape(5, n)
            else:
                base, res = rays.array[:, :n], out.array[:, :n]
            base[:] = cam[:, :n]
            res[:] = 0
            whole = res.view(np.int32)
            r = _capi.Rays(*[base[k].ctypes.data for k in range(7)], None)
            h = _capi.Hits(*[res[k].ctypes.data for k in range(5)])  # t u v, patch object
            _capi.check(g.lib.cgs_intersect_host(g.h, C.byref(r), n, 0, 0, rt.DEFAULT_TOL, int(any_hit), C.byref(h), None),
                        "cgs_intersect_host")
            assert np.array_equal(whole[3], want["patch"])
            if not any_hit:
                assert np.array_equal(res[:3], np.stack([want[k] for k in "tuv"])) and np.array_equal(whole[4], want["object"])
        finally:
            rays.close()
            out.close()
    g.close()
