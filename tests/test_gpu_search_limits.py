"""Searches that reach their iteration limit (4,096 clipping iterations, 16,384
bisections): lanes lend intervals of long searches to idle lanes, and where such a
search stops must not depend on it.  Grazing rays whose searches pass the limits,
each alone, in sets and among many, at tolerances that make them longer still,
give the hits and the error of a search that runs in one piece: bit for bit the
oracle's under the same limits."""
import numpy as np
import pytest

from cgspline_gb300 import scenes as S

pytestmark = pytest.mark.gpu

# of 2^20 seeded grazing rays over the 16,384-patch torus, those with more than 4,096 clipping iterations
LONG = [7761, 37982, 72346, 221682, 546097, 603592, 723236, 733904, 769604, 890358, 909653, 967140]


@pytest.fixture(scope="module")
def grazing():
    sc = S.scene_c2()
    rays = S.grazing_rays(sc.surfaces[0], 1 << 20, seed=3)
    at = np.unique(np.concatenate([np.arange(i - 8, i + 9) for i in LONG]))
    return sc, np.ascontiguousarray(rays[:, at]), np.searchsorted(at, LONG)


@pytest.mark.parametrize("exponent", [-12, -16, -20])
@pytest.mark.parametrize("method,any_hit", [(0, False), (1, False), (1, True)])
def test_a_search_stops_at_its_limit_whatever_else_runs(grazing, method, any_hit, exponent, oracle_mod):
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import _capi, rt
    sc, rays, long_ones = grazing
    tol = 2.0 ** exponent
    ref = oracle_mod.OracleScene(sc).intersect(rays, method=oracle_mod.SUBDIV if method else oracle_mod.CLIP_DEVICE,
                                               any_hit=any_hit, tol=tol, search_limits=oracle_mod.SEARCH_LIMITS)
    g = rt.GpuScene(sc, lib_path=_capi.LIB_NOFMA_PATH)
    keys = ["t", "u", "v", "patch", "object"]
    errors = 0

    def same(at):
        h = g.intersect(torch.from_numpy(np.ascontiguousarray(rays[:, at])).cuda(), method=method, any_hit=any_hit, tol=tol)
        if any_hit:
            got = h["patch"].cpu().numpy() >= 0
            assert np.array_equal(got, ref["patch"][at] >= 0), int((got != (ref["patch"][at] >= 0)).sum())
        else:
            for k in keys:
                got = h[k].cpu().numpy()
                assert np.array_equal(got, ref[k][at]), (k, at[got != ref[k][at]][:8])
        return g.counters()["device_errors"]

    n = rays.shape[1]
    for i in range(n):
        errors |= same(np.array([i]))
    assert errors in (0, 2)
    if not any_hit and (method, exponent) in ((0, -12), (0, -16), (0, -20), (1, -20)):
        assert errors == 2  # the limit was reached
    for size in (3, 33):
        for a in range(0, n, size):
            same(np.arange(a, min(a + size, n)))
    for order in (np.arange(n), np.arange(n)[::-1], np.concatenate([long_ones, np.arange(n)]),
                  np.tile(np.arange(n), 66000 // n + 1)):  # the last: past the one-launch queries' size
        assert same(order) == errors
    g.close()


@pytest.mark.parametrize("exponent", [-12, -16, -20])
def test_pairs_stop_at_their_limit_whatever_else_runs(grazing, exponent, oracle_mod):
    """The same of explicit (ray, patch) pairs: each long ray with the patches that it hits with and without the
    limit and their neighbours, alone and among many."""
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import _capi, rt
    sc, rays, long_ones = grazing
    scene = oracle_mod.OracleScene(sc)
    few = np.ascontiguousarray(rays[:, long_ones])
    hit = np.stack([scene.intersect(few, method=oracle_mod.CLIP_DEVICE, search_limits=limits)["patch"]
                    for limits in ((0, 0), oracle_mod.SEARCH_LIMITS)])
    pids = np.clip(np.concatenate([hit + k for k in range(-3, 4)]), 0, sc.surfaces[0].indices.size // 16 - 1)
    at = np.tile(np.arange(len(long_ones)), pids.shape[0])
    pids = pids.reshape(-1)
    g = rt.GpuScene(sc, lib_path=_capi.LIB_NOFMA_PATH)

    def run(which):
        out = rt.do_bezier_clipping(g, 0, torch.from_numpy(np.ascontiguousarray(few[:, at[which]])).cuda(),
                                    torch.from_numpy(pids[which].astype(np.int32)).cuda(), tol=2.0 ** exponent)
        return [x.cpu().numpy() for x in out], g.counters()["device_errors"]

    n = pids.size
    alone = [run(np.array([i])) for i in range(n)]
    want = [np.concatenate([a[0][k] for a in alone]) for k in range(4)]
    errors = np.bitwise_or.reduce([a[1] for a in alone])
    assert errors in (0, 2) and want[0].any()
    for which in (np.arange(n), np.arange(n)[::-1], np.tile(np.arange(n), 60)):
        got, e = run(which)
        assert e == errors
        for a, b in zip(got, want):
            assert np.array_equal(a, b[which])
    g.close()
