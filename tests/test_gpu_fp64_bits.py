"""The near-grazing search's FP64 bounds take conversions, comparisons and signs
from the numbers' bits and round their own quotients, with other ranges of
exponents left to the operators: grazing rays at scales on both sides, against
the oracle's restatement of the same search in plain double arithmetic."""
import numpy as np
import pytest

from cgspline_gb300 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [-6, -3, 0, 3])
def test_grazing_rays_at_scales(exponent, oracle_mod):
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import _capi, rt
    sc = S.scene_c2(nu=32, nv=32)
    rays = S.grazing_rays(sc.surfaces[0], 3001, seed=exponent + 50)
    k = np.float32(2.0 ** exponent)
    sc.surfaces[0].points[:, :3] *= k
    rays[0:3] *= k
    o = oracle_mod.OracleScene(sc).intersect(rays, method=oracle_mod.CLIP_GRAZE64, precision=oracle_mod.FP32_POLISH64,
                                             graze_sin=oracle_mod.GRAZE_30)
    g = rt.GpuScene(sc, lib_path=_capi.LIB_NOFMA_PATH)
    h = {a: v.cpu().numpy() for a, v in g.intersect(torch.from_numpy(rays).cuda(), precision=rt.FP32_GRAZE64).items()}
    g.close()
    hit = o["patch"] >= 0
    assert hit.mean() > 0.3
    # the bar of the same comparison at scale 1 (test_gpu_precision.py), and of t on hits of the same patch
    assert ((h["patch"] >= 0) != hit).mean() <= 2e-3
    same = hit & (h["patch"] == o["patch"])
    assert same.sum() >= 0.98 * hit.sum()
    assert np.quantile(np.abs(h["t"][same] - o["t"][same]) / o["t"][same], 0.99) < 1e-5
