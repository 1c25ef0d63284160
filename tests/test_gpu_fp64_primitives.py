"""The FP64 arithmetic of the near-grazing search and of the polish, which works on
the numbers' bits where it can: each primitive against CUDA's operator, bit for
bit, on random operands and at the edges (significands of all ones, the limits of
the exponents that it treats itself, ties, signed zeros, denormals, infinities,
NaN), and the two forms of the clip bounds and of the polish against each other,
without contraction bit for bit."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from cgspline_gb300 import scenes as S

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module", params=["product", "parity"])
def prim(request, tmp_path_factory):
    """The primitives compiled as in the product library (contracted) and as in the parity build."""
    pytest.importorskip("torch")
    from cgspline_gb300 import build
    out = str(tmp_path_factory.mktemp("prim") / f"prim_{request.param}.so")
    extra = [] if request.param == "product" else ["--fmad=false"]
    r = subprocess.run([build.nvcc(), *build.ARCH, *build.NVCC_FLAGS, *extra, "-shared",
                        os.path.join(HERE, "fp64_primitives.cu"), "-o", out], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(out)
    lib.kind = request.param
    return lib


def call(lib, what, a, b):
    a, b = np.ascontiguousarray(a, np.float64), np.ascontiguousarray(b, np.float64)
    got, want = np.zeros((a.size, 4)), np.zeros((a.size, 4))
    p = [x.ctypes.data_as(C.c_void_p) for x in (a, b, got, want)]
    assert lib.primitive(what, a.size, *p) == 0
    return got, want


def same(got, want, a, b):
    nan = np.isnan(got) & np.isnan(want)
    bad = ~nan & (got.view(np.uint64) != want.view(np.uint64))
    rows = np.flatnonzero(bad.any(axis=1))
    assert rows.size == 0, (rows.size, [(float(a[i]).hex(), float(b[i]).hex(), got[i].tolist(), want[i].tolist())
                                        for i in rows[:4]])


def doubles(bits):
    return np.ascontiguousarray(bits, np.uint64).view(np.float64)


def edges():
    """Doubles at the edges: every exponent near the limits of the bit paths with significands of zeros, ones and ties."""
    exps = np.array(sorted({0, 1, 2, 522, 523, 524, 896, 897, 898, 922, 923, 924, 1022, 1023, 1024, 1121, 1122, 1123, 1124, 1149,
                            1150, 1151, 1521, 1522, 1523, 1524, 2045, 2046, 2047}), np.uint64)
    one = np.uint64(1)
    top = (one << np.uint64(52)) - one
    sig = [np.uint64(0), one, np.uint64(2), top, top - one, one << np.uint64(51), (one << np.uint64(51)) + one,
           one << np.uint64(28), (one << np.uint64(28)) + one, (one << np.uint64(28)) - one, one << np.uint64(29),
           (one << np.uint64(29)) - one, (np.uint64(3) << np.uint64(28)), ((one << np.uint64(23)) - one) << np.uint64(29),
           (((one << np.uint64(24)) - one) << np.uint64(28)), (((one << np.uint64(24)) - one) << np.uint64(28)) - one]
    v = np.array([(e << np.uint64(52)) | s for e in exps for s in sig], np.uint64)
    return doubles(np.concatenate([v, v | (one << np.uint64(63))]))


def random_doubles(n, lo, hi, seed):
    r = np.random.RandomState(seed)
    return np.ldexp(r.uniform(1.0, 2.0, n), r.randint(lo, hi + 1, n)) * np.where(r.rand(n) < 0.5, -1.0, 1.0)


def pairs(lo, hi, seed, n=4_000_000):
    e = edges()
    a, b = (x.reshape(-1) for x in np.meshgrid(e, e, indexing="ij"))
    ones = doubles(np.array([0x000FFFFFFFFFFFFF | (k << 52) for k in range(1000, 1046)], np.uint64))
    ra, rb = random_doubles(n, lo, hi, seed), random_doubles(n, lo, hi, seed + 1)
    return (np.concatenate([a, ra, np.repeat(random_doubles(2000, lo, hi, seed + 2), ones.size)]),
            np.concatenate([b, rb, np.tile(ones, 2000)]))


@pytest.mark.parametrize("lo,hi", [(-3, 3), (-40, 40), (-110, 110)])
def test_quotient(prim, lo, hi):
    a, b = pairs(lo, hi, 11)
    same(*call(prim, 0, a, b), a, b)


@pytest.mark.parametrize("what", [1, 2, 3])
def test_conversions_and_order(prim, what):
    a, b = pairs(-160, 160, 5, 1_000_000)
    if what == 3:  # the order is that of finite doubles
        keep = np.isfinite(a) & np.isfinite(b) & ~((a == 0) & (b == 0))
        a, b = a[keep], b[keep]
    same(*call(prim, what, a, b), a, b)
    if what == 3:
        x = edges()
        got, want = call(prim, 3, x, np.zeros_like(x))
        assert np.array_equal(got[:, 2:], want[:, 2:])


@pytest.mark.parametrize("lo,hi", [(-3, 3), (-30, 30), (-60, 60)])
def test_unit_vectors(prim, lo, hi):
    n = 2_000_000
    a, b = random_doubles(n, lo, hi, 21), random_doubles(n, lo, hi, 22)
    # lengths with a significand of all ones: along an axis
    ones = doubles(np.array([0x000FFFFFFFFFFFFF | (k << 52) for k in range(1010, 1040)], np.uint64))
    e = edges()
    e = e[np.isfinite(e)]
    a = np.concatenate([a, ones, np.zeros_like(ones), -ones, e, np.zeros_like(e)])
    b = np.concatenate([b, np.zeros_like(ones), ones, np.zeros_like(ones), np.zeros_like(e), e])
    same(*call(prim, 4, a, b), a, b)


def nets(n, seed, exponent):
    """Nets as the search meets them: random ones, smooth ones about the origin, thin ones, with zeros and equal distances."""
    r = np.random.RandomState(seed)
    p = r.randn(n, 16, 2)
    g = np.stack(np.meshgrid(np.arange(4) - 1.5, np.arange(4) - 1.5, indexing="ij"), -1).reshape(16, 2)
    m = r.randn(n, 2, 2)
    smooth = np.einsum("ka,nab->nkb", g, m) + 0.05 * r.randn(n, 16, 2) + 0.5 * r.randn(n, 1, 2)
    thin = smooth * np.array([1.0, 2.0 ** -18])
    p = np.where((np.arange(n) % 4 < 2)[:, None, None], smooth, p)
    p = np.where((np.arange(n) % 4 == 2)[:, None, None], thin, p)
    p[::7] = np.round(p[::7] * 4.0) / 4.0
    p[::97, 3:9] = 0.0
    return np.ascontiguousarray(np.ldexp(p, exponent), np.float32)


@pytest.mark.parametrize("exponent", [-140, -100, -20, 0, 20, 60])
def test_two_forms_of_the_clip_bounds(prim, exponent):
    if prim.kind != "parity":
        pytest.skip("contraction rounds the two forms' sums apart")
    n = 400_000
    x = nets(n, exponent + 200, exponent)
    got, want = np.zeros((n, 4)), np.zeros((n, 4))
    assert prim.bounds(n, *(v.ctypes.data_as(C.c_void_p) for v in (x, got, want))) == 0
    nan = np.isnan(got) & np.isnan(want)
    bad = ~nan & (got.view(np.uint64) != want.view(np.uint64))
    assert not bad.any(), (int(bad.any(axis=1).sum()), np.flatnonzero(bad.any(axis=1))[:8])


@pytest.mark.parametrize("precision", [1, 3])
def test_two_forms_of_a_query(precision, monkeypatch):
    """The engine's polish and near-grazing search and those of the one-thread-per-ray kernels, parity build: the same
    t, u, v, patch and object, bit for bit."""
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import _capi, rt
    sc = S.scene_c2(nu=32, nv=32)
    rays = rt.camera_rays(S.camera_c2(), 320, 180)
    graze = torch.from_numpy(S.grazing_rays(sc.surfaces[0], 4000, seed=31)).cuda()
    rays = torch.cat([rays, graze], dim=1).contiguous()
    lib = _capi.load(_capi.LIB_NOFMA_PATH)
    monkeypatch.setattr(rt._capi, "load", lambda *a: lib)
    g = rt.GpuScene(sc)
    sv = rt.Server(g, slots=1, options=rt.Options(schedule=rt.PLAIN, precision=precision))
    ticket, plain = sv.submit_query(0, rays)
    sv.wait(ticket, 120.0)
    ours = g.intersect(rays, precision=precision)
    assert (plain["patch"] >= 0).float().mean() > 0.2
    for k in ("patch", "object", "t", "u", "v"):
        a, b = plain[k].cpu().numpy(), ours[k].cpu().numpy()
        hit = plain["patch"].cpu().numpy() >= 0
        assert np.array_equal(a[hit], b[hit]), (k, int((a[hit] != b[hit]).sum()))
    assert np.array_equal(plain["patch"].cpu().numpy(), ours["patch"].cpu().numpy())
    sv.close()
    g.close()
