"""The perfect-hash build at the edges of its three forms (one thread block,
one cluster, many launches), on keys in a shuffled order, and in stores of many
BVHs that share the device, against the oracle: key sets that need several trials, key sets that no trial places, and a bucket
that overflows."""
import numpy as np
import pytest

from cgspline_gb300 import scenes as S

pytestmark = pytest.mark.gpu


def build(keys):
    torch = pytest.importorskip("torch")
    from cgspline_gb300 import rt
    h = rt.PerfectHashFunction()
    status = h.build(torch.from_numpy(keys.view(np.int32)).cuda())
    return h, status


# leaves: 2 L - 1 heap keys.  8,191 and 8,193 keys lie on both sides of the thread block's limit, 16,383 and 16,387 of a
# change of the bucket count inside the cluster's range, 131,071 and 131,073 of the cluster's limit.
@pytest.mark.parametrize("leaves", [1, 2, 3, 40, 900, 4096, 4097, 8192, 8194, 20000 - 400, 32768, 65536, 65537])
def test_shuffled_heap_keys_match_the_oracle(leaves, oracle_mod):
    keys = S.bvh_keys(leaves)
    keys = np.ascontiguousarray(keys[np.random.RandomState(leaves).permutation(keys.size)])
    o = oracle_mod.hash_build(keys)
    h, status = build(keys)
    assert status == o["status"] == 0
    assert (h.A, h.B, h.N, h.mask, h.trials) == (o["A"], o["B"], o["N"], o["mask"], o["trials"])
    assert np.array_equal(h.disp, o["disp"]) and np.array_equal(h.table, o["table"])


@pytest.mark.parametrize("leaves", [2 * 17 * 17, 2 * 93 * 93, 2 * 257 * 257])
def test_key_sets_without_a_table_fail(leaves):
    assert build(S.bvh_keys(leaves))[1] == 6  # CGS_ERR_HASH_FAILED


@pytest.mark.parametrize("n", [3000, 30000, 140000])
def test_bucket_overflow_is_reported(n):
    keys = np.arange(1, n + 1, dtype=np.uint32)
    keys[:5] = np.uint32(1 << 20) * np.arange(1, 6, dtype=np.uint32) + np.uint32(7)  # five keys of one bucket
    assert build(keys)[1] == 5  # CGS_ERR_HASH_BUCKET_OVERFLOW


# 77 BVHs of 9,247 to 69,937 keys: clusters of 2, 4, 8 and 16; 12 of them: 8 or 16 for all.
@pytest.mark.parametrize("sides", [[68] * 74 + [187, 92, 137], [68] * 9 + [92, 187, 137]])
def test_stores_of_many_bvhs_match_the_oracle(sides, oracle_mod):
    from cgspline_gb300 import rt
    fields = {n: S.heightfield(n, n=n) for n in sorted(set(sides))}
    l2w, w2l = S.IDENTITY16.copy(), S.IDENTITY16.copy()
    sc = S.Scene([fields[n] for n in sides], [S.Object(k, l2w, w2l) for k in range(len(sides))], S.scene_c1().lights,
                 name="fields")
    g = rt.GpuScene(sc)
    want = {}
    for k, n in enumerate(sides):
        b = g.bvh(k)
        if n not in want:
            want[n] = oracle_mod.hash_build(b["keys"])
            assert want[n]["status"] == 0
        o = want[n]
        assert (b["A"], b["B"], b["N"], b["mask"]) == (o["A"], o["B"], o["N"], o["mask"])
        assert np.array_equal(b["disp"], o["disp"]) and np.array_equal(b["table"][:o["N"]], o["table"][:o["N"]])
    g.close()
