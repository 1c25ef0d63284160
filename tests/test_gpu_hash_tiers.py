"""The perfect-hash build at the edges of its three forms (one thread block,
one cluster, many launches), on keys in a shuffled order, against the oracle:
key sets that need several trials, key sets that no trial places, and a bucket
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
