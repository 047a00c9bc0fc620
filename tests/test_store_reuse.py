"""One warp's visited store from search to search: small bitmaps, bitmaps of the
whole store, hash sets (ranks that fit no bitmap) and backward searches follow
one another on the same shared memory, in every order."""
import numpy as np
import pytest

from sbfs import problem as P

pytestmark = pytest.mark.gpu


def _with_ranks(rng, count, n, ra, rb):
    recs = np.zeros((count, 2 * P.RECORD_LSTRIDE), dtype=np.uint8)
    for i in range(count):
        for at, r in ((0, ra), (P.RECORD_LSTRIDE, rb)):
            image = rng.permutation(n)[:r]
            m = np.concatenate([image, image[rng.integers(0, r, n - r)]])
            recs[i, at:at + n] = rng.permutation(m)
    return recs


@pytest.mark.parametrize("n,fits", [(16, 14), (20, 15), (28, 16)])   # 2^fits + 2^fits bits: the whole store
def test_searches_of_every_kind_in_one_warp(engine, oracle_mod, n, fits):
    rng = np.random.default_rng(n)
    kinds = [_with_ranks(rng, 6, n, 3, 4), _with_ranks(rng, 6, n, fits, fits), _with_ranks(rng, 6, n, fits + 1, 4),
             _with_ranks(rng, 6, n, fits + 1, fits), np.stack([P.cerny_record(n), P.perm_merge_record(n, 5)]),
             P.uniform_maps(6, n, 9)]
    recs = np.concatenate(kinds)
    ref = oracle_mod.solve(recs, n=n, words=False, threads=8)["len"]
    # (n <= 20: 2220 and 3108 warps; 888 above) several searches per warp, in a new order each time
    order = np.concatenate([rng.permutation(len(recs)) for _ in range(400 if n <= 20 else 40)])
    r = engine.solve(recs[order], n=n)
    np.testing.assert_array_equal(r["len"], ref[order])
    assert oracle_mod.replay(recs[order], r["len"], r["words"], n=n)[0] == 0
