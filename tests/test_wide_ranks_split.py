"""n = 18..20, wide both ways: images of at most 2^17 bits are searched by k_mid,
larger ones by k_cta beside it.  Ranks on both sides of that line."""
import numpy as np
import pytest

import sbfs
from sbfs import problem as P

pytestmark = pytest.mark.gpu


def _map_of_rank(rng, n, r):
    m = rng.permutation(n)
    m[rng.choice(n, n - r, replace=False)] = -1
    kept = m[m >= 0]
    m[m < 0] = rng.choice(kept, n - r)
    return m


def _batch(n, ranks, each, seed):
    rng = np.random.default_rng(seed)
    recs = np.zeros((each * len(ranks), 2 * P.RECORD_LSTRIDE), dtype=np.uint8)
    for i in range(len(recs)):
        ra, rb = ranks[i % len(ranks)]
        recs[i, :n], recs[i, 32:32 + n] = _map_of_rank(rng, n, ra), _map_of_rank(rng, n, rb)
    return recs


def _ranks(n):
    # 2^17 bits, 2^17 + 2^15, twice that, and the plain index of a permutation
    return [(16, 16), (17, 15), (15, 17), (17, 17), (n - 1, n - 1), (n, n - 2), (n - 2, n), (16, 15)]


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("n", [18, 19, 20])
def test_ranks_about_the_line(oracle_mod, n, use_graph):
    recs = _batch(n, _ranks(n), 12, n)
    ref = oracle_mod.solve(recs, n=n, words=False, threads=8)["len"]
    with sbfs.Engine(use_graph=use_graph) as eng:
        for _ in range(4):
            r = eng.solve(recs, n=n)
            np.testing.assert_array_equal(r["len"], ref)
            assert oracle_mod.replay(recs, r["len"], r["words"], n=n)[0] == 0


def test_mixed_sizes(engine, oracle_mod):
    sizes = [13, 16, 17, 18, 19, 20, 22]
    parts = [_batch(n, _ranks(n) if n > 17 else [(n - 1, n - 1), (n, n - 2)], 4, 7 * n) for n in sizes]
    recs = np.concatenate(parts)
    ns = np.repeat(np.array(sizes, dtype=np.uint8), [len(p) for p in parts])
    ref = oracle_mod.solve(recs, ns=ns, words=False, threads=8)["len"]
    for _ in range(3):
        r = engine.solve(recs, ns=ns)
        np.testing.assert_array_equal(r["len"], ref)
        assert oracle_mod.replay(recs, r["len"], r["words"], ns=ns)[0] == 0
