"""Per-lane searches at the edges of their visited bitmaps: ranks that fill a
lane's words, that need half or all of a pool bitmap, more such lanes than the
pool holds, permutations (every subset reachable), and odd record strides."""
import numpy as np
import pytest

from sbfs import problem as P

pytestmark = pytest.mark.gpu


def _with_ranks(rng, count, n, ra, rb):
    """Records of n states whose letters have images of exactly ra and rb states."""
    recs = np.zeros((count, 2 * n), dtype=np.uint8)
    for i in range(count):
        for letter, r in ((0, ra), (1, rb)):
            image = rng.permutation(n)[:r]
            m = np.concatenate([image, image[rng.integers(0, r, n - r)]])
            recs[i, letter * n:letter * n + n] = rng.permutation(m)
    return recs


@pytest.mark.parametrize("n", [9, 11, 12, 13, 14])
def test_every_rank_pair(engine, oracle_mod, n):
    rng = np.random.default_rng(n)
    recs = np.concatenate([_with_ranks(rng, 12, n, ra, rb) for ra in range(1, n + 1) for rb in range(1, n + 1)])
    recs = recs[rng.permutation(len(recs))]
    ref = oracle_mod.solve(recs, n=n, lstride=n, words=False, threads=8)
    r = engine.solve(recs, n=n, lstride=n)
    np.testing.assert_array_equal(r["len"], ref["len"])
    assert oracle_mod.replay(recs, r["len"], r["words"], n=n, lstride=n)[0] == 0
    np.testing.assert_array_equal(engine.verify(recs, n=n, lstride=n)["len"], ref["len"])


@pytest.mark.parametrize("n", [12, 13, 14])
def test_more_large_bitmaps_than_the_pool_holds(engine, oracle_mod, n):
    """Every automaton needs a pool bitmap: all lanes of a warp but a few wait."""
    rng = np.random.default_rng(100 + n)
    recs = np.concatenate([_with_ranks(rng, 700, n, n - 1, n - 1), _with_ranks(rng, 700, n, n - 1, n - 2),
                           _with_ranks(rng, 100, n, n, n - 1)])
    ref = oracle_mod.solve(recs, n=n, lstride=n, words=False, threads=8)
    r = engine.solve(recs, n=n, lstride=n)
    np.testing.assert_array_equal(r["len"], ref["len"])
    assert oracle_mod.replay(recs, r["len"], r["words"], n=n, lstride=n)[0] == 0


@pytest.mark.parametrize("n,lstride", [(9, 9), (10, 11), (11, 13), (12, 17), (13, 13), (13, 15), (14, 14), (14, 31)])
def test_odd_record_strides(engine, oracle_mod, n, lstride):
    """Strides that are no multiple of four: records start at any alignment, and
    the first and last ones end where the batch does."""
    recs = P.repack(P.uniform_maps(1003, n, 7 * n + lstride), 32, lstride)
    ref = oracle_mod.solve(recs, n=n, lstride=lstride, words=False, threads=8)
    for first in (0, 1, 2, 3):
        r = engine.solve(recs[first:], n=n, lstride=lstride)
        np.testing.assert_array_equal(r["len"], ref["len"][first:])
    assert oracle_mod.replay(recs[3:], r["len"], r["words"], n=n, lstride=lstride)[0] == 0


def test_device_records_at_any_address(engine, oracle_mod):
    """Device batches that start at an odd address."""
    import torch
    n, count = 10, 4001
    recs = P.repack(P.uniform_maps(count, n, 3), 32, n)
    ref = oracle_mod.solve(recs, n=n, lstride=n, words=False, threads=8)["len"]
    dev = torch.device("cuda", 0)
    for off in (1, 2, 3, 7):
        buf = torch.zeros(off + recs.size, dtype=torch.uint8, device=dev)
        buf[off:] = torch.from_numpy(recs.reshape(-1)).to(dev)
        d_len = torch.empty(count, dtype=torch.int32, device=dev)
        d_fv = torch.empty(1, dtype=torch.int64, device=dev)
        engine.solve_device(buf.data_ptr() + off, n, count, n=n, d_len=d_len, d_first_violation=d_fv)
        engine.wait_device()
        np.testing.assert_array_equal(d_len.cpu().numpy(), ref)
