"""Per-lane searches of batches whose automata need more large bitmaps than the
warps' pools hold: lanes then search in the shared-memory column of a lane that
does not.  Results at every share of such automata, and their cost."""
import numpy as np
import pytest

import sbfs

pytestmark = pytest.mark.gpu


def _permutations(rng, count, n):
    return np.argsort(rng.random((count, n)), axis=1).astype(np.uint8)


def _near_permutations(rng, count, n):
    """Images of exactly n - 1 states."""
    p = _permutations(rng, count, n)
    p[:, 0] = p[:, 1]
    return np.take_along_axis(p, _permutations(rng, count, n), axis=1)


def _batch(kind, share, count, n):
    rng = np.random.default_rng(1000 * n + int(100 * share))
    a, b = (rng.integers(0, n, (count, n)).astype(np.uint8) for _ in range(2))
    large = rng.random(count) < share
    letters = {"permutation": (_permutations, None), "rank n-1": (None, _near_permutations),
               "both": (_permutations, _near_permutations), "permutations": (_permutations, _permutations)}[kind]
    for x, f in zip((a, b), letters):
        if f:
            x[large] = f(rng, count, n)[large]
    return np.ascontiguousarray(np.concatenate([a, b], axis=1))


@pytest.mark.parametrize("n", [10, 11, 12, 13, 14])
@pytest.mark.parametrize("share", [0.2, 1.0])
@pytest.mark.parametrize("ring", [0, 16])   # 16: a column is too short for the largest bitmaps at n = 12
def test_results_at_every_share(oracle_mod, n, share, ring):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    recs = np.concatenate([_batch(kind, share, 1501, n) for kind in ("permutation", "rank n-1", "both", "permutations")])
    ref = oracle_mod.solve(recs, n=n, lstride=n, words=False, threads=8)
    with sbfs.Engine(lane_ring=ring) as eng:
        r = eng.solve(recs, n=n, lstride=n)
        np.testing.assert_array_equal(r["len"], ref["len"])
        assert oracle_mod.replay(recs, r["len"], r["words"], n=n, lstride=n)[0] == 0
        np.testing.assert_array_equal(eng.verify(recs, n=n, lstride=n)["len"], ref["len"])


def test_streamed_batch(engine, oracle_mod):
    """Records that arrive while the kernel runs, stretches of them of large ranks alone."""
    n, chunk = 12, 1 << 17
    recs = _batch("rank n-1", 0.0, 3 * chunk, n)
    recs[chunk:chunk + chunk // 4] = _batch("rank n-1", 1.0, chunk // 4, n)
    recs[2 * chunk - 2000:2 * chunk + 2000] = _batch("permutation", 1.0, 4000, n)
    ref = oracle_mod.solve(recs, n=n, lstride=n, words=False, threads=8)
    r = engine.solve(recs, n=n, lstride=n)
    np.testing.assert_array_equal(r["len"], ref["len"])
    assert oracle_mod.replay(recs, r["len"], r["words"], n=n, lstride=n)[0] == 0


@pytest.mark.parametrize("n", [12, 13, 14])
def test_cost_per_subset(engine, n):
    """A batch of large ranks costs a subset about what a random batch does
    (with searches in the pools alone 5.3 and 3.2 times that at n = 13 and 14)."""
    import torch
    count = 60_000
    ns = []
    for share in (0.0, 1.0):
        d = torch.from_numpy(_batch("rank n-1", share, count, n)).cuda()
        d_len = torch.empty(count, dtype=torch.int32, device="cuda")
        d_fv = torch.empty(1, dtype=torch.int64, device="cuda")
        best = np.inf
        for _ in range(8):
            engine.solve_device(d, n, count, n=n, d_len=d_len, d_first_violation=d_fv)
            st = engine.wait_device()
            best = min(best, st["kernel_ms"] * 1e6 / st["expanded"])
        ns.append(best)
    assert ns[1] < 2.5 * ns[0], ns
