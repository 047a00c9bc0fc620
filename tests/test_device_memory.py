"""Device memory that small batches hold: working areas follow the batch."""
import numpy as np
import pytest

import sbfs
from sbfs import problem as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [[16], [13, 14, 15, 16]])
def test_small_batches_take_little_device_memory(oracle_mod, sizes):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    ns = np.array(sizes, dtype=np.uint8)
    recs = np.concatenate([P.uniform_maps(1, n, n) for n in sizes])
    with sbfs.Engine() as eng:
        eng.verify(P.uniform_maps(1, 8, 1), n=8)          # the context, the modules and the handle's plan
        before = torch.cuda.mem_get_info()[0]
        got = eng.verify(recs, ns=ns)["len"]
        used = before - torch.cuda.mem_get_info()[0]
    np.testing.assert_array_equal(got, oracle_mod.solve(recs, ns=ns, words=False, threads=2)["len"])
    assert used < 64 << 20, used


def test_wide_hand_offs_beyond_the_queue_on_chip(oracle_mod):
    """Searches that go on in the spill, more of them than there are CTAs for a
    batch this small, at both of its sizes."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(3)
    rows, ns = [], []
    for n in (14, 15, 16, 17, 18):
        for _ in range(6):
            rec = np.zeros(2 * P.RECORD_LSTRIDE, dtype=np.uint8)
            rec[:n], rec[32:32 + n] = rng.permutation(n), rng.permutation(n)
            rec[32] = rec[33]                             # two permutations but for one merged pair
            rows.append(rec)
            ns.append(n)
    recs, ns = np.stack(rows), np.array(ns, dtype=np.uint8)
    ref = oracle_mod.solve(recs, ns=ns, words=False, threads=8)["len"]
    for part in (slice(0, 3), slice(0, 18), slice(18, 30), slice(0, 30)):
        with sbfs.Engine() as eng:
            r = eng.solve(recs[part], ns=ns[part])
            np.testing.assert_array_equal(r["len"], ref[part])
            assert oracle_mod.replay(recs[part], r["len"], r["words"], ns=ns[part])[0] == 0
