"""n <= 8 on the per-lane kernel: the count of synchronizing automata, kept per
warp, and records at every stride and address (words where they are aligned,
bytes elsewhere)."""
import numpy as np
import pytest

from sbfs import problem as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,lstride", [(1, 1), (2, 4), (3, 3), (4, 4), (5, 8), (5, 5), (6, 7), (7, 8), (8, 8), (8, 9), (8, 12)])
def test_counts_and_record_addresses(engine, oracle_mod, n, lstride):
    import torch
    count = 4099
    recs = P.repack(P.uniform_maps(count, n, 17 * n + lstride), 32, lstride)
    ref = oracle_mod.solve(recs, n=n, lstride=lstride, words=False, threads=8)["len"]
    dev = torch.device("cuda", 0)
    ws = 1
    for off in (0, 1, 2, 4):
        buf = torch.zeros(off + recs.size, dtype=torch.uint8, device=dev)
        buf[off:] = torch.from_numpy(recs.reshape(-1)).to(dev)
        d_len = torch.empty(count, dtype=torch.int32, device=dev)
        d_words = torch.empty((count, ws), dtype=torch.int64, device=dev)
        d_fv = torch.empty(1, dtype=torch.int64, device=dev)
        for words in (None, d_words):
            engine.solve_device(buf.data_ptr() + off, lstride, count, n=n, d_len=d_len, d_words=words,
                                word_stride=ws if words is not None else 0, d_first_violation=d_fv)
            st = engine.wait_device()
            np.testing.assert_array_equal(d_len.cpu().numpy(), ref)
            assert st["synchronizing"] == int((ref >= 0).sum())
        assert oracle_mod.replay(recs, ref, d_words.cpu().numpy().view(np.uint64), n=n, lstride=lstride)[0] == 0
