"""Automata that reach the level slots in calls that ask for no lengths: their
violations are counted and their words stored all the same."""
import numpy as np
import pytest

import sbfs
from sbfs import problem as P

pytestmark = pytest.mark.gpu


def _wide(n, seed):
    """Two permutations but for one merged pair: more subsets than stay on chip."""
    rng = np.random.default_rng(seed)
    rec = np.zeros(2 * P.RECORD_LSTRIDE, dtype=np.uint8)
    rec[:n], rec[32:32 + n] = rng.permutation(n), rng.permutation(n)
    rec[32] = rec[33]
    return rec


@pytest.mark.parametrize("mixed", [False, True])
def test_violations_and_words_without_lengths(oracle_mod, mixed):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 22
    recs = np.concatenate([P.uniform_maps(20, n, 5), _wide(n, 0)[None], _wide(n, 1)[None], P.uniform_maps(1, n, 6)])
    ns = np.full(len(recs), n, dtype=np.uint8)
    if mixed:   # (behind the others: with this slack a smaller automaton violates its bound whatever it is)
        ns[-1], recs[-1] = 9, P.uniform_maps(1, 9, 3)[0]
    ref = oracle_mod.solve(recs, ns=ns, words=False, threads=8)["len"]
    wide = int(ref[20:22].max())
    assert ref[:20].max() < wide            # the violation below is a level-slot automaton's
    first = 20 + int(np.argmax(ref[20:22] == wide))
    with sbfs.Engine(slack=(n - 1) ** 2 - wide + 1) as eng:
        kw = dict(ns=ns) if mixed else dict(n=n)
        assert eng.verify(recs, **kw)["first_violation"] == first
        assert eng.verify(recs, lengths=False, **kw)["first_violation"] == first
        dev = torch.device("cuda", 0)
        ws = sbfs.word_stride_for(n)
        d_words = torch.full((len(recs), ws), -1, dtype=torch.int64, device=dev)
        d_fv = torch.empty(1, dtype=torch.int64, device=dev)
        eng.solve_device(torch.from_numpy(recs).to(dev), 32, len(recs), n=0 if mixed else n,
                         d_ns=torch.from_numpy(ns).to(dev) if mixed else None, max_n=n, d_len=None, d_words=d_words,
                         word_stride=ws, d_first_violation=d_fv)
        eng.wait_device()
        assert int(d_fv.item()) == first
        words = d_words.cpu().numpy().view(np.uint64)
        assert oracle_mod.replay(recs, ref, words, ns=ns)[0] == 0
