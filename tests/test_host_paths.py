"""Host calls on both sides of the rules that choose their path: small calls
(results of a pageable caller behind the counters, up to 1 MB), streamed
batches at the edges of their 2^17-automaton chunks, buffers at odd places."""
import numpy as np
import pytest

import sbfs
from sbfs import problem as P

pytestmark = pytest.mark.gpu


def _pinned(a):
    torch = pytest.importorskip("torch")
    signed = a.view(np.int64) if a.dtype == np.uint64 else a
    return torch.from_numpy(signed).pin_memory().numpy().view(a.dtype)


def _mixed(count, seed, lo=2, hi=14):
    rng = np.random.default_rng(seed)
    ns = rng.integers(lo, hi + 1, count).astype(np.uint8)
    recs = np.zeros((count, 64), dtype=np.uint8)
    for n in range(lo, hi + 1):
        at = np.nonzero(ns == n)[0]
        recs[at] = P.uniform_maps(len(at), n, seed + n)
    return recs, ns


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("pin_in,pin_out", [(False, False), (True, False), (False, True)])
def test_small_calls(oracle_mod, use_graph, pin_in, pin_out):
    """Counts around one warp and around the 1 MB of results that still lie behind
    the counters (12-byte results at n <= 8, with a word of 8 bytes and its length)."""
    with sbfs.Engine(device=0, use_graph=use_graph) as eng:
        for count in (1, 2, 31, 33, 3000, 87_200, 87_400, 1):
            recs = P.repack(P.uniform_maps(count, 8, count), 32, 8)
            ref = oracle_mod.solve(recs, n=8, lstride=8, words=False, threads=8)["len"]
            out = np.full(count, -7, dtype=np.int32), np.full((count, 1), 7, dtype=np.uint64)
            if pin_out:
                out = tuple(_pinned(a) for a in out)
            r = eng.solve(_pinned(recs) if pin_in else recs, n=8, lstride=8, out=out, word_stride=1)
            np.testing.assert_array_equal(r["len"], ref)
            assert oracle_mod.replay(recs, r["len"], r["words"], n=8, lstride=8)[0] == 0
            np.testing.assert_array_equal(eng.verify(recs, n=8, lstride=8)["len"], ref)
        for count in (1, 40, 5000, 37_500):
            recs, ns = _mixed(count, count)
            ref = oracle_mod.solve(recs, ns=ns, words=False, threads=8)["len"]
            r = eng.solve(_pinned(recs) if pin_in else recs, ns=_pinned(ns) if pin_in else ns)
            np.testing.assert_array_equal(r["len"], ref)
            assert oracle_mod.replay(recs, r["len"], r["words"], ns=ns)[0] == 0
            np.testing.assert_array_equal(eng.verify(recs, ns=ns)["len"], ref)


@pytest.mark.parametrize("use_graph", [False, True])
def test_only_the_classes_of_the_sizes(oracle_mod, use_graph):
    """Ranges of sizes that begin and end in each size class, one after another with
    the same counts and buffers."""
    count = 300
    recs_at, ns_at = np.zeros((count, 64), dtype=np.uint8), np.zeros(count, dtype=np.uint8)
    with sbfs.Engine(device=0, use_graph=use_graph) as eng:
        for lo, hi in [(2, 8), (2, 9), (8, 20), (9, 12), (12, 13), (13, 16), (16, 17), (17, 20), (20, 21), (21, 22),
                       (8, 22), (13, 20), (2, 20)] * 2:
            recs_at[:], ns_at[:] = _mixed(count, 100 * lo + hi, lo, hi)
            ref = oracle_mod.solve(recs_at, ns=ns_at, words=False, threads=8)["len"]
            np.testing.assert_array_equal(eng.verify(recs_at, ns=ns_at)["len"], ref)
        ns_at[17] = 0   # a malformed size is still found
        with pytest.raises(Exception):
            eng.verify(recs_at, ns=ns_at)


@pytest.mark.parametrize("n", [7, 12, 13, 14])
@pytest.mark.parametrize("count", [2 << 17, (2 << 17) + 1, (3 << 17) - 1, (4 << 17) + 33])
def test_streamed_chunk_edges(engine, n, count):
    """Against the path that copies the batch in as one piece."""
    recs = P.repack(P.uniform_maps(count, n, n + count), 32, n)
    with sbfs.Engine(device=0, chunk=1 << 20) as whole:
        ref = whole.solve(recs, n=n, lstride=n, words=False)
    pin = _pinned(recs)
    for src in (recs, pin):
        r = engine.verify(src, n=n, lstride=n)
        np.testing.assert_array_equal(r["len"], ref["len"])
        assert r["first_violation"] == ref["first_violation"]
    out = _pinned(np.full(count, -7, dtype=np.int32)), None
    np.testing.assert_array_equal(engine.solve(pin, n=n, lstride=n, words=False, out=out)["len"], ref["len"])


@pytest.mark.parametrize("word_stride,skip", [(2, 0), (2, 1), (3, 0), (4, 0), (4, 1)])
def test_streamed_words_at_any_stride(engine, oracle_mod, word_stride, skip):
    """Late results are stored 8 or 16 bytes at a time, by stride and address."""
    n, count = 12, (2 << 17) + 5
    recs = _pinned(P.repack(P.uniform_maps(count, n, 5), 32, n))
    words = _pinned(np.full(count * word_stride + 2, 7, dtype=np.uint64))
    assert words.ctypes.data % 16 == 0
    view = words[skip:skip + count * word_stride].reshape(count, word_stride)
    out = _pinned(np.empty(count, dtype=np.int32)), view
    r = engine.solve(recs, n=n, lstride=n, out=out, word_stride=word_stride)
    assert oracle_mod.replay(recs, r["len"], np.ascontiguousarray(view), n=n, lstride=n)[0] == 0
    assert (view[:, 2:] == 0).all()
    assert (words[:skip] == 7).all() and (words[skip + count * word_stride:] == 7).all()
