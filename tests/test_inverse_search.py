"""Slow and wide automata: the searches that leave the forward hash-set search
and are settled backwards from the singletons or by their pairs of states,
against the oracle."""
import numpy as np
import pytest

from sbfs import problem as P

pytestmark = pytest.mark.gpu


def _cycle_merge(n, p, q):
    """a the n-cycle, b the identity but for p -> q: shortest words of about
    n^2 / (distance of p and q) letters, or never synchronizing."""
    rec = np.zeros(2 * P.RECORD_LSTRIDE, dtype=np.uint8)
    rec[:n] = (np.arange(n) + 1) % n
    rec[32:32 + n] = np.arange(n)
    rec[32 + p] = q
    return rec


def _two_permutations(n, seed):
    """Both letters permutations but for one merged pair: wide both ways."""
    rng = np.random.default_rng(seed)
    rec = np.zeros(2 * P.RECORD_LSTRIDE, dtype=np.uint8)
    rec[:n], rec[32:32 + n] = rng.permutation(n), rng.permutation(n)
    rec[32] = rec[33]
    return rec


def _two_components(n, seed):
    """Two halves, each closed under both letters: never synchronizing, wide."""
    h = n // 2
    lo, hi = P.uniform_maps(1, h, seed)[0], P.uniform_maps(1, n - h, seed + 1)[0]
    rec = np.zeros(2 * P.RECORD_LSTRIDE, dtype=np.uint8)
    for base in (0, 32):
        rec[base:base + h] = lo[base:base + h]
        rec[base + h:base + n] = hi[base:base + n - h] + h
    return rec


def slow_batch(n):
    rows = [P.cerny_record(n)] + [_cycle_merge(n, 0, q) for q in range(1, n)]
    rows += [_cycle_merge(n, n - 1, q) for q in range(0, n - 1, 3)]
    rows += [P.perm_merge_record(n, 100 + s) for s in range(40)]
    rows += [_two_permutations(n, s) for s in range(3)] + [_two_components(n, s) for s in range(6)]
    return np.stack(rows + list(P.uniform_maps(64, n, 5)))


@pytest.mark.parametrize("n", [13, 15, 16, 17, 18, 20, 21])
def test_slow_families(engine, oracle_mod, n):
    recs = slow_batch(n)
    # n = 13 and 14 take the per-lane kernel as uniform batches: one member of another size
    ns = np.full(len(recs), n, dtype=np.uint8)
    ns[-1] = 12
    recs[-1] = P.uniform_maps(1, 12, 3)[0]
    ref = oracle_mod.solve(recs, ns=ns, words=False, threads=8)
    r = engine.solve(recs, ns=ns)
    np.testing.assert_array_equal(r["len"], ref["len"])
    assert r["len"][0] == (n - 1) ** 2 and r["first_violation"] == -1
    assert oracle_mod.replay(recs, r["len"], r["words"], ns=ns)[0] == 0
    np.testing.assert_array_equal(engine.verify(recs, ns=ns)["len"], ref["len"])
    # uniform batches reach the same kernels without the size-class bucketing
    np.testing.assert_array_equal(engine.solve(recs[:-1], n=n)["len"], ref["len"][:-1])


def test_generations_wrap_between_searches(engine, oracle_mod):
    """More searches in one warp than the set has generations: every automaton
    takes a second generation for its inverse search."""
    n = 20
    recs = np.concatenate([slow_batch(n)[:20]] * 2 + [P.uniform_maps(40, n, 11)])
    recs = np.concatenate([recs] * 160)          # 12,800 automata
    ref = oracle_mod.solve(recs[:80], n=n, words=False, threads=8)["len"]
    np.testing.assert_array_equal(engine.solve(recs, n=n)["len"], np.tile(ref, 160))


def test_largest_slow_automaton_and_words(engine, oracle_mod):
    """C_28: 729 letters in twelve 64-bit words; a word array too narrow for them is left zero."""
    n = 28
    recs = np.stack([P.cerny_record(n), _cycle_merge(n, 0, n - 1), P.uniform_maps(1, n, 2)[0]])
    r = engine.solve(recs, n=n)
    assert r["len"][0] == (n - 1) ** 2
    assert oracle_mod.replay(recs, r["len"], r["words"], n=n)[0] == 0
    short = engine.solve(recs, n=n, word_stride=2)
    np.testing.assert_array_equal(short["len"], r["len"])
    assert not short["words"][0].any()


@pytest.mark.parametrize("n", [22, 24])
def test_wide_large_automata(engine, oracle_mod, n):
    """Random automata past a warp's set (3072 subsets), and two-permutation
    automata past a CTA's (24,576), beside slow and malformed ones."""
    rows = [_two_permutations(n, s) for s in range(2)] + [_two_components(n, 7)]
    recs = np.concatenate([np.stack(rows), P.uniform_maps(400, n, 77)])
    ns = np.full(len(recs), n, dtype=np.uint8)
    ns[-1] = 9                                   # mixed sizes: the members come from the bucketing
    recs[-1] = P.uniform_maps(1, 9, 3)[0]
    ref = oracle_mod.solve(recs, ns=ns, words=False, threads=8)
    r = engine.solve(recs, ns=ns)
    np.testing.assert_array_equal(r["len"], ref["len"])
    assert oracle_mod.replay(recs, r["len"], r["words"], ns=ns)[0] == 0
    np.testing.assert_array_equal(engine.solve(recs[:-1], n=n, words=False)["len"], ref["len"][:-1])
    # lengths that nobody asked for still count for the violation index
    assert engine.verify(recs, ns=ns, lengths=False)["first_violation"] == -1
