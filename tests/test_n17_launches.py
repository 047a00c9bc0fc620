"""n = 17 alone: what k_mid cannot hold starts at n = 18, so nothing is launched
for it."""
import numpy as np
import pytest

import sbfs
from sbfs import problem as P

pytestmark = pytest.mark.gpu


def _near_permutations(rng, n):
    rec = np.zeros(2 * P.RECORD_LSTRIDE, dtype=np.uint8)
    rec[:n], rec[32:32 + n] = rng.permutation(n), rng.permutation(n)
    rec[32] = rec[33]
    return rec


def _batch(n, seed):
    rng = np.random.default_rng(seed)
    return np.concatenate([np.stack([_near_permutations(rng, n) for _ in range(8)]), P.uniform_maps(200, n, seed),
                           P.cerny_record(n)[None]])


@pytest.mark.parametrize("n,launches", [(17, 2), (18, 3)])
def test_kernels_launched_and_results(engine, oracle_mod, n, launches):
    recs = _batch(n, n)
    ref = oracle_mod.solve(recs, n=n, words=False, threads=8)["len"]
    r = engine.solve(recs, n=n)
    np.testing.assert_array_equal(r["len"], ref)
    assert oracle_mod.replay(recs, r["len"], r["words"], n=n)[0] == 0
    assert r["stats"]["launches"] == launches


@pytest.mark.parametrize("most", [17, 18])
def test_mixed_host_batches(engine, oracle_mod, most):
    sizes = list(range(13, most + 1))
    recs = np.concatenate([_batch(n, n) for n in sizes])
    ns = np.repeat(np.array(sizes, dtype=np.uint8), len(recs) // len(sizes))
    ref = oracle_mod.solve(recs, ns=ns, words=False, threads=8)["len"]
    r = engine.solve(recs, ns=ns)
    np.testing.assert_array_equal(r["len"], ref)
    assert oracle_mod.replay(recs, r["len"], r["words"], ns=ns)[0] == 0


def test_device_batch_larger_than_its_caller_says(oracle_mod):
    """max_n of a device batch is not checked against its sizes: a larger member
    of the same class gets its result or an error, never a stale one."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    recs = np.concatenate([_batch(17, 1), _batch(18, 2)])
    ns = np.repeat(np.array([17, 18], dtype=np.uint8), len(recs) // 2)
    ref = oracle_mod.solve(recs, ns=ns, words=False, threads=8)["len"]
    dev = torch.device("cuda", 0)
    d_len = torch.full((len(recs),), -99, dtype=torch.int32, device=dev)
    d_fv = torch.empty(1, dtype=torch.int64, device=dev)
    with sbfs.Engine() as eng:
        eng.solve_device(torch.from_numpy(recs).to(dev), 32, len(recs), d_ns=torch.from_numpy(ns).to(dev), max_n=17,
                         d_len=d_len, d_first_violation=d_fv)
        try:
            eng.wait_device()
        except sbfs.SbfsError as e:
            assert e.status == 1
    got = d_len.cpu().numpy()
    assert ((got == ref) | (got == -2)).all()
