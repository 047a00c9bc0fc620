"""An error of the kernels that try large requests on chip reaches the requests
of that try, as a mini-batch's error reaches its requests.  (The host sets the
error word, SBFS_SERVER_FAIL_TRY=k; no GPU fault is involved.)"""
import os

import numpy as np
import pytest

from sbfs import problem as P
from sbfs.server import Server

pytestmark = pytest.mark.gpu


def _wide(n, seed):
    """Two permutations but for one merged pair: left to the level slots."""
    rng = np.random.default_rng(seed)
    rec = np.zeros(2 * P.RECORD_LSTRIDE, dtype=np.uint8)
    rec[:n], rec[32:32 + n] = rng.permutation(n), rng.permutation(n)
    rec[32] = rec[33]
    return rec


def test_failed_try_completes_with_an_error(oracle_mod):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 22
    recs = np.concatenate([P.uniform_maps(6, n, 9), P.cerny_record(n)[None], _wide(n, 0)[None]])
    ref = oracle_mod.solve(recs, n=n, words=False, threads=8)["len"]
    os.environ["SBFS_SERVER_FAIL_TRY"] = "1"
    try:
        srv = Server(device=0)
    finally:
        del os.environ["SBFS_SERVER_FAIL_TRY"]
    with srv:
        first = srv.submit_record(recs[0], n)
        assert srv.wait_all([first], timeout_s=60)[first]["status"] == 4          # SBFS_ECUDA
        ids = [srv.submit_record(r, n) for r in recs]                             # later tries are their own
        res = srv.wait_all(ids, timeout_s=60)
    assert all(res[i]["status"] == 0 for i in ids)
    np.testing.assert_array_equal([res[i]["len"] for i in ids], ref)


def test_what_a_failed_try_leaves_is_solved(oracle_mod):
    """The slots that the try did not settle start from their records."""
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 22
    rec = _wide(n, 0)
    ref = oracle_mod.solve(rec[None], n=n, words=False, threads=8)["len"][0]
    os.environ["SBFS_SERVER_FAIL_TRY"] = "1"
    try:
        srv = Server(device=0)
    finally:
        del os.environ["SBFS_SERVER_FAIL_TRY"]
    with srv:
        rid = srv.submit_record(rec, n)
        r = srv.wait_all([rid], timeout_s=60)[rid]
    assert r["status"] == 0 and r["len"] == ref
