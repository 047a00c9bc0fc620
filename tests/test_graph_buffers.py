"""CUDA graphs and the buffers behind them.

A captured launch sequence is replayed only while the lane's buffers are the very
allocations it was captured with.  CPU: an allocator that hands out the same
address again must still change the signature (csrc/buffers.hpp).  GPU: a handle
with graphs solves batches whose buffers grow, and repeat, in every order, and
pinned results go to buffers that were freed and allocated anew."""
import os
import shutil
import subprocess

import numpy as np
import pytest

import sbfs
from sbfs import problem as P

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gpgpu-binary-automaton-synchronizing-algorithms_b200", "csrc")

DRIVER = r"""
#include <cstdio>
#include "buffers.hpp"
static char area[1 << 16];
extern "C" {
cudaError_t cudaMalloc(void **p, size_t) { *p = area; return cudaSuccess; }
cudaError_t cudaFree(void *) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t, unsigned) { *p = area + 4096; return cudaSuccess; }
cudaError_t cudaFreeHost(void *) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
}
int main() {
    sbfs::DevBuf d;
    sbfs::HostBuf h;
    if (d.reserve(300) || h.reserve(300)) return 1;
    const auto s0 = sbfs::buffers_signature({&d, &h});
    if (d.reserve(200) || h.reserve(300) || sbfs::buffers_signature({&d, &h}) != s0) return 2;   // kept
    void *const at = d.ptr;
    if (d.reserve(5000) || d.ptr != at) return 3;                 // grown, at the same address
    const auto s1 = sbfs::buffers_signature({&d, &h});
    if (s1 == s0) return 4;
    if (h.reserve(5000)) return 5;
    if (sbfs::buffers_signature({&d, &h}) == s1) return 6;
    std::puts("ok");
    return 0;
}
"""


def test_signature_tells_allocations_apart(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("g++ is not installed")
    inc = "/usr/local/cuda/include"
    if not os.path.exists(os.path.join(inc, "cuda_runtime_api.h")):
        pytest.skip("no CUDA headers")
    src, exe = tmp_path / "driver.cpp", str(tmp_path / "driver")
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", inc, str(src), "-o", exe], check=True,
                   capture_output=True, text=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "ok", out.returncode


@pytest.mark.gpu
def test_growing_and_repeating_batches(oracle_mod):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(5)
    cases = {}
    for n in (7, 10, 13, 16, 18):
        for count in (1, 40, 72, 500, 3000, 9000):
            recs = P.repack(P.uniform_maps(count, n, 31 * n + count), 32, n)
            cases[n, count] = recs, oracle_mod.solve(recs, n=n, lstride=n, words=False, threads=8)["len"]
    with sbfs.Engine(use_graph=True) as eng:
        for most in (40, 72, 500, 3000, 9000):            # each step grows the handle's buffers
            some = [k for k in cases if k[1] <= most]
            for i in rng.integers(0, len(some), 60):
                n, count = some[i]
                recs, ref = cases[n, count]
                r = eng.solve(recs, n=n, lstride=n) if i % 2 else eng.verify(recs, n=n, lstride=n)
                np.testing.assert_array_equal(r["len"], ref)


@pytest.mark.gpu
def test_pinned_results_at_a_reused_address(oracle_mod):
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n, count = 11, 4000
    batches = [P.repack(P.uniform_maps(count, n, s), 32, n) for s in range(6)]
    refs = [oracle_mod.solve(b, n=n, lstride=n, words=False, threads=8)["len"] for b in batches]
    ws = sbfs.word_stride_for(n)
    with sbfs.Engine(use_graph=True) as eng:
        for _ in range(3):
            for recs, ref in zip(batches, refs):
                p_recs = torch.from_numpy(recs).pin_memory()
                p_len = torch.empty(count, dtype=torch.int32).pin_memory()
                p_words = torch.empty((count, ws), dtype=torch.int64).pin_memory()
                r = eng.solve(p_recs.numpy(), n=n, lstride=n, out=(p_len.numpy(), p_words.numpy().view(np.uint64)))
                np.testing.assert_array_equal(r["len"], ref)
                assert oracle_mod.replay(recs, r["len"], r["words"], n=n, lstride=n)[0] == 0
                del p_recs, p_len, p_words, r
