"""The allocation-free Q4_K product (knj_q4k_matmul_noalloc_launch) through the
C-ABI. Some callers cannot allocate device memory at call time and have no
workspace to pass -- a serving loop whose pool is fully given to resident
experts, a plug-in host handed only inputs and outputs. The entry point needs no
scratch at all. The tests check its results against the CPU product, that calls
on two streams may overlap, that it takes its largest row count and refuses the
next, and that no device allocation happens during the calls.

Collected last on purpose (file name sorts after the other tests)."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle_lib as ol
from gpu_util import SENTINEL, report
from kanjoos_b200 import synth

pytestmark = pytest.mark.gpu

TOL_F32 = 1e-5  # f32 sums, as for the workspace-taking entry point


def _call(L, W, x, y):
    m, n_in = x.shape
    return L.knj_q4k_matmul_noalloc_launch(C.c_void_p(W.data_ptr()), n_in, W.shape[0], C.c_void_p(x.data_ptr()), 0, n_in, m,
                                           C.c_void_p(y.data_ptr()), W.shape[0],
                                           C.c_void_p(torch.cuda.current_stream().cuda_stream))


def _problem(rng, m, n_out, n_in):
    W = synth.q4k_rows(rng, n_out, n_in)
    x = rng.standard_normal((m, n_in)).astype(np.float32)
    y = torch.full((m, n_out), SENTINEL, dtype=torch.float32, device="cuda")
    return W, x, torch.from_numpy(W).cuda(), torch.from_numpy(x).cuda(), y


def _check(y, W, x, what):
    st = report(y.cpu().numpy(), ol.matmul_q4k(W, x), what)
    assert st["unwritten"] == 0 and st["rel_rmse"] <= TOL_F32


def test_noalloc_matches_the_cpu_product_and_allocates_nothing():
    from kanjoos_b200 import _lib, ops
    L = _lib.lib()
    _lib.check(L.knj_dev_open(0))
    rng = np.random.Generator(np.random.Philox(99))
    probs = [_problem(rng, m, 768, 2048) for m in (1, 5)]
    _lib.check(_call(L, probs[0][2], probs[0][3], probs[0][4]))  # loads the kernel
    probs[0][4].fill_(SENTINEL)
    torch.cuda.synchronize()
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    free_before = torch.cuda.mem_get_info()[0]
    for _, _, W, x, y in probs:
        _lib.check(_call(L, W, x, y))
    torch.cuda.synchronize()
    assert torch.cuda.memory_stats()["allocation.all.allocated"] == before
    assert torch.cuda.mem_get_info()[0] == free_before, "device memory was allocated during the calls"
    for W, x, Wd, xd, y in probs:
        _check(y, W, x, f"noalloc product, {x.shape[0]} rows")
        assert torch.equal(y, ops.q4k_matmul(Wd, xd))  # the same kernel on the same inputs


def test_noalloc_calls_may_overlap():
    """Two problems of different shapes, each on a stream of its own, launched in turn without a wait between them."""
    from kanjoos_b200 import _lib
    L = _lib.lib()
    rng = np.random.Generator(np.random.Philox(98))
    probs = [_problem(rng, 301, 768, 1024), _problem(rng, 7, 2048, 2048)]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    torch.cuda.synchronize()
    for _ in range(8):
        for (_, _, W, x, y), s in zip(probs, streams):
            with torch.cuda.stream(s):
                y.fill_(SENTINEL)
                _lib.check(_call(L, W, x, y))
    torch.cuda.synchronize()
    for W, x, _, _, y in probs:
        _check(y, W, x, "noalloc product, two streams")


def test_noalloc_largest_row_count_and_the_next():
    from kanjoos_b200 import _lib
    L = _lib.lib()
    rng = np.random.Generator(np.random.Philox(97))
    W, x, Wd, xd, y = _problem(rng, 16320, 16, 256)
    _lib.check(_call(L, Wd, xd, y))
    _check(y, W, x, "noalloc product, 16320 rows")
    big = torch.zeros((16321, 256), dtype=torch.float32, device="cuda")
    out = torch.full((16321, 16), SENTINEL, dtype=torch.float32, device="cuda")
    assert _call(L, Wd, big, out) == -4
    torch.cuda.synchronize()
    assert (out == SENTINEL).all(), "a refused call must not write"
