"""Q4_K decode and single-matrix products on the GPU against the CPU restatement
and the golden vectors. Bit-exact for the decode; rel-RMSE <= 1e-5 over every
output for the f32-accumulate products (the tolerance the task states for the
GEMV path)."""
import numpy as np
import pytest
import torch

import oracle_lib as ol
from gpu_util import SENTINEL, dev, report
from kanjoos_b200 import synth

pytestmark = pytest.mark.gpu

TOL_F32 = 1e-5


def product_into(W, x, y):
    """knj_q4k_matmul_launch into the caller's y (which the tests poison first)."""
    import ctypes as C
    from kanjoos_b200 import _lib, ops
    L = _lib.lib()
    (m, n_in), n_out = x.shape, W.shape[0]
    nbytes = L.knj_q4k_matmul_workspace_bytes(m, n_in)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    _lib.check(L.knj_q4k_matmul_launch(C.c_void_p(W.data_ptr()), n_in, n_out, C.c_void_p(x.data_ptr()), ops._DT[x.dtype],
                                       n_in, m, C.c_void_p(y.data_ptr()), n_out, C.c_void_p(ws.data_ptr()), nbytes,
                                       C.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return y


def test_dequant_crafted_blocks_bit_exact(golden):
    from kanjoos_b200 import ops
    got = ops.q4k_dequant(dev(golden["q4k_blocks"])).cpu().numpy()
    assert np.array_equal(got.view(np.uint32), golden["q4k_blocks_f32"].view(np.uint32))


def test_dequant_cfg1_bit_exact(golden):
    """Config 1: the whole [768 x 2048] tensor, 1,572,864 weights."""
    from kanjoos_b200 import ops
    W = synth.q4k_rows(synth.stream(1, "gate"), synth.FFN, synth.HIDDEN)
    got = ops.q4k_dequant(dev(W)).cpu().numpy()
    want = ol.dequant_q4k(W)
    assert (got == SENTINEL).sum() == 0
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    assert np.array_equal(got.ravel()[:512].view(np.uint32), golden["cfg1_dequant_head"].view(np.uint32))


def test_dequant_empty_and_q6k():
    from kanjoos_b200 import ops
    assert ops.q4k_dequant(torch.empty((0, 144), dtype=torch.uint8, device="cuda")).numel() == 0
    rng = np.random.Generator(np.random.Philox(5))
    blk = rng.integers(0, 256, size=(64, 210), dtype=np.uint8)
    blk[:, 208:210] = (np.abs(rng.standard_normal((64, 1))) * 0.01).astype(np.float16).view(np.uint8)
    want = np.empty((64, 256), np.float32)
    ol.oracle().knj_or_dequant_q6k(ol.ptr(blk, ol.u8p), ol.ptr(want, ol.f32p), want.size)
    got = ops.q6k_dequant(dev(blk)).cpu().numpy()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    # and the reference's own decode of crafted blocks (all-0x00, all-0xFF, extreme scales, fp16 corners of d)
    import os
    g6 = np.load(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "golden_q6k.npz"))
    got = ops.q6k_dequant(dev(g6["q6k_blocks"])).cpu().numpy()
    assert np.array_equal(got.view(np.uint32), g6["q6k_blocks_f32"].view(np.uint32))


def test_cfg1_gemv(golden):
    """Config 1: y[768] = W[768 x 2048] . x, x f32 ~ N(0,1)."""
    from kanjoos_b200 import ops
    W = synth.q4k_rows(synth.stream(1, "gate"), synth.FFN, synth.HIDDEN)
    x = synth.stream(1, "x").standard_normal(synth.HIDDEN).astype(np.float32)
    y = torch.full((1, synth.FFN), SENTINEL, dtype=torch.float32, device="cuda")
    got = product_into(dev(W), dev(x[None]), y).cpu().numpy()[0]
    assert np.array_equal(ops.q4k_matmul(dev(W), dev(x[None])).cpu().numpy()[0], got)
    st = report(got, golden["cfg1_y"], "cfg1 GEMV vs reference dequant_dot_f32")
    assert st["unwritten"] == 0 and st["rel_rmse"] <= TOL_F32
    # and against an exact (float64) product of the bit-exact decode
    exact = (ol.dequant_q4k(W).reshape(synth.FFN, -1).astype(np.float64) @ x.astype(np.float64)).astype(np.float32)
    st = report(got, exact, "cfg1 GEMV vs float64 product")
    assert st["rel_rmse"] <= TOL_F32


@pytest.mark.parametrize("m", [1, 2, 4, 5, 15, 16, 17, 64])
@pytest.mark.parametrize("n_in,n_out", [(256, 16), (768, 48), (2048, 64)])
def test_matmul_ragged_row_counts(m, n_in, n_out):
    rng = np.random.Generator(np.random.Philox([m, n_in, n_out]))
    W = synth.q4k_rows(rng, n_out, n_in)
    x = rng.standard_normal((m, n_in)).astype(np.float32)
    got = product_into(dev(W), dev(x), torch.full((m, n_out), SENTINEL, dtype=torch.float32, device="cuda")).cpu().numpy()
    want = ol.matmul_q4k(W, x)
    st = report(got, want, f"matmul m={m} {n_out}x{n_in}")
    assert st["unwritten"] == 0 and st["rel_rmse"] <= TOL_F32


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_matmul_16bit_activations(dtype):
    from kanjoos_b200 import ops
    rng = np.random.Generator(np.random.Philox(11))
    W = synth.q4k_rows(rng, 32, 1024)
    x = torch.from_numpy(rng.standard_normal((3, 1024)).astype(np.float32)).to(dtype)
    got = ops.q4k_matmul(dev(W), x.cuda()).cpu().numpy()
    want = ol.matmul_q4k(W, x.float().numpy())
    assert report(got, want, f"matmul {dtype}")["rel_rmse"] <= TOL_F32


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("m,n_in,n_out", [(7, 768, 48), (9, 4096, 4096), (65, 512, 2048), (301, 768, 432), (512, 256, 256)])
def test_matmul_16bit_rows_in_jobs_of_eight(m, n_in, n_out, dtype):
    """Enough 16-bit rows travel as one plane, eight to a job (the first case: too few, jobs of four): full and ragged jobs,
    odd and even superblock counts, K split and not, rows over eight decades of magnitude (float16: subnormal ones
    included), against a float64 product of the decode."""
    from kanjoos_b200 import ops
    rng = np.random.Generator(np.random.Philox([m, n_in, n_out]))
    W = synth.q4k_rows(rng, n_out, n_in)
    scale = 10.0 ** (rng.integers(-4, 4, size=(m, 1)) if dtype == torch.bfloat16 else rng.integers(-6, 2, size=(m, 1)))
    x = torch.from_numpy((rng.standard_normal((m, n_in)) * scale).astype(np.float32)).to(dtype)
    got = product_into(dev(W), x.cuda(), torch.full((m, n_out), SENTINEL, dtype=torch.float32, device="cuda")).cpu().numpy()
    want = x.double().numpy() @ ol.dequant_q4k(W).reshape(n_out, n_in).astype(np.float64).T
    err = np.sqrt(((got - want) ** 2).mean(1)) / np.sqrt((want ** 2).mean(1))
    assert (got != SENTINEL).all() and err.max() <= 2e-6, f"row {err.argmax()}: {err.max():.2e}"   # f32 sums of n_in products


def test_matmul_wide_dynamic_range():
    """Activations spanning 12 orders of magnitude, a zero row and tiny rows: the
    per-vector scaling of the activation planes must keep f32-level accuracy."""
    from kanjoos_b200 import ops
    rng = np.random.Generator(np.random.Philox(13))
    W = synth.q4k_rows(rng, 32, 512)
    x = rng.standard_normal((6, 512)).astype(np.float32)
    x[0] *= 1e6
    x[1] *= 1e-6
    x[2] = 0.0
    x[3, ::2] *= 1e4
    x[4] *= 3e4
    x[5] *= 1e-20
    got = ops.q4k_matmul(dev(W), dev(x)).cpu().numpy()
    want = ol.matmul_q4k(W, x)
    for r in range(6):
        if r == 2:
            assert np.all(got[r] == 0.0)
            continue
        assert report(got[r], want[r], f"row {r}")["rel_rmse"] <= 2e-5


@pytest.mark.parametrize("m,n_out,nan_rows", [
    (5, 4096, 4),   # two jobs of 256 tiles over the SMs: the first block holds the first tiles of rows 0..3
    (1, 4096, 1),   # one job, K split over the warps of a tile
])
def test_a_wait_that_gives_up_leaves_nan(m, n_out, nan_rows):
    """The product has no status word: where a bounded wait runs out the outputs must be NaN, not what the buffer
    held before, and everything the other blocks computed stays right. The hook withholds one arrival, the copy
    itself lands."""
    from kanjoos_b200 import _lib, ops
    L = _lib.lib()
    rng = np.random.Generator(np.random.Philox([m, n_out]))
    W = dev(synth.q4k_rows(rng, n_out, 1024))
    x = dev(rng.standard_normal((m, 1024)).astype(np.float32))
    want = ops.q4k_matmul(W, x)
    y = torch.full((m, n_out), SENTINEL, dtype=torch.float32, device="cuda")
    L.knj_decode_wait_limit(2_000_000)  # about a millisecond
    L.knj_q4k_matmul_test_stall(1)
    try:
        product_into(W, x, y)
        torch.cuda.synchronize()
    finally:
        L.knj_q4k_matmul_test_stall(0)
        L.knj_decode_wait_limit(0)
    bad = torch.isnan(y)
    assert bad[:nan_rows, :16].all(), "outputs of a given-up tile must be NaN"
    assert not (y == SENTINEL).any() and int(bad.sum()) < y.numel() // 16
    assert torch.equal(y[~bad], want[~bad])
    product_into(W, x, y)  # the context and the kernel stay usable
    assert torch.equal(y, want)


@pytest.mark.parametrize("m,n_in,n_out,nan_rows", [
    (17, 1024, 8192, 8),   # three jobs of eight (five of four: 2560 tiles), the last of one row; the first block's tiles are rows 0..7's
    (9, 4096, 4096, 8),    # two jobs (three of four: 768 tiles of sixteen superblocks), K split over the warps of a tile
])
def test_a_wait_that_gives_up_leaves_nan_in_jobs_of_eight(m, n_in, n_out, nan_rows):
    """The same for 16-bit rows in jobs of eight: NaN in all eight rows of a given-up tile, in no row behind the last, and
    everything else right."""
    from kanjoos_b200 import _lib, ops
    L = _lib.lib()
    rng = np.random.Generator(np.random.Philox([m, n_out]))
    W = dev(synth.q4k_rows(rng, n_out, n_in))
    x = dev(rng.standard_normal((m, n_in)).astype(np.float32)).to(torch.bfloat16)
    want = ops.q4k_matmul(W, x)
    guard = torch.full((m + 8, n_out), SENTINEL, dtype=torch.float32, device="cuda")
    y = guard[:m]
    L.knj_decode_wait_limit(2_000_000)
    L.knj_q4k_matmul_test_stall(1)
    try:
        product_into(W, x, y)
        torch.cuda.synchronize()
    finally:
        L.knj_q4k_matmul_test_stall(0)
        L.knj_decode_wait_limit(0)
    bad = torch.isnan(y)
    assert bad[:nan_rows, :16].all() and not bad[nan_rows:, :16].any()
    assert not (y == SENTINEL).any() and int(bad.sum()) < y.numel() // 16
    assert torch.equal(y[~bad], want[~bad]) and (guard[m:] == SENTINEL).all()
    product_into(W, x, y)
    assert torch.equal(y, want)


def test_refusals_do_not_launch():
    from kanjoos_b200 import _lib, ops
    W = torch.zeros((16, 1, 144), dtype=torch.uint8, device="cuda")
    x = torch.zeros((1, 256), dtype=torch.float32, device="cuda")
    y = torch.zeros((1, 16), dtype=torch.float32, device="cuda")
    L = _lib.lib()
    import ctypes as C
    rc = L.knj_q4k_matmul_launch(C.c_void_p(W.data_ptr()), 256, 16, C.c_void_p(x.data_ptr()), 0, 256, 1,
                                 C.c_void_p(y.data_ptr()), 16, None, 0, None)
    assert rc == -4 and b"workspace" in L.knj_last_error_string()
    rc = L.knj_q4k_matmul_launch(C.c_void_p(W.data_ptr() + 8), 256, 16, C.c_void_p(x.data_ptr()), 0, 256, 1,
                                 C.c_void_p(y.data_ptr()), 16, C.c_void_p(x.data_ptr()), 1 << 20, None)
    assert rc in (-1, -4)
    with pytest.raises(_lib.KnjError):
        ops.q4k_matmul(torch.zeros((16, 1, 144), dtype=torch.uint8, device="cuda")[1:], x)  # 15 rows: not a multiple of 16


@pytest.mark.parametrize("E,N,K,counts", [
    (3, 80, 768, [5, 0, 11]),     # ragged last block (loads instead of bulk copies), passes of 8 + 3 rows
    (2, 64, 256, [1, 9]),         # one row (scalar form), 8 + 1
    (2, 192, 768, [2, 4]),        # bulk copies over three blocks; two rows (scalar form), four (one MMA column group)
    (2, 128, 1024, [7, 3]),       # four superblocks per row; two column groups, one
])
def test_q6k_projection(E, N, K, counts):
    """Q6_K down projection of the mixed-format path against the CPU decoder + a double-precision product, the
    activation rows spread over six decades of magnitude (every row has its own power-of-two scale in the MMA form)."""
    from kanjoos_b200 import ops
    rng = np.random.Generator(np.random.Philox([E, N, K]))
    nblk = K // 256
    W = rng.integers(0, 256, size=(E, N, nblk, 210), dtype=np.uint8)
    W[..., 208:210] = (np.abs(rng.standard_normal((E, N, nblk, 1))) * 0.01).astype(np.float16).view(np.uint8)
    Wf = np.empty((E * N * nblk, 256), np.float32)
    ol.oracle().knj_or_dequant_q6k(ol.ptr(W, ol.u8p), ol.ptr(Wf, ol.f32p), Wf.size)
    Wf = Wf.reshape(E, N, K)
    P = int(sum(counts))
    pe = np.concatenate([np.full(c, e, np.int32) for e, c in enumerate(counts)])
    pe = pe[rng.permutation(P)]
    A = (rng.standard_normal((P, K)) * (10.0 ** (np.arange(P) % 7 - 3))[:, None]).astype(np.float32)
    pair_idx, pair_cnt, exp_list, n_active = ops.moe_permute(dev(pe), E, P)
    Y = ops.q6k_proj(dev(A), dev(W), pair_idx, pair_cnt, exp_list, n_active, P).cpu().numpy()
    want = np.stack([(Wf[pe[p]].astype(np.float64) @ A[p].astype(np.float64)) for p in range(P)]).astype(np.float32)
    st = ol.compare(Y, want)
    print("[parity] q6k projection", st)
    assert (Y == -12345.0).sum() == 0 and st["rel_rmse"] <= 1e-5
    row_err = np.sqrt(((Y.astype(np.float64) - want) ** 2).mean(1)) / np.sqrt((want.astype(np.float64) ** 2).mean(1))
    assert row_err.max() <= 1e-5, f"worst row {row_err.argmax()}: {row_err.max():.3e}"
