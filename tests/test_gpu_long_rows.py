"""Matrices whose rows are long, all of them or where a sample of the rows does
not show it: every row is summed in an order that its length alone decides."""
import numpy as np
import pytest
import torch

import oracle
from finchgb import _lib as L
from finchgb import device as dev
from helpers import abs_terms, assert_close, bf16_bits, oracle_spmv, to_dev, to_host, upload
from test_gpu_tiles import csr_of_lengths

pytestmark = pytest.mark.gpu


def strided_sums(b, x, rows, parts=32):
    """The rows' sums as `parts` running sums, entry p of a row in sum
    p mod parts, folded as a tree; products and sums each rounded."""
    out = []
    for r in rows:
        p0, p1 = b.ptr[r] - 1, b.ptr[r + 1] - 1
        t = b.val[p0:p1] * x[b.idx[p0:p1] - 1]
        t = np.concatenate([t, np.zeros(-t.size % parts, t.dtype)]).reshape(-1, parts)
        acc = np.zeros(parts, t.dtype)
        for row in t:
            acc = acc + row
        while acc.size > 1:
            acc = acc[:acc.size // 2] + acc[acc.size // 2:]
        out.append(acc[0])
    return np.array(out)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m,length", [(3000, 28), (3000, 63), (3000, 100), (600, 129), (500, 161), (300, 400), (40, 2048),
                                      (50_000, 40)])
def test_spmv_evenly_long_rows(gpu_lib, m, length, dtype):
    """Rows of one length over 24: 32 sums a row, whichever lanes hold them,
    and one running sum in Finch's order."""
    rng = np.random.default_rng(length)
    b = csr_of_lengths(rng, np.full(m, length), 5000, dtype)
    A, x = upload(b), rng.standard_normal(5000).astype(dtype)
    rows = np.unique(np.concatenate([[0, m - 1], rng.integers(0, m, 60)]))
    got = to_host(dev.spmv(A, to_dev(x), flags=L.NO_FMA))
    assert np.array_equal(got[rows], strided_sums(b, x, rows))
    assert_close(got, oracle_spmv(L.PLUS_TIMES, b, x), abs_terms(b, x), dtype)
    got = to_host(dev.spmv(A, to_dev(x), flags=L.FINCH_ORDER))
    assert np.array_equal(got, oracle_spmv(L.PLUS_TIMES, b, x, fma=True))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m,short,length", [(320_000, 2, 40), (90_000, 6, 300), (60_000, 20, 300)])
def test_spmv_unsampled_long_rows(gpu_lib, m, short, length, dtype):
    """More long rows together, between the sampled ones, than a block's list
    holds: each is summed as if it were alone, so twice the same."""
    rng = np.random.default_rng(short)
    lengths = np.full(m, short)
    long = np.arange(m // 64, m // 64 + 700)  # half a sampling step from the windows
    lengths[long] = length
    b = csr_of_lengths(rng, lengths, 9000, dtype)
    A, x = upload(b), rng.standard_normal(9000).astype(dtype)
    got = to_host(dev.spmv(A, to_dev(x), flags=L.NO_FMA))
    rows = rng.choice(long, 200, replace=False)
    assert np.array_equal(got[rows], strided_sums(b, x, rows))
    assert_close(got, oracle_spmv(L.PLUS_TIMES, b, x), abs_terms(b, x), dtype)
    assert np.array_equal(got, to_host(dev.spmv(A, to_dev(x), flags=L.NO_FMA)))
    got = to_host(dev.spmv(A, to_dev(x), flags=L.FINCH_ORDER))
    assert np.array_equal(got, oracle_spmv(L.PLUS_TIMES, b, x, fma=True))


@pytest.mark.parametrize("mean", [3, 12])
def test_spmv_short_rows_of_skewed_fp32(gpu_lib, mean):
    """Rows of at most 32 entries beside long ones: FP32 keeps four sums a row,
    also where the rows around it are nearly empty."""
    rng = np.random.default_rng(mean)
    lengths = np.where(rng.random(60_000) < 0.2, rng.integers(5, 33, 60_000), mean // 3)
    lengths[::500] = 900
    b = csr_of_lengths(rng, lengths, 9000, np.float32)
    A, x = upload(b), rng.standard_normal(9000).astype(np.float32)
    got = to_host(dev.spmv(A, to_dev(x), flags=L.NO_FMA))
    rows = rng.choice(np.flatnonzero((lengths > 4) & (lengths <= 32)), 300, replace=False)
    assert np.array_equal(got[rows], strided_sums(b, x, rows, parts=4))
    assert_close(got, oracle_spmv(L.PLUS_TIMES, b, x), abs_terms(b, x), np.float32)


def swallowing(lengths, n, dtype):
    """Rows whose first product swallows every later one that is added to it,
    one by one: 2^24 (FP64: 2^53), then ones.  What a row's sum lacks is how
    many entries shared a running sum with the first."""
    b = csr_of_lengths(np.random.default_rng(1), lengths, n, dtype)
    b.val[:] = 1
    b.val[(b.ptr[:-1] - 1)[np.asarray(lengths) > 0]] = 2.0 ** (24 if dtype == np.float32 else 53)
    return b, np.ones(n, dtype)


@pytest.mark.parametrize("nk", [4, 16, 20, 48, 64, 128])
def test_spmm_fp32_rows_have_four_sums(gpu_lib, nk):
    """The default for aligned operands, rows of at most 64 entries: no more
    than a quarter of a row shares its first entry's sum."""
    lengths = np.repeat([64, 48, 32, 16], 100)
    b, _ = swallowing(lengths, 300, np.float32)
    C = to_host(dev.spmm(upload(b), to_dev(np.ones((300, nk), np.float32))))
    assert (C.astype(np.float64) >= 2.0 ** 24 + (lengths - lengths / 4)[:, None]).all()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("nk", [4, 32, 64, 128, 132])
def test_spmm_hub_rows_are_cut(gpu_lib, nk, dtype):
    """Rows of far more entries than a block's share of the steps: a share's
    entries at most (2,048) share a sum with the first, and the parts of every
    row meet in a fixed order; rows before, between and after them, a second
    slab of columns, accumulating into strided rows."""
    hub = {32: 200_000, 64: 120_000}.get(nk, 60_000)  # from nk = 32 on 64 MB of gathers, the size from which rows are cut
    lengths = np.full(3000, 5)
    lengths[[0, 700, 701, 2999]] = (hub, hub // 2, hub // 3 + 1000, hub)
    n = hub + 10_000
    b, _ = swallowing(lengths, n, dtype)
    big = 2.0 ** (24 if dtype == np.float32 else 53)
    B = torch.ones((n, nk + 4), dtype=torch.float32 if dtype == np.float32 else torch.float64, device="cuda")[:, :nk]
    for ptr in (lambda t: t, lambda t: t.long()):
        A = upload(b)
        A = dev.DeviceSparse(A.nrows, A.ncols, ptr(A.ptr), A.idx, A.val, A.orient, A.base)
        C = torch.full((3000, nk + 4), 7.0, dtype=B.dtype, device="cuda")
        dev.spmm(A, B, C[:, :nk])
        got = to_host(C)[:, :nk].astype(np.float64) - big
        lack = (lengths - 1)[:, None] - got
        # adding the parts to the first rounds to even, once an addition: 3 + 3 + 7 + 1 of them at most
        assert lack.min() >= -14 and lack.max() <= 2048 + 14
        dev.spmm(A, B, C[:, :nk])
        assert np.array_equal(to_host(C)[:, :nk].astype(np.float64) - big, got)
        assert (to_host(C)[:, nk:] == 7).all()
    A = upload(b)
    A.val = torch.ones_like(A.val)
    C = torch.full((3000, nk), 3.0, dtype=B.dtype, device="cuda")
    dev.spmm(A, B, C, flags=L.ACCUMULATE)
    assert np.array_equal(to_host(C), np.broadcast_to((lengths + 3.0)[:, None], (3000, nk)))
    g, s = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s), torch.cuda.graph(g, stream=s):
        dev.spmm(A, B, C)
    C.zero_()
    g.replay()
    assert np.array_equal(to_host(C), np.broadcast_to(lengths[:, None], (3000, nk)))


@pytest.mark.parametrize("dtype,bf16", [(np.float32, False), (np.float64, False), (np.float32, True)])
@pytest.mark.parametrize("nk", [16, 32, 64, 128])
@pytest.mark.parametrize("length", [64, 65, 127, 129, 257, 512, 513, 1500])
def test_spmm_evenly_long_rows(gpu_lib, length, nk, dtype, bf16):
    """Rows of one length: by the groups, by the warps, by the block, cut."""
    rng = np.random.default_rng(length)
    m = 40_000 // length
    r = csr_of_lengths(rng, np.full(m, length), 6000, dtype)
    B = rng.standard_normal((6000, nk)).astype(dtype)
    A, Bd = upload(r, as_bf16=bf16), to_dev(B)
    val = bf16_bits(r.val) if bf16 else r.val
    want = oracle.spmm_csr(m, 6000, r.ptr, r.idx, val, B, bf16=bf16)
    scale = oracle.spmm_csr(m, 6000, r.ptr, r.idx, np.abs(r.val).astype(np.float64), np.abs(B).astype(np.float64))
    C = to_host(dev.spmm(A, Bd))
    assert_close(C, want, scale, dtype)
    assert np.array_equal(C, to_host(dev.spmm(A, Bd)))
