"""Kernels whose work is cut by size (column slabs, tiles of rows and entries)
at the sizes where a cut can go wrong, against the oracle."""
import numpy as np
import pytest
import torch

import oracle
from finchgb import _lib as L
from finchgb import device as dev
from finchgb.workloads import SparseBuffers, _fibers_from_lengths, _ptr
from helpers import abs_terms, assert_close, bf16_bits, oracle_spmv, to_dev, to_host, upload

pytestmark = pytest.mark.gpu


def csr_of_lengths(rng, lengths, n, dtype):
    lengths = np.asarray(lengths, dtype=np.int64)
    cols = _fibers_from_lengths(rng, lengths, n)
    b = SparseBuffers(lengths.size, n, _ptr(lengths), cols + 1, None, "csr")
    if np.dtype(dtype).kind == "i":
        info = np.iinfo(dtype)
        b.val = rng.integers(info.min // 2, info.max // 2, size=b.nnz, dtype=dtype)
    else:
        b.val = rng.standard_normal(b.nnz).astype(dtype)
    return b


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("nk", [1, 5, 9, 17, 31, 33, 37, 47, 65])
def test_spmm_odd_widths_bit_exact(gpu_lib, dtype, nk):
    """Widths that fit no vector: whole 32-column slabs, then the narrowest
    group of lanes that covers the rest.  Rows of 0 to 70 entries, so every
    mix of batches of 8, 4, 2 and 1; one running sum per output, bit for bit."""
    rng = np.random.default_rng(nk)
    r = csr_of_lengths(rng, np.arange(71), 200, dtype)
    B = rng.standard_normal((200, nk)).astype(dtype)
    C0 = rng.standard_normal((71, nk)).astype(dtype)
    A, Bd = upload(r), to_dev(B)
    for fma, flags in ((True, 0), (False, L.FINCH_ORDER | L.NO_FMA)):
        want = oracle.spmm_csr(71, 200, r.ptr, r.idx, r.val, B, fma=fma)
        assert np.array_equal(to_host(dev.spmm(A, Bd, flags=flags)), want)
        Cd = to_dev(C0)
        dev.spmm(A, Bd, Cd, flags=flags | L.ACCUMULATE)
        want = oracle.spmm_csr(71, 200, r.ptr, r.idx, r.val, B, C=C0.copy(), init=False, fma=fma)
        assert np.array_equal(to_host(Cd), want)


def spmv_lengths(kind, rng):
    if kind == "hidden":  # short rows; the long ones lie outside the sampled windows, 100 of them together
        n = rng.integers(0, 4, 320_000)
        n[5000:5100] = 40
        n[[123_456, 200_111, 319_999]] = (9000, 2049, 2048)
    elif kind == "skewed":
        n = np.minimum(rng.zipf(1.5, 60_000), 3000)
        n[rng.choice(60_000, 20_000, replace=False)] = 0
        n[[0, 7, 59_999]] = (7000, 33, 32)
    elif kind == "mid":  # rows that average over 14 entries, some long
        n = rng.poisson(20, 8000)
        n[:40] = 300
    elif kind == "few":
        n = np.array([31_000, 0, 9999, 33, 30_000])
    else:
        n = np.zeros(70_001, dtype=np.int64)
    return n.astype(np.int64)


@pytest.mark.parametrize("ptr64", [False, True])
@pytest.mark.parametrize("kind", ["hidden", "skewed", "mid", "few", "empty"])
def test_spmv_sampled_rows(gpu_lib, kind, ptr64):
    """The pull that samples row lengths: equal to the nest bit for bit in
    Finch's order (both contractions) and over an exact semiring, within the
    bound otherwise, accumulating or not, whatever the sample missed."""
    rng = np.random.default_rng(len(kind))
    lengths, n = spmv_lengths(kind, rng), 40_000

    def device_of(b):
        A = upload(b)
        if ptr64:
            A = dev.DeviceSparse(A.nrows, A.ncols, A.ptr.long(), A.idx, A.val, A.orient, A.base)
        return A

    for dtype in (np.float64, np.float32):
        b = csr_of_lengths(rng, lengths, n, dtype)
        A, x = device_of(b), rng.standard_normal(n).astype(dtype)
        y0 = rng.standard_normal(b.nrows).astype(dtype)
        want, scale = oracle_spmv(L.PLUS_TIMES, b, x), abs_terms(b, x)
        assert_close(to_host(dev.spmv(A, to_dev(x))), want, scale, dtype)
        yd = to_dev(y0)
        dev.spmv(A, to_dev(x), yd, flags=L.ACCUMULATE)
        assert_close(to_host(yd), want.astype(np.float64) + y0, scale + np.abs(y0), dtype)
        for fma, flag in ((True, 0), (False, L.NO_FMA)):
            got = to_host(dev.spmv(A, to_dev(x), flags=L.FINCH_ORDER | flag))
            assert np.array_equal(got, oracle_spmv(L.PLUS_TIMES, b, x, fma=fma))
    b = csr_of_lengths(rng, lengths, n, np.int32)
    x = rng.integers(-(1 << 30), 1 << 30, size=n, dtype=np.int32)
    y0 = rng.integers(-(1 << 30), 1 << 30, size=b.nrows, dtype=np.int32)
    want = oracle_spmv(L.MIN_PLUS, b, x)
    assert np.array_equal(to_host(dev.spmv(device_of(b), to_dev(x), semiring=L.MIN_PLUS)), want)
    yd = to_dev(y0)
    dev.spmv(device_of(b), to_dev(x), yd, semiring=L.MIN_PLUS, flags=L.ACCUMULATE)
    assert np.array_equal(to_host(yd), np.minimum(want, y0))


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("shape", ["edges", "wide", "ragged"])
def test_spgemm_merged_rows(gpu_lib, dtype, shape):
    """Rows that one thread merges, beside rows of the hash tiers: 0 to 10
    lists, bounds about 64, blocks of 128 rows with more outputs than the
    staging array holds, a last block that is not full.  The product is the
    serial nest's bit for bit, also where the lists are not ascending."""
    rng = np.random.default_rng(len(shape))
    if shape == "edges":
        la, lb, n = np.arange(700) % 11, np.full(300, 8), 5000
    elif shape == "wide":  # 8 lists of 8: 64 products, nearly as many outputs
        la, lb, n = np.full(257, 8), np.full(300, 8), 100_000
    else:
        la, lb, n = rng.integers(0, 9, 1000), rng.integers(0, 30, 300), 900
    A, B = csr_of_lengths(rng, la, 300, dtype), csr_of_lengths(rng, lb, n, dtype)
    for fma, flags in ((True, 0), (False, L.NO_FMA)):
        ptr, idx, val = dev.spgemm(upload(A), upload(B), flags=flags).to_host()
        wp, wi, wv = oracle.spgemm_csr(la.size, n, A.ptr, A.idx, A.val, B.ptr, B.idx, B.val, fma=fma)
        assert np.array_equal(ptr, wp) and np.array_equal(idx, wi) and np.array_equal(val, wv)
    order = np.lexsort((rng.random(B.nnz), np.repeat(np.arange(300), lb)))  # each list shuffled
    S = SparseBuffers(300, n, B.ptr, B.idx[order], B.val[order], "csr")
    ptr2, idx2, val2 = dev.spgemm(upload(A), upload(S), flags=L.NO_FMA).to_host()
    assert np.array_equal(ptr2, ptr) and np.array_equal(idx2, idx) and np.array_equal(val2, val)


def ewise_pair(kind, rng, dtype):
    """Two matrices of one shape that share about half their places."""
    n = 20_000
    if kind == "short":  # several staged tiles, the last one not full
        la = rng.integers(0, 17, 3001)
    elif kind == "long":  # long pairs in staged tiles and beyond them
        la = rng.integers(0, 6, 500)
        la[[3, 4, 100, 499]] = (33, 64, 700, 9000)
    elif kind == "rare":  # short fibers on average, read where they lie, and a few long pairs among them
        la = rng.integers(0, 5, 5003)
        la[[3, 4, 90, 700, 5002]] = (33, 64, 300, 9000, 700)
    elif kind == "one":
        la = np.array([5000])
    else:  # nothing, or nothing in one of the two
        la = np.zeros(200, dtype=np.int64)
        la[7] = 40
    A = csr_of_lengths(rng, la, n, dtype)
    f = np.repeat(np.arange(la.size), la)
    keep = rng.random(A.nnz) < 0.5
    key = np.unique(np.concatenate([f[keep] * n + A.idx[keep] - 1,
                                    rng.integers(0, la.size * n, int((~keep).sum()) if kind != "none" else 0)]))
    lb = np.bincount(key // n, minlength=la.size)
    B = csr_of_lengths(rng, lb, n, dtype)
    B.idx = key % n + 1
    return A, B


@pytest.mark.parametrize("dtype", [np.float64, np.float32, np.int32, np.int64])
@pytest.mark.parametrize("kind", ["short", "long", "rare", "one", "none"])
def test_ewise_tiles(gpu_lib, kind, dtype):
    """Merges of short pairs (a thread each, staged) and long ones (a warp
    each, staged or not), with ptr widths and index bases of their own:
    structure and values equal the two-finger merge's; sums are within the
    bound, over every dimension."""
    rng = np.random.default_rng(len(kind))
    A, B = ewise_pair(kind, rng, dtype)
    for a, b in ((A, B), (B, A)):
        da, db = upload(a), upload(b)
        db = dev.DeviceSparse(db.nrows, db.ncols, db.ptr.long() - 1, db.idx - 1, db.val, "csr", 0)
        for op in (L.EW_MUL, L.EW_ADD):
            ptr, idx, val = dev.ewise(op, da, db).to_host()
            wp, wi, wv = oracle.ewise(op, a.nrows, a.ptr, a.idx, a.val, b.ptr, b.idx, b.val)
            assert np.array_equal(ptr, wp) and np.array_equal(idx, wi) and np.array_equal(val, wv)
        if np.dtype(dtype).kind == "f":
            for dims in (0, 1, 2):
                args = (dims, a.nrows, a.ncols, a.ptr, a.idx)
                want = oracle.ewise_reduce(*args, a.val, b.ptr, b.idx, b.val)
                scale = oracle.ewise_reduce(*args, np.abs(a.val), b.ptr, b.idx, np.abs(b.val))
                assert_close(to_host(dev.ewise_reduce(dims, da, db)), want, scale, dtype)


@pytest.mark.parametrize("dtype,bf16", [(np.float32, False), (np.float64, False), (np.float32, True)])
@pytest.mark.parametrize("nk", [4, 12, 32, 60, 128, 132])
def test_spmm_whole_rows(gpu_lib, dtype, bf16, nk):
    """The default for aligned operands: groups of 4 to 32 lanes, lanes beyond
    nk, a second slab of columns, rows at both sides of the length from which
    the block folds a row, empty rows, blocks whose share lies inside one row;
    within the bound, accumulating into strided rows too, and the same twice."""
    rng = np.random.default_rng(nk)
    lengths = rng.integers(0, 40, 3000)
    lengths[100:140] = rng.integers(62, 68, 40)
    lengths[[0, 7, 1500, 2999]] = (9000, 600, 65, 64)
    lengths[2000:2300] = 0
    r = csr_of_lengths(rng, lengths, 9500, dtype)
    B = rng.standard_normal((9500, nk + 4)).astype(dtype)[:, :nk]
    A, Bd = upload(r, as_bf16=bf16), to_dev(np.pad(B, ((0, 0), (0, 4))))[:, :nk]
    Bc = np.ascontiguousarray(B)
    val = bf16_bits(r.val) if bf16 else r.val
    want = oracle.spmm_csr(3000, 9500, r.ptr, r.idx, val, Bc, bf16=bf16)
    scale = oracle.spmm_csr(3000, 9500, r.ptr, r.idx, np.abs(r.val).astype(np.float64), np.abs(Bc).astype(np.float64))
    C = to_host(dev.spmm(A, Bd))
    assert_close(C, want, scale, dtype)
    assert np.array_equal(C, to_host(dev.spmm(A, Bd)))
    C0 = rng.standard_normal((3000, nk + 4)).astype(dtype)
    Cd = to_dev(C0)
    dev.spmm(A, Bd, Cd[:, :nk], flags=L.ACCUMULATE)
    got = to_host(Cd)
    assert_close(got[:, :nk], want.astype(np.float64) + C0[:, :nk], scale + np.abs(C0[:, :nk]), dtype)
    assert np.array_equal(got[:, nk:], C0[:, nk:])


@pytest.mark.parametrize("kind", ["dense", "hollow", "long"])
@pytest.mark.parametrize("val", ["f64", "i32", "bf16", "bool", "pattern"])
def test_transpose_and_scale_runs(gpu_lib, kind, val):
    """Kernels that find the fiber of every entry of a run of 2,048: runs with
    few fibers, with more than their shared memory holds (mostly empty), and
    inside one fiber; first and last fibers empty, a last run not full.
    Transposes and masked scalings equal numpy's, every payload width."""
    rng = np.random.default_rng(len(kind))
    if kind == "dense":
        lengths = rng.integers(0, 30, 900)
    elif kind == "hollow":
        lengths = (rng.random(60_000) < 0.1).astype(np.int64)
    else:
        lengths = np.array([0, 0, 5000, 0, 1, 2047, 0])
    lengths[[0, -1]] = 0
    n = 5200
    b = csr_of_lengths(rng, lengths, n, np.float64)
    f = np.repeat(np.arange(lengths.size), lengths)
    t = {"f64": torch.float64, "i32": torch.int32, "bf16": torch.bfloat16, "bool": torch.uint8, "pattern": None}[val]
    A = upload(b)
    if t is None:
        A = dev.DeviceSparse(A.nrows, A.ncols, A.ptr, A.idx, None, "csr", 1)
        v = np.ones(b.nnz)
    else:
        A.val = (A.val * 3).to(torch.int64).clamp(0, 1).to(t) if t == torch.uint8 else (A.val * 3).to(t)
        v = A.val.double().cpu().numpy()
    T = A.transposed_storage()
    order = np.lexsort((f, b.idx))
    assert np.array_equal(T.idx.cpu().numpy(), f[order])
    assert np.array_equal(np.diff(T.ptr.cpu().numpy()), np.bincount(b.idx - 1, minlength=n))
    if t is not None:
        assert np.array_equal(T.val.double().cpu().numpy(), v[order])
    if val == "bf16":
        return
    keep = rng.integers(0, 3, n).astype(np.float64)
    by = rng.integers(1, 9, lengths.size).astype(np.float64)
    S, changed = dev.sparse_scale(A, to_dev(by), L.AXIS_ROW, to_dev(keep), L.AXIS_COL, L.MAP_MUL)
    kept = keep[b.idx - 1] != 0
    assert changed == 0 and np.array_equal(S.idx.cpu().numpy(), b.idx[kept] - 1)
    assert np.array_equal(S.val.cpu().numpy(), (v * by[f])[kept])
    assert np.array_equal(np.diff(S.ptr.cpu().numpy()), np.bincount(f[kept], minlength=lengths.size))
