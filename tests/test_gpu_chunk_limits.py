"""Kernels that take another number of blocks from a size on, at both sides of
that size."""
import numpy as np
import pytest
import torch

import oracle
from finchgb import _lib as L
from finchgb import device as dev
from helpers import assert_close, to_dev, to_host, upload
from test_gpu_tiles import csr_of_lengths

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("val", ["f64", "pattern"])
@pytest.mark.parametrize("over", [-1, 0, 3])
def test_runs_of_entries(gpu_lib, over, val):
    """Transposes and masked scalings by runs of 256 entries a block, and of
    2,048 from as many entries as give every SM one: equal numpy's."""
    rng = np.random.default_rng(5)
    n, nnz = 3000, 2048 * torch.cuda.get_device_properties(0).multi_processor_count + over
    lengths = rng.multinomial(nnz - 5000, np.full(1200, 1 / 1200))
    lengths = np.concatenate([[0, 2500], lengths, [0, 2500, 0]])
    b = csr_of_lengths(rng, lengths, n, np.float64)
    assert b.nnz == nnz
    f, A = np.repeat(np.arange(lengths.size), lengths), upload(b)
    if val == "pattern":
        A = dev.DeviceSparse(A.nrows, A.ncols, A.ptr, A.idx, None, "csr", 1)
    T, order = A.transposed_storage(), np.lexsort((f, b.idx))
    assert np.array_equal(to_host(T.idx), f[order])
    assert np.array_equal(np.diff(to_host(T.ptr)), np.bincount(b.idx - 1, minlength=n))
    if val == "f64":
        assert np.array_equal(to_host(T.val), b.val[order])
    v = b.val if val == "f64" else np.ones(nnz)
    by, keep = rng.integers(1, 9, lengths.size).astype(np.float64), rng.integers(0, 3, n).astype(np.float64)
    S, changed = dev.sparse_scale(A, to_dev(by), L.AXIS_ROW, to_dev(keep), L.AXIS_COL, L.MAP_MUL)
    kept = keep[b.idx - 1] != 0
    assert changed == 0 and np.array_equal(to_host(S.idx), b.idx[kept] - 1)
    assert np.array_equal(to_host(S.val), (v * by[f])[kept])
    assert np.array_equal(np.diff(to_host(S.ptr)), np.bincount(f[kept], minlength=lengths.size))


@pytest.mark.parametrize("nf", [1024, 24 * 1024, 24 * 1024 + 1, 40_000])
def test_fold_of_partials(gpu_lib, nf):
    """sum(A .* B) over everything: one block's fold, and two levels of it."""
    rng = np.random.default_rng(nf)
    b = csr_of_lengths(rng, rng.integers(0, 4, nf), 500, np.float64)
    want = oracle.ewise_reduce(0, nf, 500, b.ptr, b.idx, b.val, b.ptr, b.idx, b.val)
    got = to_host(dev.ewise_reduce(0, upload(b), upload(b)))
    assert_close(got, want, np.abs(want), np.float64)


@pytest.mark.parametrize("m", [63, 64, 65, 128])
def test_spgemm_blocks_of_rows(gpu_lib, m):
    """Rows merged by one thread each, 64 a block: a block that is full, one row
    short and one row over, the last row another tier's."""
    rng = np.random.default_rng(m)
    A, B = csr_of_lengths(rng, [5] * (m - 1) + [40], 300, np.float64), csr_of_lengths(rng, np.full(300, 7), 900, np.float64)
    ptr, idx, val = dev.spgemm(upload(A), upload(B)).to_host()
    wp, wi, wv = oracle.spgemm_csr(m, 900, A.ptr, A.idx, A.val, B.ptr, B.idx, B.val, fma=True)
    assert np.array_equal(ptr, wp) and np.array_equal(idx, wi) and np.array_equal(val, wv)
