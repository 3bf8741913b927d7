"""Kernels whose work is cut by size (column slabs, tiles of rows and entries)
at the sizes where a cut can go wrong, against the oracle."""
import numpy as np
import pytest

import oracle
from finchgb import _lib as L
from finchgb import device as dev
from finchgb.workloads import SparseBuffers, _fibers_from_lengths, _ptr
from helpers import to_dev, to_host, upload

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
