"""Virtual-row schedules keep 32-bit indices and scan two counts to a word: a
matrix with more virtual rows is refused, also where the words have run over."""
import ctypes
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "finch.jl_gb300" / "csrc"
SHIM = r"""
#include "vrow_counts.h"
extern "C" int fits(const unsigned long long* rows, int n) { return fgb::vrow_fits(rows, n); }
extern "C" long long scanned(const long long* lo, const long long* hi, int n, int high) {
  int64_t all = 0;
  for (int k = 0; k < n; ++k) all += fgb::vr_pack(lo[k], hi[k]);
  return high ? fgb::vr_hi(all) : fgb::vr_lo(all);
}
"""


@pytest.fixture(scope="module")
def shim(tmp_path_factory):
    d = tmp_path_factory.mktemp("vrow_shim")
    (d / "shim.cpp").write_text(SHIM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(CSRC), str(d / "shim.cpp"), "-o",
                    str(d / "shim.so")], check=True)
    lib = ctypes.CDLL(str(d / "shim.so"))
    lib.scanned.restype = ctypes.c_longlong
    return lib


@pytest.mark.parametrize("rows,slots", [([5, 2**31 - 6], [4, 2**31 - 7]), ([2**31], [0]), ([2**32, 7], [0, 3]),
                                        ([2**31, 2**31, 9], [2**31, 2**31, 0]), ([2**63, 2**63, 3], [0, 0, 2])])
def test_more_rows_than_indices_are_refused(shim, rows, slots):
    n, total = len(rows), sum(rows)
    assert bool(shim.fits((ctypes.c_ulonglong * n)(*rows), n)) == (total < 2**31)
    if total < 2**31:  # the words then hold both counts
        lo, hi = (ctypes.c_longlong * n)(*rows), (ctypes.c_longlong * n)(*slots)
        assert shim.scanned(lo, hi, n, 0) == total and shim.scanned(lo, hi, n, 1) == sum(slots)
    elif total < 2**63:  # what the low half alone would say
        lo, hi = (ctypes.c_longlong * n)(*rows), (ctypes.c_longlong * n)(*slots)
        assert shim.scanned(lo, hi, n, 0) == total % 2**32
