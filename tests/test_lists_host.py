"""Index arithmetic of the quartet lists (csrc/lists.cuh), compiled for the
host: positions past 2^31 entries come out whole.

A class of a large molecule passes 2^31 quartets at 17 GB of list, which fits
the GPU; the sizes here are only counted, nothing of that length is made."""
import ctypes
import hashlib
import os
import subprocess
import tempfile

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "hfcode_b200", "csrc")


@pytest.fixture(scope="module")
def lists():
    srcs = [os.path.join(ROOT, "tests", "hostcheck", "host_lists.cpp"), os.path.join(CSRC, "lists.cuh"),
            os.path.join(CSRC, "types.cuh")]
    h = hashlib.sha1(b"".join(open(s, "rb").read() for s in srcs)).hexdigest()[:16]
    out = os.path.join(tempfile.gettempdir(), f"hfgpu_hostlists_{h}.so")
    if not os.path.exists(out):
        subprocess.check_call(["g++", "-O1", "-std=c++20", "-fPIC", "-shared", "-pthread", "-w", "-I", CSRC, "-o",
                               out + ".tmp", srcs[0]])
        os.replace(out + ".tmp", out)
    return ctypes.CDLL(out)


def ll(a):
    return np.ascontiguousarray(a, dtype=np.int64).ctypes.data_as(ctypes.POINTER(ctypes.c_longlong))


def i32(a):
    return np.ascontiguousarray(a, dtype=np.int32).ctypes.data_as(ctypes.POINTER(ctypes.c_int))


@pytest.mark.parametrize("nt,most", [(1, 2048), (127, 2048), (128, 2048), (300, 2048), (513, 1 << 23)])
def test_entries_before_each_tile(lists, nt, most):
    # most < 2^24: one step of 128 tiles stays below 2^31, as 128 tiles of
    # 2048 candidates do; 513 tiles of 2^23 pass 2^32 in all
    rng = np.random.default_rng(nt)
    counts = rng.integers(most // 2, most + 1, size=(nt, 2))
    got = counts.copy()
    lists.hl_scan_tiles(got.ctypes.data_as(ctypes.POINTER(ctypes.c_longlong)), nt)
    want = np.concatenate([np.zeros((1, 2), dtype=np.int64), np.cumsum(counts, 0)[:-1]])
    assert np.array_equal(got, want)
    if most > 2048:
        assert want[-1].min() > 2**31


def class_list(cnt, lanes, prec, n64, coff):
    """Offsets and units of sub-classes with `cnt` entries over 2^lgb x 2^lgk lanes."""
    cnt = np.array(cnt, dtype=np.int64)
    lgb, lgk = np.array(lanes).T
    per = 32 >> (lgb + lgk)
    units = -(-cnt // per)
    off = coff + (n64 if prec else 0) + np.cumsum(cnt) - cnt
    return cnt, off, np.cumsum(units) - units, lgb, lgk, per, int(units.sum())


@pytest.mark.parametrize("prec,n64", [(0, 0), (1, 0), (1, 3 * 2**31 + 7)])
@pytest.mark.parametrize("cnt,lanes", [
    ([70, 0, 33, 1], [(0, 0), (1, 1), (2, 1), (2, 3)]),                       # small lists, an empty sub-class
    ([2**31 + 5, 100], [(0, 0), (1, 0)]),                                     # one sub-class past 2^31
    ([2**31 - 40, 90, 2**32 + 3, 17], [(0, 0), (0, 0), (0, 0), (3, 1)]),      # the class past it in the middle
])
def test_units_and_chunks(lists, cnt, lanes, prec, n64):
    coff = 12345
    cnt, off, unit, lgb, lgk, per, nunit = class_list(cnt, lanes, prec, n64, coff)
    args = [ll(cnt), ll(off), i32(unit), i32(lgb), i32(lgk), len(cnt), nunit, ctypes.c_longlong(coff), prec,
            ctypes.c_longlong(n64)]
    start = coff + (n64 if prec else 0)
    total = int(cnt.sum())
    out = np.zeros((32, 3), dtype=np.int64)
    po = out.ctypes.data_as(ctypes.POINTER(ctypes.c_longlong))
    us = {0, nunit - 1} | {int(unit[k]) + d for k in range(len(cnt)) for d in (-1, 0, 1)}
    us |= {nunit * k // 17 for k in range(17)}
    for u in sorted(x for x in us if 0 <= x < nunit):
        k = max(j for j in range(len(cnt)) if unit[j] <= u)
        assert lists.hl_unit(*args, u, po) == 1
        lg = int(lgb[k] + lgk[k])
        for lane in range(32):
            i = (u - int(unit[k])) * int(per[k]) + (lane >> lg)
            at = int(off[k]) + min(i, int(cnt[k]) - 1)
            stored = i < cnt[k] and lane % (1 << lg) == 0
            assert tuple(out[lane]) == (at, at - start, stored), (u, lane)
    assert lists.hl_unit(*args, nunit, po) == 0
    # the units of a chunk [q0, q0 + n) hold its first and last entry
    got = (ctypes.c_int * 2)()
    for q0 in {0, total // 2, max(0, total - 130), max(0, int(cnt[0]) - 3)}:
        n = min(128, total - q0)
        lists.hl_units_of(*args, ctypes.c_longlong(q0), ctypes.c_longlong(n), got)
        for end, e in ((0, q0), (1, q0 + n - 1)):
            k = max(j for j in range(len(cnt)) if cnt[j] and off[j] - start <= e)
            assert got[end] - end == unit[k] + (e - (off[k] - start)) // per[k]
