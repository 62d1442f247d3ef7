"""Which launches may begin before the one ahead of them has completed: the library's host code runs over a
stand-in for the CUDA runtime (launch_recorder.cpp) that notes its launches.  A kernel that reads what an
earlier kernel wrote without waiting by itself has to come behind an ordinary launch."""
from __future__ import annotations

import ctypes as C
import glob
import itertools
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def recorded(tmp_path_factory):
    from torch.utils import cpp_extension as ext

    from scorch_b200 import _lib, build
    build.build()
    path = str(tmp_path_factory.mktemp("recorder") / "librecorded.so")
    include = [f"-I{d}" for d in ext.include_paths("cuda") + ["/usr/local/cuda/include"]]
    subprocess.check_call([build._host_cxx(), "-O1", "-std=c++17", "-shared", "-fPIC", "-Wl,-Bsymbolic", *include,
                           os.path.join(ROOT, "tests", "launch_recorder.cpp"),
                           *sorted(glob.glob(os.path.join(build.OBJDIR, "*.o"))), "-o", path])
    lib = C.CDLL(path)
    for name, (res, args) in _lib.SIGNATURES.items():
        getattr(lib, name).restype, getattr(lib, name).argtypes = res, args
    lib.recorder_kernel.restype = C.c_char_p

    class Recorded:
        abi = lib
        file = path

        @staticmethod
        def call(fn, *args):
            """(kernel name, begins early, CTAs per cluster) of the call's launches."""
            lib.recorder_reset()
            assert fn(*args) == 0, lib.sb_last_error()
            return [(lib.recorder_kernel(i).decode(), bool(lib.recorder_early(i)), lib.recorder_cluster(i))
                    for i in range(lib.recorder_count())]
    return Recorded


def _ptr(a):
    return a.ctypes.data


@pytest.mark.parametrize("dtype", [0, 1, 2, 3])
@pytest.mark.parametrize("n", [1000, 30000])
def test_spgemm_rows_begin_behind_max_abs(recorded, dtype, n):
    # the first kernel of the bins, whichever it is, is an ordinary launch: it and those that begin beside it
    # read max |b| and the operands without a wait
    m = 64
    i32, i64 = (lambda k: np.zeros(k, np.int32)), (lambda k: np.zeros(k, np.int64))
    ws = np.zeros(recorded.abi.sb_spgemm_workspace_bytes(m, n, dtype) + 16, np.uint8)
    pos, crd, val, off, tcrd, tval, cpos = i32(m + 1), i32(4), i64(4), i32(m + 1), i32(4), i64(4), i32(m + 1)
    for bins in itertools.product((0, 7), repeat=5):
        if not any(bins) or (n > 24576 and bins[4]):        # (the bucket path reads its rows back)
            continue
        got = recorded.call(recorded.abi.sb_spgemm_rows, dtype, m, m, n, _ptr(pos), _ptr(crd), _ptr(val), _ptr(pos),
                            _ptr(crd), _ptr(val), _ptr(off), (C.c_int64 * 5)(*bins), _ptr(tcrd), _ptr(tval),
                            _ptr(cpos), C.byref(C.c_int64(0)), (_ptr(ws) + 15) // 16 * 16, ws.size - 16, None)
        rows = [g for g in got if any(k in g[0] for k in ("warp_kernel", "cta_kernel", "split_kernel", "smem_kernel"))]
        assert len(rows) == sum(b > 0 for b in bins)
        assert [early for _, early, _ in rows] == [False] + [True] * (len(rows) - 1), rows
        assert ("max_abs" in got[0][0]) == (bins[4] > 0 and dtype < 2) and not got[0][1]
        assert ("smem_kernel" in rows[-1][0]) == (bins[4] > 0) and rows[-1][2] == (8 if bins[4] else 1)
        assert "scan" in got[-1][0] and not got[-1][1]       # behind all of them


@pytest.mark.parametrize("dtype", [0, 1, 2, 3])
@pytest.mark.parametrize("k", [1, 16, 77, 600])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_spmm_without_entries_begins_behind_its_operands(recorded, dtype, k, accumulate):
    # the second kernel reads the row pointers before its wait: behind the tile kernel that is sound, alone it
    # has to be an ordinary launch
    pos, val, out = np.zeros(10, np.int32), np.zeros(4, np.int64), np.zeros(9 * k, np.int64)
    ws = np.zeros(recorded.abi.sb_spmm_csr_once_workspace_bytes(dtype, k, 4) + 16, np.uint8)
    for nnz in (0, 4):
        got = recorded.call(recorded.abi.sb_spmm_csr_once, dtype, 9, 4, k, nnz, _ptr(pos), _ptr(pos), _ptr(val),
                            _ptr(out), k, None, 0, accumulate, _ptr(out), k, (_ptr(ws) + 15) // 16 * 16, ws.size - 16,
                            None)
        assert "spmm_tile_rows_kernel" in got[-1][0]
        assert [early for _, early, _ in got] == ([True, True] if nnz else [False]), got


@pytest.mark.parametrize("k,per_sm", [(64, 3), (256, 4)])
def test_spmm_windows_fill_the_device_at_hand(recorded, k, per_sm):
    # one wave of windows for a matrix that does not need more, on 148 SMs and on 60
    nnz = 100_000
    pos, x = np.zeros(10, np.int32), np.zeros(64, np.float32)
    ws = np.zeros(recorded.abi.sb_spmm_csr_once_workspace_bytes(0, k, nnz) + 16, np.uint8)
    for device, sms in ((0, 148), (1, 60)):
        recorded.abi.recorder_device(device)
        try:
            recorded.call(recorded.abi.sb_spmm_csr_once, 0, 9, 4, k, nnz, _ptr(pos), _ptr(pos), _ptr(x), _ptr(x) // 32 * 32,
                          k, None, 0, 0, _ptr(x) // 32 * 32, k, (_ptr(ws) + 15) // 16 * 16, ws.size - 16, None)
            assert sms * per_sm * 0.8 < recorded.abi.recorder_grid(0) <= sms * per_sm
        finally:
            recorded.abi.recorder_device(0)


def test_spgemm_reports_missing_host_memory(recorded):
    # the list of the long rows (2 GB for 2^27 of them) does not fit the process: a status, not an exception
    # through the C entry point, which would end the process
    import sys

    from scorch_b200._lib import SIGNATURES
    m = 1 << 27
    script = f"""
import ctypes as C, resource
L = C.CDLL({recorded.file!r})
L.sb_spgemm_workspace_bytes.restype, L.sb_spgemm_workspace_bytes.argtypes = C.c_size_t, [C.c_int64, C.c_int64, C.c_int]
L.sb_last_error.restype = C.c_char_p
need = L.sb_spgemm_workspace_bytes({m}, 30000, 2)
resource.setrlimit(resource.RLIMIT_AS, (1 << 30, 1 << 30))
p = [C.c_void_p(16)] * 9                  # never dereferenced: the list comes first
counts, total = (C.c_int64 * 5)(0, 0, 0, 0, {m}), C.c_int64(0)
I = C.c_int64
rc = L.sb_spgemm_rows(C.c_int(2), I({m}), I({m}), I(30000), *p[:7], counts, p[7], p[8], p[0], C.byref(total),
                      p[1], C.c_size_t(need), None)
print(rc, L.sb_last_error().decode())
"""
    assert len(SIGNATURES["sb_spgemm_rows"][1]) == 19
    r = subprocess.run([sys.executable, "-c", script], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    assert r.stdout.startswith("2 ") and "host memory" in r.stdout
