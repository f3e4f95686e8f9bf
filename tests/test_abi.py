"""The C-ABI library loads and exports every entry point declared in include/ptn_gb300.h."""
import ctypes
import os
import re

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "include", "ptn_gb300.h")


def declared():
    src = open(HEADER).read()
    src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
    return sorted(set(re.findall(r"\b(ptn_\w+)\s*\(", src)))


def test_header_declares_entry_points():
    names = declared()
    assert "ptn_zcontract" in names and "ptn_zqr_keep" in names


def test_library_exports_all_declared_symbols():
    from pytreenet_gb300 import build
    lib_path = build.build()
    lib = ctypes.CDLL(lib_path)
    missing = [n for n in declared() if not hasattr(lib, n)]
    assert not missing, missing


def test_binding_signatures_cover_header():
    from pytreenet_gb300 import _lib
    assert set(declared()) <= set(_lib.SIGNATURES)


def test_zcontract_split_rule_covers_k_exactly():
    """The K split of the FP64 contraction (host arithmetic of the library):
    chunks are multiples of the K step, cover [0, K) exactly, number about
    304 CTAs in all, and only skinny outputs with a long K are split."""
    import ctypes
    from pytreenet_gb300 import _lib
    lib = _lib.load()
    chunk = ctypes.c_int64()
    for tiles in (1, 2, 3, 7, 38, 39, 400):
        for K in (1, 64, 2047, 2048, 4550, 65536, 10 ** 6 + 3):
            s = int(lib.ptn_zcontract_splits(tiles, K, ctypes.byref(chunk)))
            c = chunk.value
            if tiles > 38 or K < 2048:
                assert s == 1 and c == K
                continue
            assert s >= 1 and (s == 1 or c % 8 == 0)
            assert (s - 1) * c < K <= s * c
            assert tiles * s <= 304 + tiles
            assert s == 1 or c >= 256 - 8


def test_zcontract_scratch_rule():
    """Scratch of the tensor-core complex128 path (host arithmetic): none below
    its least size, and bounded by the digits of B, one GiB of digits of A (or
    one row tile) and the partial sums."""
    import ctypes
    from pytreenet_gb300 import _lib
    lib = _lib.load()

    def need(M, N, K):
        d = _lib.ContractDesc()
        for g, n in ((d.m, M), (d.n, N), (d.k, K)):
            g.n = 1
            g.dim[0] = n
        return int(lib.ptn_zcontract_work_bytes(ctypes.byref(d)))
    assert need(16, 16, 16) == 0 and need(1, 1, 1) == 0
    assert need(3000, 64, 64) == need(64, 3000, 64) > 0           # either operand may lead
    for M, N, K in ((640, 128, 128), (1 << 22, 10, 10), (90, 31, 8100), (655360, 256, 1280)):
        stages = (K + 15) // 16
        a = max(1 << 30, stages * 57344)
        b = (min(M, N) + 31) // 32 * stages * 28672
        assert 0 < need(M, N, K) <= a + b + 16 * 152 * 128 * 64 + 16 * M + (1 << 24)
