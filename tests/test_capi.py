"""The C ABI without a GPU: the library loads and exports every entry point
include/illatio_b200.h declares, and the argument checks that need no device."""
import ctypes
import os
import re

import pytest

from illatio_b200 import _lib, build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "illatio_b200.h")).read()
    return re.findall(r"ILL_API\s+[\w\s\*]+?\b(ill_\w+)\s*\(", text)


def test_library_builds_and_exports_every_declared_symbol():
    build.build()
    L = ctypes.CDLL(_lib.LIB_PATH)
    names = declared_symbols()
    assert len(names) >= 12
    for n in names:
        assert hasattr(L, n), "libillatio_b200.so does not export %s" % n
        assert n in _lib.SIGNATURES, "no ctypes signature for %s" % n


def test_block_geometry_and_error_text():
    L = _lib.lib()
    assert L.ill_b200_version() >= 100
    assert [L.ill_block_bytes(f) for f in range(6)] == [34, 144, 210, 84, 66, 0]
    assert [L.ill_block_weights(f) for f in range(6)] == [32, 256, 256, 256, 256, 0]
    assert L.ill_error_string(0) == b"ok"
    for code in range(1, 7):
        assert len(L.ill_error_string(code)) > 4


def test_argument_checks_need_no_device():
    # bad format, bad sizes, null and misaligned pointers are rejected before any CUDA call
    s = _lib.status
    assert s("ill_mv", 9, 16, 4, 256, 16, 16, 16, 16, 0, 0, 1, None) == 1
    assert s("ill_mv", 1, 16, 4, 100, 16, 16, 16, 16, 0, 0, 1, None) == 1   # cols not a multiple of 256
    assert s("ill_mv", 1, 16, 4, 256, 16, 16, 0, 16, 0, 0, 1, None) == 1    # Q4_K needs the sums
    assert s("ill_mv", 1, 16, 4, 256, 17, 16, 16, 16, 0, 0, 1, None) == 2   # xq not 16-byte aligned
    assert s("ill_mv", 0, 16, 4, 256, 16, 16, 0, 16, 0, 0, 0, None) == 1    # no tokens
    assert s("ill_quant_q8_k", 8, 16, 16, 16, 1, None) == 2
    assert s("ill_dequant_rows", 4, 16, 100, 0, 0, 1, 16, None) == 1


def test_argument_checks_of_the_chunk_and_peer_entry_points():
    s = _lib.status
    # ill_mm_chunk: Q8_0 has no tcgen05 form; null pointers; a misaligned Q4_K matrix
    assert s("ill_mm_chunk", 0, 16, 4, 256, 16, 16, 16, 8, 16, 0, None) == 3
    assert s("ill_mm_chunk", 1, 0, 4, 256, 16, 16, 16, 8, 16, 0, None) == 1
    assert s("ill_mm_chunk", 1, 24, 4, 256, 16, 16, 16, 8, 16, 0, None) == 2
    assert s("ill_mm_chunk", 1, 16, 4, 256, 16, 0, 16, 8, 16, 0, None) == 1      # Q4_K needs the sums' tile
    assert s("ill_mm_chunk2", 3, 16, 32, 4, 256, 16, 16, 16, 8, 16, 32, None) == 3
    assert s("ill_mm_chunk2", 1, 16, 24, 4, 256, 16, 16, 16, 8, 16, 32, None) == 2  # the second matrix 8 bytes off
    # the peer-storing product and the all-gather by peer stores
    assert s("ill_mv_peers", 2, 16, 4, 256, 16, 16, 16, 0, 0, 0, 16, 16, 2, 0, 2, 1, 0, None) == 1      # no table of buffers
    assert s("ill_mv_peers", 2, 16, 4, 256, 16, 16, 16, 16, 0, 0, 16, 16, 2, 2, 2, 1, 0, None) == 1     # rank >= world
    assert s("ill_peer_put", 16, 64, 16, 0, 16, 16, 65, 0, 2, 1, 0, None) == 1                          # more ranks than flags
    assert s("ill_peer_put", 18, 64, 16, 0, 16, 16, 2, 0, 2, 1, 0, None) == 2                           # SRC not a multiple of 4
    assert s("ill_ep_dispatch", 4, 33, 256, 16, 16, 16, 16, 16, 1, 2, 8, 0, 16, 16, 16, 16, 1, None) == 1   # more than 32 slots
    assert s("ill_quant_q8_k_f16", 16, 16, 16, 16, 0, 16, 1, None) == 1
    # the table of a pointer a row for the one-token kernels: no experts, a misaligned table
    assert s("ill_moe_row_ptrs", 0, 16, 16, 16, 8, 16, None) == 1
    assert s("ill_moe_row_ptrs", 4, 16, 16, 16, 8, 20, None) == 1
    assert s("ill_moe_row_ptrs", 4, 16, 16, 16, 0, 16, None) == 0   # no rows: nothing to do


@pytest.mark.parametrize("fmt", [0, 1, 2, (1, 2)])
@pytest.mark.parametrize("n", [2, 4, 8, 9, 16])
def test_launches_of_few_tokens_stay_within_a_cta(fmt, n):
    """Every launch of two to sixteen tokens has barriers (0 to 15), warps and shared memory that a CTA has, over all numbers of blocks a
    row and the numbers of tiles around whole rounds of 148 SMs: short rows of many rows get up to fifteen groups."""
    two = isinstance(fmt, tuple)
    f = fmt if two else (fmt, 0)
    out, seen = (ctypes.c_int * 8)(), set()
    for blocks in list(range(1, 42)) + [48, 56, 57, 64, 68, 152, 256, 544]:
        cols = blocks * (32 if fmt == 0 else 256)
        for rounds in list(range(1, 20)) + [31, 32, 33, 47, 48, 49, 64, 110]:
            for rows in (16 * rounds, 16 * 148 * rounds - 1600, 16 * 148 * rounds, 16 * 148 * rounds + 1):
                rc = _lib.status("ill_test_few_tokens_plan", 2 if two else 1, f[0], f[1], 0, rows, rows if two else 0, 0, cols, n, 148, out)
                assert rc in (0, 3)
                if rc == 0:
                    warps, groups, barrier, stages, ctas, smem, regs, _ = out
                    seen.add((warps, groups))
                    assert warps >= 1 and groups >= 1 and warps * groups <= 16 and 2 <= stages <= 4 and ctas >= 1
                    assert 1 <= barrier <= 15
                    assert warps * groups >= 8 or cols > 1280  # (all warps bring the activations)
                    per_sm = 1 if ctas <= 148 else 2
                    assert ctas <= 296 and per_sm * (smem + 1024) <= 228 * 1024 and per_sm * 32 * warps * groups * regs <= 65536
    assert (1, 15) in seen


@pytest.mark.parametrize("rows,cols,n,bm,shares,i8", [
    (151936, 896, 17, 32, False, False), (151936, 896, 32, 32, False, False), (151552, 896, 17, 32, False, False), (9728, 2560, 512, 64, True, False),
    (9700, 2560, 505, 64, True, False), (17300, 5120, 399, 64, True, False), (1536, 5120, 8192, 64, True, False), (5120, 1536, 2048, 64, False, False), (896, 4864, 8192, 64, True, False),
    (4096, 2048, 8192, 128, False, False), (36000, 1024, 300, 64, False, False),
    (151936, 896, 80, 80, False, True), (17408, 5120, 160, 64, False, True), (4864, 896, 512, 48, False, True), (896, 4864, 777, 48, False, False)])
def test_tiles_of_a_q8_0_chunk(rows, cols, n, bm, shares, i8):
    """Few tokens of many rows keep the tile that their number asks for on both sides of eight rounds; even shares where they save enough;
    and which of the two kernels takes the chunk."""
    out = (ctypes.c_int * 4)()
    assert _lib.status("ill_test_q8_chunk_plan", rows, cols, n, 148, out) == 0
    assert (out[0], out[1] != 0, bool(out[3])) == (bm, shares, i8) and 1 <= out[2] <= 148
