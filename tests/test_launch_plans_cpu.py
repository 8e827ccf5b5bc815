"""The host rules that lay launches out, on CPU: they are functions of sizes alone and need no device."""
import ctypes as C

import pytest

from tl_b200 import _lib, synth

SMS, SMEM = 148, 227 * 1024          # a B200

TYPES = [synth.Q4_0, synth.Q8_0, synth.Q4_K, synth.Q6_K]


def matvec_slices(t, n, k, m, few=0):
    f = _lib.lib().tlb_matvec_slices
    f.restype, f.argtypes = C.c_int, [C.c_int, C.c_int64, C.c_int64, C.c_int, C.c_int, C.c_int, C.c_size_t]
    return f(t, n, k, m, few, SMS, SMEM)


@pytest.mark.parametrize("t", TYPES)
def test_matvec_takes_every_row_length(t):
    """One row fits for K up to 56 units of 256 and any number of outputs, so groups of up to four, halved until they fit, do;
    a slice count divides K."""
    for units in range(1, 57):
        for n in (1, 16, 1000, 4096, 14336, 32000, 128256, 320000):
            for m in (1, 2, 3, 4):
                kb = matvec_slices(t, n, 256 * units, m)
                assert kb > 0 or m > 1, (units, n)
                assert kb == 0 or units % kb == 0 and kb <= 16, (units, n, m)


def test_matvec_rows_that_go_in_smaller_groups():
    """Lengths of tests/test_gpu_quant.py that fit two rows or one, but neither three nor four."""
    for t, units, n, most in [(synth.Q8_0, 41, 40, 3), (synth.Q8_0, 43, 300, 3), (synth.Q8_0, 46, 2048, 3), (synth.Q8_0, 53, 128256, 1), (synth.Q6_K, 53, 40, 3)]:
        assert [matvec_slices(t, n, 256 * units, m) > 0 for m in (1, 2, 3, 4)] == [m <= most for m in (1, 2, 3, 4)], (t, units, n)


def test_chains_of_short_launches_as_measured():
    """Eight warps a CTA where a decode layer was faster with them: rows of 2048 or less, launches of up to 140 units per SM."""
    f = _lib.lib().tlb_matvec_few
    f.restype, f.argtypes = C.c_int, [C.c_int64, C.c_int64, C.c_int]
    for d_model, units, few in [(1024, 14, 1), (1536, 21, 1), (2048, 38, 1), (2048, 76, 1), (2048, 138, 1), (2048, 194, 0), (2304, 35, 0), (2560, 35, 0), (3072, 83, 0), (4096, 28, 0), (4096, 38, 0)]:
        assert f(d_model, units * SMS, SMS) == few, (d_model, units)
    # gate|up of width 1536 (31.9 us a layer unsliced, 34.8 in two slices), down of width 2048 (sliced: 34.8, unsliced: 39)
    assert matvec_slices(synth.Q4_K, 2 * 4096, 1536, 1, few=1) == 1
    assert matvec_slices(synth.Q4_K, 2048, 5632, 1, few=1) > 1


def gemm_form(m, n, k):
    """(activation rows per tile, K ranges, whether two CTAs share a tile)"""
    f = _lib.lib().tlb_gemm_plan
    f.restype, f.argtypes = None, [C.c_int64] * 4 + [C.c_int] + [C.POINTER(C.c_int)] * 3
    nt, splits, pair = C.c_int(), C.c_int(), C.c_int()
    f(m, (n + 127) // 128, k // 256, n, SMS, C.byref(nt), C.byref(splits), C.byref(pair))
    return nt.value, splits.value, bool(pair.value)


def gemm_plan(m, n, k):
    return gemm_form(m, n, k)[:2]


def gemm_ranges(m, n, k):
    """(rows of a tile, K ranges in one cluster, by pairs) where a product takes that form, or None"""
    f = _lib.lib().tlb_gemm_ranges
    f.restype, f.argtypes = C.c_int, [C.c_int64] * 4 + [C.c_int] + [C.POINTER(C.c_int)] * 3
    nt, splits, pair = C.c_int(), C.c_int(), C.c_int()
    found = f(m, (n + 127) // 128, k // 256, n, SMS, C.byref(nt), C.byref(splits), C.byref(pair))
    return (nt.value, splits.value, bool(pair.value)) if found else None


def gemm_dispatch(m, n, k):
    """(rows of a tile, K ranges, by pairs, ranges in one cluster): the form that a product of more than 16 rows runs in"""
    ranges = gemm_ranges(m, n, k)
    return (ranges or gemm_form(m, n, k)) + (ranges is not None,)


def test_gemm_ranges_are_launchable():
    """Clusters of two to six CTAs, two units or more a range, and the other ranges' sums of a CTA's columns fit the activation ring."""
    for n in (1, 128, 256, 1000, 2048, 4096, 5632, 14336, 28672, 128256):
        for k in (256, 768, 1024, 2048, 2304, 4096, 8192, 14336, 28672):
            for m in (17, 31, 64, 65, 100, 128, 129, 160, 255, 256, 257, 300, 333, 384, 385, 512, 513, 769, 1000, 1536, 2048, 2821, 4096, 10000, 9000000):
                form = gemm_ranges(m, n, k)
                if form is None:
                    continue
                nt, splits, pair = form
                assert nt == (m + 15) // 16 * 16 if m <= 128 else nt in ((320, 384) if pair else (128, 160, 192, 224, 256)), (n, k, m)
                assert splits in (2, 3, 4, 6) and splits * (1 + pair) <= 6 and 2 * splits <= k // 256, (n, k, m)
                stage = (nt // 2 if pair else nt) * 128 * (4 if not pair and nt <= 64 else 1)
                ring = max(3 if nt <= 64 else 4, min(16, 192 * 1024 // stage)) * stage
                assert (splits - 1) * -(-(nt // 8) // splits) * 4096 <= ring, (n, k, m)
                assert (m + nt - 1) // nt <= 65535, (n, k, m)


def test_gemm_plans_are_launchable():
    """Tiles that an MMA takes (columns in steps of 16, of 64 where two CTAs halve two accumulators), K ranges of four units or
    more, scratch for the partial sums that stays small beside the outputs' own size or a wave of tiles, a grid within its limit."""
    for n in (1, 128, 256, 1000, 2048, 4096, 5632, 14336, 28672, 128256):
        for k in (256, 768, 1024, 2048, 2304, 4096, 8192, 14336, 28672):
            for m in (17, 31, 64, 65, 100, 128, 129, 160, 255, 256, 257, 300, 333, 384, 385, 512, 513, 769, 1000, 1536, 2048, 2821, 4096, 10000, 9000000):
                nt, splits, pair = gemm_form(m, n, k)
                assert pair == (nt > 256 or m > 128 and k >= 4096 and 2 * m * n * (k // 256 * 256) >= 5e10) and (not pair or nt % 32 == 0), (n, k, m)
                assert nt == (m + 15) // 16 * 16 if m <= 128 else nt in (128, 160, 192, 224, 256, 320, 384), (n, k, m)
                assert splits == 1 or 4 * splits <= k // 256 and splits <= (16 if m <= 128 else 8), (n, k, m)
                assert splits * m * n <= max(2 * m * n, 16 * SMS * 128 * 384), (n, k, m)
                assert (m + nt - 1) // nt <= 65535, (n, k, m)


@pytest.mark.parametrize("n,k,m,plans", [
    # plans within 2 % of the fastest of all measured for Q4_K on a B200, and one that took the time given
    (256, 2048, 4096, [(128, 1)]),                          # 34.0 us; 384 rows: 44.5
    (2048, 2048, 768, [(128, 1)]),                          # 26.8 us; 256 rows: 28.8
    (2048, 2048, 4096, [(256, 1)]),                         # 60.5 us; 320 rows: 73.9
    (5632, 2048, 4096, [(256, 1)]),                         # 128 us; 384 rows: 137
    (4096, 4096, 384, [(128, 1)]),                          # 39.2 us; 192 rows: 41.1
    (4096, 4096, 1536, [(384, 1)]),                         # 60.2 us; 256 rows: 80.4
    (14336, 4096, 333, [(384, 1)]),                         # 55.7 us; 192 rows: 74.1
    (14336, 4096, 512, [(256, 1)]),                         # 79.9 us; 192 rows: 107
    (14336, 4096, 1024, [(256, 1)]),                        # 149 us; 384 rows: 154
    (14336, 4096, 4096, [(384, 1)]),                        # 461 us; 256 rows: 488
    (4096, 14336, 256, [(256, 4)]),                         # 62 us; in one K range: 104
    (4096, 14336, 512, [(256, 2)]),                         # 90.6 us; in one K range: 111
    (4096, 14336, 4096, [(256, 1)]),                        # 512 us; 320 rows: 534
])
def test_gemm_plans_as_measured(n, k, m, plans):
    assert gemm_plan(m, n, k) in plans


def dense_matvec_plan(n, k, slots=1):
    """(chunks in flight, most chunks of a tile per warp, most tiles per CTA) of a bf16 layer of one row"""
    f = _lib.lib().tlb_dense_matvec_plan
    f.restype, f.argtypes = C.c_int, [C.c_int] * 4 + [C.c_size_t] + [C.POINTER(C.c_int)] * 3
    warps, chunks, rounds = C.c_int(), C.c_int(), C.c_int()
    depth = f(n, k, slots, SMS, SMEM, C.byref(warps), C.byref(chunks), C.byref(rounds))
    return depth, chunks.value, rounds.value


def dense_gemm_ranges(T, n, k, gated=False, transposed=False):
    """K ranges of a 16-bit product without experts (n: weight rows, gates and ups both), as launch_dense_gemm asks for them"""
    kt = (k + 63) // 64
    two = kt <= 16 or gated                              # CTAs share an SM
    nt = 128 if transposed else min(128 if two else 256, (T + 31) // 32 * 32)
    stages = min(8, (104 if two else 216) * 1024 // (16384 + nt * 128))
    f = _lib.lib().tlb_dense_gemm_ranges
    f.restype, f.argtypes = C.c_int, [C.c_int] * 7
    s = f(T, n, kt, nt, two, stages, SMS)
    assert s == 1 or (s - 1) * -(-(-(-nt // 32)) // s) * 16384 <= stages * (16384 + nt * 128), (T, n, k)      # the exchange fits the ring
    return s


def test_dense_gemm_ranges_are_launchable():
    for k in (64, 512, 1024, 1100, 2048, 5632, 14336):
        for n in (128, 1000, 2048, 3072, 5632, 10368, 32768):
            for T in (1, 17, 32, 33, 64, 100, 128, 250, 256, 512, 800, 2048):
                for form in ({}, {"gated": True}, {"transposed": True}):
                    s = dense_gemm_ranges(T, n, k, **form)
                    assert s in (1, 2, 3, 4) and (s == 1 or (k + 63) // 64 >= 8 * s), (T, n, k)


def test_dense_matvec_rings_fit():
    for k in list(range(1, 49153, 997)) + [8192, 45056, 45312, 45568, 49152]:
        for n in (1, 40, 1000, 2048, 4096, 8192, 32768):
            depth = dense_matvec_plan(n, k)[0]
            row = (k + 255) // 256 * 1024
            assert depth in (1, 2, 3) and row + depth * 16384 + 4096 <= SMEM, (n, k)      # 4 KB: the kernel's static part at most
