"""The host rules that lay launches out, on CPU: they are functions of sizes alone and need no device."""
import ctypes as C

import pytest

from tl_b200 import _lib, synth

SMS, SMEM = 148, 227 * 1024          # a B200

TYPES = [synth.Q4_0, synth.Q8_0, synth.Q4_K, synth.Q6_K]


def matvec_slices(t, n, k, m):
    f = _lib.lib().tlb_matvec_slices
    f.restype, f.argtypes = C.c_int, [C.c_int, C.c_int64, C.c_int64, C.c_int, C.c_int, C.c_size_t]
    return f(t, n, k, m, SMS, SMEM)


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
