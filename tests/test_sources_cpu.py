"""Rules of the sources that no result shows reliably."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tl_b200", "csrc")


def lines(pattern):
    """(file, line) of every line of code that has the pattern"""
    found = []
    for f in sorted(glob.glob(os.path.join(CSRC, "*"))):
        for s in open(f, encoding="utf-8"):
            if re.search(pattern, s.split("//")[0]):
                found.append((os.path.basename(f), s.strip()))
    return found


def test_quantised_models_divide_exactly():
    """__fdividef (two units in the last place) is for the sigmoids of layered models, whose sessions state it."""
    assert {f for f, _ in lines(r"\b__(fdividef|expf)\(")} <= {"act.cuh"}


def test_non_coherent_loads_read_weights_and_tables():
    """Kernels start while the one before them ends, and such a load may be moved ahead of the wait for it."""
    table = r"__ldg\((cs|sn|src) \+|__ldg\(reinterpret_cast<const (uint4|__half|float4) \*>\((p|norm_w|p\.norm_w|emb)\b"
    assert [s for s in lines(r"\b__ldg\(") if len(re.findall(r"\b__ldg\(", s[1])) != len(re.findall(table, s[1]))] == []


def test_device_memory_is_filled_in_stream_order():
    """cudaMemset fills on the default stream, which the library's stream does not wait for."""
    assert lines(r"\bcudaMemset(2D|3D)?\(") == []
