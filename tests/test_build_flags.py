"""The engine's build gives the same code for the same sources."""
from pangu_b200 import build


def test_units_are_not_split_before_ptxas():
    """nvcc's -split-compile divides a unit differently from one compile to the next:
    two compiles of engine.cu gave objects of 33.2 and 37.0 MB, with other registers and
    spills, times 8 % apart and (mixed form) other contractions. ptxas's is harmless."""
    flags = build.NVCC_FLAGS
    for i, f in enumerate(flags):
        if "split-compile" in f:
            assert i > 0 and flags[i - 1] == "-Xptxas", f
