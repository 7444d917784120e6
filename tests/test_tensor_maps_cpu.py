"""Tensor maps that a launch leaves empty are not touched by its kernel."""
import re
from pathlib import Path

from terapipe_b200.ops import lib

SRC = (Path(lib.__file__).resolve().parent / "csrc" / "gemm_sm100.cu").read_text()


def test_all_reduce_kernels_leave_the_output_map_alone():
    """The fused all-reduce passes no output map: a prefetch of a descriptor that nobody encoded is undefined, so
    every kernel that can be launched that way (one whose prefetches mention the epilogue's maps) guards it."""
    assert re.search(r"const EpiMaps tmE = \{\};.*all-reduce", SRC)
    lines = [line.strip() for line in SRC.splitlines() if "prefetch_tmap(&tmE" in line]
    assert len(lines) == 2 and all(line.startswith("if (!AR) ") for line in lines)
