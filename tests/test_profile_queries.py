"""The launch profile counts launches only: entry points that answer questions pass through untimed (kernels/profile.py)."""
import re
from pathlib import Path

import llama_rs_metal_b200
from llama_rs_metal_b200.kernels import profile


def test_entry_points_that_return_sizes_are_not_timed():
    """Every entry point with a 64-bit result answers a question (launches return an int code)."""
    sources = Path(llama_rs_metal_b200.__file__).parent / "csrc"
    names = {n for f in sources.glob("*.cu") for n in re.findall(r'LRM_API long long (lrm_\w+)\(', f.read_text())}
    assert "lrm_gemm_f32_umma_scratch" in names
    assert all(any(q in name for q in profile._QUERIES) for name in names)


def test_what_has_a_row_of_work_is_launched_from_here():
    """The profile stands between the wrappers and the library: entry points that only other entry points call never pass it."""
    kernels = Path(profile.__file__).parent
    called = {n for f in kernels.glob("*.py") if f.name != "profile.py" for n in re.findall(r"\b(lrm_\w+)", f.read_text())}
    assert set(profile.WORK) <= called, sorted(set(profile.WORK) - called)
