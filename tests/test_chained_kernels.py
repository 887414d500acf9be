"""Kernels launched by launch_chained are set up while their predecessor still writes what
they read: their parameters carry no __restrict__, which would promise the compiler that
nothing else writes it during the kernel."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "thesiscode_b200" / "csrc"
KERNEL = re.compile(r"__global__ void (?:__launch_bounds__\([^;{]*?\)\s*)?(\w+)\(([^{]*?)\)\s*\{\s*(tcb::)?chain_begin\(\);")


def test_no_restrict_on_chained_kernels():
    found = {}
    for f in sorted(CSRC.glob("*.cu*")):
        for name, params, _ in KERNEL.findall(f.read_text()):
            found[name] = "__restrict__" in params
    for name in ("pack_kernel", "velocity_epilogue_kernel", "stage_epilogue_kernel", "ke_finalize_kernel",
                 "small_order_kernel", "stage_copy_kernel", "adj_row_kernel", "adj_combine_row_kernel",
                 "adj_prepare_kernel", "adj_begin_kernel", "pair_fp64_kernel", "pair_fp32c_kernel"):
        assert name in found, name
    assert not [name for name, restricted in found.items() if restricted]
