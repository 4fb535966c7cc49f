"""The kernel the benchmark names for its end-to-end run (CPU test)."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

from bench import host_kernel  # noqa: E402

NAMES = ("rtb_fused_x_scheme", "k_fused_x")


def test_end_to_end_kernel_is_the_one_launched():
    def never():
        raise AssertionError("a mixed host trace takes no compiled kernel")

    assert host_kernel(NAMES, False, never) == NAMES[1]
    assert host_kernel(NAMES, True, lambda: (0, "")) == NAMES[0]
    assert host_kernel(NAMES, True, lambda: (3, "no NVRTC")) == "k_fused_x (no NVRTC)"
