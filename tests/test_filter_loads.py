"""The filters' loads of the levels before them: a kernel that begins while its predecessor runs may not read what that
one writes through the non-coherent path (ld.global.nc, __ldg), which is for memory that is read-only for the kernel's
whole lifetime."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nvidia-texture-tools_gb300", "csrc")


def test_levels_are_not_read_through_ldg():
    text = open(os.path.join(CSRC, "ntg_mip.cu")).read()
    early = text[:text.index("launch_after(")]  # every kernel that may be launched early stands before the launchers
    assert early.count("after_previous(njobs, order)") == 6
    assert not re.findall(r"__ldg\([^;]{0,40}\.src\b", early)
