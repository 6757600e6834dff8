"""The dense work of the host engine (host/dense.cpp) on the CPU."""
import os
import re
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = os.path.join(HERE, "..", "nutrlan_b200", "csrc", "host", "dense.cpp")


def _preprocessed(tmp_path, *flags):
    """dense.cpp as the compiler's later stages see it, its includes empty."""
    for name in re.findall(r'#include [<"]([^>"]+)', open(SRC).read()):
        (tmp_path / name).write_text("")
    shutil.copy(SRC, tmp_path / "dense.cpp")
    return subprocess.run(["g++", "-E", "-P", "-nostdinc", "-I", str(tmp_path), *flags, str(tmp_path / "dense.cpp")],
                          check=True, capture_output=True, text=True).stdout


def test_no_x86_attribute_on_other_hosts(tmp_path):
    other = _preprocessed(tmp_path, "-U__x86_64__", "-U__i386__", "-D__aarch64__")
    assert "apply_sweep" in other and "avx" not in other
    if os.uname().machine == "x86_64":
        assert "avx2" in _preprocessed(tmp_path)
