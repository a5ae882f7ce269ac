"""CPU test of the rule that picks the requests whose pinned buffers a kernel
copies: the buffer lies inside one registered range (a buffer whose two ends
are registered apart has a hole that only the copy engine may meet)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_range_covers(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not available")
    out = str(tmp_path / "pinned_check")
    subprocess.run([cxx, "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror",
                    os.path.join(ROOT, "tests", "native", "pinned_check.cc"), "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout


def test_kernel_copies_ask_for_the_range():
    """The request's buffers go through that rule, with the range the driver
    reports."""
    with open(os.path.join(ROOT, "multians_gb300", "csrc", "mans_server.cc")) as f:
        src = f.read()
    body = src[src.index("void* kernel_address("): src.index("struct Table")]
    for want in ("RANGE_START_ADDR", "RANGE_SIZE", "range_covers"):
        assert want in body
