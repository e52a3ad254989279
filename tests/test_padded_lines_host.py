"""The padded y pass of the smoothing (rows of 4k + 1 .. 4k + 3 samples),
checked on the CPU: launch_smooth, launch_smooth_y_padded and its copy kernel
are taken verbatim from libapr_b200/csrc/pipeline.cu and compiled with g++ behind
the stand-ins of tests/cpp/padded_prelude.hpp; tests/cpp/padded_main.cpp looks at
the runs it makes, at the size of the padded copy, at the copy and at what
happens where the TMA pass does not take a run."""
import os
import re
import shutil
import subprocess

import pytest

from tests.conftest import ROOT

CPP = os.path.join(ROOT, "tests", "cpp")


def _function(src, name):
    """The definition whose first line holds `name`, through its closing brace at column 0."""
    a = src.index(name)
    a = src.rindex("\n", 0, a) + 1
    if src[:a].endswith("template <typename IT>\n"):
        a -= len("template <typename IT>\n")
    return src[a:src.index("\n}\n", a) + 3]


def _translation_unit():
    with open(os.path.join(ROOT, "libapr_b200", "csrc", "pipeline.cu")) as f:
        src = f.read()
    body = "".join(_function(src, n) for n in ("void pad_lines_kernel(", "launch_smooth_y_padded(const uint16_t",
                                                  "launch_smooth(const uint16_t"))
    body, n = re.subn(r"pad_lines_kernel<<<.*?>>>\(", "run_pad(", body, flags=re.S)
    assert n == 1
    with open(os.path.join(CPP, "padded_prelude.hpp")) as f:
        prelude = f.read()
    with open(os.path.join(CPP, "padded_main.cpp")) as f:
        main = f.read()
    return prelude + body + main


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_padded_runs_and_copy(tmp_path):
    src = tmp_path / "padded_check.cpp"
    src.write_text(_translation_unit())
    exe = str(tmp_path / "padded_check")
    subprocess.run(["g++", "-std=c++17", "-O2", "-o", exe, str(src)], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "faults 0" in r.stdout, r.stdout + r.stderr
