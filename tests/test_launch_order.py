"""The host-side rules of which kernel lets its successor start when (csrc/launch_order.h), without a GPU."""
import os
import shutil
import subprocess

from conftest import ROOT


def _run(tmp_path, body):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    assert cxx, "g++ not found: set CXX"
    (tmp_path / "rules.cpp").write_text('#include <cstdio>\n#include "launch_order.h"\nint main() {\n' + body + "\n}\n")
    subprocess.run([cxx, "-std=c++17", "-pthread", f"-I{ROOT}/yan_b200/csrc", str(tmp_path / "rules.cpp"), "-o", str(tmp_path / "rules")],
                   check=True)
    return subprocess.run([str(tmp_path / "rules")], check=True, capture_output=True, text=True).stdout.split()


def test_a_cast_completes_what_is_in_front_of_it_under_the_promise(tmp_path):
    out = _run(tmp_path, 'std::printf("%d %d", yan::cast_releases_early(false), yan::cast_releases_early(true));')
    assert out == ["1", "0"]
