"""The host-side rules of which kernel lets its successor start when (csrc/launch_order.h), without a GPU."""
import glob
import os
import re
import shutil
import subprocess

from conftest import ROOT


def _run(tmp_path, body):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    assert cxx, "g++ not found: set CXX"
    (tmp_path / "rules.cpp").write_text('#include <cstdio>\n#include <initializer_list>\n#include "launch_order.h"\nint main() {\n' + body + "\n}\n")
    subprocess.run([cxx, "-std=c++17", "-pthread", f"-I{ROOT}/yan_b200/csrc", str(tmp_path / "rules.cpp"), "-o", str(tmp_path / "rules")],
                   check=True)
    return subprocess.run([str(tmp_path / "rules")], check=True, capture_output=True, text=True).stdout.split()


def test_which_casts_let_their_successor_start_early(tmp_path):
    """None under the promise that the call in front of a GEMM does not write its weights; otherwise those of the small batches."""
    out = _run(tmp_path, """for (unsigned m : {1u, 64u, 65u, 8192u})
        std::printf("%d%d ", yan::cast_releases_early(m, false), yan::cast_releases_early(m, true));""")
    assert out == ["10", "10", "00", "00"]


def test_the_first_gemm_of_a_place_waits_after_the_promise_is_made(tmp_path):
    """A quantizer launched while the promise was off may still let what follows it start early: on every stream, in every capture
    and after every switch the first GEMM does not rely on the promise, the ones behind it do."""
    out = _run(tmp_path, """
    yan::ConstantWeights w;
    int stream[100];
    auto at = [&](int device, int s, unsigned long long capture = 0, bool known = true) {
        return yan::LaunchPlace{w.era(), device, stream + s, capture, known};
    };
    auto gemm = [&](const yan::LaunchPlace& p) {
        std::printf("%d ", w.holds(p));
        w.settle(p);
    };
    gemm(at(0, 0)); gemm(at(0, 0));
    std::printf("off ");
    w.set(true);
    gemm(at(0, 0)); gemm(at(0, 0)); gemm(at(0, 1)); gemm(at(1, 0)); gemm(at(0, 0, 7)); gemm(at(0, 0, 7)); gemm(at(0, 0));
    gemm(at(0, 2, 0, false)); gemm(at(0, 2, 0, false));
    w.set(true);
    gemm(at(0, 0));
    std::printf("on ");
    const yan::LaunchPlace before = at(0, 0);
    w.set(false);
    gemm(at(0, 0));
    w.set(true);
    w.settle(before);
    gemm(at(0, 0)); gemm(at(0, 0));
    std::printf("switched ");
    for (int s = 10; s < 90; ++s) w.settle(at(0, s));
    gemm(at(0, 89)); gemm(at(0, 10)); gemm(at(0, 10));
    std::printf("many");""")
    assert " ".join(out) == "0 0 off 0 1 0 0 0 1 1 0 0 1 on 0 0 1 switched 1 0 1 many"


def test_kernels_that_start_beside_the_one_in_front_use_coherent_loads():
    """The non-coherent path is defined for data that nobody writes while the kernel is resident: only a kernel that is launched
    plainly, after everything in front of it, may use it."""
    for path in glob.glob(f"{ROOT}/yan_b200/include/**/*.cuh", recursive=True):
        with open(path) as f:
            code = re.sub(r"//.*", "", f.read())
        plain = re.search(r"__global__[^;{]*per_block_cast_to_fp8_kernel.*?\n}\n", code, re.S)
        code = code.replace(plain.group(0), "") if plain else code
        assert not re.search(r"__ldg\b|ld\.global\S*\.nc\b", code), path
