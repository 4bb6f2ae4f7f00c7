"""Which copies from and to pageable memory go through the pieces of several
threads (csrc/hostcopy.h): the rule on its own, compiled without a GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "hostcopy.h"
int main()
{
    long mb;
    int in;
    sfh::CopyCredit c;
    while (std::scanf("%ld %d", &mb, &in) == 2) std::printf("%d", (int)c.enough((size_t)mb << 20, in != 0));
    return 0;
}
"""


def test_buffers_are_made_once_they_are_repaid(tmp_path):
    """A first upload of 36 or 190 MB, or a first download of 36, is the
    driver's, since making the pieces' buffers takes longer than it; one of a
    gigabyte makes them at once; repeated copies come to it, downloads after a
    third of the bytes; copies below 32 MB never do, nor count."""
    gxx, cuda = shutil.which("g++"), os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    if not gxx or not os.path.exists(os.path.join(cuda, "cuda_runtime.h")):
        pytest.skip("needs g++ and the CUDA headers")
    src, exe = tmp_path / "rule.cpp", tmp_path / "rule"
    src.write_text(PROGRAM)
    r = subprocess.run([gxx, "-std=c++17", "-I" + cuda, "-I" + os.path.join(ROOT, "staggered_fermions_hmc_b200", "csrc"),
                        str(src), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def taken(*copies):
        text = "".join("%d %d\n" % (mb, way == "in") for mb, way in copies)
        return subprocess.run([str(exe)], input=text, capture_output=True, text=True).stdout

    assert taken((36, "in")) == "0" and taken((190, "in")) == "0" and taken((36, "out")) == "0"
    assert taken((1208, "in")) == "1" and taken((101, "out")) == "1"
    assert taken(*[(36, "in")] * 9) == "000000011"
    assert taken(*[(36, "out")] * 4) == "0011"
    assert taken(*[(31, "in")] * 20) == "0" * 20
    assert taken((1208, "in"), (31, "out"), (32, "out")) == "101"
