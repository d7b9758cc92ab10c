"""Which kernels a class's modules hold: a sampling kernel compiles without the FP64 pass over hand-offs, which
a plain FP64 run never launches and which would double its compilation, and the pass without the other."""
import os
import re
import subprocess

import pytest

from feyntrop_gb300 import build as native


@pytest.fixture(scope="module")
def dump(tmp_path_factory):
    native.build()
    tmp, here = tmp_path_factory.mktemp("modules"), os.path.dirname(native.LIB)
    (tmp / "dump.cpp").write_text("""#include <cstdio>
#include <cstdlib>
#include "%s"
int main(int, char** a)
{
    ft::kernel_key k;
    k.E = 3; k.V = 3; k.loops = 1; k.K = 2; k.ek = {1, 2, 2}; k.el = {0, 1, 0};
    k.prec = std::atoi(a[1]); k.mode = std::atoi(a[2]); k.batch = std::atoi(a[3]); k.part = std::atoi(a[4]);
    std::fputs(ft::kernel_source(k).c_str(), stdout);
}
""" % os.path.join(native.CSRC, "jit.hpp"))
    subprocess.run([native.CXX, "-std=c++17", "-I" + os.path.join(native.CUDA, "include"), str(tmp / "dump.cpp"), "-o",
                    str(tmp / "dump"), "-L" + here, "-lfeyntrop_gb300", "-Wl,-rpath," + here], check=True)
    return str(tmp / "dump")


@pytest.mark.parametrize("prec,mode", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("batch", [0, 1])
def test_one_kernel_per_module(dump, prec, mode, batch):
    for part in range(1 if prec else 2):
        text = subprocess.run([dump] + [str(x) for x in (prec, mode, batch, part)], check=True, capture_output=True,
                              text=True).stdout
        pre = subprocess.run([native.CXX, "-E", "-P", "-x", "c++", "-"], input=text, check=True, capture_output=True,
                             text=True).stdout
        kernels = re.findall(r'extern "C" __global__.*?(ft_\w+)\(', pre, re.S)
        assert kernels == ["ft_sample" + ("_queue" if part else "") + ("_batch" if batch else "")]
