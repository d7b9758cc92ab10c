"""Launch shapes settled against a block's shared memory: whole warps (the kernels' warp-wide operations name all 32
lanes) whose tables and sums fit an SM, for every class and shape, up to more eps orders than the 30 that 12-edge
graphs took with 102 KB of staged FP64 table."""
import os
import subprocess

from feyntrop_gb300 import build as native

LIMIT = 227 * 1024


def test_blocks_are_whole_warps_that_fit(tmp_path):
    native.build()
    here = os.path.dirname(native.LIB)
    (tmp_path / "shapes.cpp").write_text("""#include <cstdio>
#include "%s"
#include "%s"
int main()
{
    for (int E = 2; E <= 14; E++)
        for (int K = 1; K <= 36; K++)
            for (int cls = 0; cls < 8; cls++)
                for (int block : {0, 384, 512, 256, 128, 96, 64, 48, 33, 32}) {
                    ft::kernel_key k;
                    k.E = E; k.V = E; k.K = K; k.mode = cls & 1; k.prec = cls >> 1 & 1; k.batch = cls >> 2;
                    k.table_global = !ft::staged_table(E);
                    ft::launch_shape s = ft::default_shape(k);
                    if (block) s.block = block;
                    ft::apply_shape(k, s);
                    std::printf("%%d %%d %%d %%d %%d %%d %%u\\n", E, K, cls, block ? block : s.block, k.block, k.minb, ft::table_smem_bytes(k));
                }
}
""" % (os.path.join(native.CSRC, "jit.hpp"), os.path.join(native.CSRC, "tune.hpp")))
    subprocess.run([native.CXX, "-std=c++17", "-I" + os.path.join(native.CUDA, "include"), str(tmp_path / "shapes.cpp"),
                    "-o", str(tmp_path / "shapes"), "-L" + here, "-lfeyntrop_gb300", "-Wl,-rpath," + here], check=True)
    text = subprocess.run([str(tmp_path / "shapes")], check=True, capture_output=True, text=True).stdout
    halved = 0
    for line in text.splitlines():
        E, K, cls, asked, block, minb, smem = map(int, line.split())
        assert block % 32 == 0 and 32 <= block <= max(asked, 32) and 1 <= minb <= 32, line
        assert smem + 64 <= LIMIT, line
        halved += block < asked
    assert halved > 100
