"""The rule for the share of a layout that solves keep in L2, compiled from the
solver's header with the host compiler."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "mille-feillue_b200", "csrc")
CUDA_INC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
L2 = 126.0 * 2 ** 20
TENSOR_MEMORY = {3, 5, 6}  # mixed CG, CG, Jacobi PCG with x and r in tensor memory


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.exists(os.path.join(CUDA_INC, "cuda_runtime.h")),
                    reason="host compiler or CUDA headers missing")
def test_only_tensor_memory_kernels_keep_slabs_in_l2(tmp_path):
    """Vectors in global memory need L2 themselves: BiCGSTAB of 110^3 lost 13 % with a share kept."""
    src, exe = tmp_path / "keep.cpp", tmp_path / "keep"
    src.write_text("""#include <cstdio>
#include <cstdlib>
#include "solver.h"
int main(int, char **a) { std::printf("%d", mf::l2_keep(atoi(a[1]), atof(a[2]), atof(a[3]), atof(a[4]))); }
""")
    subprocess.run(["g++", "-std=c++17", "-I", CUDA_INC, "-I", os.path.join(ROOT, "include"), "-I", CSRC, str(src),
                    "-o", str(exe), "-L", os.path.join(os.path.dirname(CUDA_INC), "lib64"), "-lcudart"], check=True)

    def keep(kind, n):  # a 7-point grid of n^3: about 72 bytes a row
        return int(subprocess.run([str(exe), str(kind), str(L2), str(72.0 * n ** 3), str(float(n ** 3))],
                                  check=True, capture_output=True, text=True).stdout)

    for kind in range(10):
        assert keep(kind, 75) == 0  # fits L2 with its vectors
        for n in (100, 128, 150):
            want = int(min(256.0, 64.0 * L2 / (72.0 * n ** 3))) if kind in TENSOR_MEMORY else 0
            assert keep(kind, n) == want, (kind, n)
