"""The z transform without the divide runs on the twiddles of the z solve's radix schedule, which the
FP32 single transforms do not share: the library refuses it in FP32.

A host program calls the stage without a visible device: the refusal comes before anything is
launched, and the FP64 stage gets as far as the runtime's own error.
"""
import os
import subprocess

import pytest

from mhit36_mixedp_b200 import _lib, build

CALL = r"""
#include "kernels.h"
using namespace mhit;
int main(int argc, char** argv) {
  PoissonArgs a = {};
  a.fp32 = argv[1][0] == '4';
  a.g.nx = a.g.ny = a.g.nz = atoi(argv[2]);
  a.g.nkx = a.g.nx / 2 + 1;
  a.g.pitch = a.g.nkx;
  return poisson_stage(a, PSTAGE_ZFWD, 0) == cudaErrorInvalidValue ? 3 : 4;
}
"""


@pytest.fixture(scope="module")
def call(tmp_path_factory):
    d = tmp_path_factory.mktemp("zfwd")
    (d / "call.cu").write_text(CALL)
    exe = str(d / "call")
    lib = os.path.dirname(_lib.LIB_PATH)
    subprocess.run([build.nvcc(), "-std=c++17", "--expt-relaxed-constexpr", "-I", build.CSRC,
                    "-I", os.path.join(build.ROOT, "include"), str(d / "call.cu"), "-o", exe, "-L", lib,
                    "-lmhit_b200", "-Xlinker", "-rpath," + lib], check=True, capture_output=True)
    return lambda *a: subprocess.run([exe, *map(str, a)], env=dict(os.environ, CUDA_VISIBLE_DEVICES="")).returncode


@pytest.mark.parametrize("n", [16, 256, 512, 1024])
def test_forward_z_transform_is_fp64_only(call, n):
    assert call(4, n) == 3
    assert call(8, n) == 4
