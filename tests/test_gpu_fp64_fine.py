"""The fine logarithm and exponential of csrc/fp64_math.cuh (the stochastic transport's)
where the quick ones are tested: the same arguments, edges and bound against CUDA's."""
import subprocess

import pytest
from test_gpu_fp64_math import SOURCE

pytestmark = pytest.mark.gpu


def test_fine_functions_against_cuda(tmp_path):
    import build
    src, exe = tmp_path / "check.cu", tmp_path / "check"
    src.write_text(SOURCE.replace("f64::log(", "f64::log_fine(").replace("f64::exp(", "f64::exp_fine("))
    subprocess.check_call([build.nvcc(), *build.ARCH, "-O2", "-std=c++17", "-I", build.SRC, str(src), "-o", str(exe)])
    log, exp = (float(v) for v in subprocess.check_output([str(exe)], timeout=120).split()[:2])
    assert max(log, exp) <= 4.0, (log, exp)
