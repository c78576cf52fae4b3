"""The widest products that the tensor-core 'uvw' kernels accept compile: their index tables pass the 64 KB of constant memory."""
import os
import shutil
import subprocess
import time

import numpy as np
import pytest

from openequivariance_b200 import native
from openequivariance_b200.core import problems as P
from openequivariance_b200.core.descriptor import build_descriptor, descriptor_hash

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def _both(mul, lmax):
    return "+".join(f"{mul}x{l}e+{mul}x{l}o" for l in range(lmax + 1))


def _descriptor(in1, in2, out):
    return build_descriptor(P.FullyConnectedTPProblem(in1, in2, out, shared_weights=True, irrep_dtype=np.float32, weight_dtype=np.float32))


@pytest.mark.skipif(not shutil.which(NVCC), reason="needs nvcc")
@pytest.mark.parametrize("in1,in2,family", [
    (_both(128, 2), "1x0e+1x1o+1x2e+1x3o", "uvw_tc_dw"), (_both(96, 3), "1x0e+1x1o+1x2e+1x3o", "uvw_tc_dw"),
    (_both(128, 3), "1x0e+1x1o+1x2e", "uvw_tc_dw"), ("+".join(["32x0e"] * 32), "1x0e", "uvw_tc_dx_small")])
def test_the_widest_products_compile(in1, in2, family, tmp_path):
    text = _descriptor(in1, in2, in1)
    if native.query(text.encode(), descriptor_hash(text)).fast_path != 2:
        return                                                      # (not taken by these kernels)
    (tmp_path / "t.cu").write_text(native.emit_source(text.encode(), family))
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-cubin", "-o", str(tmp_path / "t.cubin"), str(tmp_path / "t.cu")],
                   check=True, stdout=subprocess.DEVNULL)


@pytest.mark.skipif(not shutil.which(NVCC), reason="needs nvcc")
def test_long_sums_compile_in_seconds(tmp_path):
    """The first call of a problem waits for the compiler: 6 s here; unrolled from templates, and with both kinds of sets in one program, 60 s."""
    text = _descriptor(_both(32, 3), "1x1e+1x1o+1x2e+1x2o", _both(32, 3))
    (tmp_path / "t.cu").write_text(native.emit_source(text.encode(), "uvw_tc_dx_parts"))
    start = time.perf_counter()
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-cubin", "-o", str(tmp_path / "t.cubin"), str(tmp_path / "t.cu")],
                   check=True, stdout=subprocess.DEVNULL)
    assert time.perf_counter() - start < 25


def test_the_sum_of_the_partial_rows_is_a_small_program():
    """Every backward with shared weights needs it, and the general kernels take a minute and more to compile."""
    text = _descriptor(_both(32, 2), "1x0e+1x1o+1x2e", _both(32, 2))
    assert "oeq_generic_dw_reduce(" not in native.emit_source(text.encode(), "generic")
    source = native.emit_source(text.encode(), "dw_reduce")
    assert "oeq_generic_dw_reduce(" in source and len(source) < 4000
