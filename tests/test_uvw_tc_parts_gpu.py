"""Tensor-core 'uvw' kernels where a tile's schedule is dealt to several CTAs: batches around one tile (64 / 128 items), few
tiles (every cut of the schedule), one tile more than there are SMs (a ragged last wave), against the fp64 oracle."""
import pytest

from openequivariance_b200.core.problem import TPProblem
from test_uvw_f64_gpu import orders_0_to_2, shared_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("batch", [1, 64, 65, 129, 1000, 2500, 128 * 148 + 1])
def test_cut_schedules(batch, wide):
    # (one tile more than there are SMs is cut where the cut's price is less than the wave that it saves)
    cut = [f"oeq_uvw_tc_{k}_parts" for k in ("forward", "backward_dx", "backward_dy")] if batch <= 2500 else []
    orders_0_to_2(shared_problem(wide), batch, cut + ["oeq_uvw_tc_backward_dw"])


@pytest.mark.parametrize("batch", [77, 47 * 128, 100 * 128 + 5])   # the small sets in parts, the large ones in parts, a whole tile per CTA
def test_weights_at_any_address_and_batches_between(batch):
    """Weights that do not start on 16 bytes are copied first; batches of too few tiles for the chip deal a tile's large sets to several
    CTAs.  Against the same product in doubles: sums of a few hundred products, split to 2^-21, in fp32."""
    import numpy as np
    import torch

    import openequivariance_b200 as oeq
    from helpers import with_dtype
    p = shared_problem(True)
    gen = torch.Generator(device="cuda").manual_seed(batch)
    x, y, g = (torch.randn(batch, n, device="cuda", generator=gen) for n in (p.irreps_in1.dim, p.irreps_in2.dim, p.irreps_out.dim))
    w = torch.randn(p.weight_numel + 1, device="cuda", generator=gen)[1:]
    assert w.data_ptr() % 16 != 0
    found = []
    for q, dt in ((p, torch.float32), (with_dtype(p, np.float64), torch.float64)):
        tp = oeq.TensorProduct(q)
        args = [t if dt == torch.float32 else t.double() for t in (x, y, w, g)]
        z = torch.ops.libtorch_tp_jit.jit_tp_forward(tp.kernel, tp.hash, *args[:3], q.irreps_out.dim)
        found.append([z, *torch.ops.libtorch_tp_jit.jit_tp_backward(tp.kernel, tp.hash, *args)])
    for a, b, bound in zip(*found, (1e-6, 1e-6, 1e-6, 4e-6)):     # (dW: sums of 64 items in the tensor cores, which truncate)
        assert float((a.double() - b).norm() / b.norm()) <= bound


def test_weight_gradient_of_a_product_whose_tables_pass_constant_memory():
    """512 weight tiles or more: the weight-gradient kernel reads its tables from global memory, in several launches of 16 groups."""
    import numpy as np
    import torch

    import openequivariance_b200 as oeq
    from helpers import kernels_launched, rel_l2, uniform_inputs
    from openequivariance_b200.core import problems as P
    from oracle import tp_oracle
    feats = "128x0e+128x0o+128x1e+128x1o+128x2e+128x2o"
    p = P.FullyConnectedTPProblem(feats, "1x0e+1x1o+1x2e+1x3o", feats, shared_weights=True, irrep_dtype=np.float32, weight_dtype=np.float32)
    tp = oeq.TensorProduct(p)
    x, y, w, g, *_ = uniform_inputs(p, 65)
    args = [torch.tensor(t, device="cuda") for t in (x, y, w, g)]
    got, ran = kernels_launched(lambda: torch.ops.libtorch_tp_jit.jit_tp_backward(tp.kernel, tp.hash, *args))
    assert "oeq_uvw_tc_backward_dw" in ran
    want = list(tp_oracle.backward(p, x, y, tp.reorder_weights_to_e3nn(w), g))
    want[2] = tp.reorder_weights_from_e3nn(want[2])
    for a, b in zip(got, want):
        assert rel_l2(a.cpu().numpy(), b) <= 1e-5


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_a_harmonic_that_is_not_finite_stays_in_its_paths(bad):
    import torch

    import openequivariance_b200 as oeq
    p = shared_problem(False)
    tp = oeq.TensorProduct(p)
    gen = torch.Generator(device="cuda").manual_seed(1)
    x, y, w, g = (torch.randn(*n, device="cuda", generator=gen) for n in
                  ((70, p.irreps_in1.dim), (70, p.irreps_in2.dim), (p.weight_numel,), (70, p.irreps_out.dim)))

    def of(first):
        y[33, 0] = first
        z = torch.ops.libtorch_tp_jit.jit_tp_forward(tp.kernel, tp.hash, x, y, w, p.irreps_out.dim)
        return z, *torch.ops.libtorch_tp_jit.jit_tp_backward(tp.kernel, tp.hash, x, y, w, g)
    (z, dx, dy, dw), (_, _, _, dw0) = of(bad), of(0.0)
    others = torch.arange(70, device="cuda") != 33
    assert all(t[others].isfinite().all() and not t[33].isfinite().all() for t in (z, dx)) and dy.isfinite().all()
    at = 0
    for ins in p.instructions:
        n = int(torch.tensor(ins.path_shape).prod())
        path, path0, at = dw[at:at + n], dw0[at:at + n], at + n
        if ins.i_in2 == 0:
            assert not path.isfinite().any()
        else:
            assert torch.equal(path, path0)


def test_a_thread_whose_first_use_of_the_device_is_a_product():
    """(Its outputs come from memory that torch keeps: nothing else has made a context current in the thread.)"""
    import threading

    import torch

    import openequivariance_b200 as oeq
    p = shared_problem(False)
    tp = oeq.TensorProduct(p)
    gen = torch.Generator(device="cuda").manual_seed(2)
    x, y, w, g = (torch.randn(*n, device="cuda", generator=gen) for n in
                  ((70, p.irreps_in1.dim), (70, p.irreps_in2.dim), (p.weight_numel,), (70, p.irreps_out.dim)))
    found = []

    def call():
        found.append(torch.ops.libtorch_tp_jit.jit_tp_forward(tp.kernel, tp.hash, x, y, w, p.irreps_out.dim))
    call()
    want = found.pop().clone()
    for backward in (False, True):
        torch.ops.libtorch_tp_jit.jit_tp_backward(tp.kernel, tp.hash, x, y, w, g)     # (compiled; its memory is free again)
        target = call if not backward else lambda: found.append(torch.ops.libtorch_tp_jit.jit_tp_backward(tp.kernel, tp.hash, x, y, w, g))
        thread = threading.Thread(target=target)
        thread.start()
        thread.join()
    assert len(found) == 2 and torch.equal(found[0], want) and all(t.isfinite().all() for t in found[1])


def test_other_operators_run_while_a_program_compiles(tmp_path):
    import os
    import threading
    import time

    import torch

    import openequivariance_b200 as oeq
    from openequivariance_b200 import native
    from openequivariance_b200.core import problems as P
    small = P.readme_problem()
    tp = oeq.TensorProduct(small)
    rnd = lambda *s: torch.randn(*s, device="cuda")  # noqa: E731
    operands = [rnd(100, small.irreps_in1.dim), rnd(100, small.irreps_in2.dim), rnd(100, small.weight_numel)]
    tp(*operands)
    feats = "32x0e+32x1e+64x2o+32x3e"                        # (a product of no other test)
    p = P.FullyConnectedTPProblem(feats, "1x0e+1x1o+1x2e", feats, shared_weights=True)
    wide = oeq.TensorProduct(p)
    leaves = [t.requires_grad_() for t in (rnd(50, p.irreps_in1.dim), rnd(50, p.irreps_in2.dim), rnd(p.weight_numel))]
    gate, done, times = threading.Event(), threading.Event(), []

    def first_use():
        gate.set()
        times.append(time.perf_counter())
        try:
            wide(*leaves).sum().backward()
        finally:
            times.append(time.perf_counter())
            done.set()

    native.set_option("cache_dir", str(tmp_path))            # empty: the programs have to be compiled
    thread = threading.Thread(target=first_use)
    thread.start()
    gate.wait()
    longest, calls = 0.0, 0
    while not done.is_set():
        start = time.perf_counter()
        tp(*operands)
        if not done.is_set():
            longest, calls = max(longest, time.perf_counter() - start), calls + 1
        time.sleep(0.001)
    thread.join()
    native.set_option("cache_dir", os.path.join(os.path.dirname(oeq.__file__), "csrc", "_cubin_cache"))
    assert times[1] - times[0] > 0.5                         # it was compiled here
    assert calls > 10 and longest < 0.25 * (times[1] - times[0]), (calls, longest, times)
    assert all(t.grad.isfinite().all() for t in leaves)


@pytest.mark.parametrize("family", ["uvw_tc", "uvw_tc_dx_parts"])      # (what 50 items of these problems run)
def test_general_kernels_serve_a_problem_whose_program_is_unusable(family, tmp_path):
    """A cubin without the kernel stands in the cache where the program's should be."""
    import ctypes
    import os
    import shutil
    import subprocess

    import torch

    import openequivariance_b200 as oeq
    from helpers import kernels_launched, rel_l2, uniform_inputs
    from openequivariance_b200 import native
    from openequivariance_b200.core.descriptor import build_descriptor
    from oracle import tp_oracle
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    if not shutil.which(nvcc):
        pytest.skip("needs nvcc")
    p = TPProblem("32x1e", "1x1e", "32x1e" if family == "uvw_tc" else "32x2e", [(0, 0, 0, "uvw", True)], shared_weights=True, internal_weights=False)
    # (the name of a cubin in the cache: a hash of the source, the compiler's options and its version)
    major, minor = ctypes.c_int(), ctypes.c_int()
    native.load()
    ctypes.CDLL("libnvrtc.so.12").nvrtcVersion(ctypes.byref(major), ctypes.byref(minor))
    key = 1469598103934665603
    for c in (native.emit_source(build_descriptor(p).encode(), family) + "--gpu-architecture=sm_100a--std=c++17-lineinfo-default-device--extra-device-vectorization"
              + str(major.value * 100 + minor.value)).encode():
        key = (key ^ c) * 1099511628211 % 2 ** 64
    (tmp_path / "t.cu").write_text('extern "C" __global__ void nothing() {}\n')
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-cubin", "-o", str(tmp_path / f"{key:016x}.cubin"), str(tmp_path / "t.cu")], check=True)
    native.set_option("cache_dir", str(tmp_path))
    try:
        x, y, w, g, x2, y2, w2 = uniform_inputs(p, 50)
        tp = oeq.TensorProduct(p)
        t = [torch.tensor(a, device="cuda") for a in (x, y, w, g, x2, y2, w2)]
        ops = torch.ops.libtorch_tp_jit
        got, ran = kernels_launched(lambda: [ops.jit_tp_forward(tp.kernel, tp.hash, *t[:3], p.irreps_out.dim), *ops.jit_tp_backward(tp.kernel, tp.hash, *t[:4]),
                                             *ops.jit_tp_double_backward(tp.kernel, tp.hash, *t)])
    finally:
        native.set_option("cache_dir", os.path.join(os.path.dirname(oeq.__file__), "csrc", "_cubin_cache"))
    assert {"oeq_generic_backward_shared", "oeq_generic_forward"} <= ran and "oeq_uvw_tc_backward_dw" not in ran, ran
    we, we2 = tp.reorder_weights_to_e3nn(w), tp.reorder_weights_to_e3nn(w2)
    want = [tp_oracle.forward(p, x, y, we), *tp_oracle.backward(p, x, y, we, g), *tp_oracle.double_backward(p, x, y, we, g, x2, y2, we2)]
    for n, (a, b) in enumerate(zip(got, want)):
        assert rel_l2(a.cpu().numpy(), tp.reorder_weights_from_e3nn(b) if n in (3, 6) else b) <= 1e-5
