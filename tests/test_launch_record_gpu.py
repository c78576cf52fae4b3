"""The library's own record of the kernels that it launched."""
import numpy as np
import pytest
import torch

from helpers import kernels_launched, single

pytestmark = pytest.mark.gpu


def test_record_holds_the_kernels_of_one_call():
    import openequivariance_b200 as oeq
    from openequivariance_b200 import native
    p = single("5x1e", "1x1e", "5x1e", "uvu")
    tp = oeq.TensorProduct(p)
    x, y, w = (torch.ones(7, n, device="cuda", requires_grad=True) for n in (p.irreps_in1.dim, p.irreps_in2.dim, p.weight_numel))
    before = native.launch_count()
    z, ran = kernels_launched(lambda: tp(x, y, w))
    assert ran == {"oeq_generic_forward"} and native.launch_count() == before + 1
    _, ran = kernels_launched(lambda: torch.autograd.grad(z, [x, y, w], torch.ones_like(z)))     # a fresh record for each call
    assert ran == {"oeq_generic_backward"}
    tp(x, y, w)                                                                                   # nothing is kept while it is off
    assert native.launched_kernels() == ran and np.isfinite(z.detach().cpu().numpy()).all()
