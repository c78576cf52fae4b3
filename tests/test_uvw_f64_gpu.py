"""'uvw' in doubles with shared weights on the FP64 matrix instruction, against the fp64 oracle: batches around the 8 items of a
warp, the 32 of a block and the chunks of the weight gradient, one and two weight tiles per block, degrees up to 3."""
import numpy as np
import pytest
import torch

from helpers import REL_L2, kernels_launched, rel_l2, with_dtype
from openequivariance_b200.core.problem import TPProblem
from oracle import tp_oracle

pytestmark = pytest.mark.gpu


def shared_problem(wide):
    # destination tiles of very different cost (1, 3 and 5 components), one input block that no path reads
    mul = 64 if wide else 32
    return TPProblem(f"{mul}x0e+32x1o+32x2e+32x3o", "1x0e+1x1o+1x2e", f"32x0e+{mul}x1o+32x2e",
                     [(0, 0, 0, "uvw", True), (1, 1, 0, "uvw", True), (0, 1, 1, "uvw", True), (1, 0, 1, "uvw", True),
                      (1, 2, 1, "uvw", True), (0, 2, 2, "uvw", True), (2, 0, 2, "uvw", True), (2, 2, 2, "uvw", True)],
                     shared_weights=True, internal_weights=False)


def orders_0_to_2(p, batch, kernels):
    """All orders against the oracle; ``kernels``: names that have to be among those that ran."""
    import openequivariance_b200 as oeq
    dt = torch.float32 if p.irrep_dtype == np.float32 else torch.float64
    tp = oeq.TensorProduct(p)
    gen = torch.Generator().manual_seed(batch)
    rnd = lambda *s: torch.randn(*s, generator=gen, dtype=dt)  # noqa: E731
    x, y, w, g = rnd(batch, p.irreps_in1.dim), rnd(batch, p.irreps_in2.dim), rnd(p.weight_numel), rnd(batch, p.irreps_out.dim)
    x2, y2, w2 = rnd(*x.shape), rnd(*y.shape), rnd(*w.shape)
    leaves = [t.cuda().requires_grad_(True) for t in (x, y, w, g)]
    def forward_and_gradients():
        z = tp(*leaves[:3])
        first = torch.autograd.grad(z, leaves[:3], leaves[3], create_graph=True)
        return z, first, torch.autograd.grad(first, leaves, [t.cuda() for t in (x2, y2, w2)])

    (z, first, second), ran = kernels_launched(forward_and_gradients)
    assert set(kernels) <= ran, ran
    again = torch.autograd.grad(tp(*leaves[:3]), leaves[:3], leaves[3])
    assert all(torch.equal(a, b) for a, b in zip(first, again))        # sums run in a fixed order
    to_e3nn = lambda t: np.asarray(tp.reorder_weights_to_e3nn(t.detach().cpu().numpy()))  # noqa: E731
    args = [x.numpy(), y.numpy(), to_e3nn(w)]
    got = [z, *first, *second]
    want = [tp_oracle.forward(p, *args), *tp_oracle.backward(p, *args, g.numpy()),
            *tp_oracle.double_backward(p, *args, g.numpy(), x2.numpy(), y2.numpy(), to_e3nn(w2))]
    for n, (a, b) in enumerate(zip(got, want)):
        a = to_e3nn(a) if n in (3, 6) else a.detach().cpu().numpy()
        assert rel_l2(a, b) <= REL_L2[p.irrep_dtype], n


F64 = ["oeq_uvw_f64_forward", "oeq_uvw_f64_backward", "oeq_uvw_f64_backward_dw"]


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("batch", [1, 7, 8, 9, 33, 1301])
def test_doubles(batch, wide):
    orders_0_to_2(with_dtype(shared_problem(wide), np.float64), batch, F64)


def test_degree_three_and_blocks_without_a_path():
    p = TPProblem("32x3o+32x0e+64x1o", "1x3o+1x1o", "32x3e+32x1o+64x0e+32x1e", [(0, 1, 0, "uvw", True), (0, 0, 2, "uvw", True),
                                                                                (2, 0, 0, "uvw", True)],
                  shared_weights=True, internal_weights=False)
    orders_0_to_2(with_dtype(p, np.float64), 45, F64)
