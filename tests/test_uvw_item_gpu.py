"""Per-item-weight 'uvw' product (one block per item, or the general kernels where that does not pay) against the fp64 oracle at the edges of its tiles: multiplicities around
the 32-wide weight tiles and the widths of an access, blocks without a path, one item and many."""
import numpy as np
import pytest

from helpers import REL_L2, kernels_launched, rel_l2, uniform_inputs, with_dtype
from openequivariance_b200.core.problem import TPProblem
from oracle import tp_oracle

pytestmark = pytest.mark.gpu


def _problem(m1, m3, l1=1, l3=1):
    # two paths into the second output block (one of them from another input block), an output block and an input block without
    # a path, and weight offsets that follow the odd sizes of the first path
    return TPProblem(f"{m1}x{l1}e+{m3}x{l1}e+3x2e", "1x1e+1x0e", f"{m3}x{l3}e+{m1}x{l1}e+2x0o",
                     [(0, 0, 0, "uvw", True), (0, 1, 1, "uvw", True), (1, 1, 1, "uvw", True)],
                     shared_weights=False, internal_weights=False)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("m1,m3,l1,l3,batch", [(1, 1, 1, 1, 1), (3, 7, 1, 1, 5), (10, 48, 1, 0, 33), (33, 31, 1, 2, 7), (65, 34, 2, 2, 3),
                                               (32, 64, 2, 3, 19), (24, 40, 1, 1, 300), (96, 5, 1, 1, 4)])
def test_item_product_orders_0_to_2(m1, m3, l1, l3, batch, dt):
    import openequivariance_b200 as oeq
    p = with_dtype(_problem(m1, m3, l1, l3), dt)
    tp = oeq.TensorProduct(p)
    x, y, w, g, x2, y2, w2 = uniform_inputs(p, batch)
    we, we2 = tp.reorder_weights_to_e3nn(w), tp.reorder_weights_to_e3nn(w2)
    z = np.zeros((batch, p.irreps_out.dim), dtype=dt)
    _, ran = kernels_launched(lambda: tp.forward_cpu(x, y, z, we))
    assert "oeq_uvw_item_forward" in ran, ran
    # sums of at most 65 * 9 positive and negative products of numbers below one: the bounds of the other product tests hold
    assert rel_l2(z, tp_oracle.forward(p, x, y, we)) <= REL_L2[dt]
    dx, dy, dw = np.zeros_like(x), np.zeros_like(y), np.zeros_like(w)
    _, ran = kernels_launched(lambda: tp.backward_cpu(x, dx, y, dy, g, we, dw))
    assert "oeq_uvw_item_backward" in ran, ran
    for a, b in zip((dx, dy, dw), tp_oracle.backward(p, x, y, we, g)):
        assert rel_l2(a, b) <= REL_L2[dt]
    want = tp_oracle.double_backward(p, x, y, we, g, x2, y2, we2)
    want = (want[0], want[1], tp.reorder_weights_from_e3nn(want[2]), want[3])
    for a, b in zip(tp.double_backward_cpu(x, y, g, w, w2, x2, y2), want):
        assert rel_l2(a, b) <= REL_L2[dt]


# a batch of the general kernels' on either side of each line: forward above 600 items with few weight rows, backward above 4,800 with
# few weights and paths
@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("batch,forward,backward", [(600, "item", "item"), (601, "generic", "item"), (4800, "generic", "item"), (4801, "generic", "generic")])
def test_narrow_products_take_the_kernel_that_pays(batch, forward, backward, dt):
    import torch

    import openequivariance_b200 as oeq
    p = with_dtype(_problem(4, 5), dt)
    tp = oeq.TensorProduct(p)
    x, y, w, g, x2, y2, w2 = uniform_inputs(p, batch)
    we, we2 = tp.reorder_weights_to_e3nn(w), tp.reorder_weights_to_e3nn(w2)
    leaves = [torch.tensor(t, device="cuda", requires_grad=True) for t in (x, y, w, g)]

    def forward_and_gradients():
        z = tp(*leaves[:3])
        first = torch.autograd.grad(z, leaves[:3], leaves[3], create_graph=True)
        return z, first, torch.autograd.grad(first, leaves, [torch.tensor(t, device="cuda") for t in (x2, y2, w2)])

    (z, first, second), ran = kernels_launched(forward_and_gradients)
    name = {"item": "oeq_uvw_item_", "generic": "oeq_generic_"}
    assert ran & {n + k for n in name.values() for k in ("forward", "backward")} == {name[forward] + "forward", name[backward] + "backward"}, ran
    want = tp_oracle.double_backward(p, x, y, we, g, x2, y2, we2)
    want = [tp_oracle.forward(p, x, y, we), *tp_oracle.backward(p, x, y, we, g), want[0], want[1], tp.reorder_weights_from_e3nn(want[2]), want[3]]
    for n, (a, b) in enumerate(zip([z, *first, *second], want)):
        a = a.detach().cpu().numpy()
        a = tp.reorder_weights_to_e3nn(a) if n == 3 else a
        assert rel_l2(a, b) <= REL_L2[dt], n
