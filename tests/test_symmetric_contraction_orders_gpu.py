"""Gradients of the symmetric contraction that are differentiated again, up to third order, against einsum in fp64."""
import pytest
import torch

from helpers import rel_l2
from test_symmetric_contraction_fused_gpu import _oracle, _setup
from test_symmetric_contraction_gpu import _einsum_contraction

pytestmark = pytest.mark.gpu

# sums of at most ~1,000 products of a handful of factors, four times over: sqrt(1000) * 1e-16 * a few
TOL = 1e-12


def _close(got, want):
    for a, b in zip(got, want):
        b = torch.zeros_like(a) if b is None else b
        assert rel_l2(a.detach().cpu().numpy(), b.detach().cpu().numpy()) <= TOL


def _three_orders(out, operands, cot, tangents, later):
    """The first gradient of <out, cot>, the second of its norm (tangents None) or of its product with constants, the third of the
    second's product with ``later``."""
    first = torch.autograd.grad(out, operands, cot, create_graph=True)
    scalar = sum((f * f).sum() for f in first) if tangents is None else sum((f * t).sum() for f, t in zip(first, tangents))
    second = torch.autograd.grad(scalar, operands + [cot], create_graph=True)
    third = torch.autograd.grad(sum((s * t).sum() for s, t in zip(second, later)), operands + [cot], allow_unused=True)
    return list(first) + list(second) + list(third)


@pytest.mark.parametrize("constant", [True, False])
def test_third_order(constant):
    sc, Us, elem, y, x, cot, rnd = _setup(4, 6, 37, 3, torch.float64, keep=0.4)
    weights = [w for c in sc.contractions for w in c._weights()]
    cot.requires_grad_(True)
    tangents = [rnd(*t.shape) for t in [x] + weights] if constant else None
    later = [rnd(*t.shape) for t in [x] + weights + [cot]]
    got = _three_orders(sc(x, y), [x] + weights, cot, tangents, later)
    want, xd, params = _oracle(sc, Us, elem, x)
    cd = cot.detach().clone().requires_grad_(True)
    _close(got, _three_orders(want, [xd] + params, cd, tangents, later))


def test_weights_made_from_the_features():
    # a gradient ends at the operand that it is for: the weights' reaches the features through the weights, and not a second time
    from openequivariance_b200._torch.symmetric_contraction import Contraction
    sc, Us, elem, _, x, _, rnd = _setup(4, 6, 37, 3, torch.float64, keep=0.4)
    elem = elem.sort().values
    cot, base = rnd(37, 6), {nu: rnd(5, U.shape[-1], 6) for nu, U in Us[0].items()}
    made = {nu: w * x.mean() for nu, w in base.items()}
    c = Contraction(Us[0], 6, 5, internal_weights=False, weights=[made[2], made[1], made[3]], dtype=torch.float64).to("cuda")
    operands = [x, made[3], made[2], made[1]]
    tangents = [rnd(*t.shape) for t in operands]
    found = []
    for out in (c(x, torch.bincount(elem, minlength=5).cpu(), elem), _einsum_contraction(Us[0], made, x, elem)):
        first = torch.autograd.grad(out, operands, cot, create_graph=True)
        second = torch.autograd.grad(first, operands, tangents, retain_graph=True)
        found.append([*torch.autograd.grad(out, operands, cot, retain_graph=True), *first, *second])
    _close(*found)
