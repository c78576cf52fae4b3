"""Gradients of the symmetric contraction that are differentiated again, up to third order, and calls that a transform maps
over or records, against einsum in fp64."""
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


def test_mapped_over_features_and_over_cotangents():
    sc, Us, elem, y, x, cot, rnd = _setup(4, 6, 37, 3, torch.float64, keep=0.4)
    weights = [w for c in sc.contractions for w in c._weights()]
    want, xd, params = _oracle(sc, Us, elem, x)
    cots = rnd(3, *cot.shape)
    got = torch.autograd.grad(sc(x, y), [x] + weights, cots, is_grads_batched=True)
    _close(got, torch.autograd.grad(want, [xd] + params, cots, is_grads_batched=True, retain_graph=True))
    xs = torch.stack([x.detach(), 2 * x.detach()])
    for p in sc.parameters():
        p.requires_grad_(False)
    _close(torch.func.vmap(lambda t: sc(t, y))(xs), [_oracle(sc, Us, elem, t)[0] for t in xs])


def test_recorded_calls_follow_the_module():
    from torch.fx.experimental.proxy_tensor import make_fx
    sc, Us, elem, y, x, _, _ = _setup(4, 6, 37, 3, torch.float64, keep=0.4)
    x = x.detach()
    for p in sc.parameters():
        p.requires_grad_(False)
    sc(x, y)
    recorded = [torch.jit.trace(sc, (x, y)), make_fx(sc)(x, y)]
    sc.contractions[0].U_matrix_2.mul_(2)
    Us[0][2] = sc.contractions[0].U_matrix_2.clone()
    for f in recorded:
        _close([f(x, y)], [_oracle(sc, Us, elem, x)[0]])


def test_tensors_that_want_a_gradient():
    sc, Us, elem, y, x, cot, _ = _setup(4, 6, 37, 3, torch.float64, keep=0.4)
    U = sc.contractions[0].U_matrix_2.requires_grad_(True)
    (got,) = torch.autograd.grad(sc(x, y), U, cot)
    Us[0][2].requires_grad_(True)
    (want,) = torch.autograd.grad(_oracle(sc, Us, elem, x)[0], Us[0][2], cot)
    _close([got], [want])


def test_compiled_calls():
    sc, Us, elem, y, x, cot, _ = _setup(4, 6, 37, 3, torch.float64, keep=0.4)
    out = torch.compile(sc, backend="aot_eager", fullgraph=True)(x, y)
    want, xd, _ = _oracle(sc, Us, elem, x)
    _close([out, *torch.autograd.grad(out, [x], cot)], [want, *torch.autograd.grad(want, [xd], cot)])
