"""The one-pass symmetric contraction against einsum in fp64 at the edges of its tiles (32 nodes, 128 channels, chunks of 56
terms or 28 in doubles), with sparse tensors like the real generalised Clebsch-Gordan ones: forward, both gradients, second order."""
import pytest
import torch

from helpers import kernels_launched, rel_l2
from test_symmetric_contraction_gpu import _einsum_contraction

pytestmark = pytest.mark.gpu

# longest sum: ~1,000 products of four factors each, summed over <= 129 nodes in the weight gradient; rounding errors of fp32
# grow like sqrt(1000 * 129) * 6e-8 = 2e-5 in the worst case of one sign, ~1e-6 for random signs
TOL = {torch.float32: 1e-5, torch.float64: 1e-12}


def _setup(ell, F, N, corr, dtype, seed=0, keep=None):
    from openequivariance_b200._torch.symmetric_contraction import SymmetricContraction
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, device="cuda", dtype=torch.float64, generator=gen)  # noqa: E731
    Us = []
    for lead in ((), (3,)):
        # integers that float32 holds exactly, most of them zero
        Us.append({nu: (rnd(*lead, *([ell] * nu), 1 + nu) * 4).round() * (rnd(*lead, *([ell] * nu), 1).abs() < (keep or min(1.0, 40 / ell ** nu)))
                   for nu in range(1, corr + 1)})
    G = 5
    sc = SymmetricContraction(Us, F, G, dtype=dtype).to("cuda")
    elem = torch.randint(0, G - 1, (N,), device="cuda", generator=gen)       # the last element has no nodes
    x = rnd(N, F, ell).to(dtype).requires_grad_(True)
    return sc, Us, elem, torch.nn.functional.one_hot(elem, G).to(dtype), x, rnd(N, 4 * F).to(dtype), rnd


def _oracle(sc, Us, elem, x):
    xd = x.detach().double().requires_grad_(True)
    params, outs = [], []
    for c, U in zip(sc.contractions, Us):
        Ws = {c.correlation - i: w.detach().double().requires_grad_(True) for i, w in enumerate(c._weights())}
        params += list(Ws.values())
        outs.append(_einsum_contraction(U, Ws, xd, elem))
    return torch.cat(outs, dim=-1), xd, params


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("ell,F,N,corr", [(16, 3, 129, 3), (9, 129, 33, 3), (4, 1, 1, 3), (5, 8, 64, 2), (25, 2, 40, 2), (1, 7, 32, 3), (3, 5, 31, 1)])
def test_one_pass_contraction_at_tile_edges(ell, F, N, corr, dtype):
    sc, Us, elem, y, x, cot, rnd = _setup(ell, F, N, corr, dtype)
    weights = [w for c in sc.contractions for w in c._weights()]
    def forward_and_gradients():
        out = sc(x, y)
        return out, torch.autograd.grad(out, [x] + weights, cot)

    (out, got), ran = kernels_launched(forward_and_gradients)
    assert sc.__dict__["_plan"].fits                         # the one-pass operator ran
    assert {"oeq_sym_forward", "oeq_sym_backward_x", "oeq_sym_backward_c"} <= ran, ran
    want, xd, params = _oracle(sc, Us, elem, x)
    ref = torch.autograd.grad(want, [xd] + params, cot.double())
    assert rel_l2(out.detach().cpu().numpy(), want.detach().cpu().numpy()) <= TOL[dtype]
    for a, b in zip(got, ref):
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= TOL[dtype]
    again = torch.autograd.grad(sc(x, y), [x] + weights, cot)
    assert all(torch.equal(a, b) for a, b in zip(got, again))   # sums over nodes run in a fixed order


def test_one_pass_contraction_second_order_and_reloaded_tensors():
    sc, Us, elem, y, x, cot, rnd = _setup(4, 6, 37, 3, torch.float64, keep=0.4)
    with torch.no_grad():
        sc(x, y)
        for c, U in zip(sc.contractions, Us):                # other tensors in the same buffers, as load_state_dict leaves them
            for nu in U:
                U[nu] = U[nu].flip(0)
                getattr(c, f"U_matrix_{nu}").copy_(U[nu])
    weights = [w for c in sc.contractions for w in c._weights()]
    cot.requires_grad_(True)
    first = torch.autograd.grad(sc(x, y), [x] + weights, cot, create_graph=True)
    tangents = [rnd(*t.shape) for t in first]
    got = torch.autograd.grad(first, [x, cot] + weights, tangents)
    want, xd, params = _oracle(sc, Us, elem, x)
    cd = cot.detach().clone().requires_grad_(True)
    ref = torch.autograd.grad(torch.autograd.grad(want, [xd] + params, cd, create_graph=True), [xd, cd] + params, tangents,
                              allow_unused=True)
    for a, b in zip(got, ref):
        b = torch.zeros_like(a) if b is None else b
        assert rel_l2(a.cpu().numpy(), b.cpu().numpy()) <= 1e-12


@pytest.mark.parametrize("dtype,terms", [(torch.float32, 55), (torch.float32, 56), (torch.float32, 57), (torch.float32, 112),
                                         (torch.float64, 27), (torch.float64, 28), (torch.float64, 29), (torch.float64, 56)])
def test_one_pass_contraction_at_the_chunks_of_its_terms(dtype, terms):
    # 1 + 3 components of 25 features to the first order, and pairs of the scalar one beyond them: `terms` of them non-zero
    from openequivariance_b200._torch.symmetric_contraction import SymmetricContraction
    gen = torch.Generator(device="cuda").manual_seed(terms)
    rnd = lambda *s: torch.randn(*s, device="cuda", dtype=torch.float64, generator=gen)  # noqa: E731
    one, two, three = torch.zeros(25, 2), torch.zeros(25, 25, 1), torch.zeros(3, 25, 2)
    places = [(one, (i,)) for i in range(25)] + [(three, (w, i)) for w in range(3) for i in range(25)] + [(two, (i, 24)) for i in range(12)]
    for U, at in places[:terms]:
        U[at] = 1 + len(at)
    Us = [{1: one.double().cuda(), 2: two.double().cuda()}, {1: three.double().cuda()}]
    sc = SymmetricContraction(Us, 5, 3, dtype=dtype).to("cuda")
    elem = torch.randint(0, 3, (70,), device="cuda", generator=gen)
    x, cot = rnd(70, 5, 25).to(dtype).requires_grad_(True), rnd(70, 20).to(dtype)
    weights = [w for c in sc.contractions for w in c._weights()]
    out = sc(x, torch.nn.functional.one_hot(elem, 3).to(dtype))
    plan = sc.__dict__["_plan"]
    assert plan.fits and plan.terms.shape[0] == terms
    want, xd, params = _oracle(sc, Us, elem, x)
    ref = torch.autograd.grad(want, [xd] + params, cot.double())
    for a, b in zip([out, *torch.autograd.grad(out, [x] + weights, cot)], [want, *ref]):
        assert rel_l2(a.detach().cpu().numpy(), b.detach().cpu().numpy()) <= TOL[dtype]
