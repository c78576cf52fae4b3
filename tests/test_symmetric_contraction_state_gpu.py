"""What the symmetric contraction keeps between calls: it has to answer for the tensors, weights and devices that a module has
now, on whatever stream and thread it is called."""
import io
import os
import threading
import time
import weakref

import pytest
import torch

from helpers import kernels_launched, rel_l2
from test_symmetric_contraction_fused_gpu import TOL, _oracle, _setup

pytestmark = pytest.mark.gpu


def _right(sc, Us, elem, x, out):
    want, _, _ = _oracle(sc, Us, elem, x)
    return rel_l2(out.detach().cpu().numpy(), want.detach().cpu().numpy()) <= TOL[x.dtype]


def _data(c, nu, new):
    c._buffers[f"U_matrix_{nu}"].data.copy_(new)


def _in_place(c, nu, new):
    with torch.no_grad():
        c._buffers[f"U_matrix_{nu}"].copy_(new)


def _replaced(c, nu, new):
    setattr(c, f"U_matrix_{nu}", new.to(c._buffers[f"U_matrix_{nu}"].dtype))


def _transposed(c, nu, new):
    # the same numbers in another order of memory, and off a 16-byte boundary
    old = c._buffers[f"U_matrix_{nu}"]
    store = torch.empty(old.numel() + 1, device=old.device, dtype=old.dtype)[1:]
    setattr(c, f"U_matrix_{nu}", store.view(old.shape[::-1]).permute(*reversed(range(old.dim()))).copy_(new))


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("change", [_data, _in_place, _replaced, _transposed])
def test_changed_tensors_are_seen(change, dtype):
    sc, Us, elem, y, x, _, _ = _setup(5, 6, 37, 3, dtype, keep=0.4)
    assert _right(sc, Us, elem, x, sc(x, y))
    new = [{nu: U.flip(0) for nu, U in U_set.items()} for U_set in Us]
    new[1] = dict(Us[1])
    new[1][3] = Us[1][3].clone()
    new[1][3].view(-1)[-1] += 1.0                                   # one number, the last of the last tensor
    for c, U_set, old in zip(sc.contractions, new, Us):
        for nu in U_set:
            if not torch.equal(U_set[nu], old[nu]):
                change(c, nu, U_set[nu])
    assert _right(sc, new, elem, x, sc(x, y))
    assert _right(sc, new, elem, x, sc(x, y))


def test_changed_tensors_of_a_module_made_in_inference_mode():
    with torch.inference_mode():
        sc, Us, elem, y, x, _, _ = _setup(5, 6, 37, 3, torch.float64, keep=0.4)
        other = _setup(5, 6, 37, 3, torch.float64, seed=1, keep=0.4)
        assert _right(sc, Us, elem, x, sc(x, y))
        sc.load_state_dict(other[0].state_dict())
        assert _right(sc, other[1], elem, x, sc(x, y))


def test_captured_call_reports_changed_tensors():
    from openequivariance_b200 import native
    sc, Us, elem, y, x, _, _ = _setup(5, 6, 37, 3, torch.float32, keep=0.4)
    x = x.detach()
    for p in sc.parameters():
        p.requires_grad_(False)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        want = sc(x, y)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = sc(x, y)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want) and native.load().oeqb_check_status() == 0
    sc.contractions[0].U_matrix_2.data.mul_(2)
    graph.replay()
    torch.cuda.synchronize()
    assert native.load().oeqb_check_status() != 0
    assert native.load().oeqb_check_status() == 0                  # reported once
    Us[0][2] = Us[0][2] * 2
    plan = weakref.ref(sc.__dict__["_plan"])
    assert _right(sc, Us, elem, x, sc(x, y))
    assert sc.__dict__["_plan"] is not plan() and plan() is not None   # the graph still reads the plan that it was captured with


def test_tensors_changed_before_a_gradient_that_is_differentiated_again():
    sc, Us, elem, y, x, cot, _ = _setup(5, 6, 37, 3, torch.float64, keep=0.4)
    out = sc(x, y)
    with torch.no_grad():
        sc.contractions[0].U_matrix_2.mul_(2)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        torch.autograd.grad(out, x, cot, create_graph=True)


@pytest.mark.parametrize("bad", [5, -6, 1 << 40])
def test_a_node_of_no_element_is_refused(bad):
    from openequivariance_b200 import native
    sc, Us, elem, y, x, _, _ = _setup(5, 6, 70, 3, torch.float64, keep=0.4)
    c, keys = sc.contractions[1], elem.sort().values
    counts = torch.bincount(keys, minlength=5).cpu()
    want = c(x, counts, keys)
    keys[-1] = bad
    with pytest.raises(RuntimeError, match="out of range"):
        c(x, counts, keys)
    assert native.load().oeqb_check_status() == 0                  # the refused call left nothing behind
    keys[-1] = int(elem.max()) - 5                                  # counted from the end, as an index may be
    assert torch.equal(c(x, counts, keys), want)


def test_captured_nodes_of_no_element_have_zero_rows():
    from openequivariance_b200 import native
    sc, Us, elem, y, x, cot, _ = _setup(5, 6, 70, 3, torch.float64, keep=0.4)
    y = y.clone()
    c, keys = sc.contractions[1], elem.sort().values
    counts = torch.bincount(keys, minlength=5).cpu()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        want = torch.autograd.grad(c(x, counts, keys), x, cot[:, :18])[0]
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = c(x, counts, keys)
        dx = torch.autograd.grad(out, x, cot[:, :18])[0]
    keys[40:] = 9
    out.detach().fill_(7.0)
    dx.fill_(7.0)
    graph.replay()
    torch.cuda.synchronize()
    assert native.load().oeqb_check_status() != 0
    assert not out[40:].any() and not dx[40:].any() and bool(out[:40].any())
    assert torch.equal(dx[:40], want[:40])


def test_counts_are_checked_and_every_index_type_is_taken():
    sc, Us, elem, y, x, _, _ = _setup(5, 6, 70, 3, torch.float64, keep=0.4)
    c, keys = sc.contractions[1], elem.sort().values
    counts = torch.bincount(keys, minlength=5).cpu()
    want = c(x, counts, keys)
    assert torch.equal(c(x, counts.to(torch.int32), keys.int()), want)
    assert torch.equal(c(x, counts.cuda(), keys), want)
    assert rel_l2(c(x, counts, keys.cpu()).detach().cpu().numpy(), want.detach().cpu().numpy()) <= TOL[x.dtype]
    wrong = counts.clone()
    wrong[0] += 1
    for bad, message in ((wrong, "sums to 71"), (counts[:4], "Shape mismatch"), (counts + torch.tensor([0, 0, 0, 1, -1]), "negative")):
        with pytest.raises(RuntimeError, match=message):
            c(x, bad, keys)


def test_a_plan_is_finished_before_another_stream_finds_it():
    from openequivariance_b200._torch import symmetric_contraction as S
    sc, Us, elem, y, x, _, _ = _setup(6, 6, 70, 3, torch.float64, keep=0.4)
    S._MONOMIALS.clear()
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(one):
        torch.cuda._sleep(200_000_000)       # about 0.1 s: whatever the first call leaves to its stream is far from done
        S._monomials(6, x.device)
        assert one.query()                    # nothing of the entry is left to do
        torch.cuda._sleep(200_000_000)
        plan = S._Plan([c._tensors() for c in sc.contractions], 5, 6)
        assert one.query()
        first = sc(x, y)
    with torch.cuda.stream(two):
        second = sc(x, y)
    torch.cuda.synchronize()
    assert torch.equal(first, second) and _right(sc, Us, elem, x, second)
    assert plan.fits


def test_a_replaced_plan_outlives_its_last_use():
    # the allocator has to know every stream that a plan was used on: while `two` is busy, memory of the plan that `one` allocated
    # is not handed to the next request on `one`
    sc, Us, elem, y, x, _, _ = _setup(6, 6, 70, 3, torch.float64, keep=0.4)
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(one):
        sc(x, y)
    one.synchronize()
    plan = sc.__dict__["_plan"]
    held = {t.data_ptr() for t in [plan.place, plan.U_rows, *plan.U]}
    sizes = [(t.numel() * t.element_size()) for t in [plan.place, plan.U_rows, *plan.U]]
    with torch.cuda.stream(two):
        sc(x, y)
        torch.cuda._sleep(200_000_000)
    del plan
    sc.__dict__.pop("_plan")
    with torch.cuda.stream(one):
        again = [torch.empty(n, dtype=torch.uint8, device="cuda") for n in sizes for _ in range(4)]
    assert not held & {t.data_ptr() for t in again}
    torch.cuda.synchronize()


def test_a_module_that_was_run_saved_and_loaded():
    sc, Us, elem, y, x, _, _ = _setup(5, 6, 37, 3, torch.float64, keep=0.4)
    want = sc(x, y)
    sc.load_state_dict(sc.state_dict())
    buffer = io.BytesIO()
    torch.save(sc, buffer)
    for where in ("cuda", "cpu"):
        buffer.seek(0)
        other = torch.load(buffer, map_location=where, weights_only=False).to("cuda")
        assert torch.equal(other(x, y), want)
        assert torch.equal(other(x, y), want)


def test_the_host_part_of_a_plan_is_checked():
    sc, Us, elem, y, x, cot, _ = _setup(5, 6, 37, 3, torch.float64, keep=0.4)
    x = x.detach()
    sc(x, y)
    plan, U = sc.__dict__["_plan"], [U for c in sc.contractions for U in c._tensors()]
    weights = [w.detach() for c in sc.contractions for w in c._weights()]
    op, back = torch.ops.oeq_b200.symmetric_contraction, torch.ops.oeq_b200.symmetric_contraction_backward
    good = dict(terms=plan.terms, place=plan.place, U_rows=plan.U_rows, meta=plan.meta)
    out, group, coef, _ = op(x, elem, weights, U, plan.U, *good.values(), plan.out_dim, True)
    assert torch.equal(out, sc(x, y))
    for name, bad in (("terms", plan.terms.cuda()), ("meta", plan.meta.cuda()), ("meta", plan.meta.long()), ("meta", plan.meta[:8]),
                      ("meta", plan.meta[:12]), ("terms", plan.terms[:-1]), ("place", plan.place.long()), ("place", plan.place[:-1]),
                      ("place", plan.place.cpu()), ("U_rows", plan.U_rows[:-1]), ("U_rows", plan.U_rows.float())):
        args = list(dict(good, **{name: bad}).values())
        with pytest.raises(RuntimeError):
            op(x, elem, weights, U, plan.U, *args, plan.out_dim, True)
        with pytest.raises(RuntimeError):
            back(cot, x, elem, group, coef, weights, U, *args)
    for bad in ((group[:-1], coef), (group, coef[:-1])):
        with pytest.raises(RuntimeError):
            back(cot, x, elem, *bad, weights, U, *good.values())


def test_a_plan_is_for_one_device():
    sc, Us, elem, y, x, cot, _ = _setup(5, 6, 37, 3, torch.float64, keep=0.4)
    want = sc(x, y)
    plan = sc.__dict__["_plan"]
    assert plan.device == x.device
    plan.device = torch.device("cuda", 1)      # as if the module had been called there before
    assert torch.equal(sc(x, y), want) and sc.__dict__["_plan"] is not plan
    if torch.cuda.device_count() > 1:
        with pytest.raises(RuntimeError):
            sc(x.detach().to("cuda:1"), y.to("cuda:1"))
        assert torch.equal(sc(x, y), want)


class _Double(torch.nn.Module):
    def forward(self, w):
        return 2 * w


def test_reparametrised_weights_and_hooks():
    sc, Us, elem, y, x, cot, _ = _setup(5, 6, 37, 3, torch.float64, keep=0.4)
    plain = sc(x, y)
    first, second = sc.contractions
    called = []
    handle = second.register_forward_hook(lambda *_: called.append(1))
    assert rel_l2(sc(x, y).detach().cpu().numpy(), plain.detach().cpu().numpy()) <= TOL[x.dtype] and called == [1]
    handle.remove()
    everywhere = torch.nn.modules.module.register_module_forward_hook(lambda m, *_: called.append(type(m).__name__))
    sc(x, y)
    everywhere.remove()
    assert called == [1, "Contraction", "Contraction", "SymmetricContraction"]
    torch.nn.utils.weight_norm(first, "weights_max")          # a hook makes the weight from its two parts before each call
    with torch.no_grad():
        first.weights_max_g.mul_(2)
    torch.nn.utils.parametrize.register_parametrization(second, "weights_max", _Double())
    out = sc(x, y)
    grads = torch.autograd.grad(out, [x, first.weights_max_g, second.parametrizations.weights_max.original], cot)
    want, xd, params = _oracle(sc, Us, elem, x)                # (the weights as they now are)
    assert rel_l2(out.detach().cpu().numpy(), want.detach().cpu().numpy()) <= TOL[x.dtype]
    ref = torch.autograd.grad(want, [xd, params[3]], cot)
    assert rel_l2(grads[0].cpu().numpy(), ref[0].cpu().numpy()) <= TOL[x.dtype]
    assert rel_l2(grads[2].cpu().numpy(), 2 * ref[1].cpu().numpy()) <= TOL[x.dtype]
    assert bool(grads[1].any())


def test_other_operators_run_while_a_contraction_compiles(tmp_path):
    import openequivariance_b200 as oeq
    from openequivariance_b200 import native
    from openequivariance_b200.core import problems
    p = problems.readme_problem()
    tp = oeq.TensorProduct(p)
    rnd = lambda *s: torch.randn(*s, device="cuda")  # noqa: E731
    operands = [rnd(100, p.irreps_in1.dim), rnd(100, p.irreps_in2.dim), rnd(100, p.weight_numel)]
    tp(*operands)
    sc, Us, elem, y, x, _, _ = _setup(9, 6, 37, 3, torch.float64, seed=7, keep=0.1)     # (terms of no other test)
    gate, done, times = threading.Event(), threading.Event(), []

    def compile_it():
        gate.set()
        times.append(time.perf_counter())
        try:
            sc(x, y)
        finally:
            times.append(time.perf_counter())
            done.set()

    native.set_option("cache_dir", str(tmp_path))            # empty: the program has to be compiled
    thread = threading.Thread(target=compile_it)
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
    assert times[1] - times[0] > 0.2                         # it was compiled here
    assert calls > 10 and longest < 0.5 * (times[1] - times[0]), (calls, longest, times)
    assert _right(sc, Us, elem, x, sc(x, y))


def test_tensors_of_too_many_terms_are_composed_at_once():
    # 1,816 terms together, 454 of them the scalar irrep's: no kernels are compiled for a part of them
    sc, Us, elem, y, x, cot, _ = _setup(12, 3, 20, 3, torch.float64, keep=100.0)
    out, ran = kernels_launched(lambda: sc(x, y))
    assert not sc.__dict__["_plan"].fits and not any("oeq_sym" in k for k in ran), ran
    assert _right(sc, Us, elem, x, out)
