"""Host side of the symmetric contraction's modules."""
import copy
import io
import pickle

import torch


def _module():
    from openequivariance_b200._torch.symmetric_contraction import SymmetricContraction
    gen = torch.Generator().manual_seed(0)
    return SymmetricContraction([{nu: torch.randn(*[4] * nu, 2, generator=gen) for nu in (1, 2, 3)}], 3, 5)


def test_plans_stay_out_of_copies_and_files():
    sc = _module()
    for m in (sc, sc.contractions[0]):
        m.__dict__["_plan"] = m.__dict__["_captured"] = "kept"
    buffer = io.BytesIO()
    torch.save(sc, buffer)
    buffer.seek(0)
    for other in (copy.deepcopy(sc), pickle.loads(pickle.dumps(sc)), torch.load(buffer, weights_only=False)):
        for m in (other, other.contractions[0]):
            assert "_plan" not in m.__dict__ and "_captured" not in m.__dict__
        assert all(torch.equal(a, b) for a, b in zip(other.state_dict().values(), sc.state_dict().values()))
    assert sc.__dict__["_plan"] == "kept"
    # files written when the plan was part of the state
    fresh = type(sc.contractions[0]).__new__(type(sc.contractions[0]))
    fresh.__setstate__(dict(sc.contractions[0].__dict__))
    assert "_plan" not in fresh.__dict__ and fresh.num_elements == 5


class _Double(torch.nn.Module):
    def forward(self, w):
        return 2 * w


def test_weights_are_read_as_attributes():
    c = _module().contractions[0]
    plain = c._weights()
    assert plain[0] is c.weights_max and plain[1:] == list(c.weights)
    torch.nn.utils.parametrize.register_parametrization(c, "weights_max", _Double())
    assert torch.equal(c._weights()[0], 2 * plain[0])
    c = _module().contractions[0]
    plain = c._weights()
    torch.nn.utils.parametrize.register_parametrization(c.weights, "0", _Double())
    assert torch.equal(c._weights()[1], 2 * plain[1])
    c = _module().contractions[0]
    plain = c.weights_max.detach().clone()
    c = torch.nn.utils.weight_norm(c, "weights_max")
    assert torch.allclose(c._weights()[0], plain)
    c = _module().contractions[0]
    replica = c._replicate_for_data_parallel()      # as DataParallel leaves it: the weights are attributes
    replica.weights_max = 3 * c.weights_max
    assert torch.equal(replica._weights()[0], 3 * c.weights_max)


def test_what_a_call_of_a_contraction_runs_besides_its_forward():
    sc = _module()
    c = sc.contractions[0]
    assert c._plainly_called()
    handle = c.register_forward_hook(lambda *_: None)
    assert not c._plainly_called()
    handle.remove()
    assert c._plainly_called()
    c.forward = lambda *_: None
    assert not c._plainly_called()
    del c.forward
    assert not torch.nn.utils.weight_norm(c, "weights_max")._plainly_called()
