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
