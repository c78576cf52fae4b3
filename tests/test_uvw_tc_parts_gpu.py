"""Tensor-core 'uvw' kernels where a tile's schedule is dealt to several CTAs: batches around one tile (64 / 128 items), few
tiles (every cut of the schedule), one tile more than there are SMs (a ragged last wave), against the fp64 oracle."""
import pytest

from test_uvw_f64_gpu import orders_0_to_2, shared_problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("batch", [1, 64, 65, 129, 1000, 2500, 128 * 148 + 1])
def test_cut_schedules(batch, wide):
    # (one tile more than there are SMs is cut where the cut's price is less than the wave that it saves)
    cut = [f"oeq_uvw_tc_{k}_parts" for k in ("forward", "backward_dx", "backward_dy")] if batch <= 2500 else []
    orders_0_to_2(shared_problem(wide), batch, cut + ["oeq_uvw_tc_backward_dw"])
