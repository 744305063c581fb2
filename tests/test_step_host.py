"""Host-side rules of the whole-step sequence: which models it covers, before any kernel is launched."""
import pytest
import torch

from cuda_mace_b200 import model, step, systems


def _model(U, dtype=torch.float64, radial="exact"):
    params = systems.init_params(32, 3, 1)
    if radial == "spline":
        model.add_spline_knots(params)
    return model.InvariantMACE(params, U, dtype=dtype, device="cpu", radial=radial)


@pytest.mark.parametrize("radial", ["exact", "spline"])
def test_a_model_that_is_not_what_it_was_built_as_is_not_covered(U, radial):
    for dtype, convert in ((torch.float64, lambda m: m.float()), (torch.float32, lambda m: m.double()),
                           (torch.float32, lambda m: m.float())):   # the last: its float64 readouts
        mace = _model(U, dtype, radial)
        assert step.covers(mace)
        assert not step.covers(convert(mace))
    mace = _model(U, radial=radial)
    con = mace.layers[1].contraction
    con.weights_2 = con.weights_2[:, :2].contiguous()
    assert not step.covers(mace)


def test_a_model_off_the_current_device_has_no_plan(U):
    assert step.plan_of(_model(U)) is None
