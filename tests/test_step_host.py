"""Host-side rules of the whole-step sequence: which models it covers, before any kernel is launched."""
import gc
import weakref

import pytest
import torch

from cuda_mace_b200 import model, ops, step, systems


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


@pytest.mark.parametrize("radial", ["exact", "spline"])
def test_what_a_plan_is_made_from(U, radial):
    """Every change that node_energies() would see makes the stamp of a plan out of date."""
    changes = [
        lambda m: setattr(m, "scale", 2.0), lambda m: setattr(m, "shift", 0.5), lambda m: setattr(m.edge_basis, "p", 6),
        lambda m: setattr(m.edge_basis, "r_max", 4.0), lambda m: m.layers[1].W_up.mul_(2.0),
        lambda m: setattr(m.layers[0], "W_prod", m.layers[0].W_prod.clone()),
        lambda m: setattr(m.layers[1], "linear", torch.nn.Identity()),
        lambda m: m.layers.append(torch.nn.Module()), lambda m: m.layers[0].linear.register_forward_hook(print)]
    if radial == "spline":
        changes += [lambda m: setattr(m.layers[0].spline, "rmax", 4.0), lambda m: m.layers[1].spline.coefficients.mul_(2.0)]
    for change in changes:
        mace = _model(U, radial=radial)
        stamp = step._Stamp(mace)
        assert stamp.current(mace) and not stamp.hooked
        change(mace)
        assert not stamp.current(mace)
    mace = _model(U)     # a weight that became a parameter is followed like a buffer
    W = mace.layers[1].W_readout2
    del mace.layers[1].W_readout2
    mace.layers[1].W_readout2 = torch.nn.Parameter(W)
    stamp = step._Stamp(mace)
    with torch.no_grad():
        W.mul_(2.0)
    assert not stamp.current(mace)


def test_a_stamp_does_not_keep_its_model(U):
    mace = _model(U)
    mace.__dict__["_step_plan"] = (step._Stamp(mace), None)
    gone = weakref.ref(mace)
    gc.collect()
    gc.disable()
    try:
        del mace
        assert gone() is None
    finally:
        gc.enable()


def test_a_model_with_parts_of_its_own_is_not_covered(U):
    class Shifted(model.InvariantMACE):
        def node_energies(self, *args, **more):
            return super().node_energies(*args, **more) + 1.0

    assert not step.covers(Shifted(systems.init_params(32, 3, 1), U, dtype=torch.float64, device="cpu"))
    mace = _model(U)

    class Doubled(ops.Linear):
        def forward(self, x):
            return 2.0 * super().forward(x)

    mace.layers[1].linear = Doubled(mace.layers[1].linear.weights)
    assert not step.covers(mace)


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_no_fp16_range_for_weights_that_are_not_finite(value):
    Ws = [torch.full((8, 64), 0.1), torch.full((64, 64), 0.1), torch.full((64, 64), 0.1)]
    bounds = step.basis_bounds(8, 5.0, 5)
    assert step.half_scales(Ws, bounds) is not None
    for W in Ws:
        old = float(W[3, 5])
        W[3, 5] = value
        assert step.half_scales(Ws, bounds) is None
        W[3, 5] = old
