"""The work that users have this package do, as cases that can be timed: energy and forces of a model in the ways a
program asks for them, and the operators that a model of another code base calls one by one.

Kinds of cases (`kind`) and what one pass is:

* ``step``: energy and forces of a periodic box (0.1 atoms/A^3, 0.9 A smallest distance, r_max 5 A: about 52 edges an
  atom) by a random-init two-layer invariant MACE, asked for in one of these ways (`how`):
    - ``model``: ``InvariantMACE(...)(data)`` with the data dictionary of the reference's model (one-hot attributes,
      atoms in the caller's order);
    - ``evaluator``: ``EnergyForceEvaluator`` on positions that are on the device, neighbour list kept;
    - ``captured``: the same, recorded as a CUDA graph once for the list;
    - ``new_list``: the neighbour list of the positions is built on the device, then the step;
    - ``host``: ``evaluate_host``: every input in pinned host memory, energy and forces back on the host.
* ``contraction``, ``messages``, ``linear``: one TorchScript class under cuda-mace's name, forward and backward, as
  cuda-mace's own Python layer calls it.
"""
import functools
import math

import numpy as np
import torch

from cuda_mace_b200 import cg, evaluator, model, ops, systems, torch_classes
from cuda_mace_b200.domain import SlabDomain

R_MAX = 5.0
DENSITY = 0.1
EDGES_PER_ATOM = 52          # 4/3 pi r_max^3 * density, less the excluded volume
DTYPES = {"f32": torch.float32, "f64": torch.float64}


def listed():
    def step(name, atoms, channels, elements, dtype, how, radial="exact"):
        return dict(name=name, kind="step", atoms=atoms, channels=channels, elements=elements, dtype=dtype, how=how,
                    radial=radial)

    return [
        # a small molecule-sized cell inside a larger program (relaxation, training-set labelling): launches count
        step("step 192 f32", 192, 64, 4, "f32", "model"),
        # the same cell in the precision that energies are validated in
        step("step 192 f64", 192, 64, 4, "f64", "model"),
        # molecular dynamics of a box of water, list kept for some steps
        step("step 3000 f32", 3000, 128, 2, "f32", "evaluator"),
        # ... with the step recorded as a graph
        step("step 3000 f32 captured", 3000, 128, 2, "f32", "captured"),
        # ... when every step needs a new list
        step("step 3000 f32 new list", 3000, 128, 2, "f32", "new_list"),
        # the same box with the reference's tabulated radial weights
        step("step 3000 f32 spline", 3000, 128, 2, "f32", "model", "spline"),
        # a large cell in float64: phonons, elastic constants
        step("step 8000 f64", 8000, 128, 4, "f64", "evaluator"),
        # a server that gets each structure from a client: host buffers in and out, a ragged size
        step("step 15999 f32 host", 15999, 128, 4, "f32", "host"),
        # the most atoms of one card's share of a large simulation
        step("step 64000 f32", 64000, 128, 4, "f32", "evaluator"),
        # single operators under cuda-mace's layers
        dict(name="contraction 4096", kind="contraction", nodes=4096, channels=128, elements=10, dtype="f32"),
        dict(name="messages 8192", kind="messages", nodes=8192, degree=30, channels=128, dtype="f32"),
        dict(name="elemental linear 3000", kind="linear", nodes=3000, channels=128, elements=4, dtype="f32"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    channels = rng.choice([32, 64, 64, 96, 128, 128, 128])
    dtype = rng.choice(["f32", "f32", "f64"])
    kind = rng.choice(["step"] * 8 + ["contraction", "messages", "messages", "linear"])
    if kind == "step":
        how = rng.choice(["model", "model", "evaluator", "evaluator", "captured", "new_list", "host"])
        radial = rng.choice(["exact", "exact", "exact", "exact", "spline"])
        most = 8000 if dtype == "f64" or how == "captured" else 16000 if how in ("host", "new_list") else 60000
        if radial == "spline":
            most = min(most, 16000)
        return dict(kind=kind, atoms=size(32, most), channels=channels, elements=rng.randint(1, 10), dtype=dtype,
                    how=how, radial=radial)
    if kind == "messages":
        return dict(kind=kind, nodes=size(64, 16384), degree=rng.randint(8, 60), channels=channels, dtype=dtype)
    if kind == "contraction":
        return dict(kind=kind, nodes=size(64, 64000), channels=channels, elements=rng.randint(1, 10), dtype=dtype)
    # cuda-mace's Linear and ElementalLinear exist in float32; elements = 0 is Linear
    return dict(kind=kind, nodes=size(64, 64000), channels=channels, elements=rng.choice([0, 2, 3, 4, 7, 10]),
                dtype="f32")


# ---------------------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=1)
def coupling():
    """The generalised Clebsch-Gordan tensors: constants of l_max = 3 and correlation 3."""
    return cg.u_matrices()


@functools.lru_cache(maxsize=1)
def model_of(channels, elements, dtype, radial):
    """A program holds one model and evaluates many structures with it, so the states of a case share the model."""
    params = systems.init_params(channels, elements, 1, r_max=R_MAX)
    if radial == "spline":
        model.add_spline_knots(params)
    return model.InvariantMACE(params, coupling(), dtype=DTYPES[dtype], device="cuda", radial=radial)


def box_of(atoms):
    """Cubic up to 20 000 atoms, then the 80 A x 80 A column of the slabs that a decomposed system is cut into."""
    if atoms <= 20000:
        return np.full(3, (atoms / DENSITY) ** (1.0 / 3.0))
    return np.array([80.0, 80.0, atoms / DENSITY / 6400.0])


def prepare_step(case, seed):
    n, Z, dtype = case["atoms"], case["elements"], DTYPES[case["dtype"]]
    box = box_of(n)
    pos = systems.random_box(n, box, 0.9, seed)
    rng = np.random.default_rng(seed + 1)
    share = np.array([0.5, 0.3] + [0.2 / 8] * 8) if Z == 10 else np.array([1.0 / (k + 1) for k in range(Z)])
    species = rng.choice(Z, size=n, p=share / share.sum())
    mace = model_of(case["channels"], Z, case["dtype"], case["radial"])
    pbc = (True, True, True)
    if case["how"] == "model":
        positions = torch.from_numpy(pos).cuda()
        edge_index, shifts, _ = ops.neighbor_list(positions, box, pbc, R_MAX)
        data = dict(positions=positions, node_attrs=systems.one_hot(species, Z, dtype).cuda(), edge_index=edge_index,
                    shifts=shifts)
        return dict(mace=mace, data=data)
    # atoms stored grouped by species, as partition_slabs() stores them
    order = np.argsort(species, kind="stable")
    pos, species = pos[order], species[order]
    none = np.zeros(0, dtype=np.int64)
    dom = SlabDomain(0, 1, n, n, order, pos, species, np.zeros_like(pos), np.zeros((2, 0), dtype=np.int64),
                     np.zeros((0, 3)), none, none, (n, 0), (n, 0), 0, 0, box, pbc)
    ev = evaluator.EnergyForceEvaluator(mace, dom, "cuda")
    positions = torch.from_numpy(pos).cuda()
    if case["how"] == "host":
        edge_index, _, shift_index = ops.neighbor_list(positions, box, pbc, R_MAX)
        code = shift_index.long() + 1
        table = np.stack(np.meshgrid(*[np.arange(-1, 2)] * 3, indexing="ij"), axis=-1).reshape(27, 3) * box
        batch = dict(positions=torch.from_numpy(pos), species=torch.from_numpy(species.astype(np.int32)),
                     edge_index=edge_index.cpu(), shift_table=torch.from_numpy(table),
                     shift_index=(code[:, 0] * 9 + code[:, 1] * 3 + code[:, 2]).to(torch.uint8).cpu())
        return dict(ev=ev, batch={k: v.pin_memory() for k, v in batch.items()},
                    forces=torch.empty(n, 3, dtype=torch.float64, pin_memory=True))
    ev.rebuild_neighbor_list(positions)
    if case["how"] == "captured":
        ev.capture(positions)
    return dict(ev=ev, positions=positions)


def prepare_contraction(case, seed):
    torch_classes.load()
    g = torch.Generator("cuda").manual_seed(seed)
    n, C, Z, dtype = case["nodes"], case["channels"], case["elements"], DTYPES[case["dtype"]]
    W = [torch.randn(Z, p, C, generator=g, device="cuda", dtype=dtype) / math.sqrt(p) for p in (23, 4, 1)]
    tables = ops.SymmetricContraction(*coupling(), *W).to("cuda")
    X = torch.randn(n, 16, C, generator=g, device="cuda", dtype=dtype).requires_grad_(True)
    types = torch.randint(0, Z, (n,), generator=g, device="cuda", dtype=torch.int32)
    G = torch.randn(n, 1, C, generator=g, device="cuda", dtype=dtype)
    return dict(op=torch.classes.symm_contract.SymmetricContraction(), t=tables, X=X, types=types, G=G)


def prepare_messages(case, seed):
    torch_classes.load()
    g = torch.Generator("cuda").manual_seed(seed)
    n, C, dtype = case["nodes"], case["channels"], DTYPES[case["dtype"]]
    rand = dict(generator=g, device="cuda", dtype=dtype)
    E = n * case["degree"]   # edges fall on the receivers as they come: degrees close to a Poisson distribution
    receiver = torch.randint(0, n, (E,), generator=g, device="cuda", dtype=torch.int32).sort()[0]
    sender = torch.randint(0, n, (E,), generator=g, device="cuda", dtype=torch.int32)
    X = torch.randn(n, C, **rand).requires_grad_(True)
    Y = torch.classes.spherical_harmonics.SphericalHarmonics().forward(torch.randn(E, 3, **rand)).requires_grad_(True)
    R = torch.randn(E, 4, C, **rand).requires_grad_(True)
    G = torch.randn(n, 16, C, **rand)
    return dict(op=torch.classes.inv_message_passing.InvariantMessagePassingTP(), X=X, Y=Y, R=R, sender=sender,
                receiver=receiver, n=n, G=G)


def prepare_linear(case, seed):
    torch_classes.load()
    g = torch.Generator("cuda").manual_seed(seed)
    n, C, Z, dtype = case["nodes"], case["channels"], case["elements"], DTYPES[case["dtype"]]
    rand = dict(generator=g, device="cuda", dtype=dtype)
    X = torch.randn(n, 16, C, **rand).requires_grad_(True)
    G = torch.randn(n, 16, C, **rand)
    if Z == 0:
        W = torch.randn(4, C, C, **rand)
        return dict(op=torch.classes.linear_wmma.Linear(), X=X, G=G, more=(W, W.transpose(-1, -2).contiguous()))
    W = torch.randn(Z, 4, C, C, **rand)
    one_hot = torch.nn.functional.one_hot(torch.randint(0, Z, (n,), generator=g, device="cuda"), Z).to(dtype)
    return dict(op=torch.classes.linear_wmma.ElementalLinear(), X=X, G=G,
                more=(W, W.transpose(-1, -2).contiguous(), one_hot))


def prepare(case, seed):
    return dict(globals()["prepare_" + case["kind"]](case, seed), kind=case["kind"], how=case.get("how"))


def run(state):
    kind, how = state["kind"], state["how"]
    if kind == "step":
        if how == "model":
            return state["mace"](state["data"])
        ev = state["ev"]
        if how == "host":
            return ev.evaluate_host(state["batch"], state["forces"])
        if how == "new_list":
            ev.rebuild_neighbor_list(state["positions"])
        return ev(state["positions"])
    if kind == "contraction":
        t = state["t"]
        out = state["op"].forward(
            state["X"], state["types"], t.u3_max_nonsparse, t.U3_num_nonsparse, t.U3_indices, t.U3_values,
            t.U2_num_nonsparse, t.U2_indices, t.U2_values, t.U1_num_values, t.U1_index, t.weights_3, t.weights_2,
            t.weights_1, t.W3_L0_size, t.W2_L0_size, t.W1_L0_size)
        return (out.detach(),) + torch.autograd.grad(out, state["X"], state["G"])
    if kind == "messages":
        out = state["op"].forward(state["X"], state["Y"], state["R"], state["sender"], state["receiver"], state["n"])
        return (out.detach(),) + torch.autograd.grad(out, (state["X"], state["Y"], state["R"]), state["G"])
    out = state["op"].forward(state["X"], *state["more"])
    return (out.detach(),) + torch.autograd.grad(out, state["X"], state["G"])


def work(case):
    """Bytes of the inputs and outputs, and the operations of the least that has to be formed.  In the first layer of a
    model the features of a sender depend on its element alone, so sums over a receiver's edges of one element are
    enough there and the [E, 4C] radial weights are needed in the second layer only."""
    s = 8 if case["dtype"] == "f64" else 4
    C = case["channels"]
    if case["kind"] == "step":
        n, Z = case["atoms"], case["elements"]
        E = EDGES_PER_ATOM * n
        edge_bytes = 0 if case["how"] == "new_list" else 9 + 24 * (case["how"] != "host")
        hidden = 2 * (8 * 64 + 2 * 64 * 64) if case["radial"] == "exact" else 0
        last = 2 * 64 * 4 * C if case["radial"] == "exact" else 8 * 4 * C
        per_edge = 2 * 2 * hidden + 2 * last + 3 * 2 * 16 * 64 + 4 * 2 * 16 * C
        per_node = 3 * 2 * 16 * C * C + 2 * 2 * 16 * 64 * C * min(Z, 4) + 2 * 3 * 430 * C + 4 * 2 * C * C
        return {"bytes": n * (24 + 4 + 24) + E * edge_bytes, "flops": E * per_edge + n * per_node}
    n = case["nodes"]
    if case["kind"] == "contraction":
        return {"bytes": s * n * C * (16 + 1 + 1 + 16) + 4 * n, "flops": n * C * 3 * 430}
    if case["kind"] == "messages":
        E = n * case["degree"]
        return {"bytes": s * (2 * 4 * E * C + 2 * 16 * E + 2 * n * C + 2 * 16 * n * C) + 8 * E,
                "flops": E * C * (40 + 100)}
    Z = max(1, case["elements"])
    return {"bytes": s * (4 * 16 * n * C + 4 * Z * C * C), "flops": 2 * 2 * 16 * n * C * C}


def tolerance(case):
    if case["dtype"] == "f64":
        return {"rel": 1e-11}
    # float32 sums; a step chains about fifteen of them, forward and back
    return {"rel": 2e-5} if case["kind"] == "step" else {"rel": 1e-5}
