"""The whole-step sequence (cmace_step_run) against the float64 oracle at the sizes where its kernels can go wrong."""
import ctypes

import numpy as np
import pytest
import torch

from cuda_mace_b200 import _abi, domain, evaluator, model, ops, step, systems
from oracle import model as omodel

pytestmark = pytest.mark.gpu


def _cluster(n, seed, stretch):
    """n atoms without periodicity, every pair within the cutoff an edge; stretch > 1 leaves some atoms alone"""
    rng = np.random.default_rng(seed)
    pos = rng.random((n, 3)) * (n / 0.1) ** (1.0 / 3.0) * stretch
    d = np.linalg.norm(pos[:, None] - pos[None], axis=-1)
    recv, send = np.nonzero((d < 5.0) & (d > 0.0))
    return pos, np.stack([recv, send]), np.zeros((recv.size, 3))


# float64 1e-10 and float32 1e-5 / 1e-4 on energy / forces: the bounds the package states.  Sizes: 1 atom (no edges),
# fewer edges than a 128-edge tile, tile remainders; elements 1, odd (half a block), 10 and the largest 16; atoms
# without edges; every channel count.
@pytest.mark.parametrize("dtype,tol_e,tol_f", [(torch.float64, 1e-10, 1e-10), (torch.float32, 1e-5, 1e-4)])
@pytest.mark.parametrize("n,C,Z,stretch", [
    (1, 32, 2, 1.0), (5, 64, 1, 1.0), (23, 96, 3, 1.0), (40, 128, 10, 1.6), (61, 32, 16, 1.3), (70, 128, 2, 1.0),
    (33, 64, 7, 3.0)])
def test_step_against_the_oracle(U, dtype, tol_e, tol_f, n, C, Z, stretch):
    pos, ei, sh = _cluster(n, n, stretch)
    species = np.random.default_rng(n + 1).integers(0, Z, n)
    params = systems.init_params(C, Z, 7)
    one_hot = systems.one_hot(species, Z)
    _, e_ref, f_ref = omodel.energy_and_forces(params, U, torch.from_numpy(pos), one_hot, torch.from_numpy(ei),
                                               torch.from_numpy(sh))
    mace = model.InvariantMACE(params, U, dtype=dtype, device="cuda")
    assert step.plan_of(mace) is not None
    data = dict(positions=torch.from_numpy(pos).cuda(), node_attrs=one_hot.to(dtype).cuda(),
                edge_index=torch.from_numpy(ei).to(torch.int32).cuda(), shifts=torch.from_numpy(sh).cuda())
    out = mace(data)
    assert abs(float(out["interaction_energy"]) - float(e_ref)) < tol_e * max(abs(float(e_ref)), 1e-3)
    scale = max(float(f_ref.abs().max()), 1e-6)
    assert float((out["forces"].cpu() - f_ref).abs().max()) < tol_f * scale
    # the element index instead of the one-hot matrix, and a changed weight: the layout has to follow
    data["species"] = torch.from_numpy(species).cuda()
    assert torch.equal(mace(data)["forces"], out["forces"])
    with torch.no_grad():
        mace.layers[1].W_readout2.mul_(2.0)
    assert n == 1 or not torch.equal(mace(data)["forces"], out["forces"])


# against the model's own autograd path (same bounds), what the oracle does not have: 16 basis functions, tabulated radial
# weights (one element and several, the C = 128 and the narrower edge passes), and a list that crosses from eight warps a
# receiver to one (1 184 receivers and channel chunks); grouping by element in one block (up to 2 048 nodes) and in several;
# float64 products with a row-wise epilogue in tiles of 32 (70 atoms), 64 (400) and 128 rows
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-10), (torch.float32, 1e-4)])
@pytest.mark.parametrize("n,C,Z,nb,radial", [(70, 64, 3, 16, "exact"), (50, 128, 3, 8, "spline"), (33, 96, 1, 8, "spline"),
                                             (1300, 32, 2, 8, "spline"), (2048, 32, 3, 8, "exact"),
                                             (4100, 64, 5, 8, "exact"), (400, 32, 2, 8, "exact")])
def test_step_against_autograd(U, dtype, tol, n, C, Z, nb, radial):
    pos, ei, sh = _cluster(n, 3, 1.0)
    species = torch.from_numpy(np.random.default_rng(4).integers(0, Z, n)).to(torch.int32).cuda()
    params = systems.init_params(C, Z, 7, num_bessel=nb)
    if radial == "spline":
        model.add_spline_knots(params)
    mace = model.InvariantMACE(params, U, dtype=dtype, device="cuda", radial=radial)
    assert step.plan_of(mace) is not None
    p = torch.from_numpy(pos).cuda()
    edges, shifts = torch.from_numpy(ei).to(torch.int32).cuda(), torch.from_numpy(sh).cuda()
    out = mace(dict(positions=p, species=species, edge_index=edges, shifts=shifts))
    p.requires_grad_(True)
    (g,) = torch.autograd.grad(mace.node_energies(p, species, edges, shifts).sum(), p)
    assert float((out["forces"] + g).abs().max()) < tol * float(g.abs().max())


# tiles of 8 nodes up to 1 184 atoms, of 16 up to 2 368 in float64 and 4 736 in float32, of 32 beyond; one node past a tile and a
# tile but one; every element's part of the matrices in turn within a tile.  Against the model's own autograd path, same bounds
@pytest.mark.parametrize("dtype,tol,n", [(torch.float64, 1e-10, 1184), (torch.float64, 1e-10, 1185), (torch.float64, 1e-10, 2367),
                                         (torch.float64, 1e-10, 2369), (torch.float32, 1e-4, 1185), (torch.float32, 1e-4, 4735),
                                         (torch.float32, 1e-4, 4737)])
def test_nodes_between_the_layers_at_tile_edges(U, dtype, tol, n):
    C, Z = 64, 9
    receiver, sender = torch.arange(n).repeat_interleave(2), torch.stack([torch.arange(n).roll(1), torch.arange(n).roll(-1)], 1).reshape(-1)
    pos = torch.stack([1.3 * torch.arange(n), torch.arange(n) % 3, torch.arange(n) % 2], 1).double()   # a crooked closed chain
    shifts = torch.zeros(2 * n, 3, dtype=torch.float64)
    shifts[0, 0], shifts[-1, 0] = -1.3 * n, 1.3 * n
    species = torch.randint(0, Z, (n,), generator=torch.Generator().manual_seed(n), dtype=torch.int32).cuda()
    mace = model.InvariantMACE(systems.init_params(C, Z, 7), U, dtype=dtype, device="cuda")
    plan = step.plan_of(mace)
    assert plan is not None
    p, edges, shifts = pos.cuda(), torch.stack([receiver, sender]).to(torch.int32).cuda(), shifts.cuda()
    _, _, _, forces = step.energy_forces(plan, p, species, None, shifts, ops.EdgeTopology(edges[1], edges[0], n))
    p.requires_grad_(True)
    (g,) = torch.autograd.grad(mace.node_energies(p, species, edges, shifts).sum(), p)
    assert float((forces + g).abs().max()) < tol * float(g.abs().max())


def _list_of(receiver, n, seed, channels=128):
    """A model's weights and a list with these receivers; a shift an edge gives any distance up to the cutoff."""
    rng = np.random.default_rng(seed)
    edges = receiver.size
    sender = rng.integers(0, n, edges)
    pos, shifts = rng.normal(size=(n, 3)), rng.normal(size=(edges, 3))
    length = rng.uniform(0.9, 4.9, edges)[:, None]
    shifts = shifts / np.linalg.norm(shifts, axis=1, keepdims=True) * length - (pos[sender] - pos[receiver])
    return systems.init_params(channels, 3, 7), pos, np.stack([receiver, sender]), shifts, rng.integers(0, 3, n)


def _step_of(U, params, pos, ei, sh, species):
    mace = model.InvariantMACE(params, U, dtype=torch.float32, device="cuda")
    out = mace(dict(positions=torch.from_numpy(pos).cuda(), species=torch.from_numpy(species.astype(np.int32)).cuda(),
                    edge_index=torch.from_numpy(ei.astype(np.int32)).cuda(), shifts=torch.from_numpy(sh).cuda()))
    assert step.plan_of(mace).model.fused_w   # the kernels meant here
    return out


# the second layer's fused kernels at the edges of their tiles (32 and 128 edges) and of their pairs and groups of edges (2, 8,
# 16): lists of so many edges with so many a receiver, and receivers without any; 40 a receiver is more than a tile of the
# forward holds, 1 more receivers than the backward stages.  Energy and forces against the oracle, with the bounds of the
# whole step above; a list shorter than its degree is that of any larger one.
@pytest.mark.parametrize("edges,degree", [(1, 1)] + [(9, d) for d in (1, 2, 3, 17)] +
                         [(e, d) for e in (127, 128, 129, 300) for d in (1, 2, 3, 17, 40)])
def test_second_layer_at_tile_edges(U, edges, degree):
    n = -(-edges // degree) + 2
    receiver = np.minimum(np.arange(edges) // degree, n - 1)
    receiver[receiver > 0] += 1          # receiver 1 and the last one have no edges
    params, pos, ei, sh, species = _list_of(receiver, n, edges * 50 + degree)
    out = _step_of(U, params, pos, ei, sh, species)
    _, e_ref, f_ref = omodel.energy_and_forces(params, U, torch.from_numpy(pos), systems.one_hot(species, 3),
                                               torch.from_numpy(ei), torch.from_numpy(sh))
    assert abs(float(out["interaction_energy"]) - float(e_ref)) < 1e-5 * max(abs(float(e_ref)), 1e-3)
    assert float((out["forces"].cpu() - f_ref).abs().max()) < 1e-4 * max(float(f_ref.abs().max()), 1e-6)


# the same kernels for fewer channels, whose rows, tiles and steps are laid out differently: an odd number of steps a tile (96
# channels) and a single one (32), one and two words of last edges, lanes without a channel; 300 edges of 1 a receiver are more
# receivers than any of them stages.  Bounds as above
@pytest.mark.parametrize("channels", [32, 64, 96])
@pytest.mark.parametrize("edges,degree", [(1, 1), (9, 2), (63, 40), (65, 3), (128, 1), (129, 17), (300, 1), (300, 40)])
def test_narrow_second_layer_at_tile_edges(U, channels, edges, degree):
    n = -(-edges // degree) + 2
    receiver = np.minimum(np.arange(edges) // degree, n - 1)
    receiver[receiver > 0] += 1
    params, pos, ei, sh, species = _list_of(receiver, n, edges * 50 + degree, channels)
    out = _step_of(U, params, pos, ei, sh, species)
    _, e_ref, f_ref = omodel.energy_and_forces(params, U, torch.from_numpy(pos), systems.one_hot(species, 3),
                                               torch.from_numpy(ei), torch.from_numpy(sh))
    assert abs(float(out["interaction_energy"]) - float(e_ref)) < 1e-5 * max(abs(float(e_ref)), 1e-3)
    assert float((out["forces"].cpu() - f_ref).abs().max()) < 1e-4 * max(float(f_ref.abs().max()), 1e-6)


# Four and five tiles of the backward a block on 148 blocks, eight and nine of the forward a set: every buffer and barrier is
# used again, its phase wraps.  Receivers of so many edges in turn: few (warps whose receivers are not staged beside those
# whose are), and a long one before many short ones.  Against the operators in float64 (the oracle's contraction of so many
# nodes takes 60 GB), same bounds.
@pytest.mark.parametrize("channels,degrees", [(128, (3,)), (128, (10,)), (128, (70,) + (1,) * 40), (32, (3,)), (64, (70,) + (1,) * 40),
                                              (96, (10,))])
def test_second_layer_over_many_tiles(U, channels, degrees):
    edges = 80_001
    receiver = np.repeat(np.arange(edges), np.resize(degrees, edges))[:edges]
    n = int(receiver[-1]) + 1
    params, pos, ei, sh, species = _list_of(receiver, n, len(degrees), channels)
    out = _step_of(U, params, pos, ei, sh, species)
    mace = model.InvariantMACE(params, U, dtype=torch.float64, device="cuda")
    p = torch.from_numpy(pos).cuda().requires_grad_(True)
    energies = mace.node_energies(p, torch.from_numpy(species.astype(np.int32)).cuda(),
                                  torch.from_numpy(ei.astype(np.int32)).cuda(), torch.from_numpy(sh).cuda())
    (g,) = torch.autograd.grad(energies.sum(), p)
    energies = energies.detach()
    assert abs(float(out["interaction_energy"] - energies.sum())) < 1e-5 * float(energies.abs().sum())
    assert float((out["forces"] + g).abs().max()) < 1e-4 * float(g.abs().max())


def _images(n, side, seed):
    """Every edge of n atoms in a cell that is hardly longer than the cutoff: several images of a neighbour in a receiver's row,
    atoms that are their own neighbours, rows of many more than 64 edges."""
    pos = np.random.default_rng(seed).uniform(0, side, (n, 3))
    cells = np.stack(np.meshgrid(*[np.arange(-2, 3)] * 3, indexing="ij"), -1).reshape(-1, 3) * side
    recv, send, shift = [], [], []
    for i in range(n):
        d = pos[None] + cells[:, None] - pos[i]
        r = np.linalg.norm(d, axis=-1)
        k, j = np.nonzero((r > 1e-9) & (r < 5.0))
        recv.append(np.full(j.size, i)), send.append(j), shift.append(cells[k])
    return pos, np.stack([np.concatenate(recv), np.concatenate(send)]), np.concatenate(shift)


# An edge and its reverse share the rows of the radial perceptrons where both are in the list: a complete list, one with every
# third edge missing (a reverse that is not there), one with edges twice and rows shuffled, one with one-way edges only.
# Against the operators in float64, which know of no pairs: rounding over the chain, in float32 as in the tests above.
@pytest.mark.parametrize("kind", ["complete", "missing", "twice", "one way"])
@pytest.mark.parametrize("channels,dtype,tol", [(32, torch.float64, 1e-12), (64, torch.float64, 1e-12), (96, torch.float64, 1e-12),
                                                (32, torch.float32, 1e-5), (64, torch.float32, 1e-5), (128, torch.float32, 1e-5)])
def test_edges_that_share_a_length(U, kind, channels, dtype, tol):
    pos, ei, sh = _images(170, 7.0, 3)
    rng = np.random.default_rng(4)
    keep = np.arange(ei.shape[1])
    if kind == "missing":
        keep = keep[rng.random(keep.size) > 0.33]
    elif kind == "one way":
        keep = keep[ei[0] <= ei[1]]
    elif kind == "twice":
        keep = np.concatenate([keep, rng.choice(keep, 2000)])
        keep = rng.permutation(keep)
    keep = keep[np.argsort(ei[0][keep], kind="stable")]
    ei, sh = torch.from_numpy(ei[:, keep].astype(np.int32)).cuda(), torch.from_numpy(sh[keep]).cuda()
    assert ei.shape[1] > 74 * 2 * 128   # where float32 looks for pairs; float64 does from 74 * 16 * 8
    params = systems.init_params(channels, 3, 7)
    mace = model.InvariantMACE(params, U, dtype=dtype, device="cuda")
    p = torch.from_numpy(pos).cuda()
    species = torch.from_numpy(rng.integers(0, 3, pos.shape[0]).astype(np.int32)).cuda()
    out = mace(dict(positions=p, species=species, edge_index=ei, shifts=sh))
    assert step.plan_of(mace) is not None
    p.requires_grad_(True)
    energies = model.InvariantMACE(params, U, dtype=torch.float64, device="cuda").node_energies(p, species, ei, sh)
    (g,) = torch.autograd.grad(energies.sum(), p)
    energies = energies.detach()
    assert abs(float(out["interaction_energy"] - energies.sum())) < tol * float(energies.abs().sum())
    assert float((out["forces"] + g).abs().max()) < 10 * tol * float(g.abs().max())


# below and above the 32 768 edges from which a new list's grouping by sender runs beside the step
@pytest.mark.parametrize("n", [300, 1100])
def test_new_list_and_host_batch(U, n):
    side = (n / 0.1) ** (1.0 / 3.0)
    pos, species = systems.random_box(n, np.full(3, side), 0.9, 5), np.zeros(n, dtype=np.int64)
    dom = domain.partition_slabs(pos, species, np.full(3, side), 1, 5.0, 0)
    mace = model.InvariantMACE(systems.init_params(64, 1, 7), U, dtype=torch.float64, device="cuda")
    ev = evaluator.EnergyForceEvaluator(mace, dom, "cuda")
    p = ev.load_domain()
    assert (dom.edge_index.shape[1] >= step._BESIDE_EDGES) == (n > 1000)
    ev.topology.sender_order()          # grouped before the step
    e, f = ev(p)
    batch = ev.host_batch()
    e_host, f_host = ev.evaluate_host(batch)
    # the same edges in the same order: the same bits
    assert e_host == float(e) and torch.equal(f_host, f.cpu())
    assert torch.equal(ev.shifts.cpu(), torch.from_numpy(dom.shifts))
    ev.rebuild_neighbor_list(p)
    e_new, f_new = ev(p)                # another order of the edges: float64 rounding over about 50 edges a node
    assert abs(float(e_new - e)) < 1e-12 * n and float((f_new - f).abs().max()) < 1e-11 * float(f.abs().max())
    batch["shift_table"] = batch["shift_table"][:1]
    with pytest.raises(RuntimeError, match="shift"):
        ev.evaluate_host(batch)
    assert bool(ev(p)[0].isnan())
    with pytest.raises(RuntimeError, match="shift"):
        ops.check_status()
    assert torch.equal(ev.rebuild_neighbor_list(p)(p)[1], f_new)   # the device goes on


def _small(U, dtype=torch.float64, n=12, C=32, Z=3, **more):
    pos, ei, sh = _cluster(n, 3, 1.0)
    mace = model.InvariantMACE(systems.init_params(C, Z, 7, **more), U, dtype=dtype, device="cuda")
    species = torch.arange(n, dtype=torch.int32) % Z
    data = dict(positions=torch.from_numpy(pos).cuda(), species=species.cuda(),
                edge_index=torch.from_numpy(ei).to(torch.int32).cuda(), shifts=torch.from_numpy(sh).cuda())
    return mace, data


# a caller of the C interface that lays fused_w_back out as earlier libraries read it, steps of 8 channels, without the word
# that names the layout: right forces, from the radial weights in memory.  Bounds of a float32 step
def test_a_layout_of_earlier_callers_gives_the_same_forces(U):
    mace, data = _small(U, torch.float32, n=70, C=128)
    ref = mace(data)
    plan = step.plan_of(mace)
    w = mace.layers[1].W_radial3.t()
    old = w.reshape(4, 16, 8, 64).transpose(0, 1).reshape(16, 32, 64)
    old = torch.stack([step.half_images(b, 1.0 / plan.model.fused_scale) for b in old]).contiguous()
    plan.model.fused_w_back, plan.model.fused_layout = old.data_ptr(), 0
    out = mace(data)
    assert mace.__dict__["_step_plan"][1] is plan
    scale = float(ref["forces"].abs().max())
    assert float((out["forces"] - ref["forces"]).abs().max()) < 1e-4 * scale
    assert abs(float(out["interaction_energy"] - ref["interaction_energy"])) < 1e-5 * abs(float(ref["interaction_energy"]))


# The same for fewer channels, whose plans name their layout too: without that name the second layer's rows leave as float32 and
# its radial weights are written.  300 edges and more than the 18 944 from which a named layout looks for pairs
@pytest.mark.parametrize("channels,layout", [(32, 0), (64, 0), (96, 0), (64, 2), (128, 3)])
def test_a_layout_without_its_name_writes_the_radial_weights(U, channels, layout):
    params, pos, ei, sh, species = _list_of(np.arange(300) // 20, 16, channels, channels)
    for many in (False, True):
        if many:
            pos, ei, sh = _images(170, 7.0, 3)
            species = np.arange(170) % 3
        data = dict(positions=torch.from_numpy(pos).cuda(), species=torch.from_numpy(species.astype(np.int32)).cuda(),
                    edge_index=torch.from_numpy(ei).to(torch.int32).cuda(), shifts=torch.from_numpy(sh).cuda())
        assert (ei.shape[1] > 74 * 2 * 128) == many
        want = model.InvariantMACE(params, U, dtype=torch.float64, device="cuda")(data)
        mace = model.InvariantMACE(params, U, dtype=torch.float32, device="cuda")
        plan = step.plan_of(mace)
        assert plan.model.fused_layout == (_abi.FUSED_LAYOUT if channels == 128 else _abi.FUSED_LAYOUT_NARROW)
        size = lambda: _abi.call("cmace_step_workspace_bytes", ctypes.byref(plan.model), len(pos), len(pos), ei.shape[1])
        named, plan.model.fused_layout = size(), layout
        assert size() >= named + ei.shape[1] * (4 * channels * 4 - 8) - 512   # less the numbers of shared rows
        out = mace(data)
        assert step.plan_of(mace) is plan
        scale = float(want["forces"].abs().max())
        assert float((out["forces"] - want["forces"]).abs().max()) < 1e-4 * scale
        assert abs(float(out["interaction_energy"] - want["interaction_energy"])) < 1e-5 * float(want["node_energy"].abs().sum())


# nothing of these calls is launched: the checks come first
@pytest.mark.parametrize("species,node_attrs", [
    (torch.zeros(12, dtype=torch.int32), None), (torch.zeros(11, dtype=torch.int32, device="meta"), None),
    (torch.zeros(12, 1, dtype=torch.int32, device="meta"), None), (None, torch.eye(3)[torch.zeros(12, dtype=torch.long)]),
    (None, torch.zeros(11, 3, device="meta")), (None, torch.zeros(13, 3, device="meta"))])
def test_elements_that_do_not_fit_the_atoms_are_refused(U, species, node_attrs):
    mace, data = _small(U)
    del data["species"]
    for name, t in (("species", species), ("node_attrs", node_attrs)):
        if t is not None:   # "meta" stands for the GPU: the parameters are made where there may be none
            data[name] = torch.zeros(t.shape, dtype=t.dtype, device="cuda") if t.is_meta else t
    with pytest.raises(RuntimeError):
        mace(data)


def test_a_model_on_another_device_or_of_another_type_is_refused(U):
    mace, data = _small(U)
    mace(data)
    mace.float()
    with pytest.raises((RuntimeError, TypeError)):
        mace(data)
    mace, data = _small(U)
    mace(data)
    mace.cpu()
    with pytest.raises(RuntimeError):
        mace(data)


# one block of nodes and several
@pytest.mark.parametrize("dtype,index,at,n", [(torch.float64, 3, 0, 12), (torch.float32, -1, 11, 12),
                                              (torch.float32, 2**31 - 1, 2100, 2200)])
def test_an_element_index_that_does_not_exist_is_reported(U, dtype, index, at, n):
    mace, data = _small(U, dtype, n)
    good = mace(data)
    data["species"] = data["species"].clone()
    data["species"][at] = index
    bad = mace(data)
    assert bool(bad["energy"].isnan()) and bool(bad["interaction_energy"].isnan())
    assert bad["node_energy"].isnan().nonzero().flatten().tolist() == [at]
    with pytest.raises(RuntimeError, match="element"):
        ops.check_status()
    data["species"][at] = at % 3
    assert torch.equal(mace(data)["forces"], good["forces"])
    ops.check_status()


def test_a_recorded_step_of_a_host_batch_keeps_its_inputs(U):
    n = 300
    side = (n / 0.1) ** (1.0 / 3.0)
    pos, species = systems.random_box(n, np.full(3, side), 0.9, 5), np.zeros(n, dtype=np.int64)
    dom = domain.partition_slabs(pos, species, np.full(3, side), 1, 5.0, 0)
    mace = model.InvariantMACE(systems.init_params(64, 1, 7), U, dtype=torch.float32, device="cuda")
    ev = evaluator.EnergyForceEvaluator(mace, dom, "cuda")
    e, f = ev.evaluate_host(ev.host_batch())
    p = torch.from_numpy(dom.positions[:n]).cuda()
    ev.capture(p)
    pair = ev._shifts
    rows = ev.shifts                               # as rows: the recording goes on reading the pair
    assert torch.equal(rows.cpu(), torch.from_numpy(dom.shifts)) and ev._shifts is pair and ev.shifts is rows
    assert any(x is pair for x in ev._graph[4])
    assert torch.equal(ev(p)[1].cpu(), f)
    ev.shifts = torch.zeros_like(rows)             # another list: no replay of the recorded one
    assert ev._graph is None
    assert not torch.equal(ev(p)[1].cpu(), f)


@pytest.mark.parametrize("how", ["model", "captured"])
def test_a_changed_model_changes_the_step(U, how):
    """scale, shift and r_max like the weights: the step agrees with node_energies() after every change, recorded or not;
    a model that the sequence has refused is taken again once it is what it was."""
    n = 300
    side = (n / 0.1) ** (1.0 / 3.0)
    pos, species = systems.random_box(n, np.full(3, side), 0.9, 5), np.zeros(n, dtype=np.int64)
    dom = domain.partition_slabs(pos, species, np.full(3, side), 1, 5.0, 0)
    mace = model.InvariantMACE(systems.init_params(32, 1, 7), U, dtype=torch.float64, device="cuda")
    ev = evaluator.EnergyForceEvaluator(mace, dom, "cuda")
    p = ev.load_domain()

    def agrees():
        q = p.clone().requires_grad_(True)
        e = mace.node_energies(q, ev.species, ev.edge_index, ev.shifts).sum()
        (g,), e = torch.autograd.grad(e, q), e.detach()
        if how == "captured":
            got = ev(p)
        else:
            out = mace(dict(positions=p, species=ev.species, edge_index=ev.edge_index, shifts=ev.shifts))
            got = out["interaction_energy"], out["forces"]
        assert abs(float(got[0] - e)) < 1e-10 * abs(float(e))
        assert float((got[1] + g).abs().max()) < 1e-10 * float(g.abs().max())

    def scale():
        mace.scale = 1.7

    def shift():
        mace.shift = -0.25

    def radius():
        mace.edge_basis.r_max = 4.5

    def weight():
        for W in (mace.layers[1].W_readout2, mace.layers[1].W_readout2_T):
            W.mul_(0.5)

    for change in (scale, shift, radius, weight):
        if how == "captured":
            ev.capture(p)
        agrees()
        change()
        agrees()
    assert step.plan_of(mace) is not None
    hook = mace.layers[1].linear.register_forward_hook(lambda *a: None)
    assert step.plan_of(mace) is None
    hook.remove()
    assert step.plan_of(mace) is not None


# what a plan is made of has to be there for every stream, and to stay for whoever still reads it
def test_a_plan_laid_out_on_one_stream_serves_another(U):
    mace, data = _small(U, torch.float32)
    want = mace(data)["forces"]
    first, second = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(3):
        mace.layers[1].W_readout2.mul_(1.0)          # another version: laid out again
        torch.cuda.synchronize()
        with torch.cuda.stream(first):
            torch.cuda._sleep(20_000_000)            # some 10 ms before the layout's kernels
            a = mace(data)["forces"]
        with torch.cuda.stream(second):
            b = mace(data)["forces"]
        torch.cuda.synchronize()
        assert torch.equal(a, want) and torch.equal(b, want)


def _record(mace, data):
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=side):
        out = mace(data)
    return graph, out


def test_a_graph_of_the_caller_keeps_the_weights_it_reads(U):
    mace, data = _small(U, torch.float32)
    want = mace(data)["forces"].clone()
    graph, out = _record(mace, data)
    old = step.plan_of(mace)
    sizes = [t.numel() * t.element_size() for t in old.keep]
    mace.layers[1].W_readout2.mul_(2.0)
    changed = mace(data)["forces"].clone()
    assert step.plan_of(mace) is not old and not torch.equal(changed, want)
    del old
    junk = [torch.full((s,), 255, dtype=torch.uint8, device="cuda") for s in sizes for _ in range(4)]
    graph.replay()
    assert torch.equal(out["forces"], want) and len(junk) > 0


@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-10), (torch.float32, 1e-4)])
def test_no_layout_while_a_graph_is_recorded(U, dtype, tol):
    mace, data = _small(U, dtype)
    mace(data)
    mace.node_energies(data["positions"], data["species"], data["edge_index"], data["shifts"])
    for W in (mace.layers[1].W_readout2, mace.layers[1].W_readout2_T):
        W.mul_(2.0)
    graph, out = _record(mace, data)
    eager = mace(data)["forces"]
    graph.replay()
    assert float((out["forces"] - eager).abs().max()) < tol * float(eager.abs().max())


# a diverged model: NaN comes out, as from the operators, instead of an error from the layout
@pytest.mark.parametrize("dtype,C", [(torch.float32, 128), (torch.float32, 32), (torch.float64, 32)])
@pytest.mark.parametrize("layer,which", [(0, 0), (1, 2), (1, 3)])
def test_weights_that_are_not_finite(U, dtype, C, layer, which):
    mace, data = _small(U, dtype, C=C)
    getattr(mace.layers[layer], f"W_radial{which}")[1, 2] = float("nan")
    out = mace(data)
    assert bool(out["energy"].isnan()) and bool(out["forces"].isnan().any())
    ops.check_status()


# Layers whose values are small everywhere: silu is linear there, so factors of two layers that cancel leave the model nearly
# as it is.  Against the same weights in float64; 1e-5 and 1e-4 are the package's float32 bounds.
@pytest.mark.parametrize("C", [32, 128])
@pytest.mark.parametrize("small,back", [(0, 1), (1, 2), (2, 3)])
def test_small_hidden_values_keep_their_digits(U, C, small, back):
    out = {}
    for dtype in (torch.float64, torch.float32):
        mace, data = _small(U, dtype, n=40, C=C)
        for L in mace.layers:
            for k, factor in ((small, 2.0**-30), (back, 2.0**30)):
                for name in (f"W_radial{k}", f"W_radial{k}_T"):
                    getattr(L, name).mul_(factor)
        assert step.plan_of(mace).model.radial_half[0][0] or dtype == torch.float64
        out[dtype] = mace(data)
    ref, got = out[torch.float64], out[torch.float32]
    assert abs(float(got["interaction_energy"] / ref["interaction_energy"]) - 1.0) < 1e-5
    assert float((got["forces"] - ref["forces"]).abs().max()) < 1e-4 * float(ref["forces"].abs().max())


def _with_hidden_weights_times(params, factor):
    for P in params["layers"]:
        P["W_radial"] = [W * factor if i < 3 else W / factor**3 for i, W in enumerate(P["W_radial"])]   # R stays as large
    return params


def _largest_factor(C, Z, nb):
    """Largest power of 2^(1/8) of the initial hidden weights whose bounds still fit fp16, seed 7"""
    bounds, k = step.basis_bounds(nb, 5.0, 5), 0
    while True:
        params = _with_hidden_weights_times(systems.init_params(C, Z, 7, num_bessel=nb), 2.0 ** ((k + 1) / 8))
        for P in params["layers"]:
            Ws = [W / W.shape[0] ** 0.5 * (model.SILU_2MOM if i else 1.0) for i, W in enumerate(P["W_radial"][:3])]
            if step.half_scales(Ws, bounds) is None:
                return 2.0 ** (k / 8)
        k += 1


# float32 on both sides of the rule that gives a model the fp16 kernels: just below the largest hidden weights that fit, and
# well beyond, where radial_pair, sums_tf32, sums_bwd_tf32 and, at 128 channels, the passes over [E, 4, C] run.  Edges around
# the kernels' tiles of 128, odd numbers of elements; the package's bounds of 1e-5 and 1e-4 on energy and forces.
@pytest.mark.parametrize("nb", [8, 16])
@pytest.mark.parametrize("C,Z,edges", [(64, 3, 127), (128, 5, 128), (96, 1, 129), (128, 2, 385), (32, 7, 1), (128, 3, 5000)])
@pytest.mark.parametrize("fits", [True, False])
def test_hidden_weights_around_the_limit_of_fp16(U, nb, C, Z, edges, fits):
    n = 180 if edges > 1000 else 40
    pos, ei, sh = _cluster(n, 3, 1.0)
    ei, sh = ei[:, :edges], sh[:edges]
    assert ei.shape[1] == edges
    factor = _largest_factor(C, Z, nb) * (1.0 if fits else 2.0)
    params = _with_hidden_weights_times(systems.init_params(C, Z, 7, num_bessel=nb), factor)
    species = torch.from_numpy(np.random.default_rng(4).integers(0, Z, n)).to(torch.int32).cuda()
    edge_index, shifts = torch.from_numpy(ei).to(torch.int32).cuda(), torch.from_numpy(sh).cuda()
    p = torch.from_numpy(pos).cuda().requires_grad_(True)
    ref = model.InvariantMACE(params, U, dtype=torch.float64, device="cuda")
    e = ref.node_energies(p, species, edge_index, shifts).sum()
    (g,), e = torch.autograd.grad(e, p), e.detach()
    mace = model.InvariantMACE(params, U, dtype=torch.float32, device="cuda")
    assert bool(step.plan_of(mace).model.radial_half[0][0]) == fits
    out = mace(dict(positions=p, species=species, edge_index=edge_index, shifts=shifts))
    assert abs(float(out["interaction_energy"] - e)) < 1e-5 * abs(float(e))
    assert float((out["forces"] + g).abs().max()) < 1e-4 * float(g.abs().max())
    ops.check_status()


def _periodic(U, n, dtype, C=64):
    side = (n / 0.1) ** (1.0 / 3.0)
    pos, species = systems.random_box(n, np.full(3, side), 0.9, 5), np.zeros(n, dtype=np.int64)
    dom = domain.partition_slabs(pos, species, np.full(3, side), 1, 5.0, 0)
    mace = model.InvariantMACE(systems.init_params(C, 1, 7), U, dtype=dtype, device="cuda")
    ev = evaluator.EnergyForceEvaluator(mace, dom, "cuda")
    return ev, ev.load_domain()


# Programmatic launches overlap the kernel before them, not what the stream waits for: positions that another stream writes
# late, and a grouping by sender that is late, both before the first kernel of a range.  (All buffers hold valid values before.)
def test_a_wait_between_launches_is_kept(U, monkeypatch):
    ev, p = _periodic(U, 300, torch.float32)
    moved = p + 0.01
    moved[0] += 0.2
    old, want = ev(p)[1].clone(), ev(moved)[1].clone()
    assert not torch.equal(old, want)
    other = torch.cuda.Stream()
    buffer = p.clone()
    for _ in range(5):
        buffer.copy_(p)
        other.wait_stream(torch.cuda.current_stream())
        ev(buffer)                                    # its last kernel lets the next one come early
        with torch.cuda.stream(other):
            torch.cuda._sleep(2_000_000)
            buffer.copy_(moved, non_blocking=True)
            written = other.record_event()
        torch.cuda.current_stream().wait_event(written)
        assert torch.equal(ev(buffer)[1], want)


def test_a_late_grouping_is_waited_for(U, monkeypatch):
    ev, p = _periodic(U, 1100, torch.float32)
    assert step._BESIDE_EDGES <= ev.topology.nedges <= 98304   # beside the step, launches chained
    ev.topology.sender_order()
    want = ev(p)[1].clone()
    buffers, group = ops.EdgeTopology.grouping_buffers, ops.EdgeTopology.group_senders

    def zeros(self):
        return tuple(t.zero_() for t in buffers(self))

    def late(self, b, stream):
        with torch.cuda.stream(torch.cuda.ExternalStream(stream)):
            torch.cuda._sleep(2_000_000)
        group(self, b, stream)

    monkeypatch.setattr(ops.EdgeTopology, "grouping_buffers", zeros)
    monkeypatch.setattr(ops.EdgeTopology, "group_senders", late)
    for _ in range(5):
        ev.set_neighbor_list(ev.species, ev.edge_index, ev.shifts)
        assert torch.equal(ev(p)[1], want)


def _programmatic_edges(graph):
    """(number of nodes, number of edges, of those programmatic) of a recorded graph"""
    class Data(ctypes.Structure):   # cudaGraphEdgeData; type 1 is programmatic
        _fields_ = [("from_port", ctypes.c_uint8), ("to_port", ctypes.c_uint8), ("type", ctypes.c_uint8),
                    ("reserved", ctypes.c_uint8 * 5)]

    cudart, raw = ctypes.CDLL("libcudart.so.12"), ctypes.c_void_p(graph.raw_cuda_graph())
    nodes, count = ctypes.c_size_t(), ctypes.c_size_t()
    assert cudart.cudaGraphGetNodes(raw, None, ctypes.byref(nodes)) == 0
    assert cudart.cudaGraphGetEdges_v2(raw, None, None, None, ctypes.byref(count)) == 0
    ends, data = (ctypes.c_void_p * (2 * count.value))(), (Data * count.value)()
    assert cudart.cudaGraphGetEdges_v2(raw, ctypes.byref(ends), ctypes.byref(ends, count.value * ctypes.sizeof(ctypes.c_void_p)), data,
                                       ctypes.byref(count)) == 0
    return nodes.value, count.value, sum(d.type == 1 for d in data)


# A caller that runs a range of steps, a kernel of its own and the other steps: the second range's first kernel, whatever step
# launches it, comes after that kernel, the others are chained.  12: one that float32 steps leave out (radial_back)
@pytest.mark.parametrize("split", [1, 2, 3, 5, 6, 7, 12, 13, 14, 16, 18])
@pytest.mark.parametrize("dtype,C", [(torch.float32, 64), (torch.float64, 128)])
def test_a_range_begins_after_what_its_caller_put_before_it(U, dtype, C, split, monkeypatch):
    mace, data = _small(U, dtype, n=70, C=C)
    want = mace(data)["forces"].clone()
    run, counter, ranges = _abi.run_steps, torch.zeros(1, device="cuda"), []

    def in_two(m, io, first, last, stream):
        for a, b in ((first, split), (split, last)):
            before = io.launches
            run(m, io, a, b, stream)
            ranges.append(io.launches - before)
            if b == split:
                counter.add_(1)

    monkeypatch.setattr(_abi, "run_steps", in_two)
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=side):
        out = mace(data)
    nodes, edges, chained = _programmatic_edges(graph)
    assert nodes == sum(ranges) + 1 and edges == nodes - 1 and min(ranges) > 0
    assert chained == sum(ranges) - 2
    graph.replay()
    assert torch.equal(out["forces"], want)


# Recorded float32 steps are chained up to 196 608 edges, live ones too: the same kernels, so the same bits, also for positions that
# the recording has not seen, several replays in a row (each begins while the one before may still run)
@pytest.mark.parametrize("channels", [64, 128])
def test_a_recorded_step_of_many_edges_is_chained_and_the_same(U, channels):
    n = 2300
    ev, p = _periodic(U, n, torch.float32, channels)
    data = dict(positions=p.clone(), species=ev.species, edge_index=ev.edge_index, shifts=ev.shifts)
    assert 98304 < ev.edge_index.shape[1] <= 196608
    mace, moved = ev.model, [p + 0.001 * k * torch.sin(p + k) for k in range(3)]
    want = []
    for q in moved:
        data["positions"].copy_(q)
        out = mace(data)
        want.append((out["energy"].clone(), out["forces"].clone()))
    side, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph(keep_graph=True)
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(graph, stream=side):
        out = mace(data)
    nodes, edges, chained = _programmatic_edges(graph)
    assert edges == chained == nodes - 1
    for _ in range(4):
        got = []
        for q in moved:
            data["positions"].copy_(q)
            graph.replay()
            got.append((out["energy"].clone(), out["forces"].clone()))
        assert all(torch.equal(a, b) for x, y in zip(got, want) for a, b in zip(x, y))


def test_results_do_not_share_memory(U):
    """An energy that is kept keeps three values, the forces their own rows."""
    mace, data = _small(U)
    out = mace(data)
    size = {k: t.untyped_storage().nbytes() for k, t in out.items()}
    assert size["energy"] <= 24 and size["interaction_energy"] <= 24
    assert size["node_energy"] == 12 * 8 and size["forces"] == 12 * 3 * 8
    ev, p = _periodic(U, 300, torch.float32)
    energy, forces = ev(p)
    assert energy.untyped_storage().nbytes() <= 24 and forces.untyped_storage().nbytes() == 300 * 3 * 8


# around the line beyond which a system of few edges and many elements takes the operators: the same energies either way
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-10), (torch.float32, 1e-4)])
def test_few_edges_and_many_elements(U, dtype, tol, monkeypatch):
    mace, data = _small(U, dtype, n=40, C=32, Z=10)
    plan = step.plan_of(mace)
    big = 400_000 // 10
    assert step.pays(plan, big, 52 * big) and not step.pays(plan, big, 8 * big) and step.pays(plan, 400, 8 * 400)
    assert step.pays(step.plan_of(_small(U, dtype, Z=4)[0]), 10 * big, 0)
    native = mace(data)
    monkeypatch.setattr(step, "pays", lambda *a: False)
    monkeypatch.setattr(step, "energy_forces", None)
    operators = mace(data)
    assert abs(float(native["energy"] / operators["energy"]) - 1.0) < tol
    assert float((native["forces"] - operators["forces"]).abs().max()) < tol * float(native["forces"].abs().max())


# A recording of operators that nothing has warmed up leaves nothing behind: their packed weights, groupings and edge orders are
# filled by a replay only, so no call outside the graph may find them.  (Without that the second call would read them unwritten.)
@pytest.mark.parametrize("dtype,tol", [(torch.float64, 1e-10), (torch.float32, 1e-4)])
def test_a_recording_leaves_no_cached_results_behind(U, dtype, tol, monkeypatch):
    mace, data = _small(U, dtype, n=40, C=64, Z=3)
    want = mace(data)["forces"]                       # native: makes the plans of the contractions
    data = {k: t.clone() for k, t in data.items()}    # tensors that no cache knows
    for L in mace.layers:
        for name, b in list(L.named_buffers()):
            b.mul_(1)                                 # nor these versions
    caches = (ops._packed_cache, ops._topology_cache, ops._grouping_cache, ops._onehot_cache)
    sizes = [set(c.entries) for c in caches]
    graph, out = _record(mace, data)                  # no layout while recording: the operators
    assert [set(c.entries) for c in caches] == sizes
    graph.replay()
    assert float((out["forces"] - want).abs().max()) < tol * float(want.abs().max())
    monkeypatch.setattr(step, "pays", lambda *a: False)
    assert float((mace(data)["forces"] - want).abs().max()) < tol * float(want.abs().max())


def test_a_recorded_step_that_takes_the_operators(U, monkeypatch):
    ev, p = _periodic(U, 300, torch.float64, C=32)
    e, f = ev(p)
    asked = []
    monkeypatch.setattr(step, "pays", lambda plan, atoms, edges, recorded=False: asked.append(recorded) or not recorded)
    ev.capture(p)
    assert set(asked) == {True} and len(asked) == 3   # twice to warm up, once recorded
    assert torch.equal(ev(p)[1], ev(p)[1]) and float((ev(p)[1] - f).abs().max()) < 1e-10 * float(f.abs().max())
    ev.shifts = ev.shifts                             # live again
    assert torch.equal(ev(p)[1], f) and asked[-1] is False
