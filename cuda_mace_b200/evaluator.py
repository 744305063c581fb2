"""Energy+force evaluation of one slab (or of the whole periodic box on a single GPU): the call a
user of the package makes per step.

    ev = EnergyForceEvaluator(model, domain, device, group)
    energy, forces = ev(positions_owned)            # tensors already on the device
    energy, forces = ev.evaluate_host(host_batch)   # pinned host buffers in, host results out

`evaluate_host` moves the step's inputs (positions, species, edge list, shifts) to the device,
rebuilds the edge topology for the list it was given, runs the model and copies energy and forces
back, so it is the end-to-end path including every host<->device byte.  The shift vectors of a periodic
neighbour list take only a handful of distinct values (lattice translations), so the host batch carries
them as a small table plus one byte per edge instead of three float64 per edge.
"""
import torch

from . import domain as _domain
from . import ops, step


class EnergyForceEvaluator:
    def __init__(self, model, dom, device, group=None):
        self.model = model
        self.dom = dom
        self.device = torch.device(device)
        self.plan = _domain.HaloPlan(dom, self.device, group).verify()
        self.species = None
        self.edge_index = None
        self._shifts = None   # [E, 3], or (index, table) as a host batch carries them
        self._shift_rows = None   # [E, 3] of an (index, table), made when somebody asks
        self.topology = None
        self._graph = None
        self._recording = False

    def set_neighbor_list(self, species, edge_index, shifts):
        """Device tensors: species [n_local] int32, edge_index [2,E] int32 (receivers sorted), shifts [E,3]."""
        return self._set_list(species, edge_index, shifts)

    def _set_list(self, species, edge_index, shifts, row_ptr=None):
        self.species = species.to(torch.int32).contiguous()
        self.edge_index = edge_index
        self._shifts, self._shift_rows = shifts, None
        self.topology = ops.EdgeTopology(edge_index[1], edge_index[0], self.dom.n_owned, self.dom.n_local, row_ptr)
        self._graph = None   # a captured step belongs to the list it was captured with
        return self

    @property
    def shifts(self):
        if not isinstance(self._shifts, tuple):
            return self._shifts
        if self._shift_rows is None:   # beside the pair, not in its place: a recorded step reads the pair
            index, table = self._shifts
            self._shift_rows = table.index_select(0, index.to(torch.int64))
        return self._shift_rows

    @shifts.setter
    def shifts(self, value):
        self._shifts, self._shift_rows = value, None
        self._graph = None

    def rebuild_neighbor_list(self, positions_owned, r_cut=None):
        """Builds the neighbour list of the current positions on the device (cell-list kernels) instead of taking
        it from the host: ghost positions come from the neighbouring slabs, receivers are the owned atoms, the
        slab's z axis is open once it carries ghosts.  One host synchronisation (edge count)."""
        d = self.dom
        if d.box is None:
            raise RuntimeError("the domain does not carry its box")
        r_cut = float(self.model.r_max if r_cut is None else r_cut)
        with torch.no_grad():
            pos_local = positions_owned.detach()
            if d.nranks > 1:
                pos_local = _domain.halo_exchange(pos_local, self.plan) + self.plan.ghost_shift(pos_local.dtype)
        lo, ext = [0.0, 0.0, 0.0], [float(v) for v in d.box]
        for ax in range(3):
            if not d.pbc[ax]:
                zmin, zmax = float(pos_local[:, ax].min()), float(pos_local[:, ax].max())
                lo[ax], ext[ax] = zmin, max(zmax - zmin, 1e-6) * (1 + 1e-12) + 1e-9
        edge_index, shifts, _, row_ptr = ops.neighbor_list_rows(pos_local, ext, d.pbc, r_cut, d.n_owned, lo=lo)
        if self.species is None:
            self.species = torch.as_tensor(d.species, dtype=torch.int32, device=self.device)
        return self._set_list(self.species, edge_index, shifts.to(positions_owned.dtype), row_ptr)

    def load_domain(self, pos_dtype=torch.float64):
        d = self.dom
        dev = self.device
        self.set_neighbor_list(torch.as_tensor(d.species, dtype=torch.int32, device=dev),
                               torch.as_tensor(d.edge_index, dtype=torch.int32, device=dev),
                               torch.as_tensor(d.shifts, dtype=pos_dtype, device=dev))
        return torch.as_tensor(d.positions[: d.n_owned], dtype=pos_dtype, device=dev)

    def capture(self, positions_owned):
        """Records the whole energy+force step for the current neighbour list as a CUDA graph; later calls copy
        the positions into the graph's input and replay it, which takes the host's part (80 to 95 us a step) out
        of a program that is short of it; the step itself is no faster (about 420 us either way at 3 000 atoms).  Single-rank
        domains only: the halo exchange of a multi-rank step is host-driven.  A new neighbour list drops the recording, and so
        does a changed model."""
        if self.dom.nranks != 1:
            raise RuntimeError("capture() needs a single-rank domain")
        self._graph, self._recording = None, True   # the warm-up takes the way that will be recorded
        try:
            return self._capture(positions_owned)
        finally:
            self._recording = False

    def _capture(self, positions_owned):
        static_pos = positions_owned.detach().clone()
        side = torch.cuda.Stream(device=self.device)
        side.wait_stream(torch.cuda.current_stream(self.device))
        with torch.cuda.stream(side):
            for _ in range(2):      # warm-up outside the recording: weight packing, caches, allocator pools
                self(static_pos)
        torch.cuda.current_stream(self.device).wait_stream(side)
        ops.check_status()
        plan = step.plan_of(self.model) if step.takes(static_pos, self._shifts) else None
        others = plan is not None and plan.recorded
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            energy, forces = self(static_pos)
        if plan is not None:
            plan.recorded = others   # kept below, by this object
        # what the recording reads by address stays alive with it, whatever the attributes become: the list, the plan's
        # weights
        reads = (plan, self.species, self.edge_index, self._shifts, self.topology)
        self._graph = (graph, static_pos, energy, forces, reads)
        return self

    def __call__(self, positions_owned):
        if self._graph is not None and not torch.cuda.is_current_stream_capturing():
            graph, static_pos, energy, forces, (plan, *_) = self._graph
            if plan is None or plan.current(self.model):
                static_pos.copy_(positions_owned)
                graph.replay()
                return energy.clone(), forces.clone()
            self._graph = None   # the model has changed: the recording has the old weights laid out

        if step.takes(positions_owned, self._shifts):
            plan = self._plan()
            if plan is not None:
                return self._evaluate_native(plan, positions_owned.detach())[:2]

        def node_energy(pos_local, exchange):
            return self.model.node_energies(pos_local, self.species, self.edge_index, self.shifts,
                                            topology=self.topology, exchange=exchange, n_owned=self.dom.n_owned)

        return _domain.distributed_energy_forces(node_energy, self.dom, self.plan, positions_owned)

    def _plan(self):
        """The model's plan for the current list, or None for the operators; every rank of a decomposition decides alike."""
        plan = step.plan_of(self.model)
        if plan is None or self.dom.nranks > 1 or step.pays(plan, self.dom.n_owned, self.topology.nedges,
                                                                   self._recording):
            return plan
        return None

    def _evaluate_native(self, plan, positions_owned):
        """Total interaction energy over all ranks, forces on the owned atoms and this rank's sums, by the library's
        own sequence."""
        many = self.dom.nranks > 1
        pos = positions_owned
        if many:
            pos = self.plan.forward_fill(pos) + self.plan.ghost_shift(pos.dtype)
        sums, _, _, forces = step.energy_forces(plan, pos, self.species, None, self._shifts, self.topology,
                                                halo=self.plan if many else None)
        energy = sums[1]
        if many:
            energy = energy.clone()
            torch.distributed.all_reduce(energy, group=self.plan.group)
        return energy, forces, sums

    # ---- end-to-end path with host buffers ----------------------------------------------------
    def host_batch(self, pos_dtype=torch.float64):
        """Pinned host copies of one step's inputs, as a data loader would hand them over."""
        import numpy as np

        d = self.dom
        pin = lambda t: t.pin_memory() if torch.cuda.is_available() else t
        batch = {
            "positions": pin(torch.as_tensor(d.positions[: d.n_owned], dtype=pos_dtype)),
            "species": pin(torch.as_tensor(d.species, dtype=torch.int32)),
            "edge_index": pin(torch.as_tensor(d.edge_index, dtype=torch.int32)),
        }
        table, index = np.unique(np.asarray(d.shifts), axis=0, return_inverse=True)
        if table.shape[0] <= 256:
            batch["shift_table"] = pin(torch.as_tensor(table, dtype=pos_dtype))
            batch["shift_index"] = pin(torch.as_tensor(index.reshape(-1).astype(np.uint8)))
        else:  # not a lattice-translation list: ship the vectors themselves
            batch["shifts"] = pin(torch.as_tensor(d.shifts, dtype=pos_dtype))
        return batch

    @staticmethod
    def h2d_bytes(batch):
        return int(sum(t.numel() * t.element_size() for t in batch.values()))

    def evaluate_host(self, batch, out_forces=None):
        dev = self.device
        moved = {k: v.to(dev, non_blocking=True) for k, v in batch.items()}
        shifts = moved["shifts"] if "shifts" in moved else (moved["shift_index"], moved["shift_table"])
        self.set_neighbor_list(moved["species"], moved["edge_index"], shifts)
        positions, plan, sums = moved["positions"], None, None
        if step.takes(positions, shifts):
            plan = self._plan()
        if plan is not None:
            energy, forces, sums = self._evaluate_native(plan, positions.detach())
        else:
            energy, forces = self(positions)
        if out_forces is None:
            out_forces = torch.empty(forces.shape, dtype=forces.dtype, pin_memory=torch.cuda.is_available())
        out_forces.copy_(forces, non_blocking=True)
        if sums is None:
            e = float(energy.cpu())  # synchronises
            ops.check_status()
            return e, out_forces
        # energies and the record of failures in one copy, the step's only synchronisation
        _, inter, failed = sums.tolist()
        if failed:
            ops.check_status()
            raise RuntimeError("cuda_mace_b200: a kernel of the step recorded a failure")
        return (inter if self.dom.nranks == 1 else float(energy)), out_forces
