"""Slab decomposition: energy and forces equal the single-GPU periodic evaluation.  Two ranks on two GPUs (NCCL), skipped
when fewer than two devices are visible: ranks are child processes that leave only after the step has finished, NVLS is
switched off for them.  Two and three ranks as threads on one GPU: the ranges of the native sequence with ghost rows."""
import os
import socket
import threading

import numpy as np
import pytest
import torch
import torch.distributed as dist
import torch.multiprocessing as mp

pytestmark = pytest.mark.gpu


def free_port():
    with socket.socket() as s:
        s.bind(("127.0.0.1", 0))
        return s.getsockname()[1]


def case():
    from cuda_mace_b200 import systems

    box = np.array([22.0, 22.0, 40.0])
    pos = systems.random_box(1800, box, 0.9, seed=3)
    rng = np.random.default_rng(3)
    species = rng.integers(0, 4, pos.shape[0])
    params = systems.init_params(64, 4, 8)
    return pos, species, box, params


def worker(rank, world, port, out_dir):
    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port), NCCL_NVLS_ENABLE="0")
    torch.cuda.set_device(rank)
    dist.init_process_group("nccl", rank=rank, world_size=world, device_id=torch.device("cuda", rank))
    try:
        from cuda_mace_b200 import cg, domain, evaluator, model, ops

        pos, species, box, params = case()
        dom = domain.partition_slabs(pos, species, box, world, 5.0, rank)
        net = model.InvariantMACE(params, cg.u_matrices(), dtype=torch.float64, device=f"cuda:{rank}")
        ev = evaluator.EnergyForceEvaluator(net, dom, f"cuda:{rank}")
        p = ev.load_domain()
        e, f = ev(p)
        ops.check_status()
        # second pass with the neighbour list of the slab (owned + ghost atoms, open z axis) rebuilt on the device
        n_edges = ev.edge_index.shape[1]
        ev.rebuild_neighbor_list(p)
        assert ev.edge_index.shape[1] == n_edges
        e2, f2 = ev(p)
        assert abs(float(e2) - float(e)) < 1e-11 * abs(float(e))
        assert float((f2 - f).abs().max()) < 1e-10 * float(f.abs().max())
        np.savez(os.path.join(out_dir, f"rank{rank}.npz"), e=e.cpu().numpy(), f=f.cpu().numpy(), ids=dom.owned_global)
        dist.barrier()
    finally:
        dist.destroy_process_group()


@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_two_gpu_slabs_equal_single_gpu(tmp_path):
    from cuda_mace_b200 import cg, model, systems

    pos, species, box, params = case()
    ei, sh = systems.neighbor_list(pos, box, (True, True, True), 5.0)
    net = model.InvariantMACE(params, cg.u_matrices(), dtype=torch.float64, device="cuda:0")
    ref = net(dict(positions=torch.from_numpy(pos).cuda(), species=torch.from_numpy(species).to(torch.int32).cuda(),
                   edge_index=torch.from_numpy(ei).to(torch.int32).cuda(), shifts=torch.from_numpy(sh).cuda()))
    mp.spawn(worker, args=(2, free_port(), str(tmp_path)), nprocs=2, join=True)
    forces = np.zeros_like(pos)
    for r in range(2):
        z = np.load(tmp_path / f"rank{r}.npz")
        assert abs(float(z["e"]) - float(ref["interaction_energy"])) < 1e-10 * abs(float(ref["interaction_energy"]))
        forces[z["ids"]] = z["f"]
    fr = ref["forces"].cpu().numpy()
    assert np.abs(forces - fr).max() < 1e-10 * np.abs(fr).max()


class _Exchanges:
    """The exchanges of ranks that are threads of this process: every rank leaves its rows, all wait on the host, every rank
    copies what its neighbours left.  All launches are on one stream, so no kernel waits for another rank's."""

    def __init__(self, world):
        from cuda_mace_b200 import domain

        self.barrier, self.rows, self.kind = threading.Barrier(world, timeout=120), {}, domain.HaloPlan

    def halo(self, dom):
        shared = self

        class Halo(self.kind):
            def verify(self):
                return self

            def _exchange(self, out_down, out_up, in_from_down, in_from_up):
                d = self.dom
                shared.rows[d.rank] = out_down, out_up
                shared.barrier.wait()
                in_from_down.copy_(shared.rows[d.down][1])
                in_from_up.copy_(shared.rows[d.up][0])
                shared.barrier.wait()

        return Halo(dom, "cuda")

    def sum(self, rank, t):
        self.rows[rank] = t.clone()
        self.barrier.wait()
        total = sum(self.rows[r] for r in sorted(self.rows))
        self.barrier.wait()
        t.copy_(total)


# The ranges of the native sequence with ghost rows, two and three slabs on one GPU against the whole box: the fused and the
# unfused second layer, float64, tabulated weights; lists below and above the 32 768 edges from which the grouping by sender
# runs beside the step; both neighbours the same rank or not; the list from the host and from the device.
@pytest.mark.parametrize("dtype,C,radial,tol_e,tol_f", [
    (torch.float64, 64, "exact", 1e-10, 1e-10), (torch.float32, 128, "exact", 1e-5, 1e-4),
    (torch.float32, 64, "exact", 1e-5, 1e-4), (torch.float64, 32, "spline", 1e-10, 1e-10)])
@pytest.mark.parametrize("world,n", [(2, 1800), (3, 1500), (2, 900)])
def test_slabs_on_one_gpu_equal_the_box(monkeypatch, dtype, C, radial, tol_e, tol_f, world, n):
    from cuda_mace_b200 import cg, domain, evaluator, model, ops, step, systems

    box = np.array([22.0, 22.0, 40.0]) if n > 1000 else np.array([16.0, 16.0, 40.0])
    pos = systems.random_box(n, box, 0.9, seed=3)
    species = np.random.default_rng(3).integers(0, 4, n)
    params = systems.init_params(C, 4, 8)
    if radial == "spline":
        model.add_spline_knots(params)
    net = model.InvariantMACE(params, cg.u_matrices(), dtype=dtype, device="cuda", radial=radial)
    whole = evaluator.EnergyForceEvaluator(net, domain.partition_slabs(pos, species, box, 1, 5.0, 0), "cuda")
    e_ref, f_ref = whole(whole.load_domain())
    want = torch.empty_like(f_ref)
    want[torch.from_numpy(whole.dom.owned_global)] = f_ref
    assert step.plan_of(net) is not None

    exchanges, ranks = _Exchanges(world), threading.local()
    monkeypatch.setattr(domain, "HaloPlan", lambda dom, device, group=None: exchanges.halo(dom))
    monkeypatch.setattr(dist, "all_reduce", lambda t, group=None: exchanges.sum(ranks.rank, t))
    results, errors = {}, []

    def run(rank):
        try:
            ranks.rank = rank
            dom = domain.partition_slabs(pos, species, box, world, 5.0, rank)
            ev = evaluator.EnergyForceEvaluator(net, dom, "cuda")
            p = ev.load_domain()
            assert dom.n_local > dom.n_owned and step.takes(p, ev.shifts)
            got = [ev(p)]
            ev.rebuild_neighbor_list(p)
            got.append(ev(p))
            e_host, f_host = ev.evaluate_host(ev.host_batch())
            results[rank] = dom.owned_global, got + [(torch.tensor(e_host, dtype=torch.float64), f_host.cuda())]
        except BaseException as error:
            errors.append(error)
            exchanges.barrier.abort()

    threads = [threading.Thread(target=run, args=(r,)) for r in range(world)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for k in range(3):
        forces = torch.empty_like(want)
        for owned, got in results.values():
            assert abs(float(got[k][0]) - float(e_ref)) < tol_e * abs(float(e_ref))
            forces[torch.from_numpy(owned)] = got[k][1]
        assert float((forces - want).abs().max()) < tol_f * float(want.abs().max())
    ops.check_status()
