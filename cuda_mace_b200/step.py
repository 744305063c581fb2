"""The whole energy+force step of an ``InvariantMACE`` on the library's own sequence of kernels (cmace_step_run).

``StepPlan`` lays a model's constant weights out once: products of constant matrices that the model applies one after
the other are multiplied in float64 (embedding, linear_up, last radial layer, Linear and skip_tp of the first layer;
product and linear_up between the layers; product, skip connection and readout), the rest is packed for the tensor
cores.  ``energy_forces`` then runs the step: no autograd graph, one workspace, no synchronisation.  The model's
autograd path (``node_energies``) stays for what the sequence does not cover: ``covers`` says why.
"""
import ctypes
import math
import os

import torch

from . import _abi, ops

SILU_2MOM = 1.676532470331092   # normalisation of the activation, 1/sqrt(E[silu(x)^2]) for x ~ N(0,1)
_H = 64                         # hidden width of the radial perceptron


def _pack(Bt):
    B3 = Bt.reshape(-1, Bt.shape[-2], Bt.shape[-1]).contiguous()
    nmat, N, K = B3.shape
    out = torch.empty(int(_abi.call("cmace_gemm_packed_floats", nmat, N, K)), dtype=torch.float32, device=Bt.device)
    _abi.call("cmace_gemm_pack_weights_f32", B3.data_ptr(), nmat, N, K, out.data_ptr(), ops._stream())
    return out


def half_images(Wt, scale):
    """fp16 hi and lo images of Wt [N, K <= 64] * scale: rows of 64 fp16 with the tensor core's 128-byte swizzle."""
    N, K = Wt.shape
    w = torch.zeros(N, 64, dtype=torch.float32, device=Wt.device)
    w[:, :K] = Wt * scale
    hi = w.half()
    images = torch.stack([hi, (w - hi.float()).half()]).view(2, N, 8, 8)
    rows = torch.arange(N, device=Wt.device)[:, None]
    chunk = torch.arange(8, device=Wt.device)[None, :]
    out = torch.empty_like(images)
    out[:, rows, chunk ^ (rows & 7)] = images
    return out


def basis_bounds(nb, r_max, p):
    """Estimates of the largest |b_n| and |db_n/dr| of the radial basis on (0, r_max): sampled on a grid far finer than the n-th wave
    (32 points per nb = 16 half-wave), plus 5 %."""
    r = torch.arange(1, 4097, dtype=torch.float64) * (r_max / 4096)
    x = r / r_max
    f = 1 - 0.5 * (p + 1) * (p + 2) * x**p + p * (p + 2) * x**(p + 1) - 0.5 * p * (p + 1) * x**(p + 2)
    df = 0.5 * p * (p + 1) * (p + 2) * (-x**(p - 1) + 2 * x**p - x**(p + 1)) / r_max
    w = torch.arange(1, nb + 1, dtype=torch.float64)[:, None] * math.pi / r_max
    pref = math.sqrt(2.0 / r_max)
    b = pref * torch.sin(w * r) / r
    db = pref * (w * torch.cos(w * r) / r - torch.sin(w * r) / r**2)
    return (1.05 * (b * f).abs().amax(dim=1), 1.05 * (db * f + b * df).abs().amax(dim=1))


def half_scales(Ws, bounds):
    """The 13 powers of two of the fp16 radial kernel and the weights' factors, or None when a bound of some layer's
    values or derivatives exceeds 2^15 or a weight is not finite.  |silu(z)| <= |z| and |silu'| < 1.1 carry the bounds from
    layer to layer."""
    if not all(bool(W.isfinite().all()) for W in Ws):
        return None

    def power(t):   # the power of two that puts the largest entry just below 2^15
        return 14 - math.floor(math.log2(max(float(t.max()), 1e-30)))

    v, d = bounds
    sv, sd = power(v), power(d)
    out = [2.0**sv, 2.0**sd]
    z, a, t, factors = [], [], [], []
    for W in Ws:
        w = W.double().abs().cpu()
        sw = power(w) - 1
        v, d = v @ w, 1.1 * (d @ w)
        nv, nd = power(v), power(d)
        if min(nv, nd, sv, sd) < 0:
            return None
        # the split's absolute error, 2^-25, has to stay small beside small values too; 2^60 is far from float32's end
        nv, nd = min(nv, 60), min(nd, 60)
        z.append(2.0 ** -(sv + sw))
        a.append(2.0 ** (nv - sv - sw))
        t.append(2.0 ** (nd - sd - sw))
        factors.append(2.0**sw)
        sv, sd = nv, nd
    return out + z + a + t + [2.0**-sv, 2.0**-sd], factors


def fused_rows(C):
    """Column of W4 [64, 4 C] in every row of the fused message kernel's W^T (header, fused_w), -1 for a row of zeros."""
    blocks = {32: 1, 64: 2, 96: 4, 128: 4}[C]
    j, q, i = torch.meshgrid(torch.arange(blocks), torch.arange(4), torch.arange(32), indexing="ij")
    if C == 32:
        degree, channel = 3 - q, i
    else:
        degree = torch.where(q < 2, torch.where(2 * j < blocks, 3, 0), torch.where(2 * j < blocks, 1, 2))
        channel = 32 * (q & 1) + i if C == 64 else 64 * (q & 1) + 2 * i + (j & 1)
    return torch.where(channel < C, degree * C + channel, -1).reshape(-1)


def _expected_buffers(model):
    """(tensor, shape, dtype) of every buffer that a plan of `model` reads."""
    C, Z, T, D = model.channels, model.num_elements, model.dtype, torch.float64
    L0, L1 = model.layers
    out = [(model.atomic_energies, (Z,), D), (model.embedding, (Z, C), T), (L0.linear.weights, (Z, 4, C, C), T),
           (L0.W_readout, (C, 1), D), (L1.linear.weights, (4, C, C), T), (L1.W_sc, (C, Z * C), T),
           (L1.W_readout1, (C, 16), D), (L1.W_readout2, (16, 1), D)]
    for L in model.layers:
        con = L.contraction
        out += [(L.W_up, (C, C), T), (L.W_prod, (C, C), T), (con.weights_3, (1, Z, con.W3_L0_size, C), T),
                (con.weights_2, (1, Z, con.W2_L0_size, C), T), (con.weights_1, (1, Z, con.W1_L0_size, C), T)]
        if model.radial == "spline":
            intervals = model.layers[0].spline.coefficients.shape[0]
            out += [(L.spline.coefficients, (intervals, 4, 4 * C), T), (L.spline.r_knots, (intervals + 1,), T)]
        else:
            nb = model.edge_basis.num_bessel
            widths = (nb, _H, _H, _H, 4 * C)
            out += [(getattr(L, f"W_radial{i}"), widths[i:i + 2], T) for i in range(4)]
    return out


# what no plan reads: the tables that a contraction's own plan is made from once, transposes that only autograd uses
_UNREAD = ("U1_", "U2_", "U3_", "weights_transposed")


class _Stamp:
    """What a plan was made from: the tensors, submodules and plain attributes of a model, by identity, version or value.
    (Edits that autograd's version counter does not see, such as those through ``.data``, are not seen here either.)
    It holds the parts, not the model, which holds it: no cycle that would keep a model's memory until it is collected."""

    def __init__(self, model):
        modules = list(model.modules())
        self.tensors = [(d, k, t, t._version) for m in modules for d in (m._buffers, m._parameters)
                        for k, t in d.items() if t is not None and not k.endswith("_T") and not k.startswith(_UNREAD)]
        self.children = [(m._modules, tuple(m._modules.values())) for m in modules]
        plain = [(m.__dict__, k, v) for m in modules for k, v in m.__dict__.items()
                 if k[0] != "_" and k != "training" and isinstance(v, (bool, int, float, str, torch.dtype))]
        self.plain = [p for p in plain if p[0] is not model.__dict__]
        self.own = [p[1:] for p in plain if p[0] is model.__dict__]
        # hooks of the parts would not run: the model's own run around forward()
        self.hooks = [h for m in modules[1:] for h in (m._forward_hooks, m._forward_pre_hooks, m._backward_hooks,
                                                       m._backward_pre_hooks)]
        self.hooked = any(self.hooks)

    def current(self, model):
        for d, k, t, v in self.tensors:
            if d.get(k) is not t or t._version != v:
                return False
        for d, v in self.children:
            if tuple(d.values()) != v:
                return False
        for d, k, v in self.plain:
            if d.get(k) != v:
                return False
        d = model.__dict__
        for k, v in self.own:
            if d.get(k) != v:
                return False
        return any(self.hooks) == self.hooked


_PARTS = ("node_energies", "_messages", "_radial_weights", "_mm")   # what forward() is made of


def _is_standard(model):
    """Whether the model's parts are the package's own: a subclass or a replaced module computes something else."""
    from .model import InvariantMACE

    L0, L1 = model.layers
    parts = [(model.edge_basis, ops.EdgeBasis), (model.spherical_harmonics, ops.SphericalHarmonics),
             (model.tp, ops.InvariantMessagePassingTP), (L0.linear, ops.ElementalLinear), (L1.linear, ops.Linear)]
    parts += [(L.contraction, ops.SymmetricContraction) for L in model.layers]
    if model.radial == "spline":
        parts += [(L.spline, ops.CubicSpline) for L in model.layers]
    return (all(type(m) is kind for m, kind in parts)
            and all(getattr(type(model), k) is getattr(InvariantMACE, k) and k not in model.__dict__ for k in _PARTS))


def covers(model):
    """Whether the sequence covers a model: the standard two-layer architecture in float32 or float64, every buffer with
    the shape and type it was built with, on one device (kernels get plain pointers: a model that was converted or
    replaced in part afterwards is left to the operators and their checks)."""
    if model.radial not in ("exact", "spline") or len(model.layers) != 2 or model.num_elements > 16:
        return False
    if model.dtype not in (torch.float32, torch.float64) or model.channels not in (32, 64, 96, 128):
        return False
    if not _is_standard(model):
        return False
    if model.radial == "exact" and model.edge_basis.num_bessel not in (8, 16):
        return False
    for L in model.layers:
        if model.radial == "spline":
            first = model.layers[0].spline
            if L.spline.h != first.h or L.spline.rmax != first.rmax:
                return False
        elif L.n_radial != 4:
            return False
    dev = model.embedding.device
    return all(t.device == dev and t.dtype == dtype and tuple(t.shape) == shape
               for t, shape, dtype in _expected_buffers(model))


class StepPlan:
    """Folded and packed weights of one model, and the C description that points at them."""

    def __init__(self, model):
        self.keep = []
        self.recorded = False   # a graph that somebody else keeps reads this plan by address
        self.stamp = _Stamp(model)
        f32 = model.dtype == torch.float32
        C, Z = model.channels, model.num_elements
        L0, L1 = model.layers
        d = lambda t: t.double()
        self.device = model.embedding.device
        m = _abi.StepModel()
        m.is_f64, m.channels, m.elements = int(not f32), C, Z
        m.nbessel, m.cutoff_p = model.edge_basis.num_bessel, model.edge_basis.p
        m.r_max, m.scale, m.shift = model.edge_basis.r_max, model.scale, model.shift

        def hold(t):
            t = t.contiguous()
            self.keep.append(t)
            return t.data_ptr()

        def matrix(W):   # [.., K, N] in the layout the products want
            W = W.to(model.dtype)
            return hold(_pack(W.transpose(-1, -2)) if f32 else W)

        x = d(model.embedding) @ d(L0.W_up)                                  # [Z, C] sender features of the first layer
        lin = d(L0.linear.weights) / math.sqrt(C)                            # [Z, 4, C, C]
        if model.radial == "spline":
            for t, L in enumerate((L0, L1)):
                m.spline[t] = hold(L.spline.coefficients)
            m.spline_knots, m.sender_table = hold(L0.spline.r_knots), hold(x.to(model.dtype))
            m.spline_width, m.spline_rmax = L0.spline.h, L0.spline.rmax
            m.spline_intervals = L0.spline.coefficients.shape[0]
            m.fold, m.fold_back[0] = matrix(lin), matrix(lin.transpose(-1, -2))
        else:
            self._radial(model, m, hold, matrix, x, lin)
        lin = d(L1.linear.weights) / math.sqrt(C)
        m.linear[0], m.linear[1] = matrix(lin), matrix(lin.transpose(-1, -2))
        for t, L in enumerate((L0, L1)):
            con = L.contraction
            if con._plan is None:
                con._plan = ops.make_plan(con.u3_max_nonsparse, con.U3_num_nonsparse, con.U3_indices, con.U3_values,
                                          con.U2_num_nonsparse, con.U2_indices, con.U2_values, con.W3_L0_size,
                                          con.W2_L0_size, con.W1_L0_size)
            weff = torch.empty(Z, 13, C, dtype=model.dtype, device=x.device)
            weights = [w.contiguous() for w in (con.weights_3, con.weights_2, con.weights_1)]
            _abi.call("cmace_symcon_effective_weights", con._plan.handle, int(not f32), *[w.data_ptr() for w in weights],
                      Z, C, weff.data_ptr(), ops._stream())
            m.weff[t] = hold(weff)
        prod0, prod1, ro1 = d(L0.W_prod), d(L1.W_prod), d(L1.W_readout1)
        up = prod0 @ d(L1.W_up)
        m.up, m.up_back = hold(up.to(model.dtype)), hold(up.t().to(model.dtype))
        sc = d(L1.W_sc).view(C, Z, C).permute(1, 0, 2)                       # [Z, C, C]
        extra = torch.cat([prod0 @ sc @ ro1, (prod0 @ d(L0.W_readout)).expand(Z, C, 1)], dim=2)   # [Z, C, 17]
        extra = torch.nn.functional.pad(extra, (0, 3))   # whole groups of four
        m.extra = hold(extra.to(model.dtype))
        m.extra_back = hold(extra.transpose(1, 2).to(model.dtype))
        m.readout1 = hold((prod1 @ ro1).t().to(model.dtype))
        m.readout2 = hold(d(L1.W_readout2)[:, 0] * SILU_2MOM)
        m.atomic_energies = hold(model.atomic_energies)
        self.model = m
        self.channels, self.dtype, self.elements = C, model.dtype, Z

    @staticmethod
    def _radial(model, m, hold, matrix, x, lin):
        """Weights of the radial perceptrons, and the first layer's element-dependent product of their hidden layers."""
        d = lambda t: t.double()
        f32 = model.dtype == torch.float32
        C, Z = model.channels, model.num_elements
        L0, L1 = model.layers
        for t, L in enumerate((L0, L1)):
            for i in range(4):
                if (t, i) != (0, 3):
                    m.radial[t][i] = matrix(getattr(L, f"W_radial{i}"))
        if f32:
            bounds = basis_bounds(m.nbessel, m.r_max, m.cutoff_p)
            scales = [half_scales([getattr(L, f"W_radial{i}") for i in range(3)], bounds) for L in (L0, L1)]
            if None not in scales and bool(L1.W_radial3.isfinite().all()):
                for t, L in enumerate((L0, L1)):
                    values, factors = scales[t]
                    m.half_scales[t][:] = values
                    for i in range(3):
                        m.radial_half[t][i] = hold(half_images(getattr(L, f"W_radial{i}").t(), factors[i]))
                w4 = torch.nn.functional.pad(L1.W_radial3.t(), (0, 0, 0, 1))   # row -1: zeros
                w = w4[fused_rows(C).to(w4.device)]
                scale = 2.0 ** (13 - math.floor(math.log2(max(float(w.abs().max()), 1e-30))))
                w = w * scale
                hi = w.half()
                m.fused_w = hold(torch.cat([hi, (w - hi.float()).half()], dim=1))
                m.fused_scale = 1.0 / scale
                m.fused_layout = _abi.FUSED_LAYOUT if C == 128 else _abi.FUSED_LAYOUT_NARROW
                # [step of 16 channels, (l, j, t, i), k]: row 8 j + 2 t + i of a degree is channel 4 t + 2 j + i of the step
                steps = C // 16
                wt = L1.W_radial3.t().reshape(4, steps, 4, 2, 2, _H).permute(1, 0, 3, 2, 4, 5).reshape(steps, 64, _H)
                m.fused_w_back = hold(torch.stack([half_images(b, scale) for b in wt]))
            m.radial_back = matrix(L1.W_radial3.t())
        w4 = d(L0.W_radial3).view(_H, 4, C)
        fold = torch.einsum("zc,klc,rlcd->rlzkd", x, w4, lin).reshape(Z, 4, Z * _H, C)
        m.fold = matrix(fold)
        blocks = [fold[:, :, 2 * b * _H: min(2 * b + 2, Z) * _H].transpose(-1, -2) for b in range((Z + 1) // 2)]
        if model.dtype == torch.float32 and Z >= 4:   # the blocks of two elements one after the other: one launch takes them
            m.fold_back[0] = matrix(torch.stack(blocks[:Z // 2]))
            first = Z // 2
        else:
            first = 0
        for b in range(first, (Z + 1) // 2):
            m.fold_back[b] = matrix(blocks[b])

    def current(self, model):
        return self.stamp.current(model)


def plan_of(model):
    """The model's plan, laid out again when the model has changed; None when the sequence does not cover the model, or
    the module-level switches of ops or the environment select other kernels.

    A plan is finished before anybody sees it and goes when nobody reads it any more, so that any stream may use it without
    an event: one synchronisation per set of weights.  While a stream is captured nothing is laid out (the kernels would be
    recorded, not run): such a step takes the operators."""
    if not ops.USE_TENSOR_CORES or ops.FUSED_RADIAL_MESSAGE_PASSING or not ops.RADIAL_GRADIENT_ON_THE_FLY:
        return None
    if os.environ.get("CMACE_SYMCON_GENERIC", "")[:1] == "1":
        return None
    stamp, plan = model.__dict__.get("_step_plan", (None, None))
    if stamp is not None and stamp.current(model):
        return plan
    dev = model.embedding.device
    if dev.type != "cuda" or dev.index != torch.cuda.current_device():
        return None   # the operators refuse such a call
    if torch.cuda.is_current_stream_capturing():
        return None
    before, plan = plan, None
    stamp = _Stamp(model)
    if not stamp.hooked and covers(model):
        try:
            with torch.no_grad():
                plan = StepPlan(model)
            stamp = plan.stamp
            torch.cuda.current_stream(dev).synchronize()
        except RuntimeError as e:
            if "not the generated program" not in str(e):
                raise
    model.__dict__["_step_plan"] = (stamp, plan)
    if before is not None:
        if before.recorded:
            model.__dict__.setdefault("_step_recorded", []).append(before)
        else:
            torch.cuda.synchronize(dev)   # steps on other streams may still read it
    return plan


# Z beyond a + b edges / atom: the operators are faster, {is_f64: {channels: (a, b)}}
_MANY_ELEMENTS = {False: {32: (2.35, 0.365), 64: (2.5, 0.58), 96: (6.3, 0.49), 128: (5.7, 0.72)},
                  True: {32: (1.05, 0.55), 64: (1.55, 0.65), 96: (2.3, 0.6), 128: (3.2, 0.675)}}


def pays(plan, atoms, edges, recorded=False):
    """Whether the sequence is the faster way for a system of this size; `recorded`: in a replayed graph.

    The first layer's sums and the products on them take 64 Z columns an atom whatever its edges are, the operators 4 C
    radial weights an edge.  Native against operators, ms, one B200, float32, 100 000 atoms of 10 edges: 32 channels 4.45; 4.43
    at 6 elements, 64 6.20; 6.32 at 8 and 7.11; 6.30 at 10, 96 9.86; 9.45 at 12, 128 11.74; 11.68 at 13 (of 5 edges 8.90; 8.51 at 10);
    50 000 atoms of 21 edges: 32 channels 3.87; 3.65 at 11, 64 5.04; 5.20 at 14 and 5.57; 5.22 at 16, 96 6.68; 6.90 at 16.  float64,
    30 000 atoms of 10 edges: 32 channels 3.61; 4.21 at 5 and 4.42; 4.24 at 7, 64 5.91; 5.94 at 8, 96 8.55; 8.75 at 8 and 9.80; 8.87 at
    10, 128 11.24; 11.17 at 10; 15 000 atoms of 21 edges: 32 4.10; 3.99 at 13, 64 5.43; 5.47 at 15, 96 7.65; 7.62 at 15, 128 9.02; 9.49
    at 16.  The lines are where both take the same; a condensed system (52 edges) stays native at any number of elements.  The
    operators' launches take the host 2.1 ms, which small systems never need natively (20 000 atoms of 10 edges, 16 elements, float32, 32 channels: 1.98;
    2.07); recorded, both take the same at 3 000 atoms of 16 elements in float32 (0.39; 0.40) and 1 000 in float64."""
    m = plan.model
    if plan.elements <= 4 or m.spline[0]:
        return True
    a, b = _MANY_ELEMENTS[bool(m.is_f64)][plan.channels]
    if plan.elements <= a + b * edges / atoms:
        return True
    least = 100_000 if m.is_f64 else 320_000
    if recorded:
        least //= 6
    return atoms * plan.elements < least


def takes(positions, shifts):
    """Inputs the sequence takes: float64 positions (at least one) and shifts, or (index, table), on the device."""
    if isinstance(shifts, tuple):
        index, shifts = shifts
        if not (index.is_cuda and index.dtype == torch.uint8):
            return False
    return (positions.is_cuda and positions.dtype == torch.float64 and positions.shape[0] > 0 and shifts.is_cuda
            and shifts.dtype == torch.float64)


_FIRST_EXCHANGE, _SENDERS, _SECOND_EXCHANGE, _END = 6, 13, 14, 19
_BESIDE_EDGES = 32768
_side_streams = {}


def _side_stream(device):
    stream = _side_streams.get(device.index)
    if stream is None:
        stream = _side_streams.setdefault(device.index, torch.cuda.Stream(device=device))
    return stream


def energy_forces(plan, positions, species, one_hot, shifts, topology, halo=None):
    """(sums [3], interaction [n_owned], node_energy [n_owned], forces): sums = (total energy, interaction energy,
    0 unless a kernel recorded a failure: check_status() tells which).

    shifts: [E, 3] float64, or (index [E] uint8, table [rows, 3] float64).  positions [n_local, 3] float64, species
    [n_local] int32 or one_hot [n_local, Z] float32 or float64.  `halo` (a HaloPlan of more than one rank) fills and
    returns the ghost rows between the ranges of steps; forces are then those of the owned atoms.

    The kernels get plain pointers, so devices, sizes and types are checked here, before the first launch."""
    index = None
    if isinstance(shifts, tuple):
        index, shifts = shifts[0].contiguous(), shifts[1]
    ops._check_cuda(positions, shifts, index, species, one_hot, topology.sender)
    positions, shifts = positions.contiguous(), shifts.contiguous()
    n, nl, E = topology.nnodes, topology.nsenders, topology.nedges
    dev = positions.device
    if plan.device != dev:
        raise RuntimeError(f"the model is on {plan.device}, the positions are on {dev}")
    if species is not None:
        species = species.contiguous()
        if species.dtype != torch.int32 or species.shape != (nl,):
            raise RuntimeError(f"species must be int32 [{nl}], got {species.dtype} {tuple(species.shape)}")
    else:
        one_hot = one_hot.contiguous()
        if one_hot.dtype not in (torch.float32, torch.float64) or one_hot.shape != (nl, plan.elements):
            raise RuntimeError(f"node attributes must be float32 or float64 [{nl}, {plan.elements}], got "
                               f"{one_hot.dtype} {tuple(one_hot.shape)}")
    if positions.shape != (nl, 3) or shifts.shape[1:] != (3,) or (shifts if index is None else index).shape[0] != E:
        raise RuntimeError(f"shape mismatch: positions {tuple(positions.shape)}, shifts {tuple(shifts.shape)} for "
                           f"{nl} atoms and {E} edges")
    capturing = torch.cuda.is_current_stream_capturing()
    plan.recorded = plan.recorded or capturing
    # results of their own: a program that keeps an energy or saves the forces does not keep the rest with them
    new = dict(dtype=torch.float64, device=dev)
    sums, interaction, node_energy, forces = (torch.empty(k, **new) for k in (3, n, n, (nl, 3)))
    m = plan.model
    nbytes = _abi.call("cmace_step_workspace_bytes", ctypes.byref(m), n, nl, E)
    workspace = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    # A new list's grouping by sender is first read two thirds into the step: beside the steps before, once it takes
    # longer (40 us at 160 000 edges) than the second stream costs the host (about 15 us).  Its launches come after those
    # of the first two steps, which keep the device busy meanwhile.
    beside = buffers = ready = None
    if topology._perm is None and E >= _BESIDE_EDGES and not capturing:
        beside = _side_stream(dev)
        buffers = topology.grouping_buffers()
        perm, send_ptr, _ = buffers
        ready = torch.cuda.current_stream(dev).record_event()
    else:
        perm, send_ptr = topology.sender_order()
    io = _abi.StepIO()
    io.n_owned, io.n_local, io.nedges = n, nl, E
    io.positions = positions.data_ptr()
    if index is None:
        io.shifts = shifts.data_ptr()
    else:
        io.shift_index, io.shift_table, io.shift_rows = index.data_ptr(), shifts.data_ptr(), shifts.shape[0]
    if species is not None:
        io.species = species.data_ptr()
    else:
        io.one_hot, io.one_hot_is_f64 = one_hot.data_ptr(), int(one_hot.dtype == torch.float64)
    io.sender, io.receiver, io.row_ptr = topology.sender.data_ptr(), topology.receiver.data_ptr(), topology.row_ptr.data_ptr()
    io.perm, io.send_ptr = perm.data_ptr(), send_ptr.data_ptr()
    io.workspace, io.workspace_bytes = workspace.data_ptr(), nbytes
    io.status = ops._status_tensor(dev).data_ptr()
    io.sums, io.interaction, io.node_energy, io.gradient = [t.data_ptr() for t in (sums, interaction, node_energy, forces)]
    io.gradient_sign = -1.0
    st = ops._stream()

    def run(first, last):
        nonlocal ready
        if ready is not None:
            _abi.run_steps(m, io, first, 2, st)
            first = 2
            beside.wait_event(ready)
            ready = None
            topology.group_senders(buffers, beside.cuda_stream)
        if beside is not None and last > _SENDERS:
            if first < _SENDERS:
                _abi.run_steps(m, io, first, _SENDERS, st)
                first = _SENDERS
            join()
        _abi.run_steps(m, io, first, last, st)

    def join():
        nonlocal beside
        torch.cuda.current_stream(dev).wait_stream(beside)
        beside = None
        if ready is None:
            topology.grouped(perm, send_ptr)

    try:
        forces = _run_ranges(run, plan, n, nl, io, halo, forces)
    finally:
        if beside is not None:   # a failed step: the grouping still owns its memory
            join()
    return sums, interaction, node_energy, forces


def _run_ranges(run, plan, n, nl, io, halo, forces):
    if halo is None:
        run(0, _END)
        return forces
    feats = dict(dtype=plan.dtype, device=forces.device)
    up = torch.empty(n, plan.channels, **feats)
    gup = torch.empty(nl, plan.channels, **feats)
    # the ghost-row pointers are set before the first range: the call checks them together
    io.up_local, io.gup_local, io.gup_owned = up.data_ptr(), gup.data_ptr(), gup.data_ptr()
    run(0, _FIRST_EXCHANGE)
    up_local = halo.forward_fill(up)
    io.up_local = up_local.data_ptr()
    run(_FIRST_EXCHANGE, _SECOND_EXCHANGE)
    gup_owned = halo.backward_reduce(gup)
    io.gup_owned = gup_owned.data_ptr()
    run(_SECOND_EXCHANGE, _END)
    return halo.backward_reduce(forces)
