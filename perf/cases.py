"""Performance cases of fasteq_b200: what its users have it do, through the public entry points.

Four kinds of work, over the range of sizes, types and directions they are used at:

* ``tp``     the ChannelwiseTensorProduct operator (gather + uvu product + scatter) through ``fast_uniform1d_jit``,
             alone (inference) or with the gradients of weights, features and edge attributes;
* ``mace``   the MACE-style model: energies and forces on a given neighbour list (``forces``), with the neighbour list
             rebuilt from the positions on every step (``rebuild``, a molecular-dynamics step), replayed from a CUDA graph
             between rebuilds (``replay``), and a force-matching training step with weight gradients (``train``);
* ``nequip`` the NequIP-style gated network on one periodic cell, energy and forces;
* ``stc`` / ``linear``  SymmetricContraction and SO3Linear alone, forward and backward with weight gradients.

``listed()`` names twelve of them; ``draw`` spreads sizes over the same ranges.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from fasteq_b200 import descriptors
from fasteq_b200.irreps import Irreps
from fasteq_b200.neighbors import radius_graph
from fasteq_b200.nn.graphed import GraphedEnergyForces
from fasteq_b200.nn.mace_style import MACEStyleModel
from fasteq_b200.nn.nequip_style import NequIPStyleModel
from fasteq_b200.ops import fast_equi_linear, fast_stc_uniform1d_jit, fast_uniform1d_jit

DEV = "cuda"
DTYPE = {"f32": torch.float32, "f64": torch.float64}
DENSITY = 0.1          # atoms per cubic Angstrom of the benchmark structures
MACE_CUTOFF, NEQUIP_CUTOFF = 5.0, 4.0
NEQUIP_SIDE_OF_20000 = 58.5
# ChannelwiseTensorProduct signatures (irreps_in1, SH lmax, lmax_out) and the types each is used in
SIGNATURES = [("128x0e+128x1o+128x2e", 3, 3, ("f32", "f64")), ("128x0e+128x1o", 3, 3, ("f32",)), ("64x0e+64x1o", 3, 3, ("f32", "f64")),
              ("32x0e+32x1o", 2, 2, ("f32", "f64")), ("33x0e+33x1o", 2, 2, ("f32",))]
MAX_TP_WEIGHTS = 644_552 * 13 * 128          # per-edge weight values of the largest listed tensor product
MID, HIDDEN = "128x0e+128x1o+128x2e+128x3o", "128x0e+128x1o"


def listed():
    return [
        # one small graph through the widest standard interaction, inference only (benchmark configuration 0): launch latency
        dict(name="tp_small_forward", kind="tp", in1=SIGNATURES[0][0], sh=3, lout=3, dtype="f32", nodes=512, edges=4096, sorted=True, grad=False),
        # the interaction of a 64-structure batch with every gradient (benchmark configuration 1, bench.py's default workload)
        dict(name="tp_batch_gradients", kind="tp", in1=SIGNATURES[1][0], sh=3, lout=3, dtype="f32", nodes=12_288, edges=644_552, sorted=True, grad=True),
        # a mid-size graph of odd extents whose edge list is not receiver-sorted, as NequIP-type data loaders emit it
        dict(name="tp_unsorted_gradients", kind="tp", in1=SIGNATURES[2][0], sh=3, lout=3, dtype="f32", nodes=3_001, edges=80_533, sorted=False, grad=True),
        # molecular dynamics of one small cell: neighbour list rebuilt and forces evaluated every step (latency bound)
        dict(name="mace_one_cell_rebuild", kind="mace", mode="rebuild", dtype="f32", structs=1, atoms_min=192, atoms_max=192),
        # the same cell between rebuilds, replayed from a CUDA graph
        dict(name="mace_one_cell_replay", kind="mace", mode="replay", dtype="f32", structs=1, atoms_min=192, atoms_max=192),
        # a batch of 64 structures on given neighbour lists (benchmark configuration 1)
        dict(name="mace_batch_forces", kind="mace", mode="forces", dtype="f32", structs=64, atoms_min=192, atoms_max=192),
        # screening: ragged batch with neighbour lists built on the way (a group of benchmark configuration 4)
        dict(name="mace_ragged_rebuild", kind="mace", mode="rebuild", dtype="f32", structs=128, atoms_min=32, atoms_max=256),
        # the large FP64 model (benchmark configuration 2)
        dict(name="mace_fp64_forces", kind="mace", mode="forces", dtype="f64", structs=32, atoms_min=384, atoms_max=384),
        # force-matching training step on a usual batch of eight structures
        dict(name="mace_train_step", kind="mace", mode="train", dtype="f32", structs=8, atoms_min=192, atoms_max=192),
        # one large periodic cell through the NequIP-style network (benchmark configuration 3)
        dict(name="nequip_large_cell", kind="nequip", atoms=20_000),
        # the product basis alone on 200,000 nodes of ten species, with weight gradients (benchmark configuration 4)
        dict(name="stc_200k_gradients", kind="stc", nodes=200_000, species=10),
        # the channel mix after the tensor product of configuration 1, with weight gradients
        dict(name="linear_after_tp_gradients", kind="linear", nodes=12_288),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tp", "tp", "tp", "mace", "mace", "mace", "mace", "nequip", "stc", "linear"])
    if kind == "tp":
        in1, sh, lout, dtypes = rng.choice(SIGNATURES)
        dtype = rng.choice(dtypes)
        d = _tp_descriptor(in1, sh, lout)
        most = MAX_TP_WEIGHTS // (d.w_seg_num * d.u_dim * (2 if dtype == "f64" else 1))
        nodes = _log_int(rng, 64, 20_000)
        edges = min(most, int(nodes * rng.uniform(4.0, 60.0)))
        return dict(kind="tp", in1=in1, sh=sh, lout=lout, dtype=dtype, nodes=nodes, edges=edges, sorted=rng.random() < 0.7, grad=rng.random() < 0.6)
    if kind == "mace":
        mode = rng.choice(["forces", "rebuild", "replay", "train"])
        dtype = "f64" if mode != "train" and rng.random() < 0.2 else "f32"
        structs = _log_int(rng, 1, {"train": 16, "f64": 16}.get(mode if mode == "train" else dtype, 96))
        lo = rng.randint(32, 256)
        return dict(kind="mace", mode=mode, dtype=dtype, structs=structs, atoms_min=lo, atoms_max=rng.randint(lo, 256))
    if kind == "nequip":
        return dict(kind="nequip", atoms=_log_int(rng, 300, 20_000))
    if kind == "stc":
        return dict(kind="stc", nodes=_log_int(rng, 100, 200_000), species=rng.randint(1, 10))
    return dict(kind="linear", nodes=_log_int(rng, 100, 20_000))


# ------------------------------------------------------------------------------------------------ inputs

@functools.lru_cache(maxsize=None)
def _tp_descriptor(in1, sh, lout):
    irreps_sh = Irreps.spherical_harmonics(sh)
    io, ins = descriptors.full_channelwise_instructions(in1, irreps_sh, lout)
    return descriptors.channelwise_tensor_product(in1, irreps_sh, io, ins)


@functools.lru_cache(maxsize=None)
def _stc_descriptor():
    return descriptors.symmetric_contraction(MID, HIDDEN)


@functools.lru_cache(maxsize=None)
def _linear_descriptor():
    irr_tp, _ = descriptors.full_channelwise_instructions(HIDDEN, Irreps.spherical_harmonics(3), 3)
    return descriptors.linear(irr_tp, MID), irr_tp.dim


def _randn(shape, dtype, g):
    return torch.randn(shape, generator=g, dtype=dtype, device=DEV)


def _structures(case, seed):
    """Positions (float64, wrapped), species, structure ids and cubic box lengths of a batch of periodic structures.
    The atom counts belong to the case (a batch of the same extents), everything else follows from the seed."""
    atoms = np.random.default_rng([case["structs"], case["atoms_min"], case["atoms_max"]]).integers(
        case["atoms_min"], case["atoms_max"] + 1, size=case["structs"])
    rng = np.random.default_rng(seed)
    side = (atoms / DENSITY) ** (1.0 / 3.0)
    ids = np.repeat(np.arange(case["structs"]), atoms)
    pos = rng.uniform(0.0, 1.0, size=(ids.size, 3)) * side[ids][:, None]
    t = lambda a: torch.from_numpy(a).to(DEV)
    return t(pos), t(rng.integers(0, 4, size=ids.size)), t(ids), side


def _mace_kwargs(case):
    return dict(channels=256, hidden_lmax=2) if case["dtype"] == "f64" else {}


def _model(cls, seed, dtype, trainable, **kw):
    """A random-weight model whose weights follow from the seed (drawn on the host, then moved)."""
    with torch.random.fork_rng(devices=[]):
        torch.manual_seed(seed)
        model = cls(**kw)
    model = model.to(device=DEV, dtype=dtype)
    for p in model.parameters():
        p.requires_grad_(trainable)
    return model


def prepare(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    if case["kind"] == "tp":
        d, dt = _tp_descriptor(case["in1"], case["sh"], case["lout"]), DTYPE[case["dtype"]]
        N, E, U = case["nodes"], case["edges"], d.u_dim
        src = torch.randint(0, N, (E,), generator=g, device=DEV, dtype=torch.int32)
        dst = torch.randint(0, N, (E,), generator=g, device=DEV, dtype=torch.int32)
        if case["sorted"]:
            dst = torch.sort(dst).values
        w, x, y = (_randn(s, dt, g) for s in ((E, d.w_seg_num * U), (N, d.x_seg_num * U), (E, d.y_seg_num)))
        state = dict(kind="tp", w=w, x=x, y=y, src={1: src}, dst={0: dst}, meta=d.meta(dt, DEV), cot=None)
        if case["grad"]:
            for t in (w, x, y):
                t.requires_grad_(True)
            state["cot"] = _randn((N, d.out_seg_num * U), dt, g)
        return state
    if case["kind"] == "mace":
        dt = DTYPE[case["dtype"]]
        pos, species, ids, side = _structures(case, seed)
        model = _model(MACEStyleModel, seed, dt, case["mode"] == "train", **_mace_kwargs(case))
        if case["mode"] == "rebuild":
            return dict(kind="rebuild", model=model, pos=pos, species=species, ids=ids, box=side, structs=case["structs"], dtype=dt)
        rg = radius_graph(pos, ids, side, MACE_CUTOFF, register_plan=False)
        args = (species, rg.edge_src, rg.edge_dst, rg.edge_shift.to(dt), ids, case["structs"])
        pos = pos.to(dt)
        if case["mode"] == "replay":
            return dict(kind="replay", step=GraphedEnergyForces(model, pos, *args), pos=pos)
        state = dict(kind=case["mode"], model=model, pos=pos, args=args)
        if case["mode"] == "train":
            state["params"] = list(model.parameters())
            state["energy"], state["forces"] = _randn((case["structs"],), dt, g), _randn(tuple(pos.shape), dt, g)
            state["per_structure"] = torch.bincount(ids, minlength=case["structs"]).to(dt)
        return state
    if case["kind"] == "nequip":
        n = case["atoms"]
        side = NEQUIP_SIDE_OF_20000 * (n / 20_000) ** (1.0 / 3.0)
        rng = np.random.default_rng(seed)
        pos = rng.uniform(0.0, side, size=(n, 3))
        ncell = max(1, int(side // NEQUIP_CUTOFF))
        cell = np.minimum((pos / (side / ncell)).astype(np.int64), ncell - 1)
        pos = torch.from_numpy(pos[np.lexsort((cell[:, 2], cell[:, 1], cell[:, 0]))]).to(DEV)
        rg = radius_graph(pos, torch.zeros(n, dtype=torch.int32, device=DEV), np.array([side]), NEQUIP_CUTOFF, register_plan=False)
        species = torch.randint(0, 2, (n,), generator=g, device=DEV)
        model = _model(NequIPStyleModel, seed, torch.float32, False)
        return dict(kind="forces", model=model, pos=pos.float(), args=(species, rg.edge_src, rg.edge_dst, rg.edge_shift.float()))
    if case["kind"] == "stc":
        d, B = _stc_descriptor(), case["nodes"]
        x1 = (_randn((B, d.x1_segs, d.u_dim), torch.float32, g) * 0.3).requires_grad_(True)
        x0 = (_randn((case["species"], d.x0_segs, d.u_dim), torch.float32, g) * 0.1).requires_grad_(True)
        i0 = torch.randint(0, case["species"], (B,), generator=g, device=DEV)
        return dict(kind="stc", x1=x1, x0=x0, i0=i0, tables=d.tensors(torch.float32, DEV), segs=d.out_segs,
                    cot=_randn((B, d.out_segs * d.u_dim), torch.float32, g))
    d, dim = _linear_descriptor()
    return dict(kind="linear", d=d, x=_randn((case["nodes"], dim), torch.float32, g).requires_grad_(True),
                w=_randn((d.num_weights,), torch.float32, g).requires_grad_(True), cot=_randn((case["nodes"], Irreps(MID).dim), torch.float32, g))


def run(s):
    kind = s["kind"]
    if kind == "tp":
        out = fast_uniform1d_jit(s["w"], s["x"], s["y"], s["src"], s["dst"], s["meta"])
        if s["cot"] is None:
            return out
        return (out.detach(),) + torch.autograd.grad(out, (s["w"], s["x"], s["y"]), s["cot"])
    if kind == "forces":
        return s["model"](s["pos"], *s["args"])
    if kind == "rebuild":
        rg = radius_graph(s["pos"], s["ids"], s["box"], MACE_CUTOFF)
        return s["model"](s["pos"].to(s["dtype"]), s["species"], rg.edge_src, rg.edge_dst, rg.edge_shift.to(s["dtype"]), s["ids"], s["structs"])
    if kind == "replay":
        return s["step"](s["pos"])
    if kind == "train":
        out = s["model"](s["pos"], *s["args"], create_graph=True)
        loss = (((out["energy"] - s["energy"]) / s["per_structure"]) ** 2).mean() + ((out["forces"] - s["forces"]) ** 2).mean()
        return [loss.detach()] + list(torch.autograd.grad(loss, s["params"]))
    if kind == "stc":
        out = fast_stc_uniform1d_jit(s["x1"], s["x0"], s["i0"], *s["tables"], s["segs"])
        return (out.detach(),) + torch.autograd.grad(out, (s["x1"], s["x0"]), s["cot"])
    out = fast_equi_linear(s["d"], s["w"], s["x"])
    return (out.detach(),) + torch.autograd.grad(out, (s["x"], s["w"]), s["cot"])


# ------------------------------------------------------------------------------------------------ work and tolerance

@functools.lru_cache(maxsize=None)
def _layer_terms(kind, dtype):
    """Per layer of a model: (tensor-product paths, weight segments, channels, weights and rows-by-weights of its SO3Linears,
    product-basis paths); and the widths of its radial network."""
    model = MACEStyleModel(**_mace_kwargs(dict(dtype=dtype))) if kind == "mace" else NequIPStyleModel()
    layers = []
    for layer in model.layers:
        d = layer.conv_tp.descriptor
        linears = [m for m in layer.modules() if hasattr(m, "output_scale")]
        node = sum(m.irreps_out.uniform_mul() * m.irreps_in.uniform_mul() * sum(p.rows for p in _linear_rows(m.descriptor)) for m in linears)
        stc = layer.product.descriptor.num_paths if kind == "mace" else 0
        widths = [lin.in_features for lin in layer.radial.layers] + [layer.radial.layers[-1].out_features]
        layers.append((len(d.i_list), d.w_seg_num, d.u_dim, node, stc, tuple(widths)))
    return layers, sum(p.numel() for p in model.parameters())


class _Rows:
    def __init__(self, rows):
        self.rows = rows


def _linear_rows(d):
    """Irrep rows (2l + 1) that each path of an SO3Linear multiplies."""
    segs = d.operands[1].segments if hasattr(d.operands[1], "segments") else d.operands[1]
    return [_Rows(int(segs[p.indices[1]][0])) for p in d.paths]


def work(case):
    """What a pass cannot do without: inputs read once, results written once; two operations for every multiply-add of the
    path tables and dense products, three times as many with one set of gradients, six times in a force-matching step."""
    if case["kind"] == "tp":
        d, e = _tp_descriptor(case["in1"], case["sh"], case["lout"]), 8 if case["dtype"] == "f64" else 4
        N, E, U = case["nodes"], case["edges"], d.u_dim
        w, x, y, o = E * d.w_seg_num * U, N * d.x_seg_num * U, E * d.y_seg_num, N * d.out_seg_num * U
        flops = 2.0 * len(d.i_list) * E * U
        if not case["grad"]:
            return {"bytes": float(e * (w + x + y + o) + 8 * E), "flops": flops}
        return {"bytes": float(e * (2 * (w + x + y) + 2 * o) + 8 * E), "flops": 3 * flops}
    if case["kind"] in ("mace", "nequip"):
        dtype = case.get("dtype", "f32")
        e = 8 if dtype == "f64" else 4
        layers, n_params = _layer_terms(case["kind"], dtype)
        if case["kind"] == "mace":
            N = case["structs"] * (case["atoms_min"] + case["atoms_max"]) // 2
            E = N * DENSITY * 4.0 / 3.0 * math.pi * MACE_CUTOFF ** 3
        else:
            N = case["atoms"]
            E = N * 20_000 / NEQUIP_SIDE_OF_20000 ** 3 * 4.0 / 3.0 * math.pi * NEQUIP_CUTOFF ** 3
        flops = 0.0
        for paths, w_segs, U, node, stc, widths in layers:
            flops += 2.0 * (E * (paths * U + sum(a * b for a, b in zip(widths[:-1], widths[1:]))) + N * (node + stc * U))
        train = case.get("mode") == "train"
        return {"bytes": float(E * (8 + 3 * e) + N * (6 * e + 16) + n_params * e * (2 if train else 1)), "flops": flops * (6 if train else 3)}
    if case["kind"] == "stc":
        d, B = _stc_descriptor(), case["nodes"]
        b = 4.0 * B * d.u_dim * (2 * d.x1_segs + 2 * d.out_segs) + 8 * B + 8.0 * case["species"] * d.x0_segs * d.u_dim
        return {"bytes": b, "flops": 3 * 2.0 * d.num_paths * B * d.u_dim}
    d, dim = _linear_descriptor()
    rows = sum(p.rows for p in _linear_rows(d))
    return {"bytes": 4.0 * case["nodes"] * (2 * dim + 2 * Irreps(MID).dim) + 8.0 * d.num_weights, "flops": 3 * 2.0 * case["nodes"] * rows * 128 * 128}


def tolerance(case):
    """About four times the largest difference seen between the FP32 path and the same path evaluated in FP64 (SO3Linear and
    the radial network multiply in 3xTF32; a batch's energies are sums of node energies of both signs); for FP64 a hundred
    units of its round-off."""
    if case.get("dtype") == "f64":
        return {"rel": 1e-13, "max": 1e-12} if case["kind"] == "mace" else {"rel": 5e-15, "max": 5e-14}
    return {"tp": {"rel": 6e-7, "max": 6e-6}, "mace": {"rel": 5e-5, "max": 2.5e-4}, "nequip": {"rel": 2.5e-5, "max": 1e-4},
            "stc": {"rel": 1e-5, "max": 1e-4}, "linear": {"rel": 4e-6, "max": 2e-5}}[case["kind"]]
