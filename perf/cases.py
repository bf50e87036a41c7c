"""Performance cases of the library: the calls a user's program makes, through the public modules, over the
range of sizes, layouts and options that such programs use.

A case is a dict of plain values: ``kind`` selects the call, the other entries its size and options.

* ``md``           one step of a molecular-dynamics loop: neighbour list of the moved atoms, interaction block, forces
                   (box at 0.05 atoms per cubic Angstrom, 5 Angstrom cutoff, about 26 neighbours per atom)
* ``train``        one training step of a hidden interaction block on a stored graph: output, gradients of all
                   parameters and of the node features
* ``conv``         the fused convolution with given per-edge weights: destination-sorted edges or an unsorted edge
                   list through ``perm``, inference or with the gradients of weights, edge vectors and features
* ``sh``           spherical harmonics of edge vectors, alone or with the gradient w.r.t. the vectors
* ``tp``           fully connected tensor product, inference or with the gradients of both operands and the weights
* ``tp_linear``    fully connected tensor product followed by a Linear as one module, inference
* ``node_update``  Linear followed by Gate on node features, inference or with gradients
* ``csr``          destination sort of an edge list
"""
import math

import torch

import e3nn_b200
from e3nn_b200 import layouts, nn, o3

DENSITY, CUTOFF = 0.05, 5.0
BLOCK_IRREPS = "64x0e+64x1o+64x2e+64x3o"
TP_LAYOUTS = {
    "l2_32": ("32x0e+32x1o+32x2e", "1x0e+1x1o+1x2e", "32x0e+32x1o+32x2e"),
    "l3_mixed": ("128x0e+64x1o+32x2e", "0e+1o+2e+3o", "128x0e+64x1o+32x2e"),
}
CONV_LAYOUTS = ("cfg3_11", "cfg3_15", "cfg5_23")     # 11 and 15 paths up to l = 2, 23 paths up to l = 3


def listed():
    return [
        # a small molecule or unit cell: every launch is short, the step is latency
        {"name": "md_256", "kind": "md", "atoms": 256},
        # a solvated molecule, an odd number of atoms
        {"name": "md_4k", "kind": "md", "atoms": 4001},
        # a large simulation cell on one GPU
        {"name": "md_262k", "kind": "md", "atoms": 262144},
        # a minibatch of small molecules
        {"name": "train_600", "kind": "train", "atoms": 603},
        # a minibatch of periodic cells
        {"name": "train_16k", "kind": "train", "atoms": 16384},
        # message passing in inference on a large random graph, edges sorted once
        {"name": "conv_l2_2m", "kind": "conv", "layout": "cfg3_15", "nodes": 65536, "edges": 2097152, "sorted": True, "grad": False},
        # training on an edge list as it comes from a graph library (unsorted), through csr_from_dst's perm
        {"name": "conv_perm_150k", "kind": "conv", "layout": "cfg3_11", "nodes": 10007, "edges": 150001, "sorted": False, "grad": True},
        # angular embedding of the edges of one large batch, with its gradient
        {"name": "sh_1m", "kind": "sh", "vectors": 1000003, "lmax": 3, "grad": True},
        # fully connected product of a training step at the default arithmetic
        {"name": "tp_10k", "kind": "tp", "layout": "l2_32", "rows": 10000, "mode": "fp32", "grad": True},
        # the same product followed by the channel mixing on tensor cores, a large batch in inference
        {"name": "tp_linear_1m", "kind": "tp_linear", "layout": "l3_mixed", "rows": 1048576, "mode": "tf32"},
        # node update of a hidden layer in training at the default arithmetic
        {"name": "node_update_20k", "kind": "node_update", "rows": 20011, "mode": "fp32", "grad": True},
        # sorting the edges of a large graph
        {"name": "csr_2m", "kind": "csr", "nodes": 65536, "edges": 2097152},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["md", "train", "conv", "sh", "tp", "tp_linear", "node_update", "csr"])
    if kind == "md":
        return {"kind": kind, "atoms": _log_int(rng, 200, 200_000)}
    if kind == "train":
        return {"kind": kind, "atoms": _log_int(rng, 200, 20_000)}
    if kind == "conv":
        grad = rng.random() < 0.5
        edges = _log_int(rng, 2_000, 600_000 if grad else 2_000_000)
        return {"kind": kind, "layout": rng.choice(CONV_LAYOUTS), "nodes": max(64, int(edges / rng.uniform(8, 40))),
                "edges": edges, "sorted": rng.random() < 0.6, "grad": grad}
    if kind == "sh":
        return {"kind": kind, "vectors": _log_int(rng, 1_000, 4_194_304), "lmax": rng.randint(1, 6), "grad": rng.random() < 0.5}
    if kind == "tp":
        return {"kind": kind, "layout": rng.choice(sorted(TP_LAYOUTS)), "rows": _log_int(rng, 200, 60_000),
                "mode": rng.choice(["fp32", "fp32", "tf32x3"]), "grad": rng.random() < 0.6}
    if kind == "tp_linear":
        return {"kind": kind, "layout": "l3_mixed", "rows": _log_int(rng, 1_000, 1_048_576),
                "mode": rng.choice(["tf32", "tf32x3"])}
    if kind == "node_update":
        return {"kind": kind, "rows": _log_int(rng, 300, 200_000), "mode": rng.choice(["fp32", "tf32x3"]), "grad": rng.random() < 0.6}
    edges = _log_int(rng, 2_000, 4_000_000)
    return {"kind": kind, "nodes": max(64, int(edges / rng.uniform(8, 40))), "edges": edges}


# ---- what a user's program holds before the call -----------------------------------------------------------
def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev).manual_seed(seed)
    return _PREPARE[case["kind"]](case, gen, dev, seed)


def _randn(gen, *shape):
    return torch.randn(*shape, device=gen.device, generator=gen)


def _set_weights(module, gen):
    """Every parameter ~ N(0, 1), as the modules initialise themselves, from the case's own generator."""
    with torch.no_grad():
        for p in module.parameters():
            p.copy_(_randn(gen, *p.shape))
    return module


def _block(gen, dev):
    # about 26 neighbours: 0.05 * 4/3 pi 5^3
    return _set_weights(nn.InteractionBlock(BLOCK_IRREPS, 3, num_basis=8, hidden=64, r_max=CUTOFF, num_neighbors=26.0).to(dev), gen)


def _atoms(case, gen):
    box = (case["atoms"] / DENSITY) ** (1.0 / 3.0)
    pos = torch.rand(case["atoms"], 3, device=gen.device, generator=gen) * box
    return box, pos, _randn(gen, case["atoms"], o3.Irreps(BLOCK_IRREPS).dim)


def _prepare_md(case, gen, dev, seed):
    box, pos, x = _atoms(case, gen)
    block = _block(gen, dev)
    for p in block.parameters():
        p.requires_grad_(False)
    return {"kind": "md", "block": block, "box": box, "pos": pos, "x": x, "grad_out": _randn(gen, *x.shape)}


def _prepare_train(case, gen, dev, seed):
    box, pos, x = _atoms(case, gen)
    src, dst, shift, rowptr = nn.neighbor_list_pbc(pos, box, CUTOFF)
    return {"kind": "train", "block": _block(gen, dev), "pos": pos, "x": x.requires_grad_(True), "src": src, "dst": dst,
            "shift": shift, "rowptr": rowptr, "grad_out": _randn(gen, *x.shape)}


def _prepare_conv(case, gen, dev, seed):
    nodes, edges, grad = case["nodes"], case["edges"], case["grad"]
    tp = layouts.bench_conv_tp(case["layout"])
    src = torch.randint(0, nodes, (edges,), device=dev, generator=gen)
    dst = torch.randint(0, nodes, (edges,), device=dev, generator=gen)
    if case["sorted"]:
        dst = dst.sort().values
    perm, rowptr = e3nn_b200.csr_from_dst(dst, nodes)
    state = {"kind": "conv", "tp": tp, "src": src, "rowptr": rowptr, "perm": None if case["sorted"] else perm,
             "x": _randn(gen, nodes, tp.irreps_in1.dim), "vec": _randn(gen, edges, 3),
             "w": _randn(gen, edges, tp.weight_numel), "scale": (edges / nodes) ** -0.5}
    if grad:
        for name in ("x", "vec", "w"):
            state[name].requires_grad_(True)
        state["grad_out"] = _randn(gen, nodes, tp.irreps_out.dim)
    return state


def _prepare_sh(case, gen, dev, seed):
    vec = _randn(gen, case["vectors"], 3)
    state = {"kind": "sh", "irreps": o3.Irreps.spherical_harmonics(case["lmax"]), "vec": vec}
    if case["grad"]:
        vec.requires_grad_(True)
        state["grad_out"] = _randn(gen, case["vectors"], (case["lmax"] + 1) ** 2)
    return state


def _prepare_tp(case, gen, dev, seed):
    tp = _set_weights(o3.FullyConnectedTensorProduct(*TP_LAYOUTS[case["layout"]], math_mode=case["mode"]).to(dev), gen)
    state = {"kind": "tp", "tp": tp, "x": _randn(gen, case["rows"], tp.irreps_in1.dim), "y": _randn(gen, case["rows"], tp.irreps_in2.dim)}
    if case["grad"]:
        state["x"].requires_grad_(True)
        state["y"].requires_grad_(True)
        state["grad_out"] = _randn(gen, case["rows"], tp.irreps_out.dim)
    return state


def _prepare_tp_linear(case, gen, dev, seed):
    tp = o3.FullyConnectedTensorProduct(*TP_LAYOUTS[case["layout"]], math_mode=case["mode"])
    lin = o3.Linear(tp.irreps_out, tp.irreps_out, math_mode=case["mode"])
    module = _set_weights(o3.TensorProductLinear(tp, lin).to(dev), gen)
    return {"kind": "tp_linear", "module": module, "x": _randn(gen, case["rows"], tp.irreps_in1.dim),
            "y": _randn(gen, case["rows"], tp.irreps_in2.dim)}


def _gate():
    return nn.Gate("64x0e", [torch.nn.functional.silu], "192x0e", [torch.sigmoid], "64x1o+64x2e+64x3o")


def _prepare_node_update(case, gen, dev, seed):
    gate = _gate().to(dev)
    lin = _set_weights(o3.Linear(BLOCK_IRREPS, gate.irreps_in, math_mode=case["mode"]).to(dev), gen)
    state = {"kind": "node_update", "lin": lin, "gate": gate, "x": _randn(gen, case["rows"], lin.irreps_in.dim)}
    if case["grad"]:
        state["x"].requires_grad_(True)
        state["grad_out"] = _randn(gen, case["rows"], gate.irreps_out.dim)
    return state


def _prepare_csr(case, gen, dev, seed):
    return {"kind": "csr", "nodes": case["nodes"], "dst": torch.randint(0, case["nodes"], (case["edges"],), device=dev, generator=gen)}


_PREPARE = {"md": _prepare_md, "train": _prepare_train, "conv": _prepare_conv, "sh": _prepare_sh, "tp": _prepare_tp,
            "tp_linear": _prepare_tp_linear, "node_update": _prepare_node_update, "csr": _prepare_csr}


# ---- one pass ----------------------------------------------------------------------------------------------
def run(state):
    return _RUN[state["kind"]](state)


def _run_md(s):
    pos = s["pos"].detach().requires_grad_(True)
    src, dst, shift, rowptr = nn.neighbor_list_pbc(pos, s["box"], CUTOFF)
    out = s["block"](pos, s["x"], src, dst, rowptr, shift)
    (grad,) = torch.autograd.grad(out, pos, s["grad_out"])
    return {"out": out.detach(), "grad_pos": grad}


def _run_train(s):
    block = s["block"]
    out = block(s["pos"], s["x"], s["src"], s["dst"], s["rowptr"], s["shift"])
    grads = torch.autograd.grad(out, [s["x"]] + list(block.parameters()), s["grad_out"])
    return {"out": out.detach(), "grads": list(grads)}


def _run_conv(s):
    def conv():
        return e3nn_b200.conv_uvu(s["tp"], s["x"], s["vec"], s["src"], s["rowptr"], s["w"], perm=s["perm"], scale=s["scale"],
                                  edge_attr_is_vector=True)

    if "grad_out" not in s:
        with torch.no_grad():
            return conv()
    out = conv()
    return {"out": out.detach(), "grads": list(torch.autograd.grad(out, [s["x"], s["vec"], s["w"]], s["grad_out"]))}


def _run_sh(s):
    out = o3.spherical_harmonics(s["irreps"], s["vec"], normalize=True, normalization="component")
    if "grad_out" not in s:
        return out
    (grad,) = torch.autograd.grad(out, s["vec"], s["grad_out"])
    return {"out": out.detach(), "grad_vec": grad}


def _run_tp(s):
    if "grad_out" not in s:
        with torch.no_grad():
            return s["tp"](s["x"], s["y"])
    out = s["tp"](s["x"], s["y"])
    return {"out": out.detach(), "grads": list(torch.autograd.grad(out, [s["x"], s["y"], s["tp"].weight], s["grad_out"]))}


def _run_tp_linear(s):
    with torch.no_grad():
        return s["module"](s["x"], s["y"])


def _run_node_update(s):
    if "grad_out" not in s:
        with torch.no_grad():
            return s["gate"](s["lin"](s["x"]))
    out = s["gate"](s["lin"](s["x"]))
    return {"out": out.detach(), "grads": list(torch.autograd.grad(out, [s["x"], s["lin"].weight], s["grad_out"]))}


def _run_csr(s):
    return e3nn_b200.csr_from_dst(s["dst"], s["nodes"])


_RUN = {"md": _run_md, "train": _run_train, "conv": _run_conv, "sh": _run_sh, "tp": _run_tp, "tp_linear": _run_tp_linear,
        "node_update": _run_node_update, "csr": _run_csr}


# ---- the work a pass cannot do without ---------------------------------------------------------------------
def _uvu_flops(tp):
    """Multiply-adds of one row: per path and channel the coupling terms of x (x) y and the weight."""
    total = 0
    for ins in tp.instructions:
        a, b, c = tp.irreps_in1[ins.i_in1], tp.irreps_in2[ins.i_in2], tp.irreps_out[ins.i_out]
        terms = int((o3.wigner_3j(a.ir.l, b.ir.l, c.ir.l).abs() > 1e-9).sum())
        total += a.mul * (4 * terms + 2 * c.ir.dim)
    return total


def _uvw_flops(irreps1, irreps2, irreps_out):
    """Channel mixing of every path on the smaller side of its coupling."""
    tp = o3.FullyConnectedTensorProduct(irreps1, irreps2, irreps_out, internal_weights=False)
    return sum(2 * i.path_shape[0] * i.path_shape[1] * i.path_shape[2]
               * min(tp.irreps_in1[i.i_in1].ir.dim * tp.irreps_in2[i.i_in2].ir.dim, tp.irreps_out[i.i_out].ir.dim) for i in tp.instructions)


def _linear_flops(irreps_in, irreps_out):
    return sum(2 * a.mul * b.mul * a.ir.dim for a in o3.Irreps(irreps_in) for b in o3.Irreps(irreps_out) if a.ir == b.ir)


def work(case):
    kind = case["kind"]
    if kind in ("md", "train"):
        n = case["atoms"]
        edges = n * DENSITY * 4.0 / 3.0 * math.pi * CUTOFF**3
        tp = layouts.bench_conv_tp("cfg5_23")
        radial = 2.0 * (8 * 64 + 64 * tp.weight_numel)
        per_edge, per_node = radial + _uvu_flops(tp), _linear_flops(tp.irreps_out, BLOCK_IRREPS)
        dim = tp.irreps_in1.dim
        if kind == "md":      # forward, and once more for the gradient w.r.t. the edges
            return {"bytes": 4.0 * n * (3 + 2 * dim + dim + 3), "flops": edges * (2 * radial + 3 * _uvu_flops(tp)) + 2.0 * n * per_node}
        return {"bytes": 4.0 * n * (3 + 2 * dim + 2 * dim) + 28.0 * edges, "flops": 3.0 * (edges * per_edge + n * per_node)}
    if kind == "conv":
        n, e, tp = case["nodes"], case["edges"], layouts.bench_conv_tp(case["layout"])
        d1, dout, wn = tp.irreps_in1.dim, tp.irreps_out.dim, tp.weight_numel
        nbytes = 4.0 * (n * (d1 + dout) + e * (wn + 3)) + 8.0 * (e + n) + (0.0 if case["sorted"] else 8.0 * e)
        if case["grad"]:
            nbytes += 4.0 * (n * (dout + d1) + e * (wn + 3))
        return {"bytes": nbytes, "flops": (3.0 if case["grad"] else 1.0) * e * _uvu_flops(tp)}
    if kind == "sh":
        n, k = case["vectors"], (case["lmax"] + 1) ** 2
        return {"bytes": 4.0 * n * ((3 + k) + ((k + 3) if case["grad"] else 0)), "flops": n * k * (12.0 if case["grad"] else 4.0)}
    if kind == "tp":
        a, b, c = (o3.Irreps(t) for t in TP_LAYOUTS[case["layout"]])
        n, f = case["rows"], _uvw_flops(*TP_LAYOUTS[case["layout"]])
        return {"bytes": 4.0 * n * ((a.dim + b.dim + c.dim) * (2 if case["grad"] else 1)), "flops": n * f * (4.0 if case["grad"] else 1.0)}
    if kind == "tp_linear":
        a, b, c = (o3.Irreps(t) for t in TP_LAYOUTS[case["layout"]])
        return {"bytes": 4.0 * case["rows"] * (a.dim + b.dim + c.dim), "flops": case["rows"] * float(_uvw_flops(*TP_LAYOUTS[case["layout"]]))}
    if kind == "node_update":
        gate = _gate()
        n, din, dout = case["rows"], o3.Irreps(BLOCK_IRREPS).dim, gate.irreps_out.dim
        return {"bytes": 4.0 * n * (din + dout) * (2 if case["grad"] else 1),
                "flops": n * _linear_flops(BLOCK_IRREPS, gate.irreps_in) * (3.0 if case["grad"] else 1.0)}
    return {"bytes": 16.0 * case["edges"] + 8.0 * case["nodes"], "flops": 0.0}


def tolerance(case):
    kind, mode = case["kind"], case.get("mode")
    if kind == "csr":
        return "exact"
    # about four times the differences from a 64-bit evaluation of the same inputs (sizes 256 to 50,000)
    if mode == "tf32":                      # one product of 11-bit operands: 4.7e-4, 3.7e-3
        return {"rel": 2e-3, "max": 1.5e-2}
    if kind in ("md", "train") or mode == "tf32x3":
        # sums of split operands in tensor memory: 3.7e-6 (first radial layer's gradient), 1.1e-5
        return {"rel": 1.5e-5, "max": 1e-4}
    return {"rel": 2e-6, "max": 4e-5}       # 32-bit sums: 4.4e-7, 5.3e-6
