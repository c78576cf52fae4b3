"""The work that the speed of this package is judged by: batched tensor products, fused graph convolutions and symmetric
contractions at the sizes and with the options of equivariant interatomic potentials (training, molecular dynamics,
inference) and of docking models, each through the public modules and torch autograd.

A case names a problem of ``openequivariance_b200.core.problems``, its size and what is done with it:

* ``"forward"``: the product alone, without gradients (energies, embeddings);
* ``"train"``: forward, and the gradients of every input (forces in molecular dynamics, training on energies);
* ``"double"``: forward, gradients kept differentiable, and the gradients of those (training on forces).
"""

import math

import numpy as np
import torch

import openequivariance_b200 as oeq
from openequivariance_b200._torch.symmetric_contraction import SymmetricContraction
from openequivariance_b200.core import problems as P
from openequivariance_b200.core.graph import periodic_radius_graph, sort_edges, spherical_harmonics
from openequivariance_b200.core.wigner import wigner_3j

CONV_PROBLEMS = ("mace-like", "mace-large", "mace-medium", "nequip-lips", "nequip-revmd17-aspirin", "nequip-revmd17-toluene",
                 "nequip-revmd17-benzene", "nequip-water")


def _problem(name, dtype="float32"):
    if name == "readme":
        p = P.readme_problem()
    elif name == "mace-like":
        p = P.mace_like_problem()
    elif name == "nequip-like":
        p = P.nequip_like_problem()
    else:
        every = P.mace_problems() + P.nequip_problems() + P.diffdock_problems() + P.e3nn_torch_tetris_poly_problems()
        p = next(q for q in every if q.label == name)
    p = p.clone()
    p.irrep_dtype = p.weight_dtype = np.dtype(dtype).type
    return p


def _tp(problem, batch, what, dtype="float32"):
    return {"kind": "tp", "problem": problem, "batch": batch, "pass": what, "dtype": dtype}


def _conv(problem, nodes, degree, what, deterministic, dtype="float32"):
    return {"kind": "conv", "problem": problem, "nodes": nodes, "degree": degree, "pass": what, "deterministic": deterministic, "dtype": dtype}


def _contraction(nodes, features, lmax, elements, what, dtype="float32"):
    return {"kind": "contraction", "nodes": nodes, "features": features, "lmax": lmax, "elements": elements, "pass": what, "dtype": dtype}


def listed():
    return [
        # the first example of the documentation: one path, a thousand items; launches and host time are all there is
        dict(_tp("readme", 1000, "train"), name="readme product, gradients"),
        # channelwise product of a MACE-like layer on an edge batch that was gathered by the caller
        dict(_tp("mace-like", 50001, "train"), name="mace-like product, gradients"),
        # fully connected product with shared weights of a NequIP-like layer, at the batch of the package's benchmark
        dict(_tp("nequip-like", 50000, "train"), name="nequip-like product, gradients"),
        # the same in double precision, as geometry optimisation and validation run it
        dict(_tp("nequip-like", 5003, "train", "float64"), name="nequip-like product, f64"),
        # the same when a network is trained on forces
        dict(_tp("nequip-like", 2500, "double"), name="nequip-like product, 2nd order"),
        # fully connected product whose weights come from an edge network: multiplicities 48 and 10
        dict(_tp("DiffDock-L=2", 8191, "train"), name="diffdock product, gradients"),
        # molecular dynamics of a few small molecules: neighbour list in any order, everything fits in the caches
        dict(_conv("nequip-revmd17-aspirin", 105, 16.0, "train", False), name="small molecules, gradients"),
        # a training step over a large periodic cell, bitwise reproducible: the package's benchmark graph
        dict(_conv("mace-like", 24000, 32.0, "train", True), name="mace-like graph, gradients"),
        # energies of a mid-sized cell, neighbour list in any order
        dict(_conv("mace-large", 4001, 32.0, "forward", False), name="mace-large graph, forward"),
        # training on forces
        dict(_conv("mace-like", 1500, 32.0, "double", True), name="mace-like graph, 2nd order"),
        # relaxation of a crystal in double precision
        dict(_conv("mace-medium", 1003, 40.0, "train", True, "float64"), name="mace-medium graph, f64"),
        # the node-wise product basis that follows the convolution in MACE
        dict(_contraction(2003, 128, 3, 10, "train"), name="symmetric contraction"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["small", "channelwise", "shared", "shared", "edge-weights", "conv", "conv", "conv", "conv", "contraction"])
    what = rng.choice(["forward", "train", "train", "double"])
    if kind == "small":
        return _tp(rng.choice(["readme", "tetris-poly-1", "tetris-poly-2"]), _log(rng, 16, 20000), what)
    if kind == "channelwise":
        most = 20000 if what == "double" else 50000
        return _tp(rng.choice(["mace-like", "mace-large", "mace-medium"]), _log(rng, 100, most), what)
    if kind == "shared":
        dtype = rng.choice(["float32", "float32", "float64"])
        return _tp("nequip-like", _log(rng, 100, 10000 if dtype == "float64" else 50000), what, dtype)
    if kind == "edge-weights":
        return _tp(rng.choice(["DiffDock-L=1", "DiffDock-L=2"]), _log(rng, 100, 10000), rng.choice(["forward", "train"]))
    if kind == "contraction":
        return _contraction(_log(rng, 50, 3000), rng.choice([32, 64, 128]), rng.choice([2, 3]), rng.randint(1, 12), rng.choice(["forward", "train"]))
    problem = rng.choice(CONV_PROBLEMS)
    dtype = rng.choice(["float32", "float32", "float32", "float64"])
    degree = float(rng.randint(12, 48))
    # second order, doubles and the widest product (a molecule of twelve atoms): cells and batches of up to 1,500 atoms
    edges = 48000 if dtype == "float64" or what == "double" or problem == "nequip-revmd17-benzene" else 24000 * 32
    return _conv(problem, _log(rng, 21, min(24000, edges / degree)), degree, what, rng.random() < 0.5, dtype)


# ---- inputs ---------------------------------------------------------------------------------------------------

def _coupling_tensors(lmax, out_l, correlation=3):
    """Generalised Clebsch-Gordan tensors of the symmetric contraction: every way of coupling nu factors of the natural-parity
    features 0e + 1o + ... + lmax to an output of degree ``out_l``, as ``{nu: U [(2 out_l + 1), ell, ..., ell, paths]}`` (the
    leading dimension only for out_l > 0)."""
    ell = (lmax + 1) ** 2
    # chains[l] = list of (parity exponent, tensor [ell] * nu + [2l + 1])
    chains = {}
    for l in range(lmax + 1):
        t = np.zeros((ell, 2 * l + 1))
        t[l * l:(l + 1) ** 2] = np.eye(2 * l + 1)
        chains[l] = [(l % 2, t)]
    out = {}
    for nu in range(1, correlation + 1):
        if nu > 1:
            grown = {}
            for l12, parts in chains.items():
                for parity, t in parts:
                    for l3 in range(lmax + 1):
                        for l in range(abs(l12 - l3), l12 + l3 + 1):
                            if l > lmax + out_l:
                                continue
                            c = np.zeros((2 * l12 + 1, ell, 2 * l + 1))
                            c[:, l3 * l3:(l3 + 1) ** 2] = wigner_3j(l12, l3, l) * math.sqrt(2 * l + 1)
                            grown.setdefault(l, []).append(((parity + l3) % 2, np.tensordot(t, c, axes=1)))
            chains = grown
        paths = [t for parity, t in chains.get(out_l, []) if parity == out_l % 2]
        u = np.stack(paths, axis=-1)                      # [ell] * nu + [2 out_l + 1, paths]
        u = np.moveaxis(u, -2, 0)
        out[nu] = torch.from_numpy(np.ascontiguousarray(u[0] if out_l == 0 else u))
    return out


_TENSORS = {}


def _tensors(lmax, out_l):
    if (lmax, out_l) not in _TENSORS:
        _TENSORS[lmax, out_l] = _coupling_tensors(lmax, out_l)
    return _TENSORS[lmax, out_l]


def _prepare_contraction(case, gen, dtype):
    n, f, g = case["nodes"], case["features"], case["elements"]
    ell = (case["lmax"] + 1) ** 2
    torch.manual_seed(gen.initial_seed() % (1 << 31))     # the module draws its own weights
    module = SymmetricContraction([_tensors(case["lmax"], 0), _tensors(case["lmax"], 1)], f, g, dtype=dtype).to("cuda")
    element = torch.randint(0, g, (n,), device="cuda", generator=gen)
    y = torch.nn.functional.one_hot(element, g).to(dtype)
    x = torch.randn(n, f, ell, device="cuda", dtype=dtype, generator=gen)
    cot = torch.randn(n, 4 * f, device="cuda", dtype=dtype, generator=gen)
    if case["pass"] == "forward":
        for p in module.parameters():
            p.requires_grad_(False)
    return {"call": lambda x: module(x, y), "inputs": [x], "more": list(module.parameters()), "cot": cot}


def _edges(case):
    """Directed edges of a case's graph: ``degree`` per node, fewer where there are not that many other nodes."""
    return 2 * int(case["nodes"] * min(case["degree"], 0.6 * (case["nodes"] - 1)) / 2)


def _graph(case, seed):
    """The closest pairs of a periodic cloud of points, so many that every seed gives the same number of edges: ``rows, cols``
    sorted by (row, col), the permutation to sender-major order, and the edges' vectors."""
    pairs = _edges(case) // 2
    g = periodic_radius_graph(case["nodes"], mean_degree=2.8 * pairs / case["nodes"], cutoff=5.0, seed=seed, device="cuda")
    once = g["rows"] < g["cols"]
    i, j, vec = g["rows"][once], g["cols"][once], g["vec"][once]
    near = vec.square().sum(1).argsort(stable=True)[:pairs]
    assert near.numel() == pairs
    rows, cols = torch.cat([i[near], j[near]]), torch.cat([j[near], i[near]])
    order, perm = sort_edges(rows, cols)
    return rows[order].contiguous(), cols[order].contiguous(), perm.contiguous(), torch.cat([vec[near], -vec[near]])[order]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = torch.float64 if case["dtype"] == "float64" else torch.float32
    if case["kind"] == "contraction":
        state = _prepare_contraction(case, gen, dtype)
    else:
        problem = _problem(case["problem"], case["dtype"])
        lmax = max(ir.l for _, ir in problem.irreps_in2)
        rand = lambda *shape: torch.randn(*shape, device="cuda", dtype=dtype, generator=gen)  # noqa: E731
        if case["kind"] == "tp":
            items = rows_x = case["batch"]
            module = oeq.TensorProduct(problem)
            vec = torch.randn(items, 3, device="cuda", dtype=torch.float64, generator=gen)
            call = module
        else:
            rows_x = case["nodes"]
            rows, cols, perm, vec = _graph(case, seed)
            items = rows.numel()
            module = oeq.TensorProductConv(problem, deterministic=case["deterministic"])
            if case["deterministic"]:
                call = lambda x, y, w: module(x, y, w, rows, cols, perm)  # noqa: E731
            else:
                shuffle = torch.randperm(items, device="cuda", generator=gen)
                rows, cols, vec = rows[shuffle].contiguous(), cols[shuffle].contiguous(), vec[shuffle]
                call = lambda x, y, w: module(x, y, w, rows, cols)  # noqa: E731
        if case["problem"] == "readme":
            y = torch.rand(items, problem.irreps_in2.dim, device="cuda", dtype=dtype, generator=gen)
        else:
            y = spherical_harmonics(lmax, vec).to(dtype).contiguous()
        x = rand(rows_x, problem.irreps_in1.dim)
        if problem.shared_weights:
            fan_in = problem.irreps_in1.dim / len(problem.irreps_in1)
            w = rand(problem.weight_numel) / math.sqrt(fan_in)
        else:
            w = rand(items, problem.weight_numel)
        state = {"call": call, "inputs": [x, y, w], "more": [], "cot": rand(rows_x, problem.irreps_out.dim)}
    state["pass"] = case["pass"]
    if case["pass"] != "forward":
        for t in state["inputs"]:
            t.requires_grad_(True)
    if case["pass"] == "double":
        state["cot"].requires_grad_(True)
        state["cot2"] = [torch.randn(t.shape, device="cuda", dtype=dtype, generator=gen) for t in state["inputs"]]
    return state


def run(state):
    out = state["call"](*state["inputs"])
    if state["pass"] == "forward":
        return out
    wanted = state["inputs"] + state["more"]
    if state["pass"] == "train":
        return [out] + list(torch.autograd.grad(out, wanted, state["cot"]))
    first = torch.autograd.grad(out, wanted, state["cot"], create_graph=True)
    second = torch.autograd.grad(first, wanted + [state["cot"]], state["cot2"])
    return [out] + list(first) + list(second)


# ---- what a pass cannot do without ----------------------------------------------------------------------------

def work(case):
    size = 8 if case["dtype"] == "float64" else 4
    times = {"forward": 1, "train": 3, "double": 10}[case["pass"]]   # forward + 2 for gradients + 3 forward, 2 x 2 gradients
    if case["kind"] == "contraction":
        n, f, ell, g = case["nodes"], case["features"], (case["lmax"] + 1) ** 2, case["elements"]
        params = sum(_tensors(case["lmax"], l)[nu].shape[-1] for l in (0, 1) for nu in (1, 2, 3)) * g * f
        values = n * f * (ell + 4) + params + n * g
        once = 2 * n * f * 4 * (ell ** 3 + ell ** 2 + ell)
        return {"bytes": size * values * (1 if case["pass"] == "forward" else 2), "flops": once * times}
    problem = _problem(case["problem"], case["dtype"])
    x, y, z, w = problem.irreps_in1.dim, problem.irreps_in2.dim, problem.irreps_out.dim, problem.weight_numel
    flops = 0
    for ins in problem.instructions:
        (u, a), (v, b), (m, o) = problem.irreps_in1[ins.i_in1], problem.irreps_in2[ins.i_in2], problem.irreps_out[ins.i_out]
        pairs = int((np.abs(wigner_3j(a.l, b.l, o.l)).max(axis=1) > 1e-12).sum())
        flops += 2 * u * v * pairs + 2 * u * v * (m if ins.connection_mode == "uvw" else 1) * (2 * o.l + 1)
    if case["kind"] == "tp":
        rows = items = case["batch"]
        index = 0
    else:
        rows, items = case["nodes"], _edges(case)
        index = 16 * items
    weights = w if problem.shared_weights else items * w
    counts = {"forward": (1, 1), "train": (2, 2), "double": (4, 3)}[case["pass"]]   # inputs and their gradients; output and its cotangents
    values = counts[0] * (rows * x + items * y + weights) + counts[1] * rows * z
    return {"bytes": size * values + index, "flops": items * flops * times}


def tolerance(case):
    # sums of 32-bit and 64-bit products in another order (and, for the fully connected product, from split operands)
    return {"rel": 1e-12} if case["dtype"] == "float64" else {"rel": 1e-5}
