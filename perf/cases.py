"""The work that is timed when the speed of this package is judged: what a message-passing interatomic
potential asks of it, through the public modules, from one small molecule to a training batch of a million edges.

A case is a dict of plain values.  ``op`` names the piece of such a model:

* ``conv``            channelwise tensor product with gather and scatter: node features (senders) x edge
                      harmonics x per-edge weights -> receivers; forward only or with all three gradients;
* ``interaction``     one convolution step as a model runs it: edge vectors -> spherical harmonics, edge lengths ->
                      radial MLP -> weights, product, backward to node features, edge vectors and MLP parameters;
* ``force_training``  energy -> gradients (forces) -> gradient of a loss on them (double backward);
* ``contraction``     symmetric contraction with species weights, forward and backward;
* ``fully_connected`` dense uvw product with shared weights, forward and backward;
* ``node_linear``     equivariant linear layer on node features, forward and backward.

Sizes: 128 channels, lmax 3, 65,536 / 1,048,576 edges, 16,384 atoms, 32,768 samples are the ones of the benchmark
configurations (``bench.py``, ``bench_configs.py``); the others are generic.
"""
from __future__ import annotations

import copy
import math
from functools import lru_cache

import numpy as np
import torch

import cuequivariance_b200 as cb
from cuequivariance_b200.dense import linear_f32x3

DEVICE = "cuda"
DTYPES = {"float32": torch.float32, "float64": torch.float64, "bfloat16": torch.bfloat16}


def listed():
    return [
        # One small molecule (21 atoms, all pairs within the cutoff): molecular dynamics calls the product and its
        # gradients thousands of times a second, and launches and host work are all there is to it.
        {"name": "conv_molecule", "op": "conv", "channels": 128, "l_in": 1, "l_sh": 3, "l_out": 3, "edges": 420, "nodes": 21,
         "layout": "mul_ir", "sorted": True, "dtype": "float32", "gradients": True},
        # Inference on a medium structure with an edge list in no particular order (configuration 0 of bench_configs.py).
        {"name": "conv_forward_unsorted", "op": "conv", "channels": 128, "l_in": 2, "l_sh": 3, "l_out": 3, "edges": 65536,
         "nodes": 4096, "layout": "mul_ir", "sorted": False, "dtype": "float32", "gradients": False},
        # The headline: a training batch of a million edges, forward and all gradients (bench.py).
        {"name": "conv_gradients_1m", "op": "conv", "channels": 128, "l_in": 3, "l_sh": 3, "l_out": 3, "edges": 1048576,
         "nodes": 32768, "layout": "mul_ir", "sorted": True, "dtype": "float32", "gradients": True},
        # A narrower model: 96 channels, lmax 2, component-major layout, odd counts, unsorted edges.
        {"name": "conv_ragged_l2", "op": "conv", "channels": 96, "l_in": 2, "l_sh": 2, "l_out": 2, "edges": 40003, "nodes": 1999,
         "layout": "ir_mul", "sorted": False, "dtype": "float32", "gradients": True},
        # Double precision, as used to validate a model or relax a structure tightly.
        {"name": "conv_gradients_f64", "op": "conv", "channels": 128, "l_in": 3, "l_sh": 3, "l_out": 3, "edges": 65536, "nodes": 4096,
         "layout": "mul_ir", "sorted": True, "dtype": "float64", "gradients": True},
        # A whole convolution step from edge vectors, as a training loop runs it (the end-to-end leg of bench.py).
        {"name": "interaction_step", "op": "interaction", "channels": 128, "l_in": 3, "l_sh": 3, "l_out": 3, "edges": 262144,
         "nodes": 8192},
        # Training on forces: double backward (configuration 4 of bench_configs.py).
        {"name": "force_training", "op": "force_training", "channels": 128, "l_in": 3, "l_sh": 3, "l_out": 3, "edges": 65536,
         "nodes": 4096},
        # The many-body step of a training batch (configuration 1 of bench_configs.py).
        {"name": "contraction_batch", "op": "contraction", "channels": 128, "l_in": 3, "l_out": 1, "degree": 3, "atoms": 16384,
         "species": 10},
        # The same step of a smaller model on a few hundred atoms: the last layer, scalars out.
        {"name": "contraction_small", "op": "contraction", "channels": 64, "l_in": 2, "l_out": 0, "degree": 3, "atoms": 213,
         "species": 10},
        # Dense products between node features (configuration 2 of bench_configs.py), in both precisions it is used in.
        {"name": "fully_connected_f32", "op": "fully_connected", "channels": 64, "l_max": 2, "batch": 32768, "dtype": "float32"},
        {"name": "fully_connected_bf16", "op": "fully_connected", "channels": 64, "l_max": 2, "batch": 32768, "dtype": "bfloat16"},
        # The linear layer in front of and behind every product, on all nodes of the million-edge batch.
        {"name": "node_linear", "op": "node_linear", "channels": 128, "l_max": 3, "nodes": 32768, "classes": 1},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges.  No drawn case is larger than the listed ones of its kind."""
    op = rng.choice(["conv", "conv", "conv", "interaction", "force_training", "contraction", "fully_connected", "node_linear"])
    if op in ("conv", "interaction", "force_training"):
        channels = rng.choice([32, 64, 64, 96, 128, 128, 128, 256])
        l_in, l_sh, l_out = rng.randint(1 if op == "force_training" else 0, 3), rng.choice([1, 2, 3, 3]), rng.choice([1, 2, 3, 3])
        dtype = "float64" if op == "conv" and rng.random() < 0.2 else "float32"
        most = 65536 if op == "force_training" or dtype == "float64" else 262144
        edges = _log_uniform(rng, 300, most * 128 // max(channels, 128))
        case = {"op": op, "channels": channels, "l_in": l_in, "l_sh": l_sh, "l_out": l_out, "edges": edges,
                "nodes": max(8, int(edges / rng.uniform(10, 40)))}
        if op == "conv":
            case.update(layout=rng.choice(["mul_ir", "mul_ir", "ir_mul"]), sorted=rng.random() < 0.5, dtype=dtype,
                        gradients=rng.random() < 0.7)
        return case
    if op == "contraction":
        return {"op": op, "channels": rng.choice([32, 64, 96, 128]), "l_in": rng.randint(1, 3), "l_out": rng.randint(0, 1),
                "degree": rng.randint(2, 3), "atoms": _log_uniform(rng, 20, 16384), "species": rng.choice([2, 4, 10])}
    if op == "fully_connected":
        dtype = rng.choice(["float32", "bfloat16"])
        channels = rng.choice([32, 64, 64, 96] if dtype == "float32" else [64, 64, 128])
        batch = _log_uniform(rng, 200, 32768 * 64 ** 3 // max(channels, 64) ** 3)
        return {"op": op, "channels": channels, "l_max": rng.randint(1, 2), "batch": batch, "dtype": dtype}
    return {"op": op, "channels": rng.choice([32, 64, 96, 128]), "l_max": rng.randint(0, 3), "nodes": _log_uniform(rng, 300, 32768),
            "classes": rng.choice([1, 1, 10])}


# ---- the modules: a program builds each once and keeps it for all its inputs --------------------------------------
def _natural(lmax):
    return [f"{l}{'eo'[l % 2]}" for l in range(lmax + 1)]  # noqa: E741


def _irreps(channels, lmax):
    return "+".join(f"{channels}x{ir}" for ir in _natural(lmax))


@lru_cache(maxsize=None)
def _conv_module(channels, l_in, l_sh, l_out, layout):
    return cb.ChannelWiseTensorProduct(_irreps(channels, l_in), "+".join(_natural(l_sh)), _natural(l_out),
                                       layout=getattr(cb, layout), shared_weights=False, internal_weights=False)


@lru_cache(maxsize=None)
def _harmonics_module(l_sh):
    return cb.SphericalHarmonics(list(range(l_sh + 1)), normalize=True)


@lru_cache(maxsize=None)
def _contraction_module(channels, l_in, l_out, degree, species):
    return cb.SymmetricContraction(_irreps(channels, l_in), _irreps(channels, l_out), degree, species, layout=cb.mul_ir,
                                   dtype=torch.float32, device=DEVICE)


@lru_cache(maxsize=None)
def _fully_connected_module(channels, l_max):
    s = _irreps(channels, l_max)
    return cb.FullyConnectedTensorProduct(s, s, s, layout=cb.mul_ir, internal_weights=False, shared_weights=True)


@lru_cache(maxsize=None)
def _linear_module(channels, l_max, classes):
    s = _irreps(channels, l_max)
    return cb.Linear(s, s, layout=cb.mul_ir, internal_weights=False, shared_weights=True, weight_classes=classes)


# ---- prepare ----------------------------------------------------------------------------------------------------
def _graph(case, gen):
    E, N = case["edges"], case["nodes"]
    snd = torch.randint(0, N, (E,), generator=gen, device=DEVICE, dtype=torch.int32)
    rcv = torch.randint(0, N, (E,), generator=gen, device=DEVICE, dtype=torch.int32)
    if case.get("sorted", True):
        rcv = torch.sort(rcv).values
    return snd, rcv


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(int(seed))

    def randn(*shape, dtype=torch.float32, scale=1.0):
        t = torch.randn(*shape, generator=gen, device=DEVICE, dtype=torch.float64 if dtype == torch.float64 else torch.float32)
        return (t * scale if scale != 1.0 else t).to(dtype)

    op = case["op"]
    s = {"op": op}
    if op in ("conv", "interaction", "force_training"):
        tp = _conv_module(case["channels"], case["l_in"], case["l_sh"], case["l_out"], case.get("layout", "mul_ir"))
        dt = DTYPES[case.get("dtype", "float32")]
        E, N = case["edges"], case["nodes"]
        s.update(tp=tp, sh=_harmonics_module(case["l_sh"]), nodes=N)
        s["snd"], s["rcv"] = _graph(case, gen)
        s["x1"] = randn(N, tp.irreps_in1.dim, dtype=dt)
        vec = torch.nn.functional.normalize(randn(E, 3, dtype=dt), dim=1)
        if op == "conv":
            s["x2"] = s["sh"](vec).detach()
            s["w"] = randn(E, tp.weight_numel, dtype=dt)
            s["gradients"] = case["gradients"]
            if case["gradients"]:
                s["cot"] = randn(N, tp.irreps_out.dim, dtype=dt)
                for k in ("x1", "x2", "w"):
                    s[k].requires_grad_(True)
        elif op == "interaction":
            length = 0.5 + 4.5 * torch.rand(E, 1, generator=gen, device=DEVICE)
            s["vec"] = (vec * length).requires_grad_(True)
            s["x1"].requires_grad_(True)
            s["cot"] = randn(N, tp.irreps_out.dim)
            s["mlp"] = [randn(64, 8, scale=8 ** -0.5).requires_grad_(True), torch.zeros(64, device=DEVICE, requires_grad=True),
                        randn(tp.weight_numel, 64, scale=0.125).requires_grad_(True),
                        torch.zeros(tp.weight_numel, device=DEVICE, requires_grad=True)]
        else:
            s["vec"] = vec.requires_grad_(True)
            s["w"] = randn(E, tp.weight_numel).requires_grad_(True)
            s["x1"].requires_grad_(True)
    elif op == "contraction":
        # the module with this state's own weights (what it knows about its polynomial is shared)
        m = copy.copy(_contraction_module(case["channels"], case["l_in"], case["l_out"], case["degree"], case["species"]))
        fan_in = m.weight_shape[0]
        m._parameters = {"weight": torch.nn.Parameter(randn(case["species"], *m.weight_shape, scale=fan_in ** -0.5))}
        s.update(m=m, x=randn(case["atoms"], m.irreps_in.dim).requires_grad_(True), cot=randn(case["atoms"], m.irreps_out.dim),
                 species=torch.randint(0, case["species"], (case["atoms"],), generator=gen, device=DEVICE))
    elif op == "fully_connected":
        m = _fully_connected_module(case["channels"], case["l_max"])
        dt, B = DTYPES[case["dtype"]], case["batch"]
        s.update(m=m, x1=randn(B, m.irreps_in1.dim, dtype=dt).requires_grad_(True), x2=randn(B, m.irreps_in2.dim, dtype=dt).requires_grad_(True),
                 w=randn(1, m.weight_numel, dtype=dt, scale=1.0 / case["channels"]).requires_grad_(True),
                 cot=randn(B, m.irreps_out.dim, dtype=dt))
    else:
        m = _linear_module(case["channels"], case["l_max"], case["classes"])
        s.update(m=m, x=randn(case["nodes"], m.irreps_in.dim).requires_grad_(True),
                 w=randn(case["classes"], m.weight_numel).requires_grad_(True), cot=randn(case["nodes"], m.irreps_out.dim), classes=None)
        if case["classes"] > 1:
            s["classes"] = torch.sort(torch.randint(0, case["classes"], (case["nodes"],), generator=gen, device=DEVICE)).values
    return s


# ---- run ----------------------------------------------------------------------------------------------------------
def _bessel(r, n=8, cutoff=5.0):
    k = torch.arange(1, n + 1, device=r.device, dtype=r.dtype)
    return (2.0 / cutoff) ** 0.5 * torch.sin(k * math.pi * r[:, None] / cutoff) / r[:, None]


def run(s):
    op = s["op"]
    grad = torch.autograd.grad
    if op == "conv":
        kw = dict(indices_1=s["snd"], indices_out=s["rcv"], size_out=s["nodes"])
        if not s["gradients"]:
            with torch.no_grad():
                return s["tp"](s["x1"], s["x2"], s["w"], **kw)
        out = s["tp"](s["x1"], s["x2"], s["w"], **kw)
        return [out.detach(), *grad(out, (s["w"], s["x1"], s["x2"]), s["cot"])]
    if op == "interaction":
        w1, b1, w2, b2 = s["mlp"]
        hidden = torch.nn.functional.silu(torch.nn.functional.linear(_bessel(s["vec"].norm(dim=1)), w1, b1))
        weights = linear_f32x3(hidden, w2, b2)
        out = s["tp"](s["x1"], s["sh"](s["vec"]), weights, indices_1=s["snd"], indices_out=s["rcv"], size_out=s["nodes"])
        return [out.detach(), *grad(out, (s["x1"], s["vec"], *s["mlp"]), s["cot"])]
    if op == "force_training":
        out = s["tp"](s["x1"], s["sh"](s["vec"]), s["w"], indices_1=s["snd"], indices_out=s["rcv"], size_out=s["nodes"])
        blocks = s["tp"].irreps_out
        n = sum(mul for mul, ir in blocks if ir.l == 0)     # the 0e blocks come first
        energy = out[:, :n].sum()
        gx, gv, gw = grad(energy, (s["x1"], s["vec"], s["w"]), create_graph=True)
        second = grad(gv.pow(2).sum(), (s["x1"], s["vec"], s["w"]), allow_unused=True)
        return [out.detach(), gx.detach(), gv.detach(), gw.detach(), *second]
    if op == "contraction":
        out = s["m"](s["x"], s["species"])
        return [out.detach(), *grad(out, (s["x"], s["m"].weight), s["cot"])]
    if op == "fully_connected":
        out = s["m"](s["x1"], s["x2"], s["w"])
        return [out.detach(), *grad(out, (s["x1"], s["x2"], s["w"]), s["cot"])]
    out = s["m"](s["x"], s["w"], s["classes"])
    return [out.detach(), *grad(out, (s["x"], s["w"]), s["cot"])]


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _coupling_pairs(e, scalars_only=False):
    """Entries (i, k) of the coupling matrices that are not zero, over all paths of a channelwise product."""
    _, d = e.polynomial.operations[0]
    return sum(int(np.count_nonzero(np.any(p.coefficients != 0.0, axis=1))) for p in d.paths
               if not scalars_only or p.coefficients.shape[2] == 1)


def work(case):
    op = case["op"]
    if op in ("conv", "interaction", "force_training"):
        tp = _conv_module(case["channels"], case["l_in"], case["l_sh"], case["l_out"], case.get("layout", "mul_ir"))
        e = cb.descriptors.channelwise_tensor_product(tp.irreps_in1, tp.irreps_in2, _natural(case["l_out"]))
        E, N, C = case["edges"], case["nodes"], case["channels"]
        w, x1, x2, out = (r.dim for r in (*e.inputs, *e.outputs))
        size = 8 if case.get("dtype") == "float64" else 4
        # a multiply-add per channel, edge and coupling entry for the product and for each of its two contractions
        # with the cotangent (one gives the x1 and w gradients, one the x2 gradient)
        mac = _coupling_pairs(e) * C * E
        if op == "conv":
            nodes = N * (x1 + out)
            edges = E * (w + x2)
            twice = 2 if case["gradients"] else 1     # each input has a gradient, the output a cotangent
            return {"bytes": twice * size * (nodes + edges) + 8 * E, "flops": 2 * mac * (3 if case["gradients"] else 1)}
        if op == "interaction":
            layer = 3 * (64 * w + 8 * 64) * E
            return {"bytes": 4 * (2 * N * (x1 + out) + 2 * 3 * E + 2 * 64 * w) + 8 * E, "flops": 2 * (3 * mac + layer)}
        # only the paths into the scalars carry energy; their two contractions of the first pass are differentiated
        # again, three terms each
        return {"bytes": 4 * (3 * (N * x1 + E * (3 + w))) + 8 * E, "flops": 2 * 9 * _coupling_pairs(e, scalars_only=True) * C * E}
    if op == "contraction":
        m = _contraction_module(case["channels"], case["l_in"], case["l_out"], case["degree"], case["species"])
        from cuequivariance_b200.static_poly import merge_symmetric_paths

        poly = merge_symmetric_paths(m.etp.polynomial.flatten_coefficient_modes().squeeze_modes())
        monomials = sum(d.num_paths for _, d in poly.operations)
        A = case["atoms"]
        w = case["species"] * m.weight_shape[0] * m.weight_shape[1]
        return {"bytes": 4 * (2 * A * (m.irreps_in.dim + m.irreps_out.dim) + 2 * w) + 8 * A, "flops": 2 * 2 * 3 * monomials * case["channels"] * A}
    if op == "fully_connected":
        m = _fully_connected_module(case["channels"], case["l_max"])
        _, d = m.f.polynomial.operations[0]
        cells = sum(p.coefficients.shape[2] for p in d.paths) * case["channels"] ** 3
        B = case["batch"]
        size = 2 if case["dtype"] == "bfloat16" else 4
        return {"bytes": 2 * size * (B * (m.irreps_in1.dim + m.irreps_in2.dim + m.irreps_out.dim) + m.weight_numel), "flops": 3 * 2 * cells * B}
    m = _linear_module(case["channels"], case["l_max"], case["classes"])
    N, C = case["nodes"], case["channels"]
    return {"bytes": 4 * (4 * N * m.irreps_in.dim + 2 * case["classes"] * m.weight_numel), "flops": 3 * 2 * N * m.irreps_in.dim * C}


def tolerance(case):
    # about four times the distance from the same pass evaluated in 64 bits.  The tensor core does not round its
    # 32-bit sums to nearest, which shows where a sum is long: the layers on float32-accurate GEMMs
    if case.get("dtype") == "float64":
        return {"rel": 2e-15}
    if case.get("dtype") == "bfloat16":
        return {"rel": 1.2e-2}
    return {"rel": {"conv": 1e-6, "interaction": 1.5e-5, "force_training": 1.5e-6, "contraction": 3e-6, "fully_connected": 4e-5,
                    "node_linear": 1.5e-5}[case["op"]]}
