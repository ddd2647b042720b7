"""Performance cases of the framework: what its users run, over the sizes they run it at.

Five kinds of pass, each through the public entry points:

  infer      ``Latticeformer.forward`` in eval mode on one batch on the GPU (property prediction, screening)
  serve      a stream of pinned host batches through ``serving.PipelinedPredictor`` (input copies and results included)
  train      one training step of ``Latticeformer``: forward, L1 loss, backward; loss and every gradient come back
  operators  the drop-in operator pair of ``cuda_funcs`` (lattice sums with the value projection, then the edge-indexed
             attention), forward and backward, as the reference's own host code calls them once per layer
  lattice    ``ops.lattice_sum_fwd`` with one Gaussian width per (pair, head): the log-sum-exp and the 64-bin expansion

Everything is float32, the framework's one data type; the options in use are the value encoding (64 bins, or none in the
simplified model), the depth, the domain of the lattice sum (real space, or half the heads in reciprocal space), and the
crystals: few or many, small cells (lattice lengths 3-15 A) or large ones (100-200 atoms, 10-25 A)."""
import math
import types

import numpy as np
import torch

from crystalformer_b200 import ops
from crystalformer_b200.cuda_funcs import (FusedDotProductAttentionCUDA, RealPeriodicEncodingWithProjFuncCUDA,
                                           compile_kernels)
from crystalformer_b200.model import Latticeformer, default_params
from crystalformer_b200.serving import PipelinedPredictor
from crystalformer_b200.synthetic import lognormal_atoms, make_crystals, uniform_atoms

HEADS, HEAD_DIM, MODEL_DIM, FF_DIM = 8, 16, 128, 512
SMALL_CELLS = dict(length_lo=3.0, length_hi=15.0)
LARGE_CELLS = dict(length_lo=10.0, length_hi=25.0)


def _case(kind, crystals, lo, hi, layers=4, bins=64, domain="real", law="uniform", batches=1, cells=SMALL_CELLS):
    return dict(kind=kind, crystals=crystals, atoms_lo=lo, atoms_hi=hi, law=law, layers=layers, bins=bins, domain=domain,
                batches=batches, **cells)


def listed():
    cases = {
        # one structure at a time, as an interactive prediction or a relaxation loop asks for: launches and host time
        "infer-single": _case("infer", 1, 8, 8),
        # the default model on a batch of ordinary size (the benchmark's own workload)
        "infer-batch": _case("infer", 128, 1, 30),
        # the simplified model: seven layers, no value encoding, crystals of log-normal size as in a materials database
        "infer-simplified": _case("infer", 256, 1, 60, layers=7, bins=0, law="lognormal"),
        # cells of a hundred and more atoms: long rows, few images of each pair
        "infer-large-cells": _case("infer", 64, 100, 200, cells=LARGE_CELLS),
        # screening of many candidates in one large batch
        "infer-screening": _case("infer", 1024, 1, 60),
        # a service or a screening loop fed from the host: a run of batches, several in flight
        "serve-stream": _case("serve", 128, 1, 30, batches=16),
        # a training step on a small batch (fine-tuning, the share of one of many GPUs)
        "train-small-batch": _case("train", 8, 1, 40),
        # a training step of the benchmark's size
        "train-batch": _case("train", 256, 1, 40),
        # a training step on large cells
        "train-large-cells": _case("train", 16, 100, 200, cells=LARGE_CELLS),
        # half the heads real-space, half reciprocal-space (domain "multihead"): the operator pair and the reciprocal sum
        "train-multihead": _case("train", 64, 1, 40, domain="multihead"),
        # the reference's host code on the drop-in operators: one layer's calls, forward and backward
        "operators-pair": _case("operators", 64, 1, 40),
        # the lattice-sum kernels by themselves, about 250,000 pairs of eight heads
        "lattice-sum": _case("lattice", 180, 1, 64),
    }
    return [dict(case, name=name) for name, case in cases.items()]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(("infer", "infer", "infer", "serve", "train", "train", "train", "operators", "lattice"))
    if kind in ("infer", "train") and rng.random() < 0.25:
        lo, hi, law, cells = rng.randint(61, 140), rng.randint(141, 200), "uniform", LARGE_CELLS
        crystals = _log_int(rng, 1, 64 if kind == "infer" else 16)
    else:
        lo, hi, cells = 1, _log_int(rng, 6, 64), SMALL_CELLS
        law = rng.choice(("uniform", "uniform", "lognormal"))
        crystals = _log_int(rng, *{"infer": (1, 1024), "serve": (16, 256), "train": (4, 256), "operators": (8, 128),
                                   "lattice": (8, 256)}[kind])
    layers, bins, domain = 4, 64, "real"
    if kind in ("infer", "serve") and rng.random() < 0.3:
        layers, bins = 7, 0
    elif kind == "train" and cells is SMALL_CELLS and rng.random() < 0.2:
        domain, crystals = "multihead", min(crystals, 64)
    elif kind == "train" and rng.random() < 0.25:
        bins = 0
    case = _case(kind, crystals, lo, hi, layers, bins, domain, law, 16 if kind == "serve" else 1, cells)
    most = max(_cost(c) for c in listed() if c["kind"] == kind and c["domain"] == domain)
    while _cost(case) > most:
        case["crystals"] = case["crystals"] * 4 // 5
    return case


# ------------------------------------------------------------------------------------------------------------------------
def _crystals(case, seed):
    lo, hi = case["atoms_lo"], case["atoms_hi"]
    atoms = lognormal_atoms(min(8.0, hi), 0.75, lo, hi) if case["law"] == "lognormal" else uniform_atoms(lo, hi)
    if case["kind"] in ("operators", "lattice"):
        # outputs per atom and per pair: the same crystal sizes, in another order, for every seed
        sizes = atoms(np.random.Generator(np.random.PCG64(17)), case["crystals"])
        atoms = lambda rng, b: rng.permutation(sizes)
    return make_crystals(seed, case["crystals"], atoms, length_range=(case["length_lo"], case["length_hi"]))


def _host_batch(cb):
    return types.SimpleNamespace(x=torch.from_numpy(cb.x), pos=torch.from_numpy(cb.pos),
                                 trans_vec=torch.from_numpy(cb.trans_vec), sizes=torch.from_numpy(cb.sizes))


def _moved(batch, move):
    return types.SimpleNamespace(**{name: move(t) for name, t in vars(batch).items()})


def _to_gpu(batch):
    return _moved(batch, lambda t: t.cuda())


def _model(case, seed, batch):
    """A model whose width statistics are set, as after its first training step."""
    torch.manual_seed(seed)
    model = Latticeformer(default_params(num_layers=case["layers"], value_pe_dist_real=case["bins"], domain=case["domain"]))
    model = model.cuda().train()
    with torch.no_grad():
        model(batch)
    return model


def _geometry(cb):
    """Edge list, relative positions and reciprocal rows of a batch, as an encoder keeps them for all of its layers."""
    dev = _to_gpu(_host_batch(cb))
    atom_start, edge_start = ops.crystal_offsets(dev.sizes)
    geo = ops.batch_prepare(dev.pos, dev.trans_vec, dev.sizes, atom_start, edge_start, cb.num_atoms, cb.num_edges)
    return dev, geo


def _widths(gen, *shape):
    """Gaussian parameters of standard deviations 1.4 (0.5 + U(0,1)) A."""
    sigma = 1.4 * (0.5 + torch.rand(shape, generator=gen, device="cuda"))
    return -0.5 / (sigma * sigma)


def prepare(case, seed):
    kind = case["kind"]
    cb = _crystals(case, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = types.SimpleNamespace(kind=kind)
    if kind == "infer":
        s.batch = _to_gpu(_host_batch(cb))
        s.model = _model(case, seed, s.batch).eval()
    elif kind == "serve":
        hosts = [cb] + [_crystals(case, seed + 1000003 * i) for i in range(1, case["batches"])]
        s.batches = [_moved(_host_batch(h), lambda t: t.pin_memory()) for h in hosts]
        model = _model(case, seed, _to_gpu(s.batches[0])).eval()
        s.runner = PipelinedPredictor(model, depth=6, streams=4)
    elif kind == "train":
        s.batch = _to_gpu(_host_batch(cb))
        s.model = _model(case, seed, s.batch)
        s.weights = {n: p for n, p in s.model.named_parameters() if p.requires_grad}
        s.target = torch.randn((cb.num_crystals, 1), generator=gen, device="cuda")
    elif kind == "operators":
        compile_kernels(2, HEADS, HEAD_DIM, case["bins"], HEAD_DIM, True)
        dev, s.geo = _geometry(cb)
        s.tvecs, s.bins = dev.trans_vec, case["bins"]
        shape = (cb.num_atoms, HEADS, HEAD_DIM)
        s.q, s.k, s.v, s.gout = (torch.randn(shape, generator=gen, device="cuda") for _ in range(4))
        s.q *= 0.25  # (a query comes divided by the root of the head width)
        s.W = torch.randn((1, HEADS, HEAD_DIM, case["bins"]), generator=gen, device="cuda") * 0.1
        s.a = _widths(gen, cb.num_atoms, HEADS)
        for t in (s.q, s.k, s.v, s.a, s.W):
            t.requires_grad_()
    else:
        dev, s.geo = _geometry(cb)
        s.tvecs, s.bins = dev.trans_vec, case["bins"]
        s.a = _widths(gen, cb.num_edges, HEADS)
    return s


def run(s):
    if s.kind == "infer":
        with torch.no_grad():
            return s.model(s.batch)
    if s.kind == "serve":
        results, tickets = [], []
        for batch in s.batches:
            if len(tickets) == s.runner.depth:
                results.append(s.runner.result(tickets.pop(0)).clone())
            tickets.append(s.runner.submit(batch))
        return results + [s.runner.result(t).clone() for t in tickets]
    if s.kind == "train":
        for w in s.weights.values():
            w.grad = None
        loss = (s.model(s.batch) - s.target).abs().mean()
        loss.backward()
        return {"loss": loss.detach(), **{n: w.grad for n, w in s.weights.items()}}
    g = s.geo
    if s.kind == "operators":
        phi, values = RealPeriodicEncodingWithProjFuncCUDA.apply(
            s.a, g["pos_ij"], None, s.tvecs, g["batch"], g["edges"], s.bins, 14.0, 1.0, s.W, g["rvlen"], -3.5)
        out = FusedDotProductAttentionCUDA.apply(s.q, s.k, s.v, phi, values, g["batch"], g["edges"])
        return [out.detach()] + list(torch.autograd.grad(out, (s.q, s.k, s.v, s.a, s.W), s.gout))
    return ops.lattice_sum_fwd(s.a, g["pos_ij"], s.tvecs, g["batch"], g["edges"], s.bins, 14.0, 1.0, rvlen=g["rvlen"],
                               cutoff_radius=-3.5, lattice_range=2, minimum_range=2, a_per_edge=True)


# ------------------------------------------------------------------------------------------------------------------------
def _expected(case):
    """Expected atoms, pairs and (pair, image) terms of a batch.  The images that count are those within 8.1 A of an
    atom, where a Gaussian of the default 1.4 A has fallen to 2^-24 (a float32's precision), and one per pair at least."""
    lo, hi, count = case["atoms_lo"], case["atoms_hi"], case["crystals"]
    sample = make_crystals(17, 2000, lambda rng, b: np.ones(b, dtype=np.int64),
                           length_range=(case["length_lo"], case["length_hi"]))
    density = float(np.mean(1.0 / np.abs(np.linalg.det(sample.trans_vec.astype(np.float64)))))
    if case["law"] == "lognormal":
        n = lognormal_atoms(min(8.0, hi), 0.75, lo, hi)(np.random.Generator(np.random.PCG64(17)), 20000).astype(np.float64)
    else:
        n = np.arange(lo, hi + 1, dtype=np.float64)
    atoms, pairs = count * float(np.mean(n)), count * float(np.mean(n * n))
    return atoms, pairs, pairs * (1.0 + density * 4.0 / 3.0 * math.pi * 8.07 ** 3)


def work(case):
    """Each input read once, each output written once.  A term costs an exponential and an addition per head and, with a
    value encoding, the 13 bins on which the basis is not negligible: an exponential each and a product-sum per head."""
    atoms, pairs, terms = _expected(case)
    K, kind = case["bins"], case["kind"]
    per_term = 2.0 * HEADS + (13 * (1 + 2 * HEADS) if K else 0)
    attention = pairs * HEADS * 4.0 * HEAD_DIM  # q.k and p.v
    projected = 2.0 * HEADS * HEAD_DIM * K      # W psi, once per atom or per pair
    if kind == "lattice":
        return {"bytes": pairs * (4 * HEADS + 12 + 16) + 4 * pairs * HEADS * (1 + K), "flops": terms * per_term}
    if kind == "operators":
        return {"bytes": pairs * (12 + 16) + 4 * atoms * (9 * HEADS * HEAD_DIM + 2 * HEADS) + 4 * 2 * HEADS * HEAD_DIM * K,
                "flops": 3.0 * (terms * per_term + attention + atoms * projected)}
    weights = 98 * MODEL_DIM + case["layers"] * (4 * MODEL_DIM ** 2 + 2 * MODEL_DIM * FF_DIM + MODEL_DIM * K) \
        + MODEL_DIM ** 2
    dense = 2.0 * atoms * (4 * MODEL_DIM ** 2 + 2 * MODEL_DIM * FF_DIM)
    layer = dense + attention + terms * per_term + atoms * projected
    passes, reads = (3.0, 2.0) if kind == "train" else (1.0, 1.0)
    inputs = atoms * (98 * 4 + 12) + case["crystals"] * (36 + 8 + 4)
    return {"bytes": case["batches"] * inputs + reads * 4 * weights,
            "flops": case["batches"] * passes * case["layers"] * layer}


def _cost(case):
    """Of a draw against the listed cases: operations, and pairs (whose tables fill the large cells' time)."""
    return work(case)["flops"] + 1e4 * case["batches"] * case["layers"] * _expected(case)[1]


def tolerance(case):
    # Sums of float32 products in another order, exponentials of a few units in the last place.  The derivative of the ReLU
    # is a step: among a million hidden units the few within rounding of zero may fall on either side, each of which moves
    # a column of a gradient (a 1e-6 change of the weights moves gradients by up to 2.6e-3, single values by 0.18).
    if case["kind"] == "train":
        return {"rel": 4e-3, "max": 0.3}
    if case["kind"] == "operators":
        return {"rel": 5e-5, "max": 2e-3}
    if case["kind"] == "lattice":
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 5e-5, "max": 2e-3}  # (one value per crystal, at times a small difference of larger terms)
