"""Training step of the model shell in two library calls (cf_train_forward / cf_train_backward) behind one autograd node.

``Latticeformer.forward`` takes it whenever gradients are enabled, the configuration is the one the calls implement and the
submodules are the model's own (they are not called: a hook, a parametrisation or another class in their place would not
take effect): the node's inputs are the model's parameters, its backward returns all of their gradients.  Same values as the
operation-by-operation autograd path (models/latticeformer.py:211-302 and its backward), which stays for everything else."""
from __future__ import annotations

import ctypes
from operator import is_
from typing import Optional, Tuple

import numpy as np
import torch
from torch.autograd import forward_ad

from . import _lib


class OfThisModel:
    """A cache that belongs to one model object: copies and pickles of the model carry None instead (addresses and ctypes
    structures cannot be copied)."""

    def __init__(self, *values):
        self.values = values

    def __deepcopy__(self, memo):
        return None

    def __reduce__(self):
        return type(None), ()


class ModelWatch:
    """Notices when a model is no longer the one a plan was made for: a submodule, parameter or buffer replaced, moved or
    (with ``versions``) modified in place, or a setting changed."""

    def __init__(self, model, versions: bool, modules=None):
        modules = list(model.modules()) if modules is None else modules
        children = [(m._modules, n, c) for m in modules for n, c in m._modules.items()]
        places = [(d, n, t) for m in modules for d in (m._parameters, m._buffers) for n, t in d.items() if t is not None]
        self.tensors = [t for _, _, t in places]
        self.dicts, self.names, self.values = zip(*(children + places))
        self.versions = versions
        self.settings = model.encoder.lattice_params
        self.layer_settings = [layer.self_attn.params for layer in model.encoder.layers]
        self.dropouts = [m for m in modules if isinstance(m, torch.nn.Dropout)]
        self.attentions = [layer.self_attn for layer in model.encoder.layers]
        self.key = self.now()

    def now(self) -> list:
        P = self.settings  # the scalar settings that the plans of a model contain
        key = [P.lattice_range, P.minimum_range, P.adaptive_cutoff_sigma, P.gauss_lb_real, str(P.scale_real), P.value_pe_dist_real,
               P.value_pe_width_scale, P.value_pe_dist_max]
        for Q in self.layer_settings:
            key += (Q.positive_func, Q.gauss_lb_real, Q.scale_real, Q.value_pe_dist_max, Q.gauss_lb_reci, Q.scale_reci)
        key += [m.p for m in self.dropouts] + [m.dropout for m in self.attentions]
        key += map(torch.Tensor.data_ptr, self.tensors)
        return key + [t._version for t in self.tensors] if self.versions else key

    def current(self) -> bool:
        return all(map(is_, map(dict.get, self.dicts, self.names), self.values)) and self.now() == self.key


DOMAINS = ("real", "reci", "RECI", "multihead")  # in the order of the library's codes


class TrainPlan:
    """What a step needs and the batch does not change: the parameters in the library's order with their addresses, the
    scalar settings, and where every gradient lies in one flat buffer.  Valid while the parameters keep their storage."""

    def __init__(self, model, modules):
        enc = model.encoder
        P = enc.lattice_params
        ordered, scalars = [], []
        for layer in enc.layers:
            att, Q = layer.self_attn, layer.self_attn.params
            ordered += [att.q_proj_weight, att.k_proj_weight, att.v_proj_weight, att.in_proj_bias, att.lattice_pos_weights,
                        att.pe_dist_proj, att.out_proj.weight, att.out_proj.bias, layer.linear1.weight, layer.linear1.bias,
                        layer.linear2.weight, layer.linear2.bias]
            beta = float(Q.positive_func.split("=")[1]) if "=" in Q.positive_func else 1.0
            dist_max = Q.value_pe_dist_max if Q.value_pe_dist_max >= 0 else -Q.value_pe_dist_max * Q.scale_real
            gs = att.gauss_scale.detach().cpu().tolist()
            real, reci = (-0.5 * Q.scale_real ** -2, Q.gauss_lb_real), (-0.5 * Q.scale_reci ** 2, Q.gauss_lb_reci)
            low, high = {"real": (real, real), "multihead": (real, reci)}.get(Q.domain, (reci, reci))
            scalars += [gs[0], gs[1], low[0], beta, low[1], dist_max, *high, DOMAINS.index(Q.domain)]
        ordered += [model.input_embeddings.weight, model.mlp[0].weight, model.mlp[0].bias, model.mlp[3].weight, model.mlp[3].bias]
        self.params = [p for p in ordered if p is not None]
        self.watch = ModelWatch(model, False, modules)
        self.submodules = [m.__dict__ for m in modules if m is not model]
        self.scales = [layer.self_attn.gauss_scale for layer in enc.layers]
        self.scale_versions = [g._version for g in self.scales]
        sizes = [p.numel() for p in self.params]
        # gradients lie one after the other in one buffer
        offsets, at = [], 0
        for n in sizes:
            offsets.append(at)
            at += n
        self.floats = at
        self.like = [p.detach() for p in self.params]  # (and keeps the storage that the addresses name)
        where = iter(range(len(self.params)))
        self.slots = [None if p is None else next(where) for p in ordered]
        # the gradients' places as byte offsets in the library's order (0 and not `present` for a parameter that is not there)
        self.present = np.array([s is not None for s in self.slots], dtype=np.int64)
        self.offsets = np.array([0 if s is None else 4 * offsets[s] for s in self.slots], dtype=np.int64)
        self.pointers = (ctypes.c_void_p * len(ordered))(*[None if p is None else p.data_ptr() for p in ordered])
        self.scalars = (ctypes.c_double * len(scalars))(*scalars)
        self.targets = model.mlp[3].out_features
        order_reach = model.native_reach()
        self.desc = _lib.TrainDesc(
            num_layers=len(enc.layers), lattice_range=int(P.lattice_range),
            minimum_range=int(P.lattice_range) if P.minimum_range else 0, feature_dim=model.input_embeddings.in_features,
            K=int(P.value_pe_dist_real), ff_dim=enc.layers[0].linear1.out_features, hidden=model.mlp[0].out_features,
            targets=self.targets, wscale=float(P.value_pe_width_scale), cutoff_radius=enc._cutoff(), order_reach=order_reach,
            weights=ctypes.cast(self.pointers, ctypes.c_void_p), scalars=ctypes.cast(self.scalars, ctypes.c_void_p))

    def current(self) -> bool:
        return self.watch.current() and [g._version for g in self.scales] == self.scale_versions

    def untouched(self) -> bool:
        """Whether calling the submodules would do nothing but their own forward (hooks of the model itself run in any case)."""
        for d in self.submodules:
            if d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"] or "forward" in d:
                return False
        return not torch.nn.modules.module._has_any_global_hook()

    def versions(self) -> list:
        return [p._version for p in self.params]


def usable(p: torch.Tensor, device) -> bool:
    return p.dtype == torch.float32 and p.is_contiguous() and p.device == device and p.data_ptr() % 16 == 0


def supported(model, modules) -> bool:
    """Whether the submodules are the model's own (a parametrised one has a class of its own) and the parameters what the
    kernels read: float32, contiguous, 16-byte aligned (a parameter may be a view into a longer one), on one GPU, one
    projection per head."""
    from .attention import CrystalformerMultiheadAttentionCUDA, NonDynamicallyQuantizableLinear
    from .encoder import CrystalformerEncoderCUDA, CrystalformerEncoderLayerCUDA
    own = {torch.nn.Linear, NonDynamicallyQuantizableLinear, torch.nn.Identity, torch.nn.ReLU, torch.nn.Dropout, torch.nn.Sequential,
           torch.nn.ModuleList, CrystalformerEncoderCUDA, CrystalformerEncoderLayerCUDA, CrystalformerMultiheadAttentionCUDA}
    if any(type(m) not in own for m in modules if m is not model):
        return False
    enc = model.encoder
    ff = enc.layers[0].linear1.out_features if len(enc.layers) else 0
    hidden = model.mlp[0].out_features
    dev = model.input_embeddings.weight.device
    if dev.type != "cuda" or not 1 <= len(enc.layers) <= 32 or ff % 128 or not 0 < ff <= 3328 or hidden % 128 \
            or not 0 < hidden <= 1024 or model.input_embeddings.in_features > 128:
        return False
    for layer in enc.layers:
        att = layer.self_attn
        Q = att.params
        bins = Q.value_pe_dist_real if Q.domain in ("real", "multihead") else 0
        if layer.linear1.out_features != ff or bins not in (0, 64) or Q.gauss_lb_real <= 0 or Q.gauss_lb_reci <= 0 \
                or isinstance(Q.scale_real, (list, tuple)) or isinstance(Q.scale_reci, (list, tuple)) \
                or (Q.domain != "real" and Q.lattice_range > 6) or att.out_proj.bias is None \
                or (tuple(att.pe_dist_proj.shape) if att.pe_dist_proj is not None else None) != ((1, 8, 16, 64) if bins else None):
            return False
        if any(isinstance(m, torch.nn.Dropout) and m.p > 0 for m in (layer.dropout, layer.dropout1, layer.dropout2)) or att.dropout > 0:
            return False
    return all(usable(p, dev) for m in modules for p in m._parameters.values() if p is not None)


class NotThisBatch(Exception):
    """The calls do not take the batch (a crystal of more than 1024 atoms, atoms outside every crystal)."""


class TrainStep(torch.autograd.Function):
    @staticmethod
    def forward(ctx, plan: TrainPlan, inputs, counts: Optional[Tuple[int, int, int]], *params):
        feats, pos, trans, sizes = inputs
        dev = pos.device
        N, B = pos.shape[0], sizes.shape[0]
        lib = _lib.load()
        desc = ctypes.byref(plan.desc)
        saved = torch.empty(int(lib.cf_train_saved_bytes(desc, N, B)), dtype=torch.uint8, device=dev)
        batch = _lib.TrainBatch(features=feats.data_ptr(), pos=pos.data_ptr(), trans=trans.data_ptr(), sizes=sizes.data_ptr(), N=N, B=B,
                                saved=saved.data_ptr())
        known, event = (ctypes.c_int64 * 3)(*((-1, 0, 0) if counts is None else counts)), ctypes.c_void_p()
        y = torch.empty((B, plan.targets), dtype=torch.float32, device=dev)
        with torch.cuda.device(dev):
            stream = torch.cuda.current_stream(dev).cuda_stream
            _lib.call("cf_train_begin", desc, ctypes.byref(batch), known, ctypes.byref(event), stream)
            try:
                if known[0] != N or known[2] > 1024:
                    raise NotThisBatch
                batch.E, batch.max_atoms = known[1], known[2]
                edges = torch.empty(int(lib.cf_train_edge_bytes(desc, N, B, batch.E)), dtype=torch.uint8, device=dev)
                batch.saved_edges = edges.data_ptr()
                _lib.call("cf_train_forward", desc, ctypes.byref(batch), event, y.data_ptr(), stream)
            except BaseException:  # (the first block still writes to `saved`, on a stream of the library's)
                lib.cf_begin_abandon(event, stream)
                raise
        # (no address is kept: what saved-tensor hooks give back in the backward may lie elsewhere, or be a recomputation)
        ctx.save_for_backward(saved, edges, feats, trans)
        ctx.step = (plan, (N, B, batch.E, batch.max_atoms), batch.floor_log2, plan.versions())
        return y

    @staticmethod
    @torch.autograd.function.once_differentiable
    def backward(ctx, gy):
        plan, (N, B, E, max_atoms), floor, versions = ctx.step
        saved, edges, feats, trans = ctx.saved_tensors
        if plan.versions() != versions:
            raise RuntimeError("a parameter of the model was modified by an in-place operation between the forward and the "
                               "backward of a training step")
        dev = gy.device
        gy = gy.contiguous()
        desc = plan.desc
        batch = _lib.TrainBatch(feats.data_ptr(), None, trans.data_ptr(), None, N, B, E, max_atoms, saved.data_ptr(), edges.data_ptr(), floor)
        scratch = torch.empty(int(_lib.load().cf_train_scratch_bytes(ctypes.byref(desc), N, B, E)), dtype=torch.uint8, device=dev)
        flat = torch.empty(plan.floats, dtype=torch.float32, device=dev)
        where = plan.offsets + flat.data_ptr() * plan.present
        with torch.cuda.device(dev):
            _lib.call("cf_train_backward", ctypes.byref(desc), ctypes.byref(batch), gy.data_ptr(), scratch.data_ptr(),
                      where.ctypes.data, torch.cuda.current_stream(dev).cuda_stream)
        return (None, None, None, *torch._utils._unflatten_dense_tensors(flat, plan.like))


def train_step(model, data, counts: Optional[Tuple[int, int, int]]) -> Optional[torch.Tensor]:
    """The model's output on ``data`` with the step's autograd node behind it, or None when the calls do not apply."""
    cache = getattr(model, "_train_plan", None)
    plan = None if cache is None else cache.values[0]
    if plan is None or not plan.current():
        modules = list(model.modules())
        if not supported(model, modules):
            return None
        plan = TrainPlan(model, modules)
        model._train_plan = OfThisModel(plan)
    if not plan.untouched() or not all([att.term_lists for att in plan.watch.attentions]):
        return None
    if data.x.requires_grad or data.pos.requires_grad or data.trans_vec.requires_grad or torch.is_autocast_enabled() \
            or forward_ad._current_level >= 0:  # (forward-mode derivatives are on: an input may carry a tangent)
        return None
    # the kernels get addresses: what does not have the model's shapes and types, or lies elsewhere, is left to the operators' own checks
    dev, sizes = data.pos.device, data.sizes
    if data.x.device != dev or data.trans_vec.device != dev or data.x.dtype != torch.float32 or data.trans_vec.dtype != torch.float32 \
            or sizes.dim() != 1 or sizes.shape[0] < 1 or data.pos.dim() != 2 or data.pos.shape[1] != 3 \
            or tuple(data.x.shape) != (data.pos.shape[0], plan.desc.feature_dim) \
            or data.trans_vec.numel() != 9 * sizes.shape[0]:
        return None
    f32 = lambda t: t if (t.dtype == torch.float32 and t.is_contiguous()) else t.detach().float().contiguous()
    feats, pos, trans = f32(data.x), f32(data.pos), f32(data.trans_vec)
    if sizes.device != dev or sizes.dtype != torch.int64 or not sizes.is_contiguous():
        sizes = sizes.to(device=dev, dtype=torch.int64).contiguous()
    if pos.shape[0] < 1 or feats.data_ptr() % 16 or plan.params[0].device != dev or (counts is not None and (
            counts[0] != pos.shape[0] or counts[2] > 1024)):
        return None
    try:
        return TrainStep.apply(plan, (feats, pos, trans, sizes), counts, *plan.params)
    except NotThisBatch:
        return None
