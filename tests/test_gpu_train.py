"""The training step in two library calls (crystalformer_b200.training) against the autograd path of the same model."""
import copy
import types

import numpy as np
import pytest
import torch

from crystalformer_b200.synthetic import make_crystals

pytestmark = pytest.mark.gpu


def step(model, data, target, native):
    model.native = native
    for p in model.parameters():
        p.grad = None
    y = model(data)
    (y - target).abs().mean().backward()
    return y.detach(), {n: p.grad for n, p in model.named_parameters() if p.requires_grad}


def setup(sizes, lengths=(4.0, 12.0), **params):
    from crystalformer_b200.model import Latticeformer, default_params
    torch.manual_seed(len(sizes))
    model = Latticeformer(default_params(**params)).cuda().train()
    for p in model.parameters():
        if p.requires_grad:
            p.data.add_(torch.randn_like(p) * 0.02)
    cb = make_crystals(5, len(sizes), lambda rng, b: np.array(sizes), length_range=lengths)
    t = lambda x: torch.as_tensor(x).cuda()
    data = types.SimpleNamespace(x=t(cb.x), pos=t(cb.pos), trans_vec=t(cb.trans_vec), sizes=t(cb.sizes))
    with torch.no_grad():
        model(data)  # sets the width statistics
    return model, data, torch.randn((len(sizes), model.mlp[3].out_features), device="cuda")


@pytest.mark.parametrize("params", [dict(num_layers=2), dict(num_layers=3, value_pe_dist_real=0), dict(num_layers=1, ff_dim=128),
                                    dict(num_layers=2, ff_dim=256, targets=["a", "b", "c"], embedding_dim=[256]),
                                    dict(num_layers=2, domain="multihead"), dict(num_layers=1, domain="multihead", value_pe_dist_real=0),
                                    dict(num_layers=2, domain="reci"), dict(num_layers=2, domain="RECI"),
                                    dict(num_layers=2, domain="real-reci")])
@pytest.mark.parametrize("sizes", [[1], [3, 60, 64], [33] * 4 + [1], [100, 128, 129], [7] * 130])
def test_gradients_equal_the_autograd_path(params, sizes):
    """Row tiles of 128 (one row, a full tile, one more), chunks of 64 rows, crystals of one atom and of more than 64."""
    model, data, target = setup(sizes, lengths=(8.0, 14.0) if max(sizes) > 64 else (4.0, 12.0), **params)
    y0, ref = step(model, data, target, native=False)
    y1, got = step(model, data, target, native=True)
    assert getattr(model, "_train_plan", None) is not None
    assert (y0 - y1).abs().max() < 2e-6
    # (a single atom's soft-max has no gradient: what is left of q's and k's is rounding of the others)
    noise = 1e-6 * max(float(g.norm()) for g in ref.values())
    for name in ref:
        scale = ref[name].norm()
        # a hidden unit within rounding of zero may fall on either side of the ReLU: one column of one gradient moves
        assert (got[name] - ref[name]).norm() <= 2e-3 * scale + noise, (name, float((got[name] - ref[name]).norm() / scale))
    again = step(model, data, target, native=True)[1]
    assert all(torch.equal(got[n], again[n]) for n in got)  # no atomics in any sum


@pytest.mark.parametrize("bins", [64, 0])
@pytest.mark.parametrize("sizes,lengths", [([8] * 80, (3.0, 9.0)), ([8] * 79, (3.0, 9.0)), ([12] * 80, (3.0, 9.0)),
                                           (list(range(1, 41)) * 2, (3.0, 12.0)), ([64] * 20, (6.0, 14.0)), ([65] + [64] * 20, (8.0, 14.0)),
                                           (list(range(1, 41)) * 6 + [30] * 16, (3.0, 15.0))])
def test_gradients_over_pair_grids(sizes, lengths, bins):
    """On either side of the rule by which a step's attention goes over pair grids (640 or 960 rows, 64 atoms) and at 256 crystals, with
    some rows left over (a narrow head): as the autograd path, whose attention enumerates; two steps' graphs at once.  With no
    hidden unit near the step of its ReLU the two differ by float32 rounding: 5e-6
    of a gradient (sums over thousands of rows) and 2^-24 of the largest one, whose terms cancel in the attention's."""
    model, data, target = setup(sizes, lengths=lengths, num_layers=2, value_pe_dist_real=bins)
    with torch.no_grad():  # one head's widths from narrow to wide, by the atom; no hidden unit near the step of its ReLU
        model.encoder.layers[1].self_attn.q_proj_weight[:16].mul_(6.0)
        for b in [model.mlp[0].bias] + [layer.linear1.bias for layer in model.encoder.layers]:
            b.copy_(torch.sign(torch.randn_like(b)) * 3.0)
    nearest = []
    hooks = [layer.linear1.register_forward_hook(lambda m, i, o: nearest.append(float(o.detach().abs().min()))) for layer in model.encoder.layers]
    y0, ref = step(model, data, target, native=False)
    for hook in hooks:
        hook.remove()
    y1, got = step(model, data, target, native=True)
    assert model._train_plan is not None
    assert (y0 - y1).abs().max() < 2e-6 * max(1.0, float(y0.abs().max()))
    assert min(nearest) > 1e-5 and len(nearest) == 2
    noise = 2.0 ** -24 * max(float(g.norm()) for g in ref.values())
    for name in ref:
        assert (got[name] - ref[name]).norm() <= 5e-6 * ref[name].norm() + noise, name
    for p in model.parameters():
        p.grad = None
    first, second = (model(data) for _ in range(2))
    (second - target).abs().mean().backward()
    again = {n: p.grad.clone() for n, p in model.named_parameters() if p.requires_grad}
    (first - target).abs().mean().backward()
    assert all(torch.equal(got[n], again[n]) for n in got)
    assert all(torch.equal(2 * again[n], p.grad) for n, p in model.named_parameters() if p.requires_grad)


@pytest.mark.parametrize("crystals", [2048, 2049])
def test_batches_with_and_without_an_order_of_rows(crystals):
    """The preparation orders the rows of up to 2048 crystals; forward and backward agree on whether it has."""
    model, data, target = setup([2] * crystals, num_layers=1)
    ref, got = step(model, data, target, native=False)[1], step(model, data, target, native=True)[1]
    assert model._train_plan is not None
    for name in ref:
        assert (got[name] - ref[name]).norm() <= 2e-3 * ref[name].norm() + 1e-9, name


def test_step_follows_the_model():
    """In-place updates, replaced parameters, copies and frozen parameters; a modified weight between the two halves."""
    model, data, target = setup([9, 20, 5], num_layers=2)
    step(model, data, target, native=True)
    with torch.no_grad():
        for p in model.parameters():
            if p.requires_grad:
                p.sub_(0.01 * p.grad)
    model.mlp[3].weight = torch.nn.Parameter(model.mlp[3].weight.detach() * 1.5)
    model.encoder.layers[0].linear1.weight.requires_grad_(False)
    clone = copy.deepcopy(model)
    for m in (model, clone):
        ref, got = step(m, data, target, native=False)[1], step(m, data, target, native=True)[1]
        assert "encoder.layers.0.linear1.weight" not in got
        for name in ref:
            assert (got[name] - ref[name]).norm() <= 2e-3 * ref[name].norm() + 1e-9, name
    loss = model(data).sum()
    with torch.no_grad():
        model.mlp[0].bias.add_(1.0)
    with pytest.raises(RuntimeError, match="in-place"):
        loss.backward()


@pytest.mark.parametrize("bins", [0, 64])
@pytest.mark.parametrize("sizes,lengths", [([64, 65], (8.0, 14.0)), ([200], (10.0, 20.0)), ([201, 65, 1], (10.0, 20.0)),
                                           ([1, 2, 3, 4, 5, 8, 9, 16, 17], (3.0, 4.0)), ([33] * 40, (5.0, 11.0)),
                                           ([30] * 320, (5.0, 11.0))])
def test_forward_at_the_edges_of_its_dispatch(sizes, lengths, bins):
    """The one-call forward and the training step's against the autograd path: blocks of rows (65 to 200 atoms) or not, rows of
    few keys whose boxes are dealt over lanes, two warps per row (1,200 rows), heavy rows to one warp each (9,500 rows)."""
    model, data, target = setup(sizes, lengths=lengths, num_layers=2, value_pe_dist_real=bins)
    model.native = False
    y0 = model(data).detach()
    model.native = True
    y1 = model(data).detach()
    with torch.no_grad():
        y2 = model.eval()(data)
    scale = max(1.0, float(y0.abs().max()))
    assert (y0 - y1).abs().max() < 2e-6 * scale
    assert (y0 - y2).abs().max() < 2e-6 * scale


def test_saved_tensors_that_come_back_elsewhere():
    """Saved-tensor hooks (offloading, checkpointing) and parameters whose storage is replaced between forward and backward."""
    from torch.autograd.graph import save_on_cpu, saved_tensors_hooks
    from torch.utils.checkpoint import checkpoint
    model, data, target = setup([9, 20, 5, 66], lengths=(8.0, 14.0), num_layers=2)
    ref = step(model, data, target, native=True)[1]

    def grads(y):
        for p in model.parameters():
            p.grad = None
        fill = [torch.full((64 << 20,), 255, dtype=torch.uint8, device="cuda") for _ in range(2)]  # what the forward freed is reused
        (y - target).abs().mean().backward()
        del fill
        return {n: p.grad for n, p in model.named_parameters() if p.requires_grad}

    def with_hooks():
        with save_on_cpu():
            return model(data)

    def with_copies():
        with saved_tensors_hooks(lambda t: t.clone(), lambda t: t.clone()):
            return model(data)

    def replaced():
        y = model(data)
        for p in model.parameters():
            p.data = p.data.clone()
        return y

    for forward in (with_hooks, with_copies, lambda: checkpoint(model, data, use_reentrant=False), replaced, lambda: model(data)):
        got = grads(forward())
        assert all(torch.equal(got[n], ref[n]) for n in ref)
    # the positions are not needed any more after the forward
    y = model(data)
    data.pos.add_(0.0)
    assert all(torch.equal(g, ref[n]) for n, g in grads(y).items())


@pytest.mark.parametrize("bins", [0, 64])
@pytest.mark.parametrize("sizes", [[65] * 12, [64] * 12, [210, 100, 1] * 4, [211, 100, 1] * 4, [66] + [31] * 30, [66] + [32] * 30, [150] * 4 + [139],
                                   [150] * 4 + [140], [200, 3, 77] * 8])
def test_forward_by_blocks_of_rows_or_not(sizes, bins):
    """Both sides of every line of the rule: crystals of 64 and 65, of 210 and 211 atoms, 32 atoms on average, 740 rows."""
    test_forward_at_the_edges_of_its_dispatch(sizes, (10.0, 20.0), bins)


def test_parameters_that_are_views_at_odd_places():
    """Parameters flattened into one vector: what the kernels' wide loads cannot read takes the operation-by-operation path."""
    model, data, target = setup([9, 20, 5], num_layers=2, value_pe_dist_real=0)
    ref = step(model, data, target, native=False)
    trained = [p for p in model.parameters() if p.requires_grad]
    flat = torch.empty(sum(p.numel() for p in trained) + 1, device="cuda")
    at = 1
    for p in trained:
        flat[at:at + p.numel()] = p.data.reshape(-1)
        p.data = flat[at:at + p.numel()].view(p.shape)
        at += p.numel()
    model._train_plan = None
    got = step(model, data, target, native=True)
    assert model._train_plan is None
    assert (got[0] - ref[0]).abs().max() < 2e-6
    for n, g in ref[1].items():
        assert (got[1][n] - g).norm() <= 2e-3 * g.norm() + 1e-9, n


class Scaled(torch.nn.Linear):
    def forward(self, x):
        return 1.5 * super().forward(x)


class Doubled(torch.nn.Module):
    def forward(self, W):
        return 2.0 * W


def _hook(model, seen):
    model.encoder.layers[1].linear1.register_forward_hook(lambda m, i, o: (seen.append(1), o * 1.5)[1])


def _pre_hook(model, seen):
    model.encoder.register_forward_pre_hook(lambda m, i: seen.append(1))


def _backward_hook(model, seen):
    model.encoder.layers[0].linear2.register_full_backward_hook(lambda m, gi, go: seen.append(1))


def _parametrised(model, seen):
    torch.nn.utils.parametrize.register_parametrization(model.encoder.layers[0].linear2, "weight", Doubled())


def _subclass(model, seen):
    old = model.encoder.layers[0].linear1
    new = Scaled(old.in_features, old.out_features).cuda()
    new.load_state_dict(old.state_dict())
    model.encoder.layers[0].linear1 = new


def _own_forward(model, seen):
    layer = model.encoder.layers[1].linear2
    layer.forward = lambda x: (seen.append(1), 0.5 * torch.nn.functional.linear(x, layer.weight, layer.bias))[1]


def _layer_norm(model, seen):
    model.encoder.layers[0].norm2 = torch.nn.LayerNorm(128).cuda()


@pytest.mark.parametrize("change", [_hook, _pre_hook, _backward_hook, _parametrised, _subclass, _own_forward, _layer_norm])
def test_changed_submodules_take_effect(change):
    """What a user hangs on a submodule after the first step: the steps follow it, with updates of the weights in between."""
    import torch.nn.utils.parametrize  # noqa: F401
    model, data, target = setup([9, 20, 5], num_layers=2)
    step(model, data, target, native=True)
    assert model._train_plan is not None
    seen = []
    change(model, seen)
    for _ in range(2):
        (y0, ref), calls = step(model, data, target, native=False), len(seen)
        y1, got = step(model, data, target, native=True)
        assert len(seen) == 2 * calls
        seen.clear()
        assert torch.equal(y0, y1) and all(torch.equal(ref[n], got[n]) for n in ref)
        with torch.no_grad():
            for n, p in model.named_parameters():
                if p.requires_grad:
                    p.sub_(0.01 * got[n])


def test_hooks_of_all_modules_and_dropout():
    model, data, target = setup([9, 20, 5], num_layers=2)
    for layer in model.encoder.layers:
        layer.dropout2 = torch.nn.Dropout(0.0)
    step(model, data, target, native=True)
    assert model._train_plan is not None
    seen = []
    handle = torch.nn.modules.module.register_module_forward_hook(lambda m, i, o: seen.append(type(m)))
    step(model, data, target, native=True)
    handle.remove()
    assert torch.nn.Linear in seen
    model.encoder.layers[1].dropout2.p = 0.9  # the next step drops units
    a, b = (step(model, data, target, native=True)[0] for _ in range(2))
    assert not torch.equal(a, b)


def test_directional_derivatives_are_not_dropped():
    """A tangent on an input is refused by the operators (they define none) and not ignored."""
    import torch.autograd.forward_ad as fwad
    model, data, target = setup([9, 5], num_layers=1)
    with fwad.dual_level():
        data.x = fwad.make_dual(data.x, torch.ones_like(data.x))
        with pytest.raises((RuntimeError, NotImplementedError)):
            model(data)


@pytest.mark.parametrize("sizes", [[12] * 80, [9, 20, 5]])
def test_the_weight_floor_of_a_step(sizes):
    """A floor that nodes cannot serve (-1000: every term) keeps a step off the pair grids, and a floor that changes between the halves
    of a step does not change the way that its second half takes (80 crystals: grids, three: term lists)."""
    from crystalformer_b200 import ops
    model, data, target = setup(sizes, lengths=(4.0, 9.0), num_layers=2)
    rows = torch.zeros(4, dtype=torch.int64, device="cuda")

    def gradients(first, second):
        rows.zero_()
        ops.set_row_stats(rows)
        try:
            ops.set_weight_floor_log2(first)
            for p in model.parameters():
                p.grad = None
            loss = (model(data) - target).abs().mean()
            ops.set_weight_floor_log2(second)
            loss.backward()
        finally:
            ops.set_weight_floor_log2(-30.0)
            ops.set_row_stats(None)
        return {n: p.grad for n, p in model.named_parameters() if p.requires_grad}, int(rows[2])

    usual, by_grid = gradients(-30.0, -30.0)
    whole, enumerated = gradients(-1000.0, -1000.0)
    assert model._train_plan is not None
    assert enumerated == 0 and (by_grid > 0) == (len(sizes) > 3)
    noise = 1e-6 * max(float(g.norm()) for g in whole.values())
    for halves, ref in (((-30.0, -1000.0), usual), ((-1000.0, -30.0), whole), ((-40.0, -30.0), usual)):
        got, _ = gradients(*halves)
        for n in ref:  # (as between two kernels: a hidden unit within rounding of zero)
            assert (got[n] - ref[n]).norm() <= 2e-3 * ref[n].norm() + noise, (halves, n)
