"""The training step's dense products against 64 bits, beside the operator path (float32 GEMMs) on the same inputs.

Crystals of one atom and no value encoding: the soft-max has one entry, so the attention passes v through and the model is its dense
part, which plain torch computes in float64.  Biases of the hidden units are +-3 so that no unit is near the step of its ReLU."""
import types

import pytest
import torch

pytestmark = pytest.mark.gpu


def dense_model(ff, layers, spread):
    from crystalformer_b200.model import Latticeformer, default_params
    torch.manual_seed(ff + layers)
    model = Latticeformer(default_params(num_layers=layers, ff_dim=ff, value_pe_dist_real=0, targets=["a", "b", "c"])).cuda().train()
    with torch.no_grad():
        for n, p in model.named_parameters():
            if p.requires_grad:
                p.add_(torch.randn_like(p) * spread)
            if n.endswith("linear1.bias") or n == "mlp.0.bias":
                p.copy_(torch.sign(torch.randn_like(p)) * 3.0)
    return model


def exact(model, x, gy):
    """Outputs and gradients of the dense part in float64."""
    P = {n: p.detach().double().requires_grad_() for n, p in model.named_parameters()}
    lin = torch.nn.functional.linear
    z = lin(x.double(), P["input_embeddings.weight"])
    for i in range(len(model.encoder.layers)):
        w = lambda n: P[f"encoder.layers.{i}.{n}"]
        v = lin(z, w("self_attn.v_proj_weight"), w("self_attn.in_proj_bias")[256:])
        z = z + lin(v, w("self_attn.out_proj.weight"), w("self_attn.out_proj.bias"))
        z = z + lin(torch.relu(lin(z, w("linear1.weight"), w("linear1.bias"))), w("linear2.weight"), w("linear2.bias"))
    y = lin(torch.relu(lin(z, P["mlp.0.weight"], P["mlp.0.bias"])), P["mlp.3.weight"], P["mlp.3.bias"])
    y.backward(gy.double())
    return y.detach(), {n: p.grad for n, p in P.items() if p.grad is not None}


@pytest.mark.parametrize("ff,layers,atoms,spread", [(512, 4, 189, 0.0), (512, 4, 2425, 0.0), (512, 2, 5321, 0.02), (512, 2, 9600, 0.0),
                                                    (128, 2, 5000, 0.02), (384, 3, 700, 0.0), (640, 2, 300, 0.0)])
def test_errors_are_those_of_float32_products(ff, layers, atoms, spread):
    model = dense_model(ff, layers, spread)
    x = torch.randn((atoms, 98), device="cuda")
    data = types.SimpleNamespace(x=x, pos=torch.rand((atoms, 3), device="cuda"), sizes=torch.ones(atoms, dtype=torch.int64, device="cuda"),
                                 trans_vec=(6.0 * torch.eye(3, device="cuda")).repeat(atoms, 1, 1))
    with torch.no_grad():
        model(data)
    gy = torch.randn((atoms, 3), device="cuda")
    y64, g64 = exact(model, x, gy)
    rel = lambda a, b: float((a.double() - b).norm() / b.norm())
    off = {}
    for native in (False, True):
        model.native = native
        model.zero_grad(set_to_none=True)
        y = model(data)
        y.backward(gy)
        off[native] = {"y": rel(y.detach(), y64)}
        for n, p in model.named_parameters():
            if p.grad is not None and n in g64 and float(g64[n].norm()) > 0 and "in_proj" not in n:
                off[native][n] = rel(p.grad, g64[n])
    assert model._train_plan is not None
    print({n: (f"{e:.2e}", f"{e / off[False][n]:.2f}") for n, e in off[True].items()})
    for n, e in off[True].items():
        assert e <= BOUND(off[False][n]), (n, e, off[False][n])


# No further off than the float32 products, a tenth for chance (norms over thousands of values; a bias gradient is a few
# values or a hundred, each a few roundings of 2^-24).  Sums in a tensor-core accumulator are 2 to 40 times as far off.
BOUND = lambda float32: max(1.1 * float32, 4 * 2.0 ** -24)
