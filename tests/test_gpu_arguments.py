"""Batches that do not fit the model: the one-call paths hand addresses to kernels, so the host has to refuse them."""
import types

import numpy as np
import pytest
import torch

from crystalformer_b200.synthetic import make_crystals

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def model_and_batch():
    from crystalformer_b200.model import Latticeformer, default_params
    torch.manual_seed(1)
    model = Latticeformer(default_params(num_layers=1)).cuda()
    cb = make_crystals(5, 3, lambda rng, b: np.array([4, 7, 2]), length_range=(4.0, 9.0))
    t = lambda x: torch.as_tensor(x).cuda()
    data = dict(x=t(cb.x), pos=t(cb.pos), trans_vec=t(cb.trans_vec), sizes=t(cb.sizes))
    model.train()(types.SimpleNamespace(**data))  # sets the width statistics
    return model, data


CHANGES = {
    "features on the host": dict(x=lambda t: t.cpu()),
    "cells on the host": dict(trans_vec=lambda t: t.cpu()),
    "features too wide": dict(x=lambda t: torch.cat((t, torch.zeros((t.shape[0], 40), device=t.device)), 1)),
    "rows of features missing": dict(x=lambda t: t[:-1]),
    "positions missing": dict(pos=lambda t: t[:-1], x=lambda t: t[:-1]),
    "cells missing": dict(trans_vec=lambda t: t[:-1]),
    "features of one dimension": dict(x=lambda t: t.reshape(-1)),
}


@pytest.mark.parametrize("training", [True, False])
@pytest.mark.parametrize("change", sorted(CHANGES))
def test_batches_that_do_not_fit_are_refused(model_and_batch, change, training):
    model, data = model_and_batch
    bad = types.SimpleNamespace(**dict(data, **{n: f(data[n]) for n, f in CHANGES[change].items()}))
    model.train(training)
    counts = (13, 16 + 49 + 4, 7)
    for kw in ({}, {"counts": counts}):
        with torch.set_grad_enabled(training), pytest.raises((RuntimeError, ValueError, IndexError, TypeError)):
            model(bad, **kw)
    with torch.set_grad_enabled(training):  # and nothing is left behind
        assert torch.isfinite(model(types.SimpleNamespace(**data))).all()


def test_narrow_features(model_and_batch):
    """Training refuses a narrower x as its Linear does; inference with packed weights takes the missing columns for zeros."""
    model, data = model_and_batch
    narrow = types.SimpleNamespace(**dict(data, x=data["x"][:, :60].contiguous()))
    padded = types.SimpleNamespace(**dict(data, x=torch.cat((data["x"][:, :60], torch.zeros((13, 38), device="cuda")), 1)))
    with pytest.raises(RuntimeError):
        model.train()(narrow)
    with torch.no_grad():
        model.eval()
        assert torch.allclose(model(narrow), model(padded), rtol=0.0, atol=1e-6)


@pytest.mark.parametrize("name", ["x", "trans_vec"])
def test_other_types_in_training(model_and_batch, name):
    """Training refuses features and cells of another type, as its operators do; positions are converted."""
    model, data = model_and_batch
    model.train()
    with pytest.raises((RuntimeError, TypeError)):
        model(types.SimpleNamespace(**dict(data, **{name: data[name].double()})))
    y = model(types.SimpleNamespace(**dict(data, pos=data["pos"].double())))
    assert torch.equal(y, model(types.SimpleNamespace(**data)))


def test_atoms_beyond_the_crystals(model_and_batch):
    """Rows that no crystal owns are not part of the batch (inference)."""
    model, data = model_and_batch
    more = types.SimpleNamespace(**dict(data, x=torch.cat((data["x"], data["x"][:3])), pos=torch.cat((data["pos"], data["pos"][:3]))))
    with torch.no_grad():
        model.eval()
        assert torch.allclose(model(more), model(types.SimpleNamespace(**data)), rtol=0.0, atol=1e-6)
