"""Bounded waits of the dense kernels: one that runs out is reported as an error, once, and the device stays usable."""
import types

import numpy as np
import pytest
import torch

from crystalformer_b200.synthetic import make_crystals

pytestmark = pytest.mark.gpu


def run_out():
    from crystalformer_b200 import _lib
    _lib.call("cf_wait_probe", 2_000_000, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()


@pytest.fixture(scope="module")
def setup():
    from crystalformer_b200.model import Latticeformer, default_params
    torch.manual_seed(1)
    model = Latticeformer(default_params(num_layers=1)).cuda()
    cb = make_crystals(5, 3, lambda rng, b: np.array([4, 7, 2]), length_range=(4.0, 9.0))
    host = types.SimpleNamespace(x=torch.as_tensor(cb.x), pos=torch.as_tensor(cb.pos), trans_vec=torch.as_tensor(cb.trans_vec),
                                 sizes=torch.as_tensor(cb.sizes))
    data = types.SimpleNamespace(**{n: t.cuda() for n, t in vars(host).items()})
    with torch.no_grad():
        model.train()(data)
    return model, data, host


def test_reported_once():
    from crystalformer_b200 import _lib, ops
    ops.check_waits()
    run_out()
    with pytest.raises(_lib.CrystalformerB200Error, match="ran out") as e:
        ops.check_waits()
    assert e.value.code == -5
    ops.check_waits()


@pytest.mark.parametrize("training", [False, True])
def test_the_next_call_raises_it(setup, training):
    from crystalformer_b200 import _lib
    model, data, _ = setup
    model.train(training)
    with torch.set_grad_enabled(training):
        ref = model(data).detach()
        run_out()
        with pytest.raises(_lib.CrystalformerB200Error, match="ran out"):
            model(data)
        assert torch.equal(model(data).detach(), ref)


def test_backward_raises_it(setup):
    from crystalformer_b200 import _lib
    model, data, _ = setup
    y = model.train()(data)
    run_out()
    with pytest.raises(_lib.CrystalformerB200Error, match="ran out"):
        y.sum().backward()
    model(data).sum().backward()


def test_results_of_a_pipeline_raise_it(setup):
    from crystalformer_b200 import _lib
    from crystalformer_b200.serving import PipelinedPredictor
    model, data, host = setup
    model.eval()
    runner = PipelinedPredictor(model, depth=2)
    ticket = runner.submit(host)
    run_out()
    with pytest.raises(_lib.CrystalformerB200Error, match="ran out"):
        runner.result(ticket)
    run_out()
    with pytest.raises(_lib.CrystalformerB200Error, match="ran out"):
        runner.submit(host)
    out = runner.result(runner.submit(host))
    with torch.no_grad():
        assert torch.equal(out, model(data).cpu())
