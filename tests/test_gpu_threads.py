"""Several host threads on one stream: memory that a call allocates after it has begun its batch may have just been freed to the
stream by another thread whose kernels have not run yet."""
import threading
import types

import numpy as np
import pytest
import torch

from crystalformer_b200.synthetic import make_crystals

pytestmark = pytest.mark.gpu


def setup(bins, sizes=(30, 17, 40, 64, 1, 9)):
    from crystalformer_b200.model import Latticeformer, default_params
    torch.manual_seed(2)
    model = Latticeformer(default_params(num_layers=2, value_pe_dist_real=bins)).cuda()
    cb = make_crystals(8, len(sizes), lambda rng, b: np.array(sizes), length_range=(4.0, 9.0))
    t = lambda x: torch.as_tensor(x).cuda()
    data = types.SimpleNamespace(x=t(cb.x), pos=t(cb.pos), trans_vec=t(cb.trans_vec), sizes=t(cb.sizes))
    with torch.no_grad():
        model.train()(data)  # sets the width statistics
    return model, data, cb


def run(model, data, training):
    """The outputs, and in training every gradient (by torch.autograd.grad: nothing is accumulated in the shared model)."""
    if not training:
        with torch.no_grad():
            return [model(data)]
    y = model(data)
    return [y.detach(), *torch.autograd.grad(y.abs().mean(), [p for p in model.parameters() if p.requires_grad])]


@pytest.mark.parametrize("training", [False, True])
@pytest.mark.parametrize("bins", [0, 64])
def test_memory_freed_to_the_stream_after_the_batch_was_begun(monkeypatch, bins, training):
    """What another thread may do while this one waits for the sizes, done at that place: kernels queued on the stream that
    write a block, and the block freed.  The call is then handed that block."""
    from crystalformer_b200 import _lib
    model, data, cb = setup(bins)
    model.train(training)
    ref = run(model, data, training)
    call, seen = _lib.call, {}
    begin, finish, at = ("cf_train_begin", "cf_train_forward", None) if training else ("cf_model_begin", "cf_model_finish", 11)

    def intruded(name, *args):
        out = call(name, *args)
        if name == begin:
            if training:
                nbytes = int(_lib.load().cf_train_edge_bytes(args[0], cb.num_atoms, cb.num_crystals, cb.num_edges))
            else:
                nbytes = int(_lib.load().cf_model_workspace_bytes(cb.num_atoms, cb.num_crystals, cb.num_edges, 512))
            block = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
            torch.cuda._sleep(4_000_000)  # (about two milliseconds: longer than the batch takes)
            block.fill_(255)
            seen["block"] = block.data_ptr()
        if name == finish:
            seen["used"] = args[1]._obj.saved_edges if training else args[at]
        return out

    monkeypatch.setattr(_lib, "call", intruded)
    torch.cuda.synchronize()
    got = run(model, data, training)
    monkeypatch.undo()
    assert seen["used"] == seen["block"]  # the call was given the very block
    assert all(torch.equal(a, b) for a, b in zip(ref, got))


@pytest.mark.parametrize("training", [False, True])
def test_two_threads_on_one_stream(training):
    model, _, _ = setup(64)
    model.train(training)
    t = lambda x: torch.as_tensor(x).cuda()
    batches = []
    for i in range(6):
        sizes = np.array([[30, 2, 9], [64] * 5, [1], [17] * 20, [40, 41], [5] * 60][i])
        cb = make_crystals(20 + i, len(sizes), lambda rng, b: sizes, length_range=(4.0, 9.0))
        batches.append(types.SimpleNamespace(x=t(cb.x), pos=t(cb.pos), trans_vec=t(cb.trans_vec), sizes=t(cb.sizes)))
    ref = [run(model, b, training) for b in batches]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    wrong, rounds = [], 10

    def work(first):
        try:
            with torch.cuda.stream(stream):
                for r in range(rounds):
                    for i in range(len(batches)):
                        j = (first + i) % len(batches)
                        got = run(model, batches[j], training)
                        if not all(torch.equal(a, b) for a, b in zip(ref[j], got)):
                            wrong.append((first, r, j))
        except BaseException as e:
            wrong.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 3)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert not wrong, wrong[:3]


def test_weights_packed_behind_other_work():
    """A pipeline is built on a stream that is busy, and its streams of its own do not wait for that one."""
    from crystalformer_b200.serving import PipelinedPredictor
    model, data, cb = setup(64)
    with torch.no_grad():
        ref = model.eval()(data).cpu()
        model.input_embeddings.weight.mul_(1.0)  # (a new version: the embedding is packed again)
    host = types.SimpleNamespace(x=torch.as_tensor(cb.x).pin_memory(), pos=torch.as_tensor(cb.pos).pin_memory(),
                                 trans_vec=torch.as_tensor(cb.trans_vec).pin_memory(), sizes=torch.as_tensor(cb.sizes).pin_memory())
    torch.cuda.synchronize()
    torch.cuda._sleep(4_000_000)
    runner = PipelinedPredictor(model, depth=2, streams=2)
    assert torch.equal(runner.result(runner.submit(host)), ref)


@pytest.mark.parametrize("bins", [0, 64])
def test_steps_in_a_graph(bins):
    """With the sizes given a training step queues work only, on two streams that meet again: it can be captured."""
    model, data, cb = setup(bins)
    model.train()
    counts = (cb.num_atoms, cb.num_edges, int(cb.sizes.max()))
    weights = [p for p in model.parameters() if p.requires_grad]

    def step():
        y = model(data, counts=counts)
        return [y.detach(), *torch.autograd.grad(y.abs().mean(), weights)]

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    with torch.no_grad():
        data.pos.mul_(1.01)
        weights[0].mul_(1.1)
    graph.replay()
    assert all(torch.equal(a, b) for a, b in zip(captured, step()))
