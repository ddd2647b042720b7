"""The dense kernels of the encoder (block-level tensor instructions) against plain float32 GEMMs of the same model."""
import types

import numpy as np
import pytest
import torch

from conftest import rel_err
from crystalformer_b200.synthetic import make_crystals

pytestmark = pytest.mark.gpu



@pytest.mark.parametrize("ff", [128, 256, 512])
@pytest.mark.parametrize("sizes", [[1], [127], [128], [100, 29], [200] * 7 + [3], [5] * 60])
def test_one_call_forward_with_images_equals_the_gemm_path(ff, sizes):
    """Tiles of 128 rows: a single row, one short of a tile, a full tile, one row more, many tiles; every chunk count."""
    from crystalformer_b200.model import Latticeformer, default_params
    torch.manual_seed(len(sizes) + ff)
    model = Latticeformer(default_params(num_layers=2, ff_dim=ff)).cuda()
    for p in model.parameters():  # biases away from zero, weights of ordinary size
        if p.requires_grad:
            p.data.add_(torch.randn_like(p) * 0.05)
    cb = make_crystals(3, len(sizes), lambda rng, b: np.array(sizes), length_range=(8.0, 14.0))
    t = lambda x: torch.as_tensor(x).cuda()
    data = types.SimpleNamespace(x=t(cb.x), pos=t(cb.pos), trans_vec=t(cb.trans_vec), sizes=t(cb.sizes))
    model.train()
    with torch.no_grad():
        model(data)
    model.eval()
    from crystalformer_b200.encoder import BatchGeometry
    geo = BatchGeometry(data.pos, data.trans_vec, data.sizes)
    out = {}
    with torch.no_grad():
        for fused in (True, False):
            model.encoder.dense_fused = fused
            emb = model.input_embeddings(data.x)
            out[fused] = (model(data), model.encoder(emb, data.pos, geo.batch, data.trans_vec, geo.sizes, geometry=geo))
    assert rel_err(out[True][1].cpu().numpy(), out[False][1].cpu().numpy()) < 3e-6
    assert (out[True][0] - out[False][0]).abs().max() < 1e-6  # (embedding, pooling and head included)


@pytest.mark.parametrize("ff", [128, 384, 512, 640])
@pytest.mark.parametrize("atoms", [1, 33, 4737, 9600])
def test_boundaries_of_every_tile_height(ff, atoms):
    """Tiles of 32 rows (one row; a tile and one row), of 64 (the first batch with more than 32 rows per SM) and of 128 (more than 64 per
    SM); one to five chunks of hidden units."""
    from crystalformer_b200.model import Latticeformer, default_params
    torch.manual_seed(atoms + ff)
    model = Latticeformer(default_params(num_layers=2, ff_dim=ff)).cuda()
    for p in model.parameters():
        if p.requires_grad:
            p.data.add_(torch.randn_like(p) * 0.05)
    sizes = [1] * min(atoms, 7) + [30] * ((atoms - 7) // 30) + [(atoms - 7) % 30 or 1] if atoms > 7 else [1] * atoms
    cb = make_crystals(4, len(sizes), lambda rng, b: np.array(sizes), length_range=(8.0, 14.0))
    t = lambda x: torch.as_tensor(x).cuda()
    data = types.SimpleNamespace(x=t(cb.x), pos=t(cb.pos), trans_vec=t(cb.trans_vec), sizes=t(cb.sizes))
    model.train()
    with torch.no_grad():
        model(data)
    model.eval()
    out = {}
    with torch.no_grad():
        for fused in (True, False):
            model.encoder.dense_fused = fused
            out[fused] = model(data)
    assert (out[True] - out[False]).abs().max() < 2e-6
    # the training step's boundaries, forward and backward, against the layer-by-layer step
    model.encoder.dense_fused = True
    model.train()
    grads = {}
    for native in (True, False):
        model.native = native
        model.zero_grad(set_to_none=True)
        model(data).abs().mean().backward()
        grads[native] = {n: p.grad for n, p in model.named_parameters() if p.requires_grad}
    noise = 1e-6 * max(float(g.norm()) for g in grads[False].values())
    for n, g in grads[False].items():
        # (a hidden unit within rounding of zero may fall on either side of the ReLU)
        assert (grads[True][n] - g).norm() <= 2e-3 * g.norm() + noise, n


@pytest.mark.parametrize("ff", [128, 512, 640])
@pytest.mark.parametrize("rows", [32, 64])
def test_tiles_of_32_64_and_128_rows(ff, rows):
    """A tile of so many rows on every SM, and one row more (tiles of twice as many): the same bits for the rows that both have, and for
    batches whose last tile has one row or all but one."""
    from crystalformer_b200.model import Latticeformer, default_params
    torch.manual_seed(ff)
    model = Latticeformer(default_params(num_layers=2, ff_dim=ff)).cuda()
    most = rows * torch.cuda.get_device_properties(0).multi_processor_count
    cb = make_crystals(6, most + 1, lambda rng, b: np.ones(b, dtype=np.int64), length_range=(8.0, 14.0))
    t = lambda x: torch.as_tensor(x).cuda()
    batch = lambda n: types.SimpleNamespace(x=t(cb.x)[:n], pos=t(cb.pos)[:n], trans_vec=t(cb.trans_vec)[:n], sizes=t(cb.sizes)[:n])
    model.train()
    with torch.no_grad():
        model(batch(most))
    model.eval()
    with torch.no_grad():
        whole = model(batch(most + 1))
        for n in (most, most - 1, most - rows + 1):
            assert torch.equal(model(batch(n)), whole[:n]), n
    # the step's gradients: sums over the rows in float32, in another order of shares
    model.train()
    grads = {}
    for n in (most, most + 1):
        x = batch(n)
        model.zero_grad(set_to_none=True)
        (model(x)[:most].abs().sum()).backward()
        grads[n] = {k: p.grad.clone() for k, p in model.named_parameters() if p.requires_grad}
    noise = 1e-6 * max(float(g.norm()) for g in grads[most].values())
    for k, g in grads[most].items():
        assert (grads[most + 1][k] - g).norm() <= 2e-6 * g.norm() + noise, k


@pytest.mark.parametrize("ff", [128, 384, 512])
@pytest.mark.parametrize("atoms", [1, 33, 200, 2000])
def test_outputs_do_not_depend_on_how_a_batch_is_issued(ff, atoms):
    """A forward in tiles of 32 rows, and the serving pipeline on several streams, whose tiles have 128."""
    from crystalformer_b200.model import Latticeformer, default_params
    from crystalformer_b200.serving import PipelinedPredictor
    torch.manual_seed(atoms + ff)
    model = Latticeformer(default_params(num_layers=2, ff_dim=ff)).cuda()
    for p in model.parameters():
        if p.requires_grad:
            p.data.add_(torch.randn_like(p) * 0.05)
    sizes = [min(atoms, 20)] * max(1, atoms // 20)
    cb = make_crystals(4, len(sizes), lambda rng, b: np.array(sizes), length_range=(4.0, 12.0))
    host = types.SimpleNamespace(x=torch.as_tensor(cb.x).pin_memory(), pos=torch.as_tensor(cb.pos).pin_memory(),
                                 trans_vec=torch.as_tensor(cb.trans_vec).pin_memory(), sizes=torch.as_tensor(cb.sizes).pin_memory())
    data = types.SimpleNamespace(**{n: t.cuda() for n, t in vars(host).items()})
    with torch.no_grad():
        model.train()(data)
        direct = model.eval()(data)
    runner = PipelinedPredictor(model, depth=2, streams=2)
    assert torch.equal(runner.result(runner.submit(host)), direct.cpu())
