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
