"""The C-ABI shared library loads, exports every symbol the public header declares, and validates its arguments
before touching the device.  No GPU needed: only calls that fail validation are made."""
import ctypes
import os
import re

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def lib():
    from crystalformer_b200 import build
    build.build()
    from crystalformer_b200 import _lib
    return _lib.load()


def declared_symbols():
    text = open(os.path.join(REPO, "include", "crystalformer_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(cf_[a-z0-9_]+)\s*\(", text)))


def test_every_declared_symbol_is_exported(lib):
    names = declared_symbols()
    assert len(names) >= 14
    for name in names:
        assert hasattr(lib, name), f"{name} is declared in the header but not exported"


def test_binding_table_covers_the_header():
    from crystalformer_b200 import _lib
    bound = set(_lib.SIGNATURES) | {"cf_version", "cf_last_error", "cf_set_weight_floor_log2",
                                    "cf_get_weight_floor_log2", "cf_encoder_workspace_floats",
                                    "cf_model_workspace_bytes", "cf_term_list_workspace_bytes",
                                    "cf_row_list_workspace_bytes", "cf_set_sorted_rows", "cf_get_sorted_rows",
                                    "cf_set_row_stats", "cf_set_chained_launches"}
    assert set(declared_symbols()) <= bound


def test_version_and_knob(lib):
    assert lib.cf_version() >= 100
    lib.cf_set_weight_floor_log2(ctypes.c_double(-33.0))
    assert lib.cf_get_weight_floor_log2() == -33.0
    lib.cf_set_weight_floor_log2(ctypes.c_double(-30.0))


def test_validation_returns_codes_without_a_device(lib):
    from crystalformer_b200 import _lib
    null = ctypes.c_void_p(0)
    with pytest.raises(_lib.CrystalformerB200Error) as e:
        _lib.call("cf_lattice_sum_fwd", null, 0, null, null, null, null, 4, 4, 4, 64, 14.0, 1.0, null, 0, 0, null, 0.0,
                  2, 2, null, null, null)
    assert e.value.code == -2
    with pytest.raises(_lib.CrystalformerB200Error) as e:
        _lib.call("cf_lattice_sum_fwd", null, 0, null, null, null, null, 4, 8, 4, 32, 14.0, 1.0, null, 0, 0, null, 0.0,
                  2, 2, null, null, null)
    assert e.value.code == -2 and "K=32" in str(e.value)
    with pytest.raises(_lib.CrystalformerB200Error) as e:
        _lib.call("cf_lattice_sum_fwd", null, 0, null, null, null, null, 4, 8, 4, 64, 14.0, 1.0, null, 0, 0, null, 0.0,
                  2, 2, null, null, null)
    assert e.value.code == -1  # null pointers
    with pytest.raises(_lib.CrystalformerB200Error) as e:
        _lib.call("cf_lattice_sum_fwd", null, 0, null, null, null, null, 4, 8, 4, 64, 14.0, 1.0, null, 0, 0, null, 0.0,
                  99, 2, null, null, null)
    assert e.value.code == -4
    with pytest.raises(_lib.CrystalformerB200Error) as e:
        _lib.call("cf_fused_attn_fwd", null, null, null, null, null, null, null, 4, 8, 32, 4, null, null, null)
    assert e.value.code == -2
    with pytest.raises(_lib.CrystalformerB200Error) as e:
        _lib.call("cf_pipe_probe", 5, 1, 32, 1, null, null)
    assert e.value.code == -1


def test_package_refuses_cpu_tensors():
    import torch
    from crystalformer_b200 import ops
    with pytest.raises(RuntimeError, match="no CPU path"):
        ops.segment_mean(torch.zeros((4, 8)), torch.tensor([0, 4]))


def test_peer_gather_descriptor_matches_the_header_layout():
    """cf_peer_gather of the header: two int32, one int64, two uint32, CF_MAX_PEERS pointers, naturally aligned."""
    from crystalformer_b200 import _lib
    header = open(os.path.join(REPO, "include", "crystalformer_b200.h")).read()
    peers = int(re.search(r"#define CF_MAX_PEERS (\d+)", header).group(1))
    handle = int(re.search(r"#define CF_PEER_HANDLE_BYTES (\d+)", header).group(1))
    assert peers == _lib.MAX_PEERS and handle == _lib.PEER_HANDLE_BYTES
    D = _lib.PeerGatherDescriptor
    assert ctypes.sizeof(D) == 24 + 8 * peers
    assert (D.world.offset, D.rank.offset, D.rows_per_rank.offset, D.step.offset, D.cells.offset) == (0, 4, 8, 16, 24)


def test_workspace_of_the_maxima_holds_every_batch_below_them(lib):
    """A slot has the workspace of its three maxima (serving): no batch within them may need more, whatever kernels it takes.  Sizes on
    both sides of 64 atoms per crystal, of the smallest batch with pair grids and of the most that grids may take."""
    import numpy as np
    rng = np.random.default_rng(1)
    size = lambda n, b, e: int(lib.cf_model_workspace_bytes(n, b, e, 512))
    crystals = lambda b, n: (b * n, b, b * n * n)
    for b, large, small in ((16, 70, 60), (20, 88, 64), (64, 70, 60), (128, 70, 60), (1, 65, 64), (40000, 64, 32), (100, 1024, 64)):
        outer = np.maximum(crystals(b, large), crystals(b, small))
        assert size(*crystals(b, small)) <= size(*(int(v) for v in outer)), (b, large, small)
    for _ in range(20000):
        b = int(np.exp(rng.uniform(0, np.log(50000))))
        n = b * int(rng.integers(1, 100))
        e = int(n * rng.uniform(1, 100))
        outer = [int(v * f) for v, f in zip((n, b, e), rng.choice([1.0, 1.01, 1.25, 4.0], 3))]
        assert size(n, b, e) <= size(*outer), ((n, b, e), outer)
        assert size(n, b, min(e, 64 * n)) <= size(*outer), ((n, b, e), outer)


def test_pair_grids_lie_in_the_memory_of_the_lists(lib):
    """A batch has term lists or grids: together they take the larger one's memory, and grids are not kept for batches that never
    have them (fewer than 5,000 pairs)."""
    grid = lambda n, b, e: int(lib.cf_pair_grid_bytes(n, b, e))
    lists = lambda n, e: max(int(lib.cf_term_list_workspace_bytes(n, e)), int(lib.cf_row_list_workspace_bytes(n, e)))
    for n, b, e in ((32000, 1024, 1270000), (500000, 16000, 20000000), (9600, 64, 1500000), (2000, 128, 41000), (100, 10, 1000)):
        rest = int(lib.cf_encoder_workspace_floats(n, e, 512)) * 4 - lists(n, e) + n * 1024 + 28 * e + 100 * b + 16384
        most = max(lists(n, e), (grid(n, b, min(e, 64 * n)) or 8 << 30) if e >= 5000 else 0)
        assert int(lib.cf_model_workspace_bytes(n, b, e, 512)) <= rest + most, (n, b, e)


def test_memory_of_a_training_step_grows_with_its_sizes(lib):
    """The edge memory of a step holds its lists or its grids, whichever it takes, and never shrinks with a size (640 rows, 5,000 edges and 64
    edges per atom on both sides); without a basis the lists are the larger."""
    from crystalformer_b200 import _lib
    import numpy as np
    weights, scalars = (ctypes.c_void_p * 29)(), (ctypes.c_double * 18)()

    def desc(K):
        return _lib.TrainDesc(num_layers=2, lattice_range=2, minimum_range=2, feature_dim=98, K=K, ff_dim=512, hidden=128, targets=1, wscale=1.0,
                              weights=ctypes.cast(weights, ctypes.c_void_p), scalars=ctypes.cast(scalars, ctypes.c_void_p))

    size = lambda K, n, b, e: int(lib.cf_train_edge_bytes(ctypes.byref(desc(K)), n, b, e))
    lists = lambda n, e: int(lib.cf_term_list_workspace_bytes(n, e))
    rest = lambda e: 2 * e * 32 + 28 * e
    for n, b, e in ((5248, 256, 141696), (640, 20, 20480), (30000, 1000, 1200000)):
        grid = int(lib.cf_pair_grid_bytes(n, b, e))
        assert max(lists(n, e), grid) <= size(64, n, b, e) - rest(e) <= max(lists(n, e), grid) + 4096
        assert size(0, n, b, e) - rest(e) <= lists(n, e) + 4096
    rng = np.random.default_rng(2)
    for _ in range(2000):
        b = int(np.exp(rng.uniform(0, np.log(3000))))
        n = b * int(rng.integers(1, 100))
        e = int(n * rng.uniform(1, 100))
        outer = [int(v * f) for v, f in zip((n, b, e), rng.choice([1.0, 1.01, 1.25, 4.0], 3))]
        for K in (0, 64):
            assert size(K, n, b, e) <= size(K, *outer) and size(K, n, b, min(e, 64 * n)) <= size(K, *outer), (K, (n, b, e), outer)
