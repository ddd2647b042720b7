"""Fused attention over pair grids (csrc/pair_grid.cu, pair_attn.cu) against the float64 oracle chain and the enumerating kernel.

Tolerance: the 2-norm error against 64 bits may be 1.25 times the enumerating kernel's on the same rows plus 3e-8, what the
interpolation between the nodes leaves of a row's sums (the weights reproduce the basis functions within 2.6e-8)."""
import numpy as np
import pytest
import torch

import oracle
from crystalformer_b200.synthetic import make_crystals, uniform_atoms

pytestmark = pytest.mark.gpu
H, D, DIST_MAX, WSCALE, A_WIDEST = 8, 16, 14.0, 1.0, -0.5 * 0.5 / 1.4 ** 2


@pytest.fixture(scope="module")
def ops():
    from crystalformer_b200 import ops as o
    return o


def dev(x):
    return x if isinstance(x, torch.Tensor) else torch.as_tensor(np.ascontiguousarray(x)).cuda()


def inputs(cb, sigma, scale=0.3, seed=3):
    rng = np.random.default_rng(seed)
    N = cb.num_atoms
    a = (-0.5 / (sigma[0] + (sigma[1] - sigma[0]) * rng.random((N, H))) ** 2).astype(np.float32)
    W = (rng.standard_normal((H, D, 64)) * 0.1).astype(np.float32)
    q = (rng.standard_normal((N, H, D)) * scale).astype(np.float32)
    k, v = (rng.standard_normal((N, H, D)).astype(np.float32) for _ in range(2))
    return q, k, v, a, W


def run(ops, cb, x, K, cutoff=-3.5, minimum=2, pos=None, wscale=WSCALE, gout=None, dist_max=DIST_MAX):
    """(grid results, enumerating kernel's results, the call again); with gout: the backward's, and the rows left over"""
    q, k, v, a, W = x
    sizes = dev(cb.sizes)
    atom_start, edge_start = ops.crystal_offsets(sizes)
    g = ops.batch_prepare(dev(cb.pos if pos is None else pos), dev(cb.trans_vec), sizes, atom_start, edge_start, cb.num_atoms, cb.num_edges)
    nmax = int(cb.sizes.max())
    W = dev(W) if K else None
    args = (dev(q), dev(k), dev(v), dev(a), g["pos_ij"], dev(cb.trans_vec), g["rvlen"], g["batch"], g["edges"], g["row_start"],
            nmax, K, dist_max, wscale, W, cutoff, 2, minimum)
    grids = ops.pair_grid_build(g["pos_ij"], dev(cb.trans_vec), g["rvlen"], atom_start, edge_start, cb.num_atoms, nmax, K, dist_max,
                                wscale, cutoff, 2, minimum, A_WIDEST)
    if gout is not None:
        out, logit, lse, _, left = ops.infinite_attn_fwd_grid(*args, grids)
        out0, logit0, lse0, _ = ops.infinite_attn_fwd(*args)
        by_grid = lambda: ops.infinite_attn_bwd_grid(*args, grids, logit, lse, left, out, dev(gout))
        return by_grid(), ops.infinite_attn_bwd(*args, logit0, lse0, out0, dev(gout)), by_grid, left
    return (ops.infinite_attn_fwd_grid(*args, grids, want_psi_row=K > 0), ops.infinite_attn_fwd(*args, want_psi_row=K > 0),
            lambda: ops.infinite_attn_fwd_grid(*args, grids, want_psi_row=K > 0))


def reference(cb, x, K, cutoff, minimum, wscale=WSCALE, dist_max=DIST_MAX):
    q, k, v, a, W = x
    edges = oracle.edge_index(cb.sizes)
    pos_ij, _, _, rvlen = oracle.geometry(cb.pos, cb.trans_vec, edges)
    z, psiW = oracle.lattice_sum_fwd(a, pos_ij, cb.trans_vec, cb.batch, edges, K, dist_max, wscale, W=W[None] if K else None, rvlen=rvlen,
                                     cutoff_radius=cutoff, lattice_range=2, minimum_range=minimum, precision="f64")
    _, out = oracle.fused_attn_fwd(q, k, v, z, psiW, edges, precision="f64")
    logit = np.einsum("ehd,ehd->eh", q[edges[0]].astype(np.float64), k[edges[1]].astype(np.float64)) + z
    lse = np.full((cb.num_atoms, H), -np.inf)
    np.logaddexp.at(lse, edges[0], logit)
    return np.asarray(out).reshape(cb.num_atoms, H, D), lse


def close(x, ref, plain, rows, what):
    err, err0 = (np.linalg.norm(t.cpu().numpy().astype(np.float64)[rows] - ref[rows]) / np.linalg.norm(ref[rows]) for t in (x, plain))
    assert err <= 1.25 * err0 + 3e-8, (what, err, err0)


# sizes about the tiles of 16 keys and 8 rows; one, two and four key tiles; cells with one box per width and with several; the three
# cut-off rules; another width of the basis
@pytest.mark.parametrize("lo,hi,K,cutoff,minimum,lengths,sigma,wscale", [
    (1, 9, 64, -3.5, 2, (3.0, 9.0), (1.18, 1.6), 1.0), (15, 17, 64, -3.5, 2, (4.0, 12.0), (1.18, 1.6), 1.0),
    (31, 33, 64, -3.5, 2, (4.0, 12.0), (1.0, 1.6), 1.0), (63, 64, 64, -3.5, 2, (6.0, 12.0), (1.18, 1.6), 1.0),
    (8, 24, 64, -3.5, 0, (3.0, 9.0), (1.18, 1.6), 1.0), (4, 12, 64, 0.0, 2, (3.0, 9.0), (1.18, 1.6), 1.0),
    (4, 12, 64, 6.5, 2, (3.0, 9.0), (1.18, 1.6), 1.0), (4, 20, 64, -3.5, 2, (3.0, 4.5), (1.2, 1.7), 1.0),
    (4, 20, 64, -3.5, 2, (4.0, 9.0), (1.18, 1.6), 1.1), (1, 1, 64, -3.5, 2, (5.0, 9.0), (1.18, 1.6), 1.0),
    (1, 17, 0, -3.5, 2, (3.0, 9.0), (1.18, 1.6), 1.0), (33, 64, 0, -3.5, 2, (4.0, 12.0), (1.18, 1.9), 1.0),
    (4, 20, 0, 0.0, 2, (3.0, 9.0), (1.18, 1.6), 1.0), (4, 20, 0, -3.5, 2, (3.0, 4.5), (1.2, 1.7), 1.0)])
def test_grid_forward_against_oracle_chain(ops, lo, hi, K, cutoff, minimum, lengths, sigma, wscale):
    cb = make_crystals(41, 9, uniform_atoms(lo, hi), length_range=lengths)
    x = inputs(cb, sigma)
    (out, _, lse, psi, left), (out0, _, lse0, psi0), again = run(ops, cb, x, K, cutoff, minimum, wscale=wscale)
    ref, ref_lse = reference(cb, x, K, cutoff, minimum, wscale)
    rows = left.cpu().numpy() == 0
    assert rows.mean() > 0.9
    close(out, ref, out0, rows, "rows by nodes")
    close(out, ref, out0, slice(None), "all rows")
    # float32 logarithms of sums: a few units in the last place of either, and of the largest logit
    assert np.abs(lse.cpu().numpy() - ref_lse).max() < 1e-6 * max(1.0, np.abs(ref_lse).max()) + 1.5e-6
    # ... and on average no more than 2^-24 of a sum, half a unit in its last place, beyond twice the enumerating kernel's
    assert np.abs(lse.cpu().numpy() - ref_lse).mean() < 2 * np.abs(lse0.cpu().numpy() - ref_lse).mean() + 2.0 ** -24
    if K:  # 64 sums per (row, head), each within a few units of the row's largest
        assert float((psi - psi0).abs().max() / psi0.abs().max()) < 2e-6
    repeat = again()
    assert torch.equal(out, repeat[0]) and torch.equal(lse, repeat[2])


@pytest.mark.parametrize("K", [64, 0])
def test_rows_that_nodes_do_not_serve_are_left_over(ops, K):
    """Gaussians too narrow and too wide for the nodes, logits far above the atom's own: marked, and as good as the others."""
    cb = make_crystals(43, 8, uniform_atoms(3, 20), length_range=(4.0, 9.0))
    x = inputs(cb, (1.2, 1.5))
    rng = np.random.default_rng(1)
    kind = rng.integers(0, 4, cb.num_atoms)
    x[3][kind == 1, 5] = -0.5 / 0.3 ** 2
    x[0][kind == 2] *= 40.0
    x[3][kind == 3, 2] = -0.5 / 2.6 ** 2  # (wider than a_widest: a box beyond the crystal's, or reach beyond the nodes)
    (out, _, lse, _, left), (out0, _, lse0, _), _ = run(ops, cb, x, K)
    left = left.cpu().numpy()
    assert left[kind == 1].all() and left[kind == 3].all() and left[kind == 2].any() and not left[kind == 0].any()
    ref, _ = reference(cb, x, K, -3.5, 2)
    close(out, ref, out0, slice(None), "all rows")


@pytest.mark.parametrize("K", [64, 0])
def test_numbers_that_are_not_finite_stay_visible(ops, K):
    """A NaN or an infinity in an input shows in the rows that the enumerating kernel shows it in."""
    cb = make_crystals(44, 6, uniform_atoms(4, 18), length_range=(4.0, 9.0))
    starts = np.concatenate([[0], np.cumsum(cb.sizes)])
    x = inputs(cb, (1.2, 1.5))
    x[0][starts[0] + 1, 2, 3] = np.nan
    x[1][starts[1] + 1, 1, 0] = np.nan
    x[2][starts[2] + 2, 4, 5] = np.nan
    x[1][starts[3] + 1, 3, 3] = np.inf
    x[3][starts[4] + 1, 6] = np.nan
    pos = cb.pos.copy()
    pos[starts[5] + 2] = np.nan
    (out, *_), (out0, *_), _ = run(ops, cb, x, K, pos=pos)
    bad, bad0 = (~torch.isfinite(t).flatten(1).all(dim=1) for t in (out, out0))
    assert torch.equal(bad, bad0)


def test_crystals_beyond_the_extra_vectors(ops):
    """Cells so flat that a head's box varies by dozens: only the smallest box has vectors, all other rows are left over."""
    cb = make_crystals(45, 3, uniform_atoms(3, 6), length_range=(3.0, 6.0))
    cb.trans_vec[0] *= np.float32(0.2)
    cb.pos[:cb.sizes[0]] *= np.float32(0.2)
    x = inputs(cb, (1.2, 1.6), scale=0.1)
    (out, _, _, _, left), (out0, *_), _ = run(ops, cb, x, 64)
    assert left[:int(cb.sizes[0])].all()
    ref, _ = reference(cb, x, 64, -3.5, 2)
    close(out, ref, out0, slice(None), "all rows")


def backward_reference(cb, x, go, K, cutoff, minimum, wscale, dist_max=DIST_MAX):
    q, k, v, a, W = x
    edges = oracle.edge_index(cb.sizes)
    pos_ij, _, _, rvlen = oracle.geometry(cb.pos, cb.trans_vec, edges)
    Wn = W[None] if K else None
    common = dict(rvlen=rvlen, cutoff_radius=cutoff, lattice_range=2, minimum_range=minimum, precision="f64")
    z, psiW = oracle.lattice_sum_fwd(a, pos_ij, cb.trans_vec, cb.batch, edges, K, dist_max, wscale, W=Wn, **common)
    prob, out = oracle.fused_attn_fwd(q, k, v, z, psiW, edges, precision="f64")
    gq, gk, gv, g_phi, g_psiW = oracle.fused_attn_bwd(q, k, v, psiW, edges, prob, out, go, precision="f64")
    ga, _ = oracle.lattice_sum_bwd(a, pos_ij, cb.trans_vec, cb.batch, edges, z, g_phi, g_psiW, K, dist_max, wscale, W=Wn, **common)
    return [np.asarray(t, np.float64).reshape(cb.num_atoms, -1) for t in (gq, gk, gv, ga)]


# as the forward's, with gradients from 1e-10 to 1e10 (the columns of the products are scaled by the gradient's own size)
@pytest.mark.parametrize("lo,hi,K,cutoff,minimum,lengths,sigma,wscale,size", [
    (1, 9, 64, -3.5, 2, (3.0, 9.0), (1.18, 1.6), 1.0, 1.0), (15, 17, 64, -3.5, 2, (4.0, 12.0), (1.18, 1.6), 1.0, 1e-10),
    (31, 33, 64, -3.5, 2, (4.0, 12.0), (1.0, 1.6), 1.0, 1e10), (40, 64, 64, -3.5, 2, (6.0, 12.0), (1.18, 1.6), 1.0, 1.0),
    (8, 24, 64, -3.5, 0, (3.0, 9.0), (1.18, 1.6), 1.0, 1.0), (4, 12, 64, 0.0, 2, (3.0, 9.0), (1.18, 1.6), 1.0, 1.0),
    (4, 20, 64, -3.5, 2, (3.0, 4.5), (1.2, 1.7), 1.0, 1.0), (4, 20, 64, -3.5, 2, (4.0, 9.0), (1.18, 1.6), 1.1, 1.0),
    (1, 1, 64, -3.5, 2, (5.0, 9.0), (1.18, 1.6), 1.0, 1.0), (4, 20, 64, -3.5, 2, (3.0, 9.0), (0.3, 1.6), 1.0, 1.0),
    (1, 17, 0, -3.5, 2, (3.0, 9.0), (1.18, 1.6), 1.0, 1e-10), (33, 64, 0, -3.5, 2, (4.0, 12.0), (1.18, 1.9), 1.0, 1.0),
    (4, 20, 0, -3.5, 2, (3.0, 4.5), (1.2, 1.7), 1.0, 1e10)])
def test_grid_backward_against_oracle_chain(ops, lo, hi, K, cutoff, minimum, lengths, sigma, wscale, size):
    cb = make_crystals(41, 9, uniform_atoms(lo, hi), length_range=lengths)
    x = inputs(cb, sigma)
    go = (np.random.default_rng(5).standard_normal((cb.num_atoms, H, D)) * size).astype(np.float32)
    got, plain, again, left = run(ops, cb, x, K, cutoff, minimum, wscale=wscale, gout=go)
    assert 0.1 < left.float().mean() if sigma[0] < 0.5 else left.float().mean() < 0.1
    for name, t, t0, ref in zip(("gq", "gk", "gv", "ga"), got, plain, backward_reference(cb, x, go, K, cutoff, minimum, wscale)):
        close(t.flatten(1), ref, t0.flatten(1), slice(None), name)
    assert all(torch.equal(s, t) for s, t in zip(got, again()))


@pytest.mark.parametrize("K", [64, 0])
def test_gradients_that_are_not_finite_stay_visible(ops, K):
    """A NaN or an infinity in the gradient shows where the enumerating kernel shows it."""
    cb = make_crystals(47, 4, uniform_atoms(4, 18), length_range=(4.0, 9.0))
    starts = np.concatenate([[0], np.cumsum(cb.sizes)])
    go = np.random.default_rng(5).standard_normal((cb.num_atoms, H, D)).astype(np.float32)
    go[starts[0] + 1, 2, 3] = np.nan
    go[starts[1] + 2, 5, 0] = np.inf
    got, plain, _, _ = run(ops, cb, inputs(cb, (1.2, 1.5)), K, gout=go)
    for t, t0 in zip(got, plain):
        assert torch.equal(torch.isfinite(t), torch.isfinite(t0))


def test_tensors_off_sixteen_bytes_are_refused(ops):
    cb = make_crystals(48, 2, uniform_atoms(4, 8), length_range=(5.0, 9.0))
    x = inputs(cb, (1.2, 1.5))
    off = torch.empty(x[0].size + 1, device="cuda")[1:].copy_(dev(x[0]).flatten()).view(x[0].shape)
    with pytest.raises(RuntimeError, match="16 bytes"):
        run(ops, cb, (off,) + x[1:], 64)
    with pytest.raises(RuntimeError, match="16 bytes"):
        run(ops, cb, x, 64, gout=off)


@pytest.mark.parametrize("dist_max,wscale", [(7.0, 4.0), (5.0, 5.0), (2.0, 10.0), (3.0, 8.0), (14.0, 2.0)])
def test_wide_bases_stay_within_half_precision(ops, dist_max, wscale):
    """Bases whose functions overlap by dozens, and a gradient of one sign over all bins: sum_k u_k g_k(d) grows with the width."""
    cb = make_crystals(49, 6, uniform_atoms(6, 20), length_range=(4.0, 9.0))
    q, k, v, a, W = inputs(cb, (1.85, 1.98))
    W[:] = 0.1
    go = np.full((cb.num_atoms, H, D), 1.2437, np.float32)  # (u = 1.98995: just below a power of two)
    x = (q, k, v, a, W)
    got, plain, _, left = run(ops, cb, x, 64, wscale=wscale, gout=go, dist_max=dist_max)
    assert left.float().mean() < 0.1
    for name, t, t0, ref in zip(("gq", "gk", "gv", "ga"), got, plain, backward_reference(cb, x, go, 64, -3.5, 2, wscale, dist_max)):
        close(t.flatten(1), ref, t0.flatten(1), slice(None), name)


def test_a_high_floor_stays_within_half_precision(ops):
    """With a floor of 2^-8 the nodes reach Gaussians of 40 node spacings, whose x n^2 is beyond 1,023: nothing overflows.  The kernels leave
    terms below 2^-8 out by rules of their own, beyond 3.3 standard deviations at the least: up to P(chi2_5 > 2 ln 2 * 8) = 5 % of a sum
    weighted by d^2, of which ga is a difference of two per kernel: a fifth in all, P(chi2_3) = 1.1 % and a twentieth without d^2."""
    cb = make_crystals(49, 6, uniform_atoms(6, 20), length_range=(4.0, 9.0))
    go = np.random.default_rng(5).standard_normal((cb.num_atoms, H, D)).astype(np.float32)
    ops.set_weight_floor_log2(-8.0)
    try:
        got, plain, _, left = run(ops, cb, inputs(cb, (1.55, 1.6), scale=0.05), 64, gout=go, dist_max=8.0)
    finally:
        ops.set_weight_floor_log2(-30.0)
    assert left.float().mean() < 0.1
    for name, t, t0 in zip(("gq", "gk", "gv", "ga"), got, plain):
        assert float((t - t0).norm() / t0.norm()) < (0.2 if name == "ga" else 0.05), name


def test_projected_sums_are_as_good_as_float32(ops):
    """The value encoding's part of the rows by itself (v = 0), small logits and large cells: the products with W lose no more than float32
    sums do (a tenth for chance: 240 atoms of 8 heads and 16 channels)."""
    cb = make_crystals(52, 60, uniform_atoms(1, 7), length_range=(8.0, 15.0))
    q, k, v, a, W = inputs(cb, (0.95, 1.4), scale=0.12)
    v[:] = 0.0
    x = (q, k, v, a, W)
    (out, _, _, _, left), (out0, *_), _ = run(ops, cb, x, 64)
    assert not left.any()
    ref, _ = reference(cb, x, 64, -3.5, 2)
    err, err0 = (np.linalg.norm(t.cpu().numpy().astype(np.float64) - ref) / np.linalg.norm(ref) for t in (out, out0))
    assert err <= 1.1 * err0, (err, err0)


def test_heads_far_below_the_others_keep_their_bits(ops):
    """One head whose weights at the nodes lie 2^15 below the other heads' in every row: two atoms 5.4 to 5.7 A apart, each with its largest
    logit (14.8 bits ahead) for the other."""
    cb = make_crystals(50, 40, uniform_atoms(2, 2), length_range=(14.0, 15.0))
    cb.trans_vec[:] = np.eye(3, dtype=np.float32) * 14.5
    cb.pos[:] = 0.0
    cb.pos[1::2, 0] = np.random.default_rng(7).uniform(5.4, 5.7, 40)
    q, k, v, a, W = inputs(cb, (1.18, 1.2))
    v[:] = 0.0  # (the rows are the projected sums alone)
    q[:, 0] = k[:, 0] = 0.0
    q[0::2, 0, 0] = k[1::2, 0, 0] = q[1::2, 0, 1] = k[0::2, 0, 1] = 3.2
    x = (q, k, v, a, W)
    (out, _, _, _, left), (out0, *_), _ = run(ops, cb, x, 64)
    assert not left.any()
    ref, _ = reference(cb, x, 64, -3.5, 2)
    close(out[:, 0], ref[:, 0], out0[:, 0], slice(None), "the head below")
    close(out, ref, out0, slice(None), "all heads")


@pytest.mark.parametrize("K", [64, 0])
def test_infinities_stay_infinities(ops, K):
    """An infinity in a value, or in the value encoding's projection: the rows that meet it are the enumerating kernel's, infinite with its
    sign, and marked as left over."""
    cb = make_crystals(51, 5, uniform_atoms(4, 18), length_range=(4.0, 9.0))
    starts = np.concatenate([[0], np.cumsum(cb.sizes)])
    x = inputs(cb, (1.2, 1.5))
    x[2][starts[0] + 1, 2, 3] = np.inf
    x[2][starts[2] + 1, 7, 0] = -np.inf
    if K:
        x[4][4, 5, 9] = np.inf
    (out, _, _, _, left), (out0, *_), _ = run(ops, cb, x, K)
    assert torch.isinf(out0).any()
    for of in (torch.isposinf, torch.isneginf, torch.isnan):
        assert torch.equal(of(out), of(out0))
    assert bool(left[~torch.isfinite(out).flatten(1).all(dim=1)].all())
