"""The receptor builders at the edges of their tiles: dims that are no multiple
of a block's points, types that leave a chunk partly filled, receptors larger
than one list of kept beads, repulsive pairs and caps beyond the plateau,
records of every size.  Origins and spacings are exact in binary, so a grid
point is the same number everywhere and a potential is a double sum rounded
once: within 2^-24 of its value (twice that with the sum's own 1e-12)."""
import numpy as np
import pytest
import torch

import attract_oracle as O

pytestmark = pytest.mark.gpu


def _receptor(n, box, seed):
    return np.random.default_rng(seed).uniform(-box, box, (n, 3)).astype(np.float32).astype(np.float64)


@pytest.mark.parametrize("n_rec,types,dim,dim2,mix", [
    (0, 1, (2, 2, 2), (2, 2, 2), False), (1, 3, (5, 9, 8), (3, 4, 5), False), (40, 8, (4, 8, 8), (9, 8, 7), True),
    (257, 9, (11, 17, 3), (7, 9, 12), False), (700, 13, (9, 10, 25), (8, 6, 17), True), (1500, 2, (6, 7, 9), (5, 5, 5), True)])
def test_potentials_at_tile_edges(n_rec, types, dim, dim2, mix):
    import attract_b200 as A

    rng = np.random.default_rng(n_rec)
    n_rt = 5
    sigma, eps = rng.uniform(2.0, 4.0, (n_rt, types)), rng.uniform(0.1, 2.0, (n_rt, types))
    ivor = np.where(rng.random(sigma.shape) < 0.4, -1.0, 1.0) if mix else np.ones_like(sigma)
    cap = (sigma * (1.1 if mix else 0.6)) ** 2  # mix: caps beyond the 2.5 A plateau too
    ff = A.ForceField(eps * sigma ** 8, eps * sigma ** 6, ivor, cap)
    geom = A.GridGeom((-4.0, -3.5, -5.0), 0.5, dim, dim2, 6, 2.5, types)
    xyz, t = _receptor(n_rec, 5.0, n_rec), rng.integers(0, n_rt, n_rec)
    g = A.Grid.build(xyz, t, ff, geom, cutoff=7.0, keep_dense=True, nb_refine=1)
    pair = ff.pair_table(geom.plateau, True).astype(np.float64)  # the float32 table the kernel reads
    for got, outer in ((g.inner, False), (g.outer, True)):
        got = got.cpu().numpy()
        ref = np.zeros(got.shape) if n_rec == 0 else O.build_potential_grid(xyz, t, pair, geom.as_dict(), types, 7.0, outer)
        size = np.abs(ref).max() if n_rec else 1.0
        assert np.all(np.abs(got - ref) <= 2.0 ** -23 * np.abs(ref) + 1e-12 * size)
    ref = O.repack_bricks(g.inner.cpu().numpy(), g.outer.cpu().numpy())
    assert np.array_equal(g.bricks.cpu().numpy(), ref)


@pytest.mark.parametrize("n_rec,dim,refine,radius", [
    (0, (3, 3, 3), 1, 2.0), (5, (2, 2, 2), 4, 3.0), (90, (8, 8, 16), 1, 2.5), (300, (3, 5, 70), 2, 2.0),
    (1100, (9, 11, 13), 1, 4.0), (2100, (5, 6, 7), 2, 0.8), (60, (2, 2, 600), 1, 3.0)])
def test_lists_and_records_at_block_edges(n_rec, dim, refine, radius):
    import attract_b200 as A

    ff = A.ForceField.synthetic(4, 0)
    geom = A.GridGeom((-3.0, -2.5, -4.0), 0.7, dim, (0, 0, 0), 0, 3.0, 4)
    xyz = _receptor(n_rec, 4.0, n_rec + 1)
    g = A.Grid.build(xyz, np.zeros(n_rec, np.int64), ff, geom, list_radius=radius, potentials=False, nb_refine=refine)
    hdr = g.nb_hdr.cpu().numpy().view(np.uint32)
    lst = g.nb_list.cpu().numpy().view(np.uint16)
    if n_rec:
        c = g.nb_geom.to_c()
        rh, rl = O.build_nbgrid_f32(g.rec.cpu().numpy()[:n_rec, :3], np.array(c.origin[:], np.float32), c.spacing,
                                    c.dim[:], np.float32(radius))
        assert np.array_equal(hdr, rh) and np.array_equal(lst[: len(rl)], rl)
    else:
        assert not hdr.any()
    for rb in (32, 64, 128):
        g._pack_records(rec_bytes=rb)
        rec = g.nb_rec.cpu().numpy().reshape(-1, rb)
        inl = (rb - 6) // 2
        i = np.arange(inl)[None]
        want = np.where(i < hdr[:, 1:], lst[np.minimum(hdr[:, :1].astype(np.int64) + i, len(lst) - 1)], 65535)
        assert np.array_equal(rec[:, : 2 * inl].copy().view(np.uint16), want)
        assert np.array_equal(rec[:, 2 * inl: 2 * inl + 2].copy().view(np.uint16)[:, 0], hdr[:, 1])
        assert np.array_equal(rec[:, rb - 4:].copy().view(np.uint32)[:, 0], hdr[:, 0] + inl)


@pytest.mark.parametrize("n,top,zero,first", [(1, 3, 0.0, 1 << 24), (5, 70, 0.5, 1 << 24), (1023, 2, 0.9, 1 << 24),
                                              (1025, 300, 0.3, 1 << 24), (70_001, 14, 0.6, 1 << 24),
                                              (70_001, 60, 0.2, 1000), (70_001, 65_000, 0.5, 20_000),
                                              (3_000_000, 31, 0.9, 1 << 24), (4096, 5, 1.0, 1 << 24)])
def test_list_length_quantile_is_torchs(n, top, zero, first):
    from attract_b200.grid import list_length_quantile

    rng = np.random.default_rng(n + top)
    c = np.where(rng.random(n) < zero, 0, rng.integers(1, top + 1, n))
    hdr = torch.tensor(np.stack([np.arange(n), c], 1), dtype=torch.int32, device="cuda")
    nz = torch.tensor(c[c > 0][:first], dtype=torch.float32)
    for q in (0.99, 0.5, 0.0, 1.0):
        want = float(torch.quantile(nz, q)) if len(nz) else 0.0
        got = list_length_quantile(hdr, q, first)
        assert abs(got - want) <= 2.0 ** -22 * want  # the last step's rounding
        assert [b for b in (13, 29, 61) if b >= got] == [b for b in (13, 29, 61) if b >= want]
