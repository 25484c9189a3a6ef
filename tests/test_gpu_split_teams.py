"""Tiles of several poses (teams of 8 and 16 lanes) whose chunks a block's four
warps share: at the edges of that rule and of the chunks, the results equal those
of one warp per tile to the bit (Euler, 4x4, the adjoint's pose gradients; one grid
and two; a last tile that is partly empty), the adjoint's grid scatter equals it to float32
sums, and energies and gradients match the float64 oracle."""
import numpy as np
import pytest
import torch

import attract_oracle as O
from gpu_cases import float32_bounds, north_star_report, small_case, to_device_grid

pytestmark = pytest.mark.gpu

TILES = 148 * 5 * 2  # the most tiles that are split over a block's warps


@pytest.mark.parametrize("mode", ["reference", "analytic"])
@pytest.mark.parametrize("lanes,beads", [(8, 16), (8, 17), (8, 25), (8, 33), (8, 70), (16, 32), (16, 33), (16, 65), (16, 130)])
def test_split_tiles_are_the_same_to_the_bit(lanes, beads, mode):
    import attract_b200 as A

    few = 13  # (a last tile that is partly empty)
    last = TILES * (32 // lanes)
    c = small_case(seed=280 + beads, n_lig_beads=beads, n_poses=few)
    grid = to_device_grid(c)
    ligs = A.LigandSet([(c["lig"], c["gt"], c["lt"])])
    P = torch.tensor(c["poses"], dtype=torch.float32, device="cuda")
    M = torch.tensor(O.pose_to_mat(c["poses"]).reshape(-1, 16), dtype=torch.float32, device="cuda")
    ev = A.EvalOptions(grad_mode=mode, gravity=0.1)

    def all_of(grids, n, threads=0):
        k = -(-n // few)
        poses, mats = P.repeat(k, 1)[:n].contiguous(), M.repeat(k, 1)[:n].contiguous()
        segs = [A.Segment(0, 0, n)] if len(grids) == 1 else [A.Segment(0, 0, n // 2), A.Segment(1, 0, n - n // 2)]
        wl = A.Workload(grids, ligs, segs, lanes_per_pose=lanes)
        shape = A.LaunchShape(lanes, threads)
        E, G, S = A.energrad(wl, poses, ev, launch=shape)
        Em, Gm, Sm = A.energrad(wl, mats, ev, launch=shape)
        di, do = torch.zeros_like(grid.inner), torch.zeros_like(grid.outer)
        dP = A.energrad_backward(wl, poses, torch.ones(n, device="cuda"), ev, di, do, launch=shape) if len(grids) == 1 \
            else A.energrad_backward(wl, poses, torch.ones(n, device="cuda"), ev, launch=shape)
        return (E, G, S, Em, Gm, Sm, dP), (di, do)

    want, grids = all_of([grid], few, threads=32)  # never split
    got, scattered = all_of([grid], few)
    assert all(torch.equal(g, w) for g, w in zip(got, want))
    for g, w in zip(scattered, grids):  # every bead's eight corner weights are at most 1: u per addition
        assert (g - w).abs().max() <= 2.0 ** -23 * few * beads
    for got, _ in (all_of([grid], last), all_of([grid], last + 1), all_of([grid, grid], few)):
        for w, g in zip(want, got):
            k = len(g) // few
            assert torch.equal(g[:k * few].reshape(k, *w.shape), w.expand(k, *w.shape))
            assert torch.equal(g[k * few:], w[:len(g) - k * few])

    Eo, Go = O.energrad(c["poses"], c["lig"], c["gt"], c["lt"], c["G"], mode=mode)
    t = c["poses"][:, 3:]
    Eo, Go = Eo + 0.1 * (t ** 2).sum(1), Go + np.concatenate([np.zeros_like(t), 0.2 * t], 1)
    bounds = float32_bounds(c["poses"], c["lig"], c["gt"], c["lt"], c["G"], mode)
    north_star_report(f"{beads} beads, {lanes} lanes, {mode}", want[0].cpu().numpy(), want[1].cpu().numpy(), Eo, Go, bounds)
