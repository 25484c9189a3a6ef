"""Few poses of a large ligand are evaluated by a block of four warps each, many by
one warp: at the edges of that rule the results are the same to the bit (Euler, 4x4
and the adjoint's pose gradients; one grid and two), and the 4x4 gradients of every
team size match the float64 oracle within the counted float32 bound."""
import numpy as np
import pytest
import torch

import attract_oracle as O
from gpu_cases import float32_bounds, north_star_report, small_case, to_device_grid

pytestmark = pytest.mark.gpu

LAST = 148 * 6 * 2  # the most poses that are split over a block's warps


@pytest.mark.parametrize("mode", ["reference", "analytic"])
@pytest.mark.parametrize("beads", [64, 65, 96, 97, 129, 301])
def test_split_poses_are_the_same_to_the_bit(beads, mode):
    import attract_b200 as A

    c = small_case(seed=180 + beads, n_lig_beads=beads, n_poses=16)
    grid = to_device_grid(c)
    ligs = A.LigandSet([(c["lig"], c["gt"], c["lt"])])
    few = torch.tensor(c["poses"], dtype=torch.float32, device="cuda")
    many = few.repeat((LAST + 1 + 15) // 16, 1)[:LAST + 1]
    mats = torch.tensor(O.pose_to_mat(c["poses"]).reshape(-1, 16), dtype=torch.float32, device="cuda")
    ev = A.EvalOptions(grad_mode=mode)

    def all_of(grids, poses, mat, threads=0):
        n = len(poses)
        half = n // 2
        segs = [A.Segment(0, 0, n)] if len(grids) == 1 else [A.Segment(0, 0, half), A.Segment(1, 0, n - half)]
        wl = A.Workload(grids, ligs, segs, lanes_per_pose=32)
        shape = A.LaunchShape(32, threads)
        E, G, _ = A.energrad(wl, poses, ev, launch=shape)
        Em, Gm, _ = A.energrad(wl, mat, ev, launch=shape)
        back = A.energrad_backward(wl, poses, torch.ones(n, device="cuda"), ev, launch=shape)
        return E, G, Em, Gm, back

    want = all_of([grid], few, mats)
    whole = mats.repeat((LAST + 1 + 15) // 16, 1)
    for got in (all_of([grid], few, mats, threads=32),                         # never split
                all_of([grid], many[:LAST], whole[:LAST]),                     # the last that are
                all_of([grid], many, whole[:LAST + 1]),                        # the first that are not
                all_of([grid, grid], few, mats)):
        for w, g in zip(want, got):
            assert torch.equal(g[:16], w)
            k = len(g) // 16 * 16
            assert torch.equal(g[:k].reshape(-1, *w.shape), w.expand(k // 16, *w.shape))


@pytest.mark.parametrize("beads", [24, 70, 129])
@pytest.mark.parametrize("lanes", [8, 16, 32])
def test_matrix_gradients(lanes, beads):
    import attract_b200 as A

    c = small_case(seed=190 + beads, n_lig_beads=beads, n_poses=21)
    wl = A.Workload([to_device_grid(c)], A.LigandSet([(c["lig"], c["gt"], c["lt"])]), [A.Segment(0, 0, 21)],
                    lanes_per_pose=lanes)
    mats = O.pose_to_mat(c["poses"])
    E, dM, _ = A.energrad(wl, torch.tensor(mats.reshape(-1, 16), dtype=torch.float32, device="cuda"))
    Eo, dMo = O.energrad_mat(mats, c["lig"], c["gt"], c["lt"], c["G"])
    bounds = float32_bounds(c["poses"], c["lig"], c["gt"], c["lt"], c["G"], "reference")
    cols = lambda g: np.asarray(g).reshape(-1, 4, 4)[:, :, :3].reshape(-1, 12)
    north_star_report(f"4x4, {beads} beads, {lanes} lanes", E.cpu().numpy(), cols(dM.cpu().numpy()), Eo, cols(dMo), bounds)
