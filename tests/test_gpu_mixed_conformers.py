"""Single evaluations of conformers of different sizes in one segment (the C
interface takes them): a pose's results are those of its ligand among its like,
to the bit, whatever the chunks of the poses that share its warp -- ligands of
one, two, three and more chunks, Euler poses, matrices and the adjoint's pose
gradients, with a block's warps on one tile and with one warp per tile."""
import ctypes as C

import numpy as np
import pytest
import torch

import attract_oracle as O
from gpu_cases import small_case, to_device_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [0, 32])
@pytest.mark.parametrize("lanes", [8, 16, 32])
def test_a_pose_beside_larger_ones(lanes, threads):
    import attract_b200 as A
    from attract_b200 import _lib

    n = 23
    c = small_case(seed=310, n_lig_beads=6 * lanes, n_poses=n)
    grid = to_device_grid(c)
    sizes = [lanes - 1, 2 * lanes, lanes + 1, 6 * lanes, 2 * lanes - 1, 3 * lanes, 2 * lanes + 1]
    for largest in (7, 3):  # (with, then without a ligand of more than four chunks)
        keep = [s for s in sizes if s <= (3 if largest == 3 else 6) * lanes]
        ligs = A.LigandSet([(c["lig"][:s], c["gt"][:s], c["lt"][:s]) for s in keep])
        P = torch.tensor(c["poses"], dtype=torch.float32, device="cuda")
        M = torch.tensor(O.pose_to_mat(c["poses"]).reshape(-1, 16), dtype=torch.float32, device="cuda")
        shape, ev = A.LaunchShape(lanes, threads), A.EvalOptions(gravity=0.1)
        which = torch.tensor(np.arange(n) % len(keep), dtype=torch.int32, device="cuda")
        wl = A.Workload([grid], ligs, [A.Segment(0, 0, n)], lanes_per_pose=lanes)

        def mixed(poses, mat):
            E = torch.full((n,), float("nan"), device="cuda")
            G = torch.full((n, 16 if mat else 6), float("nan"), device="cuda")
            cfg, lc = ev.to_c(1 if mat else 0), shape.to_c()
            _lib.check(_lib.load().att_energrad(
                wl.c_grids, 1, C.byref(wl.c_ligs), wl.segs.data_ptr(), 1, wl.seg_tile.data_ptr(), wl.n_tiles, n,
                poses.data_ptr(), which.data_ptr(), C.byref(cfg), E.data_ptr(), G.data_ptr(), None, C.byref(lc),
                torch.cuda.current_stream().cuda_stream), "att_energrad")
            return E, G

        def mixed_backward():
            dP, one = torch.full((n, 6), float("nan"), device="cuda"), torch.ones(n, device="cuda")
            cfg, lc = ev.to_c(0), shape.to_c()
            _lib.check(_lib.load().att_energrad_backward(
                wl.c_grids, 1, C.byref(wl.c_ligs), wl.segs.data_ptr(), 1, wl.seg_tile.data_ptr(), wl.n_tiles, n,
                P.data_ptr(), which.data_ptr(), C.byref(cfg), one.data_ptr(), dP.data_ptr(), None, None, C.byref(lc),
                torch.cuda.current_stream().cuda_stream), "att_energrad_backward")
            return dP

        E, G = mixed(P, False)
        Em, Gm = mixed(M, True)
        dP = mixed_backward()
        for i in range(len(keep)):
            alone = A.Workload([grid], ligs, [A.Segment(0, i, n)], lanes_per_pose=lanes)
            mine = which == i
            e, g, _ = A.energrad(alone, P, ev, launch=shape)
            em, gm, _ = A.energrad(alone, M, ev, launch=shape)
            dp = A.energrad_backward(alone, P, torch.ones(n, device="cuda"), ev, launch=shape)
            for got, want in ((E, e), (G, g), (Em, em), (Gm, gm.reshape(n, 16)), (dP, dp)):
                assert torch.equal(got[mine], want[mine]), (keep[i], largest)
