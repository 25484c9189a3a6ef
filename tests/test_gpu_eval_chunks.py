"""Single evaluations take a ligand one bead per lane at a time: at the edges of
those chunks the energies and gradients (Euler, 4x4 and the adjoint's) match the
float64 oracle within the counted float32 bound, and a pose's energy is the same
to the bit alone and among others, whatever the largest ligand of the launch."""
import numpy as np
import pytest
import torch

import attract_oracle as O
from gpu_cases import float32_bounds, north_star_report, small_case, to_device_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["reference", "analytic"])
@pytest.mark.parametrize("lanes,beads", [(8, 8), (8, 9), (8, 33), (16, 17), (16, 64), (32, 31), (32, 33), (32, 64),
                                         (32, 65), (32, 129)])
def test_chunk_edges(lanes, beads, mode):
    import attract_b200 as A

    c = small_case(seed=80 + beads, n_lig_beads=beads, n_poses=21)
    grid = to_device_grid(c)
    ligs = A.LigandSet([(c["lig"], c["gt"], c["lt"])])
    wl = A.Workload([grid], ligs, [A.Segment(0, 0, 21)], lanes_per_pose=lanes)
    P = torch.tensor(c["poses"], dtype=torch.float32, device="cuda")
    ev = A.EvalOptions(grad_mode=mode)
    E, G, _ = A.energrad(wl, P, ev)
    Eo, Go = O.energrad(c["poses"], c["lig"], c["gt"], c["lt"], c["G"], mode=mode)
    bounds = float32_bounds(c["poses"], c["lig"], c["gt"], c["lt"], c["G"], mode)
    north_star_report(f"{beads} beads, {lanes} lanes, {mode}", E.cpu().numpy(), G.cpu().numpy(), Eo, Go, bounds)
    back = A.energrad_backward(wl, P, torch.ones(21, device="cuda"), ev).cpu().numpy()
    north_star_report("adjoint", E.cpu().numpy(), back, Eo, Go, bounds)
    M = torch.tensor(O.pose_to_mat(c["poses"]).reshape(-1, 16), dtype=torch.float32, device="cuda")
    north_star_report("4x4", A.energrad(wl, M, ev)[0].cpu().numpy(), None, Eo, None, bounds)
    # the same poses among 150-bead ones
    rng = np.random.default_rng(1)
    big = rng.normal(size=(150, 3)) * 2.0
    t = rng.integers(0, 4, 150)
    mix = A.Workload([grid], A.LigandSet([(big, t, t), (c["lig"], c["gt"], c["lt"])]),
                     [A.Segment(0, 0, 21), A.Segment(0, 1, 21)], lanes_per_pose=lanes)
    Em, Gm, _ = A.energrad(mix, torch.cat([P, P]), ev)
    assert torch.equal(Em[21:], E) and torch.equal(Gm[21:], G)
