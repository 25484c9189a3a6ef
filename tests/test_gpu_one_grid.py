"""A launch over one grid reads the grid's descriptor from the kernel
parameters, a launch over several from shared memory (reference gradient) or as
one launch per grid (analytic gradient): the same poses scored either way give
the same bits, in every mode, at every lane count and at 1 to 8 beads per lane
(and a ligand larger than the bead slots)."""
import numpy as np
import pytest
import torch

import attract_oracle as O
from gpu_cases import small_case, to_device_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lanes,beads", [(8, 5), (8, 16), (8, 27), (16, 16), (16, 60), (32, 32), (32, 33), (32, 300),
                                         (8, 70)])
def test_one_grid_equals_the_same_grid_among_several(lanes, beads):
    import attract_b200 as A

    c = small_case(seed=40, n_lig_beads=beads, n_poses=37)
    other = to_device_grid(small_case(seed=41, n_rec=30, n_poses=1))
    grid = to_device_grid(c)
    ligs = A.LigandSet([(c["lig"], c["gt"], c["lt"])])
    one = A.Workload([grid], ligs, [A.Segment(0, 0, 37)], lanes_per_pose=lanes)
    two = A.Workload([other, grid], ligs, [A.Segment(0, 0, 0), A.Segment(1, 0, 37)], lanes_per_pose=lanes)
    P = torch.tensor(c["poses"], dtype=torch.float32, device="cuda")
    M = torch.tensor(O.pose_to_mat(c["poses"]).reshape(-1, 16), dtype=torch.float32, device="cuda")
    Q = torch.zeros((37, 8), device="cuda")
    Q[:, :4] = torch.tensor(np.random.default_rng(0).normal(size=(37, 4)), dtype=torch.float32)
    Q[:, 4:7] = P[:, 3:]
    dL = torch.linspace(-1.0, 1.0, 37, device="cuda")
    for mode in ("reference", "analytic"):
        ev = A.EvalOptions(grad_mode=mode, gravity=0.1)
        for f in (lambda w: A.energrad(w, P, ev), lambda w: A.energrad(w, M, ev),
                  lambda w: A.minimise(w, P, 6, opts=ev)[:3],
                  lambda w: [t[..., :7] if t.dim() == 2 else t  # (column 7 is not written)
                                 for t in A.minimise_schema(w, Q, ((4, 0.5, True), (2, 0.1, False)), ev)],
                  lambda w: (A.energrad_backward(w, P, dL, ev),)):
            for a, b in zip(f(one), f(two)):
                assert torch.equal(a, b)
