"""All-pairs energies and gradients of a pose do not depend on the poses beside
it: alone, among a handful and in a library (calls that are split differently
over the GPU) they are the same to the bit -- receptors from one run of beads to
more than the tree's leaves, ligands from one bead to several passes, tables of
one form and mixed ones, with and without a cutoff, Euler poses and matrices."""
import numpy as np
import pytest
import torch

import attract_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rec,beads,rcut,mix", [
    (1, 1, 0.0, False), (64, 3, 0.0, True), (65, 24, 0.0, False), (130, 64, 9.0, True), (700, 65, 0.0, True),
    (2047, 7, 0.0, False), (2049, 130, 0.0, True), (2500, 24, 0.0, False), (2500, 24, 15.0, True), (5000, 24, 0.0, True),
    (300, 1100, 0.0, False),
    (17000, 3, 0.0, True), (33, 24, 0.0, True), (150, 24, 0.0, False), (4097, 10, 0.0, False)])
def test_a_pose_alone_and_in_a_library(n_rec, beads, rcut, mix):
    import attract_b200 as A
    from attract_b200.allpairs import AllPairs

    rng = np.random.default_rng(n_rec + beads)
    T = 6
    sigma, eps = rng.uniform(2.0, 3.0, (T, T)), rng.uniform(0.1, 2.0, (T, T))
    ivor = np.where(rng.random((T, T)) < 0.4, -1.0, 1.0) if mix else np.ones((T, T))
    ff = A.ForceField(eps * sigma ** 8, eps * sigma ** 6, ivor, (0.6 * sigma) ** 2)
    ap = AllPairs(rng.uniform(-25, 25, (n_rec, 3)), rng.integers(0, T, n_rec), rng.uniform(-8, 8, (beads, 3)),
                  rng.integers(0, T, beads), ff)
    few = np.concatenate([rng.uniform(-3, 3, (10, 3)), rng.uniform(-10, 10, (10, 3))], 1)
    most = max(60, min(16384, 400_000_000 // (n_rec * beads)))
    for X in (torch.tensor(few, dtype=torch.float32, device="cuda"),
              torch.tensor(O.pose_to_mat(few), dtype=torch.float32, device="cuda")):
        for grad in (True, False):
            run = lambda x: ap.energy(x.contiguous(), rcut=rcut or None, grad=grad)
            E, G = run(X)
            for i in range(10):
                e, g = run(X[i:i + 1])
                assert torch.equal(e, E[i:i + 1]) and (not grad or torch.equal(g, G[i:i + 1]))
            for n in (33, 300, 2000, most):
                if n > most:
                    continue
                at = torch.arange(n, device="cuda") * 7 % 10
                e, g = run(X[at])
                assert torch.equal(e, E[at]) and (not grad or torch.equal(g, G[at]))
