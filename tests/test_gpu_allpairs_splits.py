"""All-pairs rescoring over the splits of a call -- one pose to more than a
block holds, ligands that fill part of a lane's items to several passes of
them, receptors of one bead to several tiles -- against the float64 oracle,
within the tolerances of test_gpu_allpairs.py (relative to the summed
magnitudes of a pose's terms) and, for energies, the float32 positions: off by
up to 8 u (|x| + |X| + |r|) as in gpu_cases.float32_bounds, times the summed
magnitudes of the forces."""
import numpy as np
import pytest
import torch

import attract_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("poses,beads,n_rec,rcut,mix", [
    (1, 1, 1, 0.0, False), (1, 24, 2500, 0.0, True), (10, 24, 2500, 20.0, False), (130, 1, 2100, 0.0, False),
    (3, 65, 33, 0.0, True), (2, 1100, 40, 15.0, True), (257, 7, 150, 0.0, False), (40, 130, 300, 0.0, True),
    (4500, 2, 30, 12.0, True), (5, 9, 0, 0.0, False)])
def test_every_split(poses, beads, n_rec, rcut, mix):
    import attract_b200 as A
    from attract_b200.allpairs import AllPairs

    rng = np.random.default_rng(poses + beads)
    T = 6
    sigma, eps = rng.uniform(2.0, 3.0, (T, T)), rng.uniform(0.1, 2.0, (T, T))
    ivor = np.where(rng.random((T, T)) < 0.4, -1.0, 1.0) if mix else np.ones((T, T))
    cap = (0.6 * sigma) ** 2 if mix else np.zeros((T, T))
    ff = A.ForceField(eps * sigma ** 8, eps * sigma ** 6, ivor, cap)
    f32 = lambda a: np.asarray(a, np.float32).astype(np.float64)
    rec, rt = f32(rng.uniform(-25, 25, (n_rec, 3))), rng.integers(0, T, n_rec)
    lig, lt = f32(rng.uniform(-8, 8, (beads, 3))), rng.integers(0, T, beads)
    P = f32(np.concatenate([rng.uniform(-3, 3, (poses, 3)), rng.uniform(-10, 10, (poses, 3))], 1))
    ap = AllPairs(rec, rt, lig, lt, ff)
    X = torch.tensor(P, dtype=torch.float32, device="cuda")
    E, G = ap.energy(X, rcut=rcut or None, grad=True)
    E0, none = ap.energy(X, rcut=rcut or None)
    assert none is None and torch.allclose(E, E0, rtol=1e-6, atol=1e-5)
    mats = torch.tensor(O.pose_to_mat(P), dtype=torch.float32, device="cuda")
    Em, Gm = (v.cpu().numpy() for v in ap.energy(mats, rcut=rcut or None, grad=True))
    E, G = E.cpu().numpy(), G.cpu().numpy()
    if n_rec == 0:
        assert not E.any() and not G.any() and not Em.any() and not Gm.any()
        return
    pair = O.pair_table(ff.rc, ff.ac, ff.ivor, 1.0, shift_plateau=False, rcap2=ff.rcap2)
    k = np.unique(np.linspace(0, poses - 1, min(poses, 60)).astype(int))  # every block's ends among them
    Eo, Go, ea, ga, gb = O.allpairs_energrad(P[k], lig, lt, rec, rt, pair, rcut2=rcut * rcut if rcut else None,
                                             bead_grad=True)
    size = [np.linalg.norm(a, axis=-1).max() for a in (lig, O.transform(P[k], lig), rec)]
    tol = 1e-5 * ea + 1e-4 + 8 * 2.0 ** -24 * sum(size) * ga
    assert np.all(np.abs(E[k] - Eo) <= tol) and np.all(np.abs(Em[k] - Eo) <= tol)
    assert np.all(np.abs(G[k] - Go) <= 1e-4 * ga[:, None] + 1e-3)
    assert np.all(np.abs(Gm[k][:, :3, :3] - np.einsum("nr,bnc->brc", lig, gb)) <= 1e-4 * ga[:, None, None] + 1e-3)
    assert np.all(np.abs(Gm[k][:, 3, :3] - gb.sum(1)) <= 1e-4 * ga[:, None] + 1e-3)
    assert np.all(Gm[:, :, 3] == 0)
