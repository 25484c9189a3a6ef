"""Minimisations over several grids with poses on all of them, their segments
interleaved: every pose equals a launch over its own grid alone, bit for bit, in
both gradient modes (the analytic mode of several beads per lane is a launch per grid, side
by side), launched and as a captured graph, twice in a row on the same buffers, in place, on a stream
of its own, and with a segment that names no grid."""
import numpy as np
import pytest
import torch

from gpu_cases import small_case, to_device_grid

pytestmark = pytest.mark.gpu

STAGES = ((3, 0.1, True), (3, 0.05, False))


def _case(lanes, beads, n_grids=3):
    import attract_b200 as A

    c = small_case(seed=400 + beads, n_lig_beads=beads, n_poses=61)
    grids = [to_device_grid(c)] + [to_device_grid(small_case(seed=410 + i, n_rec=25 + 60 * i, n_poses=1))
                                   for i in range(1, n_grids)]
    ligs = A.LigandSet([(c["lig"], c["gt"], c["lt"])])
    counts = [0, 9, 7, 1, 13, 8, 0, 11, 12]  # 61 poses
    segs = [A.Segment(i % n_grids, 0, n) for i, n in enumerate(counts)]
    P = torch.tensor(c["poses"], dtype=torch.float32, device="cuda")
    Q = torch.zeros((61, 8), device="cuda")
    Q[:, :4] = torch.tensor(np.random.default_rng(0).normal(size=(61, 4)), dtype=torch.float32)
    Q[:, 4:7] = P[:, 3:]
    return A, grids, ligs, segs, P, Q


def _alone(A, grids, ligs, segs, lanes, f, poses):
    """f over one segment at a time, each on its own grid."""
    outs, p0 = [], 0
    for s in segs:
        if s.n_poses:
            wl = A.Workload([grids[s.grid]], ligs, [A.Segment(0, 0, s.n_poses)], lanes_per_pose=lanes)
            outs.append(f(wl, poses[p0:p0 + s.n_poses].contiguous()))
        p0 += s.n_poses
    return [torch.cat(t) for t in zip(*outs)]


@pytest.mark.parametrize("mode", ["analytic", "reference"])
@pytest.mark.parametrize("lanes,beads", [(8, 8), (8, 15), (8, 30), (8, 70), (16, 20), (16, 100), (32, 45), (32, 100)])
def test_interleaved_segments_equal_their_grids_alone(lanes, beads, mode):
    A, grids, ligs, segs, P, Q = _case(lanes, beads)
    ev = A.EvalOptions(grad_mode=mode, gravity=0.1)
    wl = A.Workload(grids, ligs, segs, lanes_per_pose=lanes)
    mini = lambda w, p: A.minimise(w, p, 6, opts=ev)[:3]
    schema = lambda w, q: [t[:, :7] if t.dim() == 2 else t for t in A.minimise_schema(w, q, STAGES, ev)]
    want = _alone(A, grids, ligs, segs, lanes, mini, P)
    for _ in range(2):
        assert all(torch.equal(a, b) for a, b in zip(mini(wl, P), want))
    assert all(torch.equal(a, b) for a, b in zip(schema(wl, Q), _alone(A, grids, ligs, segs, lanes, schema, Q)))

    # captured and replayed, in place, on a stream of its own
    plan = A.MinimisePlan(wl, 6, opts=ev)
    plan.pose_in.copy_(P)
    for _ in range(2):
        assert all(torch.equal(a, b) for a, b in zip(plan.replay(), want))
    X = P.clone()
    got = A.minimise(wl, X, 6, opts=ev, pose_out=X)[:3]
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    got = A.minimise(wl, P, 6, opts=ev, stream=side)[:3]
    torch.cuda.current_stream().wait_stream(side)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("lanes,beads", [(8, 15), (32, 45)])
def test_statistics_and_a_segment_without_a_grid(lanes, beads):
    from attract_b200 import _lib

    A, grids, ligs, segs, P, _ = _case(lanes, beads)
    ev = A.EvalOptions(grad_mode="analytic")
    wl = A.Workload(grids, ligs, segs, lanes_per_pose=lanes)
    p, E, s, st = A.minimise(wl, P, 4, opts=ev, stats=True)
    total, p0 = torch.zeros_like(st), 0
    for sg in segs:
        if sg.n_poses:
            one = A.Workload([grids[sg.grid]], ligs, [A.Segment(0, 0, sg.n_poses)], lanes_per_pose=lanes)
            total += A.minimise(one, P[p0:p0 + sg.n_poses].contiguous(), 4, opts=ev, stats=True)[3]
        p0 += sg.n_poses
    assert torch.equal(st, total)
    bad = wl.segs.clone()
    bad[4, 0] = 9  # 13 poses from the 17th on
    wl.segs = bad
    out = torch.full_like(P, 7.0)
    p2, E2, s2, _ = A.minimise(wl, P, 4, opts=ev, pose_out=out)
    keep = torch.ones(61, dtype=torch.bool, device="cuda")
    keep[17:30] = False
    assert torch.equal(p2[keep], p[keep]) and torch.equal(E2[keep], E[keep]) and torch.equal(s2[keep], s[keep])
    assert bool((p2[~keep] == 7.0).all())
    assert _lib.kernel_status(clear=True) == _lib.ATT_KERR_BAD_SEGMENT
