"""Analytic minimisations over several grids in several threads at once, each on
streams of its own and one with a higher priority, call after call: the side streams
that the library keeps between calls serve them all, and every result equals that of
a call alone, bit for bit; calls on a stream run in its order."""
import threading

import pytest
import torch

from gpu_cases import small_case, to_device_grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_grids", [2, 5, 8])
def test_threads_and_streams(n_grids):
    import attract_b200 as A

    c = small_case(seed=430, n_lig_beads=45, n_poses=60)
    grids = [to_device_grid(c)] + [to_device_grid(small_case(seed=431 + i, n_poses=1)) for i in range(n_grids - 1)]
    ligs = A.LigandSet([(c["lig"], c["gt"], c["lt"])])
    n = [60 // n_grids] * (n_grids - 1)
    segs = [A.Segment(g, 0, k) for g, k in enumerate(n + [60 - sum(n)])]
    P = torch.tensor(c["poses"], dtype=torch.float32, device="cuda")
    ev = A.EvalOptions(grad_mode="analytic", gravity=0.1)
    wl = A.Workload(grids, ligs, segs, lanes_per_pose=32)
    want = {k: A.minimise(wl, P, k, opts=ev)[:3] for k in (1, 7, 14)}
    twice = A.minimise(wl, want[7][0], 7, opts=ev)[:3]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream(priority=-1 if i == 1 else 0)):
                for k in range(12):
                    steps = (1, 7, 14)[(i + k) % 3]
                    got = A.minimise(wl, P, steps, opts=ev)[:3]
                    X = A.minimise(wl, P, 7, opts=ev)[0]
                    again = A.minimise(wl, X, 7, opts=ev)[:3]  # behind the call that makes X, with no wait between
                    for a, b in zip((*got, *again), (*want[steps], *twice)):
                        if not torch.equal(a, b):
                            wrong.append((i, k))
        except Exception as e:  # noqa: BLE001  (shown by the assertion below)
            wrong.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("steps", [3])
def test_many_tiles_one_after_another(steps):
    """More tiles than the side-by-side launches take, on a given number of blocks."""
    import attract_b200 as A

    c = small_case(seed=440, n_lig_beads=45, n_poses=50)
    grids = [to_device_grid(c), to_device_grid(small_case(seed=441, n_poses=1))]
    ligs = A.LigandSet([(c["lig"], c["gt"], c["lt"])])
    ev = A.EvalOptions(grad_mode="analytic", gravity=0.1)
    P = torch.tensor(c["poses"], dtype=torch.float32, device="cuda")
    wl = A.Workload(grids, ligs, [A.Segment(0, 0, 20), A.Segment(1, 0, 30)], lanes_per_pose=32)
    want = A.minimise(wl, P, steps, opts=ev)[:3]
    for blocks, threads in ((2, 128), (2, 96), (3, 64)):  # 8, 6 and 6 warps: 2 x 50 tiles > 3 n_grids^2 warps
        got = A.minimise(wl, P, steps, opts=ev, launch=A.LaunchShape(32, threads, blocks))[:3]
        assert all(torch.equal(a, b) for a, b in zip(got, want))
