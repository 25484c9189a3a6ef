"""The neighbour-list count's 64-bit total is true beyond 2^32 entries: the
host refuses such lists by it (``check_list_total``) before anything is
allocated or filled.  Every bead lies within the radius of every point, so
the total is points x beads, and the header of point v starts at
v x beads modulo 2^32.  Counts only: no list is filled here."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


def _count(noalloc, dim, n_rec):
    import attract_b200 as A
    from attract_b200 import _lib
    from attract_b200.grid import pack_receptor

    lib = _lib.load()
    gc = A.GridGeom((0.0, 0.0, 0.0), 1.0, dim, (0, 0, 0), 0, 3.0, 1).to_c()
    nvox = dim[0] * dim[1] * dim[2]
    rec = pack_receptor(torch.rand((n_rec, 3), generator=torch.Generator().manual_seed(1)).numpy(), [0] * n_rec, "cuda")
    hdr = torch.empty((nvox, 2), dtype=torch.int32, device="cuda")
    total = torch.zeros(1, dtype=torch.int64, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    if noalloc:
        rc = lib.att_nbgrid_count_noalloc(C.byref(gc), _lib.ptr(rec), n_rec, 1e4, _lib.ptr(hdr), _lib.ptr(total), st)
    else:
        wsb = lib.att_nbgrid_workspace_bytes(nvox)
        ws = torch.empty(wsb, dtype=torch.uint8, device="cuda")
        rc = lib.att_nbgrid_count(C.byref(gc), _lib.ptr(rec), n_rec, 1e4, _lib.ptr(hdr), _lib.ptr(total), _lib.ptr(ws),
                                  wsb, st)
    _lib.check(rc, "count")
    return nvox, int(total.item()), hdr


# one step of the scan is 8192 x 1024 points: a whole one, two of which the second is short, a fraction of one
@pytest.mark.parametrize("noalloc,dim,n_rec", [(True, (128, 256, 256), 520), (False, (129, 257, 260), 600),
                                               (False, (100, 100, 100), 4400), (True, (20, 30, 40), 7)])
def test_the_total_is_true_beyond_32_bits(noalloc, dim, n_rec):
    nvox, total, hdr = _count(noalloc, dim, n_rec)
    assert total == nvox * n_rec
    want = (torch.arange(nvox, device="cuda") * n_rec) & 0xFFFFFFFF
    assert torch.equal(hdr[:, 0].long() & 0xFFFFFFFF, want)
    assert bool((hdr[:, 1] == n_rec).all())


def test_a_list_beyond_32_bit_starts_is_refused_by_the_build(monkeypatch):
    import attract_b200 as A
    from attract_b200 import grid

    check = grid.check_list_total

    def stop(n):  # (whatever the check says, nothing may be filled here)
        check(n)
        pytest.fail(f"a list of {n} entries was not refused")

    monkeypatch.setattr(grid, "check_list_total", stop)
    geom = A.GridGeom((0.0, 0.0, 0.0), 1.0, (128, 256, 256), (0, 0, 0), 0, 3.0, 1)
    xyz = torch.rand((520, 3), generator=torch.Generator().manual_seed(1)).numpy()
    with pytest.raises(ValueError, match="32-bit"):
        A.Grid.build(xyz, [0] * 520, A.ForceField.synthetic(1, 0), geom, list_radius=1e4, potentials=False, nb_refine=1)
