"""Every minimiser and quaternion kernel that the library holds -- 8, 16 and 32
lanes with 1, 2, 4 and 8 beads per lane (and a chunked ligand), over one grid and
over several, in both gradient modes -- runs in the bounds-checked build, which
checks and guards each address it forms (copies, list and pair-buffer words, bead
slots, receptor beads, pair rows), on lists that fill the pair buffers several times.  No check
fails, and the regular build gives the same poses and energies."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

SCRIPT = r'''
import ctypes as C, json, sys
import numpy as np, torch
sys.path.insert(0, {root!r}); sys.path.insert(0, {tests!r}); sys.path.insert(0, {oracle!r})
import attract_b200 as A
from attract_b200 import _lib
from gpu_cases import small_case, to_device_grid
res = {{}}
for lanes in (8, 16, 32):
    for beads in (lanes, 2 * lanes, 3 * lanes, 7 * lanes, 8 * lanes + 3):
        # short lists, and lists of about 100 entries that continue in the CSR tail
        for n_rec in (60, 400):
            c = small_case(seed=300 + beads, n_rec=n_rec, n_lig_beads=beads, n_poses=14)
            a = to_device_grid(c)
            b = to_device_grid(small_case(seed=301 + beads, n_rec=25, n_poses=1))
            if n_rec == 400:
                a._pack_records(rec_bytes=32)
                a._att = None
            ligs = A.LigandSet([(c["lig"], c["gt"], c["lt"])])
            P = torch.tensor(c["poses"], dtype=torch.float32, device="cuda")
            Q = torch.zeros((14, 8), device="cuda"); Q[:, 3] = 1.0; Q[:, 4:7] = P[:, 3:]
            one = A.Workload([a], ligs, [A.Segment(0, 0, 14)], lanes_per_pose=lanes)
            two = A.Workload([a, b], ligs, [A.Segment(i % 2, 0, n) for i, n in enumerate((5, 4, 2, 3))],
                             lanes_per_pose=lanes)
            for name, w in (("one", one), ("two", two)):
                for mode in ("reference", "analytic"):
                    ev = A.EvalOptions(grad_mode=mode)
                    p, E, s, st = A.minimise(w, P, 4, opts=ev, stats=True)
                    q, Eq, sq = A.minimise_schema(w, Q, ((2, 0.1, True), (2, 0.05, False)), ev)
                    key = f"{{lanes}} {{beads}} {{n_rec}} {{name}} {{mode}}"
                    res[key] = [x.double().reshape(-1).cpu().tolist() for x in (p, E, s, q[:, :7], Eq, sq)]
                    torch.cuda.synchronize()
                    info = (C.c_ulonglong * 3)()
                    _lib.check(_lib.load().att_kernel_debug_info(info, 1, torch.cuda.current_stream().cuda_stream), "debug")
                    word = _lib.kernel_status(clear=True)
                    assert word == 0 and not any(info), (key, word, list(info))
print("RESULT " + json.dumps(res))
'''


def _run(lib):
    env = dict(os.environ)
    if lib:
        env["ATTRACT_B200_LIB"] = lib
    code = SCRIPT.format(root=ROOT, tests=HERE, oracle=os.path.join(ROOT, "oracle"))
    p = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr[-3000:]
    return json.loads([x for x in p.stdout.splitlines() if x.startswith("RESULT ")][-1][7:])


def test_every_minimiser_kernel_is_clean_under_checks():
    from attract_b200 import build as B

    got = _run(B.build(checked=True))  # the guarded build first
    ref = _run(None)
    assert got.keys() == ref.keys()
    for k in ref:
        for a, b in zip(got[k], ref[k]):
            assert np.allclose(a, b, rtol=1e-5, atol=1e-4, equal_nan=True), k
