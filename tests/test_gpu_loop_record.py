"""The device loop's step record (imc_loop_record_async) on its own, exact: rows of the histories and
snapshots it writes and leaves, the step index, the schedules' next entries, the last step, a step
past the last.  Sizes: one cell, one block and many, with and without groups and fiducial cells."""
import ctypes

import numpy as np
import pytest
import torch

from radtranbook_b200 import _lib, driver, imc2d, problems
from radtranbook_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,ng,n_fid", [(1, 1, 1, 1), (17, 15, 1, 0), (64, 64, 1, 300), (60, 210, 10, 5), (9, 7, 3, 0)])
def test_record_rows(cuda, nx, ny, ng, n_fid):
    nc, n, n_out = nx * ny, 4, 2
    eng = Engine("xy", np.linspace(0, 1, nx + 1), np.linspace(0, 1, ny + 1), np.ones(nc), n_groups=ng,
                 group_edges=np.geomspace(1e-2, 1.0, ng + 1) if ng > 1 else None)
    f = lambda *s: torch.full(s, -1.0, dtype=torch.float64, device=cuda)  # noqa: E731
    i64 = lambda v: torch.tensor(v, dtype=torch.int64, device=cuda)  # noqa: E731
    nsum = ctypes.sizeof(_lib.ImcStepSummary)
    b = dict(dt_sched=torch.tensor([.1, .2, .3, .4], dtype=torch.float64, device=cuda),
             step_sched=torch.arange(7, 11, dtype=torch.int32, device=cuda), nmax_sched=i64([5, 6, 7, 8]),
             out_slot=i64([1, n_out, 0, n_out]), dt=f(1), step=torch.zeros(1, dtype=torch.int32, device=cuda),
             nmax=i64([0]), k_ticket=i64([0, 0]), summary=torch.zeros(nsum, dtype=torch.uint8, device=cuda),
             hist_sum=torch.zeros((n, nsum), dtype=torch.uint8, device=cuda), T=f(nc), Tr=f(nc), Eg=f(ng * nc),
             snap_T=f(n_out + 1, nc), snap_Tr=f(n_out + 1, nc), snap_Eg=f(n_out + 1, ng * nc),
             fid=torch.randint(0, nc, (n_fid,), device=cuda), hist_T=f(n, max(n_fid, 1)), hist_Tr=f(n, max(n_fid, 1)),
             hist_Eg=f(n, ng * max(n_fid, 1)))
    ptr = {k: v.data_ptr() for k, v in b.items()}
    if ng == 1:
        for k in ("Eg", "snap_Eg", "hist_Eg"):
            ptr[k] = None
    rec = _lib.ImcLoopRecord(n_steps=n, n_out=n_out, n_fid=n_fid, **ptr)
    call = lambda: eng.lib.imc_loop_record_async(ctypes.byref(eng.cmesh), ctypes.byref(rec), eng._stream())  # noqa: E731
    ref = {k: b[k].cpu().clone() for k in ("snap_T", "snap_Tr", "snap_Eg", "hist_T", "hist_Tr", "hist_Eg", "hist_sum")}
    for k in range(n + 1):
        for key in ("T", "Tr", "Eg"):
            b[key].copy_(torch.rand_like(b[key]))
        b["summary"].copy_(torch.randint(0, 255, (nsum,), dtype=torch.uint8))
        assert call() == 0
        if k < n:
            ref["hist_sum"][k] = b["summary"].cpu()
            slot = int(b["out_slot"][k])
            keys = (("T", 1), ("Tr", 1)) + ((("Eg", ng),) if ng > 1 else ())
            for key, g in keys:
                v = b[key].cpu()
                if slot < n_out:
                    ref["snap_" + key][slot] = v
                if n_fid:
                    ref["hist_" + key][k] = v.view(g, nc)[:, b["fid"].cpu()].reshape(-1)
        for key, v in ref.items():
            assert torch.equal(b[key].cpu(), v), (k, key)
        assert b["k_ticket"].tolist() == [min(k + 1, n), 0]
        q = min(k + 1, n - 1)
        assert (float(b["dt"]), int(b["step"]), int(b["nmax"])) == (float(b["dt_sched"][q]), 7 + q, 5 + q)
    rec.T = None
    assert call() != 0


def test_fiducial_cell_outside_the_mesh_is_refused(cuda):
    p = problems.crooked_pipe(nr=6, nz=12)
    st = imc2d.init_simulation(500, p["Tinit"], p["Tr_init"], p["edges1"], p["edges2"], p["eos_dev"], p["inv_eos_dev"],
                               geometry="rz")
    with pytest.raises(ValueError):
        driver.DeviceLoop(st, Ntarget=500, Nboundary=500, Nsource=0, Nmax=2000, T_boundary=p["T_boundary"],
                          sigma_a_func=p["sigma_dev"], inv_eos=p["inv_eos_dev"], cv=p["cv_dev"], source=p["source"],
                          reflect=p["reflect"], geometry="rz", boundary_source_func=p["boundary_source_func"],
                          fiducial_cells=[(6, 0), (5, 12)])
