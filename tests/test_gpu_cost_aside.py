"""The mixed form's cost where a warp puts more than 32 muons aside (4, 8, 16 and 32 lanes
a muon, and the two-pass form), and where a block's warps keep odd numbers of them to
the end: against the FP64 form's at the same image.

Tolerance: as in test_gpu_cost.py, 1e-6 (a muon's sums carry about ten FP32 roundings).
"""
import numpy as np
import pytest

import muontomography_gb300 as M
from muontomography_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,mm,n_muons,group", [(70, 66, 8, 40.0, 700_003, 4), (40, 41, 20, 20.0, 1_000_001, 8),
                                                       (12, 12, 12, 50.0, 400_009, 16), (130, 130, 130, 4.0, 400_007, 32),
                                                       (330, 330, 160, 6.0, 400_013, 32)])
@pytest.mark.parametrize("over", [{}, {"error_xy": 0.0}])
def test_cost_of_many_muons(gpu, nx, ny, nz, mm, n_muons, group, over):
    g = M.Grid(nx, ny, nz, -nx * mm / 2, -ny * mm / 2, -nz * mm / 2, mm, mm, mm)
    x, z = 0.3 * nx * mm, 0.3 * nz * mm
    wl = W.Workload("scan", g, [M.Block((-x, -x, -z), (x, x, z), M.X0_MM["iron"])], n_muons, 93, True, 1)
    rays = wl.tracks()
    f = {}
    for prec in ("fp64", "mixed"):
        with M.MutoMLSD(wl.em_config(precision=prec, num_iteration=0, update_with_mean=True, **over)) as rec:
            rec.load_tracks(rays)
            rec.prepare()
            f[prec] = rec.nll(np.full(g.nvox, np.log(1.3e-6))), rec.status()
    n = f["fp64"][1]["n_scat_in_grid"]
    assert n == f["mixed"][1]["n_scat_in_grid"] and n > 4096 * 32 and f["mixed"][1]["muon_group"] == group
    assert abs(f["mixed"][0] - f["fp64"][0]) <= 1e-6 * max(abs(f["fp64"][0]), n)
