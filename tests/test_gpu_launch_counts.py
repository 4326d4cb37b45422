"""Kernel launches that a run reports for its snapshots: the state is
materialized by one kernel, and for the FP32 form four more widen its fields."""
import os

import pytest

import hydrofv_gb300 as H
from hydrofv_gb300 import problems as P

pytestmark = pytest.mark.gpu


def extra_launches(precision, sync, out_dir=None):
    """Launches beside those of the steps, and the snapshots stored."""
    p = P.shear_layer(64)
    storing = {"interval": 0.01, "output_dir": str(out_dir) + "/", "store_initial": False} if out_dir else None
    r = H.run_2d(p.nx, p.ny, p.g, (p.x_min, p.x_max, p.y_min, p.y_max), p.gamma, p.W, p.U, bc=p.bc,
                 slope_limiter=p.slope_limiter, cfl=p.cfl, tf=0.05, max_steps=-1,
                 options=H.default_options(precision=precision, sync_snapshots=sync), storing=storing)
    assert r.code == 0, r.message
    return r.stats["kernel_launches"] - r.stats["step_launches"], len(os.listdir(out_dir)) if out_dir else 0


@pytest.mark.parametrize("sync", [0, 1])
@pytest.mark.parametrize("precision,per_snapshot", [(H.PRECISION_FP64, 1), (H.PRECISION_FP32, 5)])
def test_launches_of_a_snapshot(gpu_available, tmp_path, precision, per_snapshot, sync):
    plain, _ = extra_launches(precision, sync)
    stored, n = extra_launches(precision, sync, tmp_path)
    assert n >= 3 and stored - plain == per_snapshot * n
