"""bench.py times the stage kernel that a handle picks by itself and names it:
the default asks for none, the reported kernel is read from the handle, and the
counts of a committed capture are used for the kernel they were taken from only."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT))

import bench  # noqa: E402


def test_captures_belong_to_their_kernels():
    tile = json.loads((ROOT / "profiles" / "stage_kernel_traffic.json").read_text())
    assert tile["kernel"].startswith(bench.STAGE_KERNELS["tile"])
    assert bench.traffic_per_launch("tile", 2048) == tile["dram_bytes_per_launch"]
    lane = ROOT / "profiles" / bench.STAGE_CAPTURES["lane"]
    assert json.loads(lane.read_text())["kernel"].startswith(bench.STAGE_KERNELS["lane"])
    assert bench.traffic_per_launch("march", 2048) is None and bench.issue_roofline("march", 2048, 1.0, None) is None


@pytest.mark.gpu
def test_default_runs_the_grids_own_kernel():
    cmd = [sys.executable, str(ROOT / "bench.py"), "--grid", "1024", "--steps", "3", "--warmup", "3", "--e2e-steps", "1",
           "--no-cpu-baseline", "--skip-3d", "--skip-ensemble", "--skip-adjoint", "--skip-ns", "--skip-eh", "--skip-ladder"]
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=300, cwd=ROOT)
    assert r.returncode == 0, r.stderr[-2000:]
    line = json.loads(r.stdout.strip().splitlines()[-1])
    assert line["roofline"]["kernel"].startswith(bench.STAGE_KERNELS["lane"]) and line["roofline"]["stage_rows"] > 0
