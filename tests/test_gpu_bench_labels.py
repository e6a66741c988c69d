"""bench.py names the phases of the kernel that ran."""
import json
import subprocess
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.mark.gpu
@pytest.mark.timeout(300)
@pytest.mark.parametrize("side,first", [(92, "search"), (100, "union")])
def test_phase_names(side, first):
    """8,464 sources run one warp each, 10,000 in tiles."""
    out = subprocess.run([sys.executable, str(ROOT / "bench.py"), "--side", str(side), "--steps", "1", "--warmup", "3",
                          "--e2e-steps", "0", "--no-cpu", "--no-extra"], capture_output=True, text=True, timeout=280,
                         cwd=str(ROOT))
    assert out.returncode == 0, out.stderr[-2000:]
    line = json.loads(out.stdout.strip().splitlines()[-1])
    assert next(iter(line["phase_share"])) == first
