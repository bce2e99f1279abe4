"""Which tile depth (coarse cells of the innermost axis, 4 or 8) the forward's launches
have, from the plan that RFBA_VERBOSE prints for each of them."""
import os
import re
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
PROG = """
import sys, torch
sys.path.insert(0, {root!r})
from rfba_gb300 import srrf
T, D, H, W, batch = {args}
ctx = srrf.Context(0)
ctx.set_time_batch(batch)
x = torch.randint(90, 700, (T, D, H, W), dtype=torch.int16, device="cuda")
ctx.forward(srrf.Config.make(mag=2, method=1, gradient_smooth=1, x_range=1, y_range=1, z_range=1), x)
torch.cuda.synchronize()
"""


def _depths(*args):
    env = dict(os.environ, RFBA_VERBOSE="1", RFBA_TUNE_MIN="0")
    r = subprocess.run([sys.executable, "-c", PROG.format(root=str(ROOT), args=args)], env=env, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    rows = re.findall(r"rfba: pass .*\bty=(\d+) cz=(\d+) .*batches=(\d+)", r.stderr)
    assert rows, r.stderr[-2000:]
    return [(int(ty), int(cz), int(n)) for ty, cz, n in rows]


@pytest.mark.parametrize("T,cz", [(64, 8), (3, 4)])
def test_schedule_search_times_the_depth_of_the_call(built_lib, T, cz):
    """45 deep tiles of 20 x 24 x 24 at mag 2: 64 volumes fill the GPU with them, the
    3 that the search times do not."""
    rows = _depths(T, 20, 24, 24, 0)
    assert {r[0] for r in rows} == {8, 16}, rows  # the search ran
    assert {r[1] for r in rows} == {cz}, rows


def test_depth_is_for_the_volumes_of_one_launch(built_lib):
    """The same map in batches of 4 of 64 volumes: each launch has 4 volumes' items."""
    rows = [r for r in _depths(64, 20, 24, 24, 4) if r[2] > 1]
    assert rows and {r[1] for r in rows} == {4}, rows
