"""What the device pool holds after mines of one dataset: twice the peak use, the block laid out by bounds counted once,
so not much more than with every array laid out exactly (counted twice it is 2.1 times as much)."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent
CHILD = """
import sys
import torch
import colo
from colo import gen
ctx = colo.Context(0)
wl = gen.config(3, scale=0.1)             # 2,000,000 points
ds = colo.Dataset.from_arrays(ctx, wl.x, wl.y, wl.fid, wl.bounds)
ds.upload()
p = colo.default_params(wl.R, wl.thr, colo.MODE_BATCHED, max_size=wl.max_size)
p.reserved[2] = int(sys.argv[1])
torch.cuda.synchronize()
free = torch.cuda.mem_get_info(0)[0]
for _ in range(3):
    n = ctx.mine(ds, p).num_candidates()
torch.cuda.synchronize()
print(n, free - torch.cuda.mem_get_info(0)[0])
"""


def test_bounds_do_not_double_what_is_held():
    pytest.importorskip("torch")
    env = dict(os.environ, PYTHONPATH=str(ROOT / "gpu-colocationmininig_gb300"))
    out = [subprocess.run([sys.executable, "-c", CHILD, str(layout)], env=env, check=True, capture_output=True, text=True,
                          timeout=300).stdout.split() for layout in (0, -1)]
    (n, held), (n_exact, exact) = ([int(v) for v in o] for o in out)
    assert n == n_exact and exact > 100 << 20
    assert held <= 1.5 * exact, (held >> 20, exact >> 20)
