"""A step that finds no memory for its buffers reports it and leaves nothing half made: the same context
steps once there is room.  Each case is a process of its own, as freed memory stays in the pool."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# 1M spheres: the grid step takes 16 MB for its position copy, then 68 MB for the candidate lists; the
# hard-contact step 17 MB for counts and colours, then 128 MB for the bodies' velocities
PROG = """
import sys
import numpy as np, torch
from pe_b200 import _abi, scenes
from pe_b200.engine import Engine, PeB200Error
torch.cuda.init()
if sys.argv[1] == "grid":
    s = scenes.dem_large(3, n=1000000, dims=(200.0, 200.0, 420.0))
    kw = dict(neighbor_lists=False)
else:
    s = scenes.nbgs_box(2, n=1000000, mu=0.0, dims=(160.0, 160.0, 490.0))
    kw = dict(solver=_abi.HCSITS, max_iterations=5, max_contacts=1024)
out = []
for short in (False, True):
    e = Engine(**kw).load_scene(s)
    if short:
        torch.cuda.synchronize()
        assert _abi.load().pe_b200_release_memory(0) == 0
        hold = torch.empty(torch.cuda.mem_get_info()[0] - 36_000_000, dtype=torch.uint8, device="cuda")
        for _ in range(2):
            try:
                e.step(s.dt)
                raise SystemExit("stepped without memory")
            except PeB200Error as err:
                assert err.code == _abi.ERR_NOMEM, err
        del hold
        torch.cuda.empty_cache()
    e.step(s.dt, 2)
    out.append(e.download())
    e.close()
assert all(np.array_equal(a, b) for a, b in zip(*out))
print("ok")
"""


@pytest.mark.parametrize("step", ["grid", "hard"])
def test_the_context_steps_once_there_is_room(step):
    r = subprocess.run([sys.executable, "-c", PROG, step], cwd=ROOT, text=True, capture_output=True,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
