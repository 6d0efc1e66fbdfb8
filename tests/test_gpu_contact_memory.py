"""The buffers of the sweeps without barriers are apart from the contact buffers: a context whose sweeps take
another form does without them, and one on a GPU with no room for them still steps, to the same bits.
Each case is a process of its own, as freed memory stays in the library's pool."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CAP = 8_000_000                     # contacts
BASE = CAP * (4 * 4 + 51 * 8 + 16)  # their FP64 records, order, colours and adjacency
MORE = CAP * (16 + 16 * 8)          # places and mailboxes
SLACK = 400_000_000

PROG = """
import sys
import numpy as np, torch
from pe_b200 import _abi, scenes
from pe_b200.engine import Engine
mode, room = int(sys.argv[1]), int(sys.argv[2])
torch.cuda.init()
s = scenes.nbgs_box(2, n=1500, mu=0.3, dims=(10.0, 10.0, 60.0), dense=True)
def run(cap):
    e = Engine(solver=_abi.HCSITS, relaxation_model=1, max_iterations=20, max_contacts=cap).load_scene(s)
    e.set_tuning(nbgs_sweeps=mode)
    e.step(s.dt, 3)
    out = e.download()
    assert e.stats()["contacts"] > 768
    return e, out
e, ref = run(0)
e.close()
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
hold = torch.empty(free - room if room else 1, dtype=torch.uint8, device="cuda")
free = torch.cuda.mem_get_info()[0]
e, out = run(%d)
torch.cuda.synchronize()
assert _abi.load().pe_b200_release_memory(0) == 0    # what a refused request left reserved
print("used", free - torch.cuda.mem_get_info()[0])
assert all(np.array_equal(a, b) for a, b in zip(ref, out))
""" % CAP


def _used(mode, room=0):
    r = subprocess.run([sys.executable, "-c", PROG, str(mode), str(room)], cwd=ROOT, text=True,
                       capture_output=True, timeout=300)
    assert r.returncode == 0, r.stderr
    return int(r.stdout.split()[-1])


def test_other_forms_do_without():
    assert _used(2) < BASE + SLACK < BASE + MORE


def test_no_room_for_them():
    assert BASE <= _used(0) < BASE + MORE + SLACK
    assert _used(0, room=BASE + SLACK + 200_000_000) < BASE + SLACK
