"""Short-lived threads that call the selections leave no pinned memory behind: the
buffers for words on their way to the host belong to the calls under way, not to the
threads.  Measured in a process of its own (each buffer and event of a thread's own
took 2 KB, and was never freed)."""

import subprocess
import sys

import pytest

from conftest import REPO

SCRIPT = """
import threading, torch
from awkward_gb300 import jagged
off = torch.tensor([0, 3, 5], device="cuda")
x = torch.arange(5.0, device="cuda")
m = torch.ones(5, dtype=torch.bool, device="cuda")

def rss():
    with open("/proc/self/status") as f:
        return int(next(l for l in f if l.startswith("VmRSS")).split()[1])

def churn(n):
    for _ in range(n):
        t = threading.Thread(target=jagged.mask_select, args=(off, x, m))
        t.start()
        t.join()

churn(200)
before = rss()
churn(3000)
print(rss() - before)
"""


@pytest.mark.gpu
def test_threads_leave_no_buffers():
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, cwd=REPO,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    assert int(r.stdout) < 2000  # KB; a buffer per thread took 6000
