"""Scratch of a sort whose long lists are nearly all of one run (up to 16384 elements):
only lists that are merged need pair buffers, so the library's pool grows by no more
than 32 bytes an element.  Measured in a process of its own (the pool keeps what it
has)."""

import subprocess
import sys

import pytest

from conftest import REPO

SCRIPT = """
import numpy as np, torch, awkward_gb300
be = awkward_gb300.backend()
rng = np.random.default_rng(1)
L = np.full(10_001, 3000); L[7000] = 20_000
off = torch.from_numpy(np.concatenate([[0], np.cumsum(L)])).cuda()
n = int(off[-1])
x = torch.randint(-1000, 1000, (n,), dtype=torch.int16, device="cuda")
out = torch.empty_like(x)
sort = be["awkward_sort", np.int16, np.int16, np.int64]
sort(out[:3000], x[:3000], 3000, off[:2], 2, True, True)  # (loads the kernels)
be.synchronize()
before = torch.cuda.mem_get_info()[0]
sort(out, x, n, off, off.numel(), True, True)
be.synchronize()
used = before - torch.cuda.mem_get_info()[0]
seg = torch.repeat_interleave(torch.arange(L.size, device="cuda"), off[1:] - off[:-1])
same = torch.equal(seg * 4096 + out, (seg * 4096 + x).sort().values)
print(used / n, same)
"""


@pytest.mark.gpu
def test_one_run_lists_take_no_pair_buffers():
    r = subprocess.run([sys.executable, "-c", SCRIPT], capture_output=True, text=True, cwd=REPO,
                       timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
    used, same = r.stdout.split()
    assert same == "True"
    assert float(used) <= 32.0
