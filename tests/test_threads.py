"""GPU: first calls of several threads at once, in a process of their own: tables that
are made on first use are whole for all of them."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

PROGRAM = """
import threading
import numpy as np
import torch
from opencuda_gb300 import _lib
from opencuda_gb300.proposal import HEAD_R, NET_IN, HoughNet
n = 8
torch.cuda.init()
nets = [HoughNet(seed=3) for _ in range(n)]
occ = (torch.rand((1, NET_IN, NET_IN), device="cuda") < 0.03).to(torch.bfloat16)
occ = occ.view(torch.int16).contiguous()
geo = (_lib.hl_coarse_geom * 1)(_lib.hl_coarse_geom(32.0, -2896.0, HEAD_R / 5793.0, 64, 64, 0))
torch.cuda.synchronize()
gate, out = threading.Barrier(n), [None] * n
def work(i):
    st = torch.cuda.Stream()
    gate.wait()
    z = nets[i].forward(occ, geo, stream=st)
    st.synchronize()
    out[i] = z.cpu().numpy()
ts = [threading.Thread(target=work, args=(i,)) for i in range(n)]
[t.start() for t in ts]
[t.join() for t in ts]
assert all(o is not None and np.array_equal(o, out[0]) for o in out)
"""


def test_first_forward_of_eight_threads(cuda):
    root = Path(__file__).resolve().parent.parent
    for _ in range(3):
        r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=root, capture_output=True,
                           text=True, timeout=120)
        assert r.returncode == 0, r.stderr[-2000:]
