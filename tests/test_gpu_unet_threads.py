"""Threads whose first network calls come at the same time: every weight gradient runs on the
tcgen05 kernel (it needs an entry point of the driver, which the first call fetches) and is right."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

FIRST_CALLS = """
import os, threading
import torch
from torch.profiler import ProfilerActivity, profile
from lbm3d_bb_b200 import unet as N

T, SHAPE, CIN, COUT = 12, (1, 4, 8, 32), 16, 16
ops = [N.Ops(torch.cuda.Stream()) for _ in range(T)]
x = torch.randint(-3, 4, (*SHAPE, CIN), device="cuda").to(torch.bfloat16)
dy = torch.randint(-3, 4, (*SHAPE, COUT), device="cuda").to(torch.bfloat16)
dw = torch.zeros((T, 27, COUT, CIN), device="cuda")
torch.cuda.synchronize()
gate = threading.Barrier(T)

def work(k):
    if os.environ["THREADS"] == "known":
        torch.cuda.synchronize()  # the thread has a current context
    gate.wait()
    ops[k].bwd_weight(x, dy, dw[k], SHAPE, CIN, COUT)

with profile(activities=[ProfilerActivity.CUDA]) as p:
    threads = [threading.Thread(target=work, args=(k,)) for k in range(T)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    torch.cuda.synchronize()
N.tc_status()
# sums of small whole numbers are exact in FP32
xp = torch.nn.functional.pad(x.double(), (0, 0, 1, 1, 1, 1, 1, 1))
n, d, h, w = SHAPE
want = torch.stack([torch.einsum("ndhwi,ndhwo->oi", xp[:, a:a + d, b:b + h, c:c + w], dy.double())
                    for a in range(3) for b in range(3) for c in range(3)])
assert all(torch.equal(dw[k].double(), want) for k in range(T))
names = [e.name for e in p.events() if "conv_bwdw" in e.name]
assert all("conv_bwdw_tc_kernel" in name for name in names), names
if len(names) < T:
    raise SystemExit(77)  # activity records were lost
"""


def _judge(r):
    if r.returncode == 77:
        pytest.skip("the profiler lost records in that process")
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("run", range(3))
def test_first_weight_gradients_of_several_threads(gpu, run):
    r = subprocess.run([sys.executable, "-c", FIRST_CALLS], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "THREADS": "known"})
    _judge(r)


def test_weight_gradients_of_threads_new_to_the_device(gpu):
    """The network's call is the first that these threads make: no context is current yet."""
    r = subprocess.run([sys.executable, "-c", FIRST_CALLS], cwd=ROOT, capture_output=True, text=True, timeout=300,
                       env={**os.environ, "THREADS": "new"})
    _judge(r)
